"""The tuning switches of the labeling that INTEGRATION.md documents are the ones that the
sources read.  No call here needs a GPU."""
import re
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_documented_switches_are_read():
    text = (ROOT / "INTEGRATION.md").read_text()
    text = text[text.index("Environment (read once per process)"):]
    documented = set(re.findall(r"`(MSC_[A-Z0-9_]+)", text[:text.index("\n\n")]))
    read = set()
    for p in (ROOT / "msceer_gb300" / "csrc").glob("*.cu"):
        read |= set(re.findall(r"(?:getenv|trips_env)\(\"(MSC_\w+)\"", p.read_text()))
    assert {"MSC_TRIPS_PER_TURN", "MSC_TRIPS_PER_TURN_PASS1", "MSC_TRIPS_PER_TURN_FP64"} <= read
    assert documented == read - {"MSC_LDIR_QUEUE_CAP"}  # (a test's, of the .grad)
