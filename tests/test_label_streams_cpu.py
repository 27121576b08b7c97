"""What runs beside the fix-up's streamlines leaves their gradient alone.  They read it
through the read-only path, which promises that nobody writes it meanwhile, on a stream of
their own while the first pass runs.  Read from the sources; no call here needs a GPU."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "msceer_gb300" / "csrc"


def body(text, head):
    """The definition that starts with `head`, comments taken out."""
    at = text.index(head)
    end = text.index("\n}\n", at)
    return re.sub(r"//[^\n]*", "", text[at:end])


def test_first_pass_does_not_write_the_gradient():
    decl = re.sub(r"//[^\n]*", "", (CSRC / "label_common.cuh").read_text())
    args = dict(re.findall(r"cudaError_t (launch_\w+)\(([^;]*)\);", decl))
    text = body((CSRC / "msc_labels_capi.cu").read_text(), "int first_pass(LabelCtx& c, DirLabels& d) {")
    # zeroed at the seeds unless the ends, which start after that, have been started already
    text, n = re.subn(r"if \(d\.n_ext > 0 && !d\.seeds_zeroed\) \{.*?\n  \}", "", text, count=1, flags=re.S)
    assert n == 1
    calls = re.findall(r"(launch_\w+)\(([^;]*c\.g32[^;]*);", text)
    assert text.count("c.g32") == len(calls) == 1
    for name, _ in calls:
        assert re.search(r"float4\s*\*", args[name]) and not re.search(r"(?<!const )float4\s*\*", args[name]), name
