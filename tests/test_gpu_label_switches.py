"""The labeling's tuning switches change no label: iterations per turn, blocks per SM, threads
of the terminal-region tiles.  The switches are read once per process, so each runs in a
child process."""
import pytest

from test_gpu_label_modes import _run

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def base(gpu):
    return _run({})


@pytest.mark.parametrize("extra", [{"MSC_TRIPS_PER_TURN": "2"}, {"MSC_TRIPS_PER_TURN": "8"},
                                   {"MSC_TRIPS_PER_TURN": "4", "MSC_EARLY_ENDS": "0"},
                                   {"MSC_TRIPS_PER_TURN_PASS1": "2"}, {"MSC_TRIPS_PER_TURN_FP64": "16"},
                                   {"MSC_LANE_CTAS_PER_SM": "1"}, {"MSC_LANE_CTAS_PER_SM": "32"},
                                   {"MSC_TERMINAL_TILES": "1", "MSC_TERMINAL_THREADS": "256"}],
                         ids=lambda e: ",".join(f"{k[4:]}={v}" for k, v in e.items()))
def test_switch_changes_no_label(base, extra):
    assert _run(extra) == base
