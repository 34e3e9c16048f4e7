import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
for p in (ROOT, ROOT / "moba-merge-cuda_b200"):
    if str(p) not in sys.path:
        sys.path.insert(0, str(p))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run on the B200 box)")


# Tests that hold a value which the code does not have any more, with the reason.  They stay as they are, and have to fail.
SUPERSEDED = {
    "test_a_plan_shows_the_next_state_until_the_allocator_moves_on":
        "refused reads of a plan's tables and pool; plans are snapshots (test_plans_are_snapshots_whatever_the_allocator_does_next)",
}


def pytest_collection_modifyitems(items):
    for item in items:
        reason = SUPERSEDED.get(item.name)
        if reason:
            item.add_marker(pytest.mark.xfail(reason=reason, strict=True))
