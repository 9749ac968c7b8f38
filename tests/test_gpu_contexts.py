"""The library used from more than one CUDA context of a process, in turn."""
import json
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

HERE = Path(__file__).resolve().parent


def _child(mode):
    r = subprocess.run([sys.executable, str(HERE / "contexts_child.py"), mode], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


def test_alternating_contexts_keep_one_pool():
    """Ten rounds of an LM update in the primary context and in another one: after the first round (module
    loading, the scratch pool's first growth) the device's free memory stays where it is, to within one
    2 MB page, and every update agrees with the FP64 normal equations to the 1e-3 bar of the split-BF16 updates."""
    out = _child("alternate")
    assert max(out["err"]) < 1e-3
    assert max(out["free"][1:]) - min(out["free"][1:]) <= 2 ** 21, out["free"]


@pytest.mark.parametrize("mode", ["trim", "destroy"])
def test_trim_gives_a_destroyed_plans_memory_back(mode):
    """A plan destroyed in its own context, and while another one is current (which stays so).  The library
    keeps a destroyed plan's memory for the next one; after a trim the device has as much free as before the
    plan, to within one 2 MB page."""
    before, plan, destroyed, trimmed = _child(mode)["free"]
    assert before - plan > 2 ** 27 and before - destroyed > 2 ** 27
    assert before - trimmed <= 2 ** 21
