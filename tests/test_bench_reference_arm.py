"""bench.py --impl reference runs the compiled reference or says that it
cannot: the repository's own code never stands in for it."""
import json
import os
import subprocess
import sys

import pytest

import pyoracle as P

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("rank", [0, 1])
def test_reference_arm_without_the_reference(rank):
    if P.ref_available():
        pytest.skip("the compiled reference is here")
    env = dict(os.environ, RANK=str(rank), WORLD_SIZE="2", LOCAL_RANK=str(rank))
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--gpus", "2", "--steps",
                        "1", "--warmup", "3"], capture_output=True, text=True, env=env, timeout=300, cwd=ROOT)
    assert r.returncode == 0, r.stderr
    if rank:
        assert r.stdout == ""
        return
    line = json.loads(r.stdout)
    assert set(line) == {"impl", "unavailable"} and line["impl"] == "reference" and line["unavailable"]
