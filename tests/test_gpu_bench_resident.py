"""bench.py's line of a resident survey says which kernel ran, and that the
tuner's fields are those of the streaming plan; one of a streaming survey does
not."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("extra,resident", [([], True), (["--tile-kernel", "2", "--tile-rows", "64"], False)])
def test_bench_line_names_the_kernel_that_ran(extra, resident):
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--shots", "4", "--nt", "60", "--steps", "1",
                        "--warmup", "3", "--no-cpu"] + extra, capture_output=True, text=True, timeout=600, cwd=ROOT)
    assert r.returncode == 0, r.stderr[-3000:]
    d = json.loads([l for l in r.stdout.splitlines() if l.startswith("{")][-1])
    c, plan, roof = d["config"], d["e2e"]["batch_plan"], d["roofline"]
    assert c["kernel"] == ("k_resident" if resident else "streaming")
    assert (c["resident_shots_per_launch"] > 0) == resident and (plan["resident_shots_per_launch"] > 0) == resident
    assert bool(c["streaming_plan"]) == resident and bool(plan["note"]) == resident
    assert ("HBM does not bound" in roof.get("note", "")) == resident
    assert ("shared memory" in c["l2"]) == resident and ("compares the two kernels" in d["plain"]["how"]) == resident
