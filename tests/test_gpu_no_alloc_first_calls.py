"""After the first no-allocation run of an engine, further ones leave the device's
free memory alone also when they are the first to need another kernel of the
engine (short and long lists take different ones).  In processes of their own, so
that nothing has loaded the kernels before."""
import os
import subprocess
import sys

import pytest

import common as C

pytestmark = pytest.mark.gpu

PROGRAM = """
import sys
import torch
import benchntt_b200 as bn

def free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info(0)[0]

layout, order = int(sys.argv[1]), sys.argv[2].split(",")
ctx = bn.Context(0)
plan = bn.Plan(ctx, 10, bn.Q_NTT, bn.MU_NTT, bn.fill_uniform(5, 1 << 10, bn.Q_NTT), layout)
engine = bn.Batch(ctx, [plan])
counts = {"short": 5, "long": 7 * ctx.sm_count + 1}
x = torch.ones((max(counts.values()) << 10, 2), dtype=torch.int64, device="cuda")
seen = []
for name in order:
    at = [x.data_ptr() + (i << 14) for i in range(counts[name])]
    jobs = bn.Batch.jobs(at, at, [0] * counts[name])
    bn.check(bn.lib().bntt_batch_run_dev_noalloc(engine.handle, jobs, len(jobs)))
    assert engine.status() == bn.OK
    seen.append(free())
print(seen[0] - seen[1], seen[1] - seen[2])
"""


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("order", ["short,long,short", "long,short,long"])
def test_later_calls_take_no_device_memory(layout, order):
    out = subprocess.run([sys.executable, "-c", PROGRAM, str(layout), order], cwd=C.ROOT, capture_output=True, text=True,
                         check=True, timeout=300, env=dict(os.environ, PYTHONPATH=C.ROOT))
    assert out.stdout.split() == ["0", "0"], out.stdout
