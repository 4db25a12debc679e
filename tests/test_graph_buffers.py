"""Captured batches after other calls have moved the engine's buffers."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

# A process of its own, whose buffers are no larger than these calls make them.  The dumps of
# sixteen dimensions need twice the words a key of the batch's eight dimensions has, so among
# dumps that grow by 3 % there are some that move the key words' buffer alone.
PROGRAM = """
import numpy as np, torch
import imagestack_b200 as ib
rng = np.random.default_rng(5)
img = rng.uniform(0, 1, (6, 48, 64)).astype(np.float32)
def filtered(graph):
    dev = [torch.from_numpy(img.copy()).cuda()]
    ib.bilateral_batch(dev, [6.0], [0.5], payload="fp64", graph=graph)
    torch.cuda.synchronize()
    return dev[0].cpu().numpy()
expect = filtered(False)
filtered(True)
n = 500.0
while n < 30000:
    k = int(n)
    pos = (rng.integers(0, 3, (k, 1)) * 2.0 + rng.normal(0, 0.2, (k, 16))).astype(np.float32)
    ib.lattice_dump(pos, pos[:, :1].copy())
    err = np.abs(filtered(True) - expect).max()
    assert err <= 1e-5, (k, err)
    n *= 1.03
print("ok")
"""


def test_captured_batch_after_dumps_of_more_dimensions(gpu):
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
