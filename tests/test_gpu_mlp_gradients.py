"""Weight gradients of all layers in one launch, at the edges of its tiles: batches below one K step, of
odd length, and of many steps, outputs off the tile size, both widths.  Against the CPU
restatement, with the tolerances of test_gpu_mlp.py (BF16 activations: 1e-2 of each tensor's norm)."""
import os
import sys

import numpy as np
import pytest

from conftest import REPO

pytestmark = pytest.mark.gpu
sys.path.insert(0, os.path.join(REPO, "oracle"))
import mlp_oracle as M  # noqa: E402


@pytest.mark.parametrize("n_in,width,n_out,m", [
    (64, 128, 132, 1), (64, 128, 132, 63), (64, 128, 132, 65), (8, 128, 1, 129), (64, 128, 131, 1000),
    (256, 256, 256, 500), (64, 256, 132, 4097), (64, 128, 132, 8192),
])
def test_gradients_shapes(n_in, width, n_out, m):
    torch = pytest.importorskip("torch")
    from souffle_gb300 import gpu
    net = gpu.Mlp(n_in, n_out, max_batch=m + 40, seed=m, width=width)
    rng = np.random.default_rng(m)
    x = rng.normal(0, 1, (m, n_in)).astype(np.float32)
    t = rng.normal(0, 0.5, (m, n_out)).astype(np.float32)
    xd, td = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    p = net.get_params()
    loss, g = net.gradients(xd.data_ptr(), td.data_ptr(), m)
    ref_loss, ref_g = M.loss_and_grads(p, x, t, n_in, width, n_out, emulate=True)
    assert loss == pytest.approx(ref_loss, rel=1e-4)
    k = 0
    for ws, bs in M.shapes(n_in, width, n_out):
        for size in (ws[0] * ws[1], bs[0]):
            a, b = g[k:k + size], ref_g[k:k + size]
            assert np.linalg.norm(a - b) <= 1e-2 * np.linalg.norm(b) + 1e-12, (k, size)
            k += size
    again = net.gradients(xd.data_ptr(), td.data_ptr(), m)
    assert again[0] == loss and np.array_equal(again[1], g)  # the same bits on every call
    assert np.array_equal(net.get_params(), p)
