"""The one-kernel forward at the edges of its dispatch: input and output widths around the 16-byte
row rule and the 160-column accumulator limit, pointers off 16 bytes, row counts around a tile and
around the tiles in flight per SM.  Against the CPU restatement with the tolerance of
test_gpu_mlp.py: hidden activations are BF16 (2^-9 relative) and SiLU adds 2^-10, which four layers
of averaging sums keep below 2e-2 of the largest output."""
import os
import sys

import numpy as np
import pytest

from conftest import REPO

pytestmark = pytest.mark.gpu
sys.path.insert(0, os.path.join(REPO, "oracle"))
import mlp_oracle as M  # noqa: E402


@pytest.mark.parametrize("n_in,width,n_out,m,off", [
    (8, 128, 132, 127, 0), (64, 128, 160, 128, 0),     # three tiles in flight, the widest output for it
    (64, 128, 164, 129, 0), (56, 256, 256, 300, 0),    # two tiles in flight
    (64, 128, 131, 257, 0), (64, 256, 1, 130, 0),      # output rows off 16 bytes: the padded route
    (64, 128, 132, 500, 1), (64, 256, 132, 500, 1),    # pointers off 16 bytes
    (72, 128, 132, 300, 0),                            # too wide an input: layer by layer
    (64, 128, 16, 152 * 128 * 3 + 1, 0),               # a fourth tile on one SM only
    (64, 128, 132, 152 * 128 * 7, 0), (64, 256, 132, 152 * 128 * 5, 0),
])
def test_forward_shapes(n_in, width, n_out, m, off):
    torch = pytest.importorskip("torch")
    from souffle_gb300 import gpu
    net = gpu.Mlp(n_in, n_out, max_batch=m, seed=n_out, width=width)
    p = net.get_params()
    rng = np.random.default_rng(m)
    x = rng.normal(0, 1, (m, n_in)).astype(np.float32)
    xd = torch.empty(m * n_in + off, device="cuda")[off:].copy_(torch.from_numpy(x).reshape(-1))
    y = torch.full((m * n_out + off + 64,), float("nan"), device="cuda")
    net.forward(xd.data_ptr(), m, y[off:].data_ptr())
    torch.cuda.synchronize()
    got = y.cpu().numpy()
    assert np.isnan(got[:off]).all() and np.isnan(got[off + m * n_out:]).all()  # nothing beside the rows
    got = got[off:off + m * n_out].reshape(m, n_out)
    rows = np.arange(m) if m <= 1024 else np.unique(np.r_[0:200, m - 200:m, rng.choice(m, 600)])
    ref = M.forward(p, x[rows], n_in, width, n_out, emulate=True)
    assert np.isfinite(got).all()
    assert np.abs(got[rows] - ref).max() <= 2e-2 * np.abs(ref).max()


@pytest.mark.parametrize("n_in,n_out,x_at,y_at", [
    (32, 64, 0, 0),          # output rows longer than input rows, from the same place
    (64, 32, 0, 0), (48, 48, 0, 0),
    (32, 64, 5000 * 64 - 4, 0), (64, 32, 0, 5000 * 64 - 4),   # a few elements shared
    (32, 64, 5000 * 64, 0), (64, 32, 0, 5000 * 64),           # neighbours, not overlapping
])
def test_forward_between_overlapping_buffers(n_in, n_out, x_at, y_at):
    """Input and output rows that share memory: bitwise the result of separate buffers."""
    torch = pytest.importorskip("torch")
    from souffle_gb300 import gpu
    m = 5000
    torch.manual_seed(n_in + n_out)
    x = torch.randn(m, n_in, device="cuda")
    want = torch.empty(m, n_out, device="cuda")
    net = gpu.Mlp(n_in, n_out, m, seed=3, width=128)
    buf = torch.zeros(m * 128, device="cuda")
    xs, ys = buf[x_at:x_at + m * n_in], buf[y_at:y_at + m * n_out]
    xs.copy_(x.reshape(-1))
    torch.cuda.synchronize()
    net.forward(x.data_ptr(), m, want.data_ptr())
    net.forward(xs.data_ptr(), m, ys.data_ptr())
    torch.cuda.synchronize()
    assert torch.equal(ys.reshape(m, n_out), want)
