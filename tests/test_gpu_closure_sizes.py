"""The closure's tensor-core backward pass at the edges of its tiles (64 samples to a
tile, two blocks an SM): loss and gradient against the oracle.

Tolerances: FP32 sums of exact products differ from the oracle's FP64 sums by a few
1e-7 of the result, but now and then such a difference moves an activation to the
neighbouring BF16 value, 2^-8 of it.  With few samples one such activation may be a
whole column of a gradient: 2^-7 of its norm; over a thousand samples or more the
moved ones average out far below 2e-4."""
import numpy as np
import pytest

from cmag_gb300.closure import Closure
from oracle import closure_oracle as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 16, 63, 64, 65, 1000, 2 * 152 * 64 + 1])
def test_gradient_at_tile_edges(gpu, n):
    import torch
    rng = np.random.default_rng(n)
    theta = C.init_params(5)
    theta[C.NPARAMS - 3:] = rng.normal(0, 0.05, 3).astype(np.float32)
    feat = (rng.normal(size=(n, 16)) * 2.0 + 0.3).astype(np.float32)
    target = rng.normal(size=(n, 3)).astype(np.float32)
    mean = rng.normal(0, 0.2, 16).astype(np.float32)
    inv = rng.uniform(0.4, 0.8, 16).astype(np.float32)
    c = Closure(theta)
    c.set_normalization(mean, inv, 1.0)
    fd, td = torch.from_numpy(feat).cuda(), torch.from_numpy(target).cuda()
    tol = 2.0 ** -7 if n < 1000 else 2e-4
    wl, wg = C.loss_and_grad(theta, feat, target, mean.astype(np.float64), inv.astype(np.float64))
    for _ in range(2):  # the second call starts from what the first left
        loss, g = c.gradient(fd, td)
        assert abs(loss - wl) <= tol * wl
        offs = np.cumsum([0] + [int(np.prod(s)) for _, s in C.SHAPES])
        for (name, _), a, b in zip(C.SHAPES, offs[:-1], offs[1:]):
            rel = np.linalg.norm(g[a:b].astype(np.float64) - wg[a:b]) / np.linalg.norm(wg[a:b])
            assert rel < tol, (name, rel)
    # a step updates the weights the network runs with (their BF16 copy and its image)
    out = torch.empty((n, 3), dtype=torch.float32, device="cuda")
    c.train_step(fd, td, 1e-3)
    c.synchronize()
    assert np.array_equal(c.bf16_params(), C.bf16(c.params).astype(np.float32))
    c.forward(fd, out)
    fresh = Closure(c.params)
    fresh.set_normalization(mean, inv, 1.0)
    want = torch.empty_like(out)
    fresh.forward(fd, want)
    assert torch.equal(out, want)
