"""The training gradient against 64 bits on the kernel's own activations.

The forward pass sums in FP32 in a fixed order, so its BF16 activations can be restated
bit for bit; the gradient that 64-bit arithmetic gives for them differs from the kernel's
by the rounding of the backward pass alone (no activation rounds the other way).

Tolerances.  Error of a matrix: its deltas keep 24 bits in three parts and sums are FP32,
a few 2^-24 each: under 1e-6 of the matrix, while a lost third part would be 2^-17.
Shrinking (the component of the error along the gradient, over 8 seeds): rounding to
nearest shifts neither way; a product level on the tensor cores may truncate each of its
sums once, by at most a unit in the last place (2^-23) and half of one on average, towards
zero: 2^-24 for each of the levels a matrix's gradient runs through (W4 and W3 one, W2
two, W1 three).  Row counts are powers of two, whose 1 / n is exact."""
import numpy as np
import pytest

from cmag_gb300.closure import Closure
from oracle import closure_oracle as C

pytestmark = pytest.mark.gpu


def on_own_activations(theta, feat, target, mean, inv):
    import torch

    def bf16(x):
        return x.to(torch.bfloat16).to(torch.float32)

    def layer(h, w, b):  # FP32, from the bias over ascending inputs (products are exact)
        s = b.expand(h.shape[0], -1).clone()
        for k in range(h.shape[1]):
            s = (s.double() + h[:, k:k + 1].double() * w[:, k].double()).float()
        return s

    def act(z):
        return bf16(z * (1.0 / (1.0 + torch.exp(-z))))

    def slope(z):
        s = torch.sigmoid(z.double())
        return s * (1 + z.double() * (1 - s))

    p = {k: bf16(torch.from_numpy(v.astype(np.float32)).cuda()) for k, v in C.unpack(theta).items()}
    x = bf16((feat - torch.from_numpy(mean).cuda()) * torch.from_numpy(inv).cuda())
    z1 = layer(x, p["W1"], p["b1"])
    a1 = act(z1)
    z2 = layer(a1, p["W2"], p["b2"])
    a2 = act(z2)
    z3 = layer(a2, p["W3"], p["b3"])
    a3 = act(z3)
    d = {k: v.double() for k, v in p.items()}
    e = (a3.double() @ d["W4"].T + d["b4"] - target.double()) / feat.shape[0]
    g = {"W4": e.T @ a3.double()}
    d3 = (e @ d["W4"]) * slope(z3)
    g["W3"] = d3.T @ a2.double()
    d2 = (d3 @ d["W3"]) * slope(z2)
    g["W2"] = d2.T @ a1.double()
    d1 = (d2 @ d["W2"]) * slope(z1)
    g["W1"] = d1.T @ x.double()
    return {k: v.cpu().numpy() for k, v in g.items()}


@pytest.mark.parametrize("n", [64, 2048, 65536])
def test_gradient_on_own_activations(gpu, n):
    import torch
    shrink = {}
    for seed in range(8):
        rng = np.random.default_rng(seed + n)
        theta = C.init_params(seed)
        theta[C.NPARAMS - 3:] = rng.normal(0, 0.05, 3).astype(np.float32)
        feat = torch.from_numpy((rng.normal(size=(n, 16)) * 2.0 + 0.3).astype(np.float32)).cuda()
        target = torch.from_numpy(rng.normal(size=(n, 3)).astype(np.float32)).cuda()
        mean = rng.normal(0, 0.2, 16).astype(np.float32)
        inv = rng.uniform(0.4, 0.8, 16).astype(np.float32)
        c = Closure(theta)
        c.set_normalization(mean, inv, 1.0)
        got = C.unpack(c.gradient(feat, target)[1])
        for name, want in on_own_activations(theta, feat, target, mean, inv).items():
            err = got[name] - want
            assert np.linalg.norm(err) < 1e-6 * np.linalg.norm(want), (name, seed)
            shrink.setdefault(name, []).append(float((err * want).sum() / (want * want).sum()))
    for name, levels in (("W4", 1), ("W3", 1), ("W2", 2), ("W1", 3)):
        assert abs(np.mean(shrink[name])) < levels * 2.0 ** -24, (name, np.mean(shrink[name]))
