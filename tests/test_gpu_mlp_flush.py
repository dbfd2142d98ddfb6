"""The training kernel's weight sums, which leave the registers every four tiles of a block: batches
of one flush, a flush and a part, and two flushes and a part, against the gradient in 64 bits.

The samples are those that float rounding cannot put on the other side of a ReLU or of the middle of
two BF16 numbers, so what is left is the sums. Tolerance: a chain of 512 float additions is off by
about sqrt(512) / sqrt(12) ulp = 4e-7 of its sum, independent over the 296 blocks and added in 64
bits: 2e-8; the result's rounding up to 6e-8. Together below 1.5e-7 of the gradient's norm."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "graphchi-cpp_b200"))

pytestmark = pytest.mark.gpu


def network(x, params, norm):
    import torch

    def bf16(v):
        return v.float().bfloat16().double()
    w1, b1, w2, b2, w3, b3 = torch.split(params, [512, 64, 4096, 64, 64, 1])
    w1, w2, w3 = bf16(w1).view(64, 8), bf16(w2).view(64, 64), bf16(w3)
    xn = bf16((x - norm[:8]) * norm[8:])  # in float, as the kernel
    a1 = xn @ w1.T + b1
    h1 = bf16(a1.clamp(min=0))
    a2 = h1 @ w2.T + b2
    return a2.clamp(min=0) @ w3 + b3, xn, a1, h1, a2, w2, w3


def clear(a1, a2):
    """Samples whose sums a1, a2 lie clear of zero, and a1 of the middles between BF16 numbers."""
    import torch
    ulp = torch.exp2(torch.floor(torch.log2(a1.abs().clamp(min=1e-30))) - 7)
    middle = (torch.remainder(a1 / ulp, 1.0) - 0.5).abs()
    return ((a1.abs() > 1e-4) & ((middle > 1e-3) | (a1 < 0))).all(1) & (a2.abs() > 1e-4).all(1)


@pytest.mark.parametrize("tiles,rest", [(4, 0), (4, 1), (5, 0), (7, 77), (8, 0), (9, 0), (9, 129)])
def test_gradient_over_flushes(tiles, rest):
    """tiles: per block, of 128 samples; two blocks to an SM."""
    import gcgpu
    import torch
    n = 128 * 2 * torch.cuda.get_device_properties(0).multi_processor_count * tiles + rest
    gen = torch.Generator(device="cuda")
    gen.manual_seed(tiles * 1000 + rest)
    with gcgpu.Mlp.load(os.path.join(os.path.dirname(gcgpu.__file__), "warm_start_rmat.npz")) as m:
        params, norm = m.get()
        params, norm = torch.from_numpy(params).cuda().double(), torch.from_numpy(norm).cuda()
        pool = torch.randn(n + n // 2, 8, generator=gen, device="cuda") / norm[8:] + norm[:8]
        x = torch.cat([xs[clear(*network(xs, params, norm)[2:5:2])] for xs in torch.split(pool, 1 << 16)])[:n]
        assert x.shape[0] == n
        t = torch.randn(n, generator=gen, device="cuda") + 1.0
        grad, loss = m.gradient(x.contiguous(), t)
    total, sq = torch.zeros(gcgpu.MLP_NPARAMS, dtype=torch.float64, device="cuda"), 0.0
    for xs, ts in zip(torch.split(x, 1 << 16), torch.split(t, 1 << 16)):
        y, xn, a1, h1, a2, w2, w3 = network(xs, params, norm)
        err = y - ts.double()
        dy = 2.0 * err / n
        d2 = dy[:, None] * w3 * (a2 > 0)
        d1 = (d2 @ w2) * (a1 > 0)
        total += torch.cat([(d1.T @ xn).reshape(-1), d1.sum(0), (d2.T @ h1).reshape(-1), d2.sum(0),
                            a2.clamp(min=0).T @ dy, dy.sum()[None]])
        sq += float((err * err).sum())
    g = torch.from_numpy(np.asarray(grad)).cuda().double()
    assert float((g - total).norm() / total.norm()) <= 1.5e-7
    for part, ref in zip(torch.split(g, [512, 64, 4096, 64, 64, 1]), torch.split(total, [512, 64, 4096, 64, 64, 1])):
        assert float((part - ref).abs().max() / ref.abs().max()) <= 1e-6
    assert abs(loss - sq / n) <= 1e-6 * sq / n
