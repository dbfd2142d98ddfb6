"""The training kernel's tiles: sample counts around one tile and one launch's blocks,
inputs that are not 16-byte aligned, against the FP64 restatement."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "graphchi-cpp_b200"))
sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "oracle"))

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 255, 4095, 128 * 296 + 1])
@pytest.mark.parametrize("offset", [0, 1])
def test_gradient_and_forward(n, offset):
    import gcgpu
    import torch
    import warm_oracle as WO
    rng = np.random.default_rng(n)
    params = rng.normal(0, 0.3, gcgpu.MLP_NPARAMS).astype(np.float32)
    norm = np.concatenate([rng.normal(0, 1, 8), rng.uniform(0.5, 2, 8)]).astype(np.float32)
    x = rng.normal(0, 1, (n, 8)).astype(np.float32)
    t = rng.normal(0, 1, n).astype(np.float32)
    room = torch.zeros(offset + n * 8, dtype=torch.float32, device="cuda")
    xd = room[offset:].view(n, 8)
    xd.copy_(torch.from_numpy(x))
    td = torch.from_numpy(t).cuda()
    with gcgpu.Mlp(seed=1) as m:
        m.set(params, norm)
        grad, loss = m.gradient(xd, td)
        y = m.forward(xd)
    # the restatement's roundings are the kernel's; what is left is FP32 summation and,
    # where an FP32 sum falls on the other side of a BF16 boundary, one such rounding
    y_ref = WO.forward(params, norm, x)
    assert np.abs(y - y_ref).max() <= 2e-2 * np.abs(y_ref).max()
    assert np.linalg.norm(y - y_ref) <= 2e-3 * np.linalg.norm(y_ref)
    g_ref, loss_ref = WO.gradient(params, norm, x, t)
    assert abs(loss - loss_ref) <= 1e-3 * loss_ref
    assert np.linalg.norm(grad - g_ref) <= 1e-2 * np.linalg.norm(g_ref)
