"""The MLP kernels at the edges of their 128-row tiles, and with rows that are
only four-byte aligned (the staging has 16-byte loads for aligned rows)."""
import ctypes

import numpy as np
import pytest

from oracle import mlp_ref


def _data(n, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    x = rng.normal(size=(n, 24)).astype(np.float32)
    return x, (np.sin(x[:, :4].sum(1)) + 0.3 * x[:, 5] * x[:, 7]).astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 1000, 4097])
def test_gpu_mlp_rows_and_alignment(gbdev, n, offset):
    import torch
    from cudapt_gb300._native import check, load
    from cudapt_gb300.mlp import MLP
    x, t = _data(n, 20 + n)
    th = mlp_ref.init(21).astype(np.float32)
    net = MLP(params=th)
    L = load()
    dx = torch.zeros(n * 24 + offset, device="cuda")
    dx[offset:] = torch.from_numpy(x.ravel()).cuda()
    dt = torch.from_numpy(t).cuda()
    dy = torch.full((n + 1,), 7.0, device="cuda")
    torch.cuda.synchronize()
    xp = dx.data_ptr() + 4 * offset
    check(L.gbpt_mlp_forward(net.handle, xp, n, dy.data_ptr(), 1))
    y = dy.cpu().numpy()
    assert y[n] == 7.0  # nothing past the last row
    want = mlp_ref.forward(th.astype(np.float64), x)
    # 88 products of BF16 operands: FP32 sums differ from the oracle's where a
    # hidden value rounds to its BF16 neighbour (2^-8 of one of 64 terms)
    ey = 2e-3 * max(np.abs(want).max(), 1.0)
    np.testing.assert_allclose(y[:n], want, rtol=2e-3, atol=ey)

    g = np.zeros(mlp_ref.N_PARAMS, np.float32)
    loss = ctypes.c_float()
    check(L.gbpt_mlp_gradients(net.handle, xp, dt.data_ptr(), n, 1, g.ctypes.data, ctypes.addressof(loss)))
    gw = mlp_ref.gradients(th.astype(np.float64), x, t)
    lw = mlp_ref.loss(th.astype(np.float64), x, t)
    # d(e^2) for an output off by ey; the gradients are products with e = y - t
    # (off by ey / rms(e) of themselves) and of two BF16 factors (2^-8 each)
    assert abs(loss.value - lw) <= 2 * ey * np.sqrt(lw) + ey * ey
    tol = 2 * 2.0 ** -8 + ey / np.sqrt(lw)
    for a, b in ((0, 1536), (1536, 1600), (1600, 5696), (5696, 5760), (5760, 5824), (5824, 5825)):
        assert np.abs(g[a:b] - gw[a:b]).max() <= 2 * tol * np.abs(gw[a:b]).max()
