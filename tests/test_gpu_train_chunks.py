"""GPU: the weight-gradient kernel at the edges of its 256-row chunks (one
chunk writes the gradient itself, more are added by the reduction) and the
Adam step that rides on the reduction.  Gradients against the FP64 network
oracle with the kernels' BF16 rounding points, 2% per layer as the other
gradient tests; Adam against its formula in FP64 from the gradient the call
returned: a handful of FP32 operations, 1e-6 relative."""
import ctypes

import numpy as np
import pytest

import oracle.mlp_oracle as M
from chysx import capi

pytestmark = pytest.mark.gpu


def _problem(rows):
    import torch

    rng = np.random.default_rng(rows)
    p = M.init_params(rng, rng.standard_normal(M.N_IN) * 0.1, rng.uniform(0.5, 2.0, M.N_IN),
                      np.array([0.1, -0.2, 0.05]), np.array([0.5, 1.5, 1.0])).astype(np.float32)
    feat = (rng.standard_normal((rows, M.N_IN)) * 1.5).astype(np.float32)
    targ = (rng.standard_normal((rows, M.N_OUT)) * 0.7).astype(np.float32)
    dev = [torch.from_numpy(a).cuda() for a in (p, feat, targ)]
    ws = torch.empty(int(capi.lib().chysx_mlp_workspace_bytes(rows)), dtype=torch.uint8, device="cuda")
    return p, feat, targ, dev, ws


@pytest.mark.parametrize("rows", [15, 255, 256, 257, 512, 513, 2305])
def test_gradient_at_chunk_edges(rows):
    import torch

    p, feat, targ, (dp, df, dt), ws = _problem(rows)
    grad = torch.full_like(dp, 7.0)
    loss = ctypes.c_double()
    capi.check(capi.lib().chysx_mlp_gradients(dp.data_ptr(), df.data_ptr(), dt.data_ptr(), rows, grad.data_ptr(),
                                              ctypes.byref(loss), ws.data_ptr(), ws.numel(), 0))
    g = grad.cpu().numpy().astype(np.float64)
    oloss, og = M.loss_and_grad(p, feat, targ, emulate_bf16=True)
    assert abs(loss.value - oloss) <= 1e-3 * oloss
    assert np.all(g[:M.OFF["w1"][0]] == 0.0)
    for k in ("w1", "b1", "w2", "b2", "w3", "b3", "w4", "b4"):
        a, b = M.OFF[k]
        assert np.linalg.norm(g[a:b] - og[a:b]) < 2e-2 * np.linalg.norm(og[a:b]), k


@pytest.mark.parametrize("rows", [40, 700])
def test_adam_step(rows):
    import torch

    p, _, _, (dp, df, dt), ws = _problem(rows)
    rng = np.random.default_rng(1)
    m1 = (1e-3 * rng.standard_normal(p.size)).astype(np.float32)
    m2 = (1e-5 * rng.uniform(0.5, 2.0, p.size)).astype(np.float32)
    d1, d2, grad = torch.from_numpy(m1).cuda(), torch.from_numpy(m2).cuda(), torch.zeros_like(dp)
    capi.check(capi.lib().chysx_mlp_train_step(dp.data_ptr(), grad.data_ptr(), d1.data_ptr(), d2.data_ptr(),
                                               df.data_ptr(), dt.data_ptr(), rows, 2e-3, 7, ws.data_ptr(), ws.numel(),
                                               None, 0))
    torch.cuda.synchronize()
    g = grad.cpu().numpy().astype(np.float64)
    w = M.OFF["w1"][0]
    e1, e2, ep = m1.astype(np.float64), m2.astype(np.float64), p.astype(np.float64)
    e1[w:] = 0.9 * e1[w:] + 0.1 * g[w:]
    e2[w:] = 0.999 * e2[w:] + 0.001 * g[w:] ** 2
    ep[w:] -= 2e-3 * (e1[w:] / (1 - 0.9 ** 7)) / (np.sqrt(e2[w:] / (1 - 0.999 ** 7)) + 1e-8)
    # c2 = 1 / (1 - 0.999^t) is formed in FP32: at t = 7 its denominator 0.007 carries 6e-8 / 0.007 = 9e-6, half of it
    # in the update's square root; 1 - 0.999 in FP32 moves m2's new part by 4.7e-5, its root by half that
    step = np.abs(ep - p).max()
    assert np.abs(dp.cpu().numpy() - ep).max() < 3e-5 * step + 2.4e-7
    assert np.abs(d1.cpu().numpy() - e1).max() < 1e-6 * np.abs(e1).max()
    assert np.abs(d2.cpu().numpy() - e2).max() < 1e-6 * np.abs(e2).max() + 1e-4 * np.abs(e2 - m2).max()


def test_workspace_alignment():
    # prediction takes a workspace at 8 bytes as at 16; what a kernel could not use is refused before any launch
    import torch

    rows = 77
    p, feat, targ, (dp, df, dt), ws = _problem(rows)
    ws = torch.empty(ws.numel() + 16, dtype=torch.uint8, device="cuda")
    n = ws.numel() - 16
    out = [torch.zeros((rows, 3), device="cuda") for _ in range(2)]
    for k, o in enumerate(out):
        capi.check(capi.lib().chysx_mlp_predict(dp.data_ptr(), df.data_ptr(), rows, o.data_ptr(),
                                                ws.data_ptr() + 8 * k, n, 0))
    assert torch.equal(out[0], out[1]) and out[0].abs().max() > 0
    grad = torch.zeros_like(dp)
    assert capi.lib().chysx_mlp_predict(dp.data_ptr(), df.data_ptr(), rows, out[0].data_ptr(), ws.data_ptr() + 4, n,
                                        0) == capi.ERR_INVALID_ARGUMENT
    assert capi.lib().chysx_mlp_gradients(dp.data_ptr(), df.data_ptr(), dt.data_ptr(), rows, grad.data_ptr(), None,
                                          ws.data_ptr() + 8, n, 0) == capi.ERR_INVALID_ARGUMENT
