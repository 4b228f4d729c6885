"""The conjugate gradients of the isotropic VJP over 2D tiles (cg_y2) against the
kernels that 3D volumes use, on the same images as volumes of one slice: sizes at
the edges of the 32 x 32 tiles and of the warps, with and without pixel weights,
in float64 solved tightly (the two solves' own errors are far below the bound),
and images that stop after different numbers of iterations in one batch."""

import numpy as np
import pytest

SHAPES = [(2, 2), (5, 31), (31, 33), (32, 32), (33, 64), (64, 65), (97, 40)]


def _vjp(op_cls, k, x, alpha, gamma, cot):
    import ctypes as C

    import torch
    from fastprox_b200 import capi
    L = capi.lib()
    op = op_cls(k, pixel_weights=alpha)
    ws = op.workspace(x, keep=True)
    z = torch.empty_like(x)
    opt = capi.options(tol=1e-13, max_iter=200000, keep=True)
    g = torch.as_tensor(gamma, device="cuda", dtype=torch.float64)
    capi.check(L.fp_prox_steps(op._op, capi.ArrayRef(g).ref(), capi.ArrayRef(x).ref(), capi.ArrayRef(z).ref(),
                               C.byref(opt), ws), "prox", (capi.FP_OK, capi.FP_ENOTCONV))
    capi.check(L.fp_workspace_set_deriv_tol(ws, 1e-13, 20000), "deriv_tol")
    gx = torch.empty_like(x)
    gp = np.zeros(op.nparams)
    capi.check(L.fp_vjp(op._op, ws, capi.ArrayRef(cot).ref(), capi.ArrayRef(gx).ref(), None, capi.ArrayRef(gp).ref()),
               "vjp")
    return z.cpu().numpy(), gx.cpu().numpy(), gp[k:]


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("weighted", [False, True])
def test_tiles_match_volume_kernels(cuda, shape, weighted):
    import torch
    from fastprox_b200 import TVIso, synth
    H, W = shape
    gamma = [0.02, 0.1, 0.3]
    x = torch.as_tensor(synth.phantom(3, H, W, seed=H + W, dtype=np.float64), device="cuda")
    cot = torch.as_tensor(np.random.default_rng(3).normal(size=(3, H, W)), device="cuda")
    alpha = synth.pixel_weights(shape, seed=4) if weighted else None
    z2, g2, p2 = _vjp(TVIso, 2, x, alpha, gamma, cot)
    z3, g3, p3 = _vjp(TVIso, 3, x[:, None].contiguous(), None if alpha is None else alpha[None], gamma,
                      cot[:, None].contiguous())
    assert np.abs(z2 - z3[:, 0]).max() <= 1e-5
    # gaps of 1e-13 certify z to 3e-7, and the curvature at an edge amplifies that by the inverse of its gradient
    assert np.linalg.norm(g2 - g3[:, 0]) <= 1e-4 * np.linalg.norm(g3)
    if weighted:
        assert np.linalg.norm(p2 - p3) <= 1e-4 * np.linalg.norm(p3)
