"""Isotropic solves of images whose values are far from one. Images between 2^-64
and 2^64 are solved as they are, so the squares of their gradients reach down among
the subnormal floats; a duality gap that loses them is too small, and the solve
stops early. Asked for:
 * always: the gap of the returned dual, formed in float64 by NumPy, is within the
   tolerance, up to the float32 rounding of the terms the solver adds up: a term
   r |g| - <g, u> with |u| <= r carries at most r times the error of g, the
   roundings of z's five (seven) terms, each at most 2^-24 of the largest value, in
   each of two (three) differences, and of the products: 32 x 2^-24 r max |x| per
   pixel;
 * down to EXACT, where the squares that the projection compares (about
   (GAMMA 2^-46)^2 = 2^-99, their last places 2^-122) are normal floats and a power
   of two therefore changes nothing but exponents: in 2D (rows of 4 n, 2 n and odd
   width, batched and ragged) the iterates and iteration counts of the same image in
   single steps (fp_b200_tv_iso_noalloc runs nothing else), in 3D the iteration
   counts of the image at scale one. Below, single steps themselves round otherwise."""

import ctypes as C

import numpy as np
import pytest

AMPLITUDES = [0, -30, -46, -56]
EXACT = -46
GAMMA, TOL = 0.1, 1e-5


def _phantom(shape, seed):
    rng = np.random.default_rng(seed)
    x = np.zeros(shape)
    x[tuple(slice(n // 3, n // 3 + max(1, n // 2)) for n in shape)] = 0.8
    return (x + 0.1 * rng.normal(size=shape)).astype(np.float32)


def _gap(x, dual, gamma):
    """The gap of u = dual (ndim, *image) in float64 at z = x - G^T u."""
    z = x.astype(np.float64)
    u = dual.astype(np.float64)
    k = x.ndim
    for a in range(k):
        prev = np.zeros_like(z)
        tail, head = [slice(None)] * k, [slice(None)] * k
        tail[a], head[a] = slice(1, None), slice(None, -1)
        prev[tuple(tail)] = u[a][tuple(head)]
        z += u[a] - prev
    g = np.zeros_like(u)
    for a in range(k):
        head = [slice(None)] * k
        head[a] = slice(None, -1)
        g[a][tuple(head)] = np.diff(z, axis=a)
    return float(np.sum(gamma * np.sqrt((g * g).sum(0)) - (g * u).sum(0)))


def _allowed(x, gamma):
    return TOL * 0.5 * float((x.astype(np.float64) ** 2).sum()) + 32 * 2.0 ** -24 * gamma * x.size * float(np.abs(x).max())


def _single_steps(x, gamma):
    import torch
    from fastprox_b200 import capi
    z = torch.empty_like(x)
    its = np.zeros(x.shape[0], np.int32)
    st = capi.lib().fp_b200_tv_iso_noalloc(C.c_void_p(x.data_ptr()), C.c_void_p(z.data_ptr()), *x.shape, gamma, TOL,
                                           5000, C.c_void_p(torch.cuda.current_stream().cuda_stream), None,
                                           its.ctypes.data_as(C.POINTER(C.c_int)))
    capi.check(st, "noalloc", (capi.FP_OK, capi.FP_ENOTCONV))
    return z, its, st == capi.FP_OK


@pytest.mark.gpu
@pytest.mark.parametrize("exponent", AMPLITUDES)
@pytest.mark.parametrize("shape", [(64, 64), (61, 66), (50, 67)])
def test_images(cuda, shape, exponent):
    import torch
    from fastprox_b200 import TVIso
    from fastprox_b200.batch import RaggedBatch
    gamma = float(np.ldexp(GAMMA, exponent))
    xs = np.ldexp(np.stack([_phantom(shape, s) for s in range(2)]), exponent)
    x = torch.as_tensor(xs, device="cuda")
    ref, its, ok = _single_steps(x, gamma)
    z, info = TVIso(2).solve(x, gamma, tol=TOL, max_iter=5000)
    assert ok and info.converged
    if exponent >= EXACT:
        assert np.array_equal(info.image_iters, its), (info.image_iters, its)
        assert torch.equal(z, ref)
    dual = info.dual.cpu().numpy()
    for b in range(2):
        assert _gap(xs[b], dual[:, b], gamma) <= _allowed(xs[b], gamma)
    batch = RaggedBatch(2, 2 * (x[0].numel() + 4))
    slots = [batch.admit(x[b], gamma, TOL, max_iter=5000) for b in range(2)]
    while batch.pending:
        for slot, zb, gap, it, conv in batch.run(steps=8):
            b = slots.index(slot)
            assert conv
            if exponent >= EXACT:
                assert it == its[b], (it, its[b])
                assert torch.equal(zb, ref[b])
            else:  # both within sqrt(2 gap) of the solution
                off = float(np.linalg.norm((zb - ref[b]).double().cpu().numpy()))
                assert off <= 2 * np.sqrt(2 * _allowed(xs[b], gamma))


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(20, 24, 32), (17, 21, 30)])
def test_volumes(cuda, shape):
    import torch
    from fastprox_b200 import TVIso
    x1 = _phantom(shape, 5)
    counts = []
    for exponent in AMPLITUDES:
        gamma = float(np.ldexp(GAMMA, exponent))
        x = np.ldexp(x1, exponent)
        _, info = TVIso(3).solve(torch.as_tensor(x, device="cuda"), gamma, tol=TOL, max_iter=5000)
        assert info.converged
        assert _gap(x, info.dual.cpu().numpy(), gamma) <= _allowed(x, gamma), exponent
        if exponent >= EXACT:
            counts.append(int(info.image_iters[0]))
    assert len(set(counts)) == 1, counts
