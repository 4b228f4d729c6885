"""The check and the polish of anisotropic TV at sizes where their kernels can go
wrong: rows of one entry, of 31, 32, 33 and 65 (the row marking works on 32
entries at a time), columns at the edges of the column marking's parts and
blocks, regions longer than a warp's run of the region sums, 3D, and images
with flat background (one large region) beside noise (many small ones). The
result is certified from outside: in float64 NumPy, the returned dual is
feasible (its running sums within their bounds, up to rounding) and the primal
minus the dual objective is within the tolerance that the solve reports."""

import numpy as np
import pytest

SHAPES = [(1, 33), (40, 1), (16, 31), (17, 32), (33, 33), (65, 65), (7, 600), (300, 5), (5, 6, 33), (9, 33, 2)]


def _image(shape, seed):
    rng = np.random.default_rng(seed)
    x = np.zeros(shape)
    x[tuple(slice(n // 3, n // 3 + max(1, n // 2)) for n in shape)] = 0.8
    noisy = x + 0.1 * rng.normal(size=shape)
    noisy[..., : shape[-1] // 2] = x[..., : shape[-1] // 2]  # half of it clean: large regions
    return noisy


def _certify(x, z, dual, lam, w):
    """(primal - dual objective, largest excess of a running sum over its bound relative to it)."""
    tv, excess = 0.0, 0.0
    for a in range(x.ndim):
        if x.shape[a] < 2:
            continue
        wa = lam * (np.ones(x.shape) if w is None else w[a])
        edge = [slice(None)] * x.ndim
        edge[a] = slice(0, x.shape[a] - 1)
        tv += float(np.sum(wa[tuple(edge)] * np.abs(np.diff(z, axis=a))))
        p = np.cumsum(dual[a], axis=a)[tuple(edge)]
        excess = max(excess, float(np.max(np.abs(p) / wa[tuple(edge)])) - 1.0)
    q = dual.sum(axis=0)
    primal = 0.5 * float(np.sum((z - x) ** 2)) + tv
    return primal - float(np.sum(x * q) - 0.5 * np.sum(q * q)), excess


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("weighted", [False, True])
def test_polished_solution_is_certified(cuda, shape, weighted):
    import torch
    from fastprox_b200 import TVAniso
    tol, lam = 1e-9, 0.15
    xs = np.stack([_image(shape, s) for s in range(3)])
    w = np.random.default_rng(9).uniform(0.5, 1.5, (len(shape),) + shape) if weighted else None
    z, info = TVAniso(len(shape), edge_weights=w).solve(torch.as_tensor(xs, device="cuda"), lam, tol=tol,
                                                        max_iter=20000)
    assert info.converged
    z, dual = z.cpu().numpy(), info.dual.cpu().numpy()
    for b in range(len(xs)):
        gap, excess = _certify(xs[b], z[b], dual[:, b], lam, w)
        target = 0.5 * tol * float(np.sum(xs[b] ** 2))
        # rounding: sums of N terms of size |x|^2 and running sums of up to 600 terms
        slack = 1e-13 * float(np.sum(xs[b] ** 2))
        assert gap <= target + slack, (b, gap, target)
        assert excess <= 1e-11, (b, excess)
