"""An edge between two parts of a column (the polish sums a column's dual in 16 parts)
is decided once. The first column of the image hangs on nothing (zero edge weights
beside it) and its entries sum to zero, so its solution is constant, its dual along
the column is its own data (up to a rounding: images where it is not exactly that are
passed over), and the test knows the running sums bit for
bit: added entry by entry within a part, and by the parts' totals. They differ in
the last place, and the edge's weight is set so that the polish's bound for a flat
edge lies between the two. Nothing else depends on that weight: the image next to
it, whose weight is 0.1 % larger (the edge is flat by either sum), takes the same
iterations to the same solution. Decided differently on its two sides, the edge
would move one of them and spoil every polish of its image."""

import math

import numpy as np
import pytest

H, W, PARTS, GAMMA = 32, 24, 16, 0.125
ETA = 1e-9  # the share of its bound within which an edge's dual counts as active (float64)


def _column(seed):
    """32 entries of size 2 to 4 with an exact sum within rounding of zero, small running sums."""
    rng = np.random.default_rng(seed)
    d = rng.uniform(2.0, 4.0, H) * np.tile([1.0, -1.0, -1.0, 1.0], H // 4)
    d[-1] = -math.fsum(d[:-1])
    return d if 2.0 <= abs(d[-1]) < 4.0 else None


def _boundary(d):
    """(edge, the larger sum) where the two ways to add up to a part's last edge differ."""
    n = H // PARTS
    pre = 0.0
    for j in range(PARTS - 1):
        total, walk = 0.0, pre
        for v in d[j * n:(j + 1) * n]:
            total, walk = total + v, walk + v
        if walk != pre + total and abs(walk) > 1.0:
            return (j + 1) * n - 1, max(abs(walk), abs(pre + total))
        pre += total
    return None


def _weight(s):
    """beta with fl(fl(GAMMA beta) (1 - ETA)) = s, or None."""
    lb = s / (1.0 - ETA)
    for _ in range(4):
        lb = np.nextafter(lb, 0.0)
    for _ in range(9):
        if lb * (1.0 - ETA) == s:
            return lb / GAMMA  # a power of two: exact
        lb = np.nextafter(lb, np.inf)
    return None


def _cases():
    for seed in range(1000):
        d = _column(seed)
        at = None if d is None else _boundary(d)
        beta = None if at is None else _weight(at[1])
        if beta is not None:
            yield seed, d, at[0], beta


def test_cases_exist():
    cases = [c for c, _ in zip(_cases(), range(4))]
    assert len(cases) == 4
    for _, d, edge, beta in cases:
        assert abs(math.fsum(d)) < 1e-15 and edge < H - 1 and GAMMA * beta > abs(math.fsum(d[: edge + 1]))


@pytest.mark.gpu
def test_an_edge_between_parts_is_decided_once(cuda):
    import torch
    from fastprox_b200 import TVAniso
    seen = 0
    for (seed, d, edge, beta), _ in zip(_cases(), range(12)):
        x = np.random.default_rng(seed).normal(size=(H, W))
        x[:, 0] = d
        res = []
        for b in (beta, beta * 1.001):
            w = np.ones((2, H, W))
            w[0, :, 0] = 1000.0  # flat
            w[0, edge, 0] = b
            w[1, :, 0] = 0.0
            z, info = TVAniso(2, edge_weights=w).solve(torch.as_tensor(x, device="cuda"), GAMMA, tol=1e-9,
                                                       max_iter=5000)
            assert info.converged
            res.append((int(info.image_iters[0]), z.cpu().numpy(), np.array_equal(info.dual[0, :, 0].cpu().numpy(), d)))
        if not (res[0][2] and res[1][2]):
            continue
        seen += 1
        assert res[0][0] == res[1][0], (seed, res[0][0], res[1][0])
        assert np.abs(res[0][1] - res[1][1]).max() <= 1e-6
    assert seen >= 4
