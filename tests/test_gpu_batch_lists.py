"""Ragged batches of images whose tiles outnumber what the batch's pixels suggest
(tall and narrow, or quad tiles of one row): the work lists hold every tile, so each
image is solved whole. Solved alone by fp_prox (another partition of the sums), z
differs by at most sqrt(2 gap) + sqrt(2 gap'); rows narrower than 32 pixels form the
gap's terms in float64 there."""

import numpy as np
import pytest

CASES = [((70000, 4), "float32", 0), ((4000, 33), "float32", 1), ((60000, 2), "float32", 0), ((40000, 2), "float64", 0)]


@pytest.mark.gpu
@pytest.mark.parametrize("shape,dtype,quad_rows", CASES)
def test_every_tile_is_listed(cuda, shape, dtype, quad_rows):
    import torch
    from fastprox_b200 import TVIso
    from fastprox_b200.batch import RaggedBatch
    rng = np.random.default_rng(shape[1])
    x = 0.2 * rng.normal(size=shape) + (np.arange(shape[0]) // 500 % 2)[:, None]
    x = torch.as_tensor(x, device="cuda").to(getattr(torch, dtype))
    ref, info = TVIso(2).solve(x, 0.2, tol=1e-6, max_iter=4000)
    small = x[:40].contiguous()
    batch = RaggedBatch(2, x.numel() + small.numel() + 8, dtype=dtype, quad_rows=quad_rows)
    slots = [batch.admit(small, 0.2, 1e-6, max_iter=4000), batch.admit(x, 0.2, 1e-6, max_iter=4000)]
    res = {}
    for _ in range(600):
        for slot, z, gap, it, conv in batch.run(steps=8, max_chunks=1):
            res[slot] = (z, gap, conv)
        if not batch.pending:
            break
    assert sorted(res) == sorted(slots)
    z, gap, conv = res[slots[1]]
    assert conv and info.converged
    off = float(torch.linalg.vector_norm(z.double() - ref.double()))
    assert off <= np.sqrt(2 * gap) + np.sqrt(2 * float(info.gaps[0])), off
