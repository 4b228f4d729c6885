"""Quad launches on rows of any width of 32 pixels or more (16-, 8- and 4-byte
copies for widths of 4 n, 2 n and odd) against single steps
(FASTPROX_B200_QUADS=0 FASTPROX_B200_PAIRS=0, in a child process: the library
reads its hints once): the same bits in z, the dual and the iteration counts,
gaps equal up to the order of their sums. Widths at the edges of the strips (one
window, its last column, two windows, the last window's overlap), heights below
and above a band and not a multiple of four rows, with and without pixel weights;
and the ragged batch on the same images."""

import os
import pathlib
import subprocess
import sys

import numpy as np
import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
SHAPES = [(2, 32), (3, 33), (5, 34), (9, 35), (40, 36), (8, 62), (17, 63), (33, 64), (64, 65), (7, 66), (61, 67),
          (12, 120), (13, 121), (70, 122), (20, 177), (31, 257)]


def _cases():
    for i, shape in enumerate(SHAPES):
        for weighted in (False, True):
            yield i, shape, weighted


def _run():
    import torch
    from fastprox_b200 import TVIso, synth
    out = {}
    for i, (H, W), weighted in _cases():
        x = torch.as_tensor(synth.phantom(2, H, W, seed=i), device="cuda")
        alpha = synth.pixel_weights((H, W), seed=50 + i) if weighted else None
        z, info = TVIso(2, pixel_weights=alpha).solve(x, 0.1, tol=1e-6, max_iter=5000)
        out[f"{i}{weighted}z"], out[f"{i}{weighted}d"] = z.cpu().numpy(), info.dual.cpu().numpy()
        out[f"{i}{weighted}n"], out[f"{i}{weighted}g"] = info.image_iters, info.gaps
    return out


@pytest.mark.gpu
def test_any_width_matches_single_steps(cuda, tmp_path):
    import torch
    from fastprox_b200 import synth
    from fastprox_b200.batch import RaggedBatch
    out = tmp_path / "single.npz"
    env = dict(os.environ, FASTPROX_B200_QUADS="0", FASTPROX_B200_PAIRS="0")
    r = subprocess.run([sys.executable, str(pathlib.Path(__file__)), str(out)], cwd=ROOT, env=env,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    ref, got = np.load(out), _run()
    for i, shape, weighted in _cases():
        k = f"{i}{weighted}"
        assert np.array_equal(got[k + "z"], ref[k + "z"]), (shape, weighted)
        assert np.array_equal(got[k + "d"], ref[k + "d"]), (shape, weighted)
        assert np.array_equal(got[k + "n"], ref[k + "n"]), (shape, weighted)
        # FP64 sums of at most 2 H W float terms, each at most |x|^2: their order, against the gap itself
        np.testing.assert_allclose(got[k + "g"], ref[k + "g"], rtol=1e-9)
    # the ragged batch takes the same quads
    imgs = [torch.as_tensor(synth.phantom(2, H, W, seed=i), device="cuda")[0] for i, (H, W) in enumerate(SHAPES)]
    b = RaggedBatch(len(imgs), sum(x.numel() + 4 for x in imgs))
    outs = [torch.empty_like(x) for x in imgs]
    slots = [b.admit(x, 0.1, 1e-6, max_iter=5000, out=o) for x, o in zip(imgs, outs)]
    its = {}
    while b.pending:
        for slot, _, gap, it, conv in b.run(steps=8):
            its[slot] = (it, gap)
    for i, slot in enumerate(slots):
        assert np.array_equal(outs[i].cpu().numpy(), ref[f"{i}Falsez"][0]), SHAPES[i]
        assert its[slot][0] == ref[f"{i}Falsen"][0], SHAPES[i]
        assert abs(its[slot][1] - ref[f"{i}Falseg"][0]) <= 1e-9 * ref[f"{i}Falseg"][0], SHAPES[i]


if __name__ == "__main__":
    sys.path.insert(0, str(ROOT))
    np.savez(sys.argv[1], **_run())
