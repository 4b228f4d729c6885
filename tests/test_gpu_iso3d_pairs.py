"""Two 3D iterations per launch against single steps (FASTPROX_B200_PAIRS=0, in a
child process: the library reads its hints once). The same float32 operations per
voxel, fused alike or not: over ITERS iterations, each of which at most triples a
difference through the momentum's two terms and adds a few roundings of 2^-24,
ITERS x 3 x 4 x 2^-24 of the largest value, 3e-5, is asked after a fixed number of
iterations. Solves to a tolerance end in the launch that forms the final iterate
again: each certifies |z - z*|^2 <= 2 gap, so two of them differ by at most
sqrt(2 gap) + sqrt(2 gap'). Extents at the edges of the windows (one window, its
last column and row, two windows, the last window's overlap) and of the chunks of
slices, with and without voxel weights, an axis weight of zero."""

import os
import pathlib
import subprocess
import sys

import numpy as np
import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
SHAPES = [(1, 12, 24), (2, 16, 32), (4, 17, 33), (5, 18, 34), (9, 31, 61), (13, 29, 62), (70, 13, 31), (20, 40, 90)]
ITERS = 41


def _run():
    import torch
    from fastprox_b200 import TVIso
    out = {}
    for i, shape in enumerate(SHAPES):
        rng = np.random.default_rng(i)
        x = np.zeros((2,) + shape, np.float32)
        x[:, :, shape[1] // 3:, shape[2] // 4:] = 1.0
        x[1, shape[0] // 2:] += 0.5
        x = torch.as_tensor(x + 0.1 * rng.standard_normal(x.shape).astype(np.float32), device="cuda")
        for weighted in (False, True):
            alpha = rng.uniform(0.0, 2.0, shape).astype(np.float32) if weighted else None
            w = (1.0, 0.0, 0.5) if i == 3 else None
            op = TVIso(3, weights=w, pixel_weights=alpha)
            z, info = op.solve(x, 0.2, tol=0.0, max_iter=ITERS)
            out[f"{i}{weighted}z"], out[f"{i}{weighted}d"] = z.cpu().numpy(), info.dual.cpu().numpy()
            out[f"{i}{weighted}n"] = info.image_iters
            z, info = op.solve(x, 0.2, tol=1e-5, max_iter=5000)
            out[f"{i}{weighted}c"], out[f"{i}{weighted}g"] = z.cpu().numpy(), info.gaps
            assert info.converged
    return out


@pytest.mark.gpu
def test_pairs_match_single_steps(cuda, tmp_path):
    out = tmp_path / "single.npz"
    env = dict(os.environ, FASTPROX_B200_PAIRS="0")
    r = subprocess.run([sys.executable, str(pathlib.Path(__file__)), str(out)], cwd=ROOT, env=env,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    ref, got = np.load(out), _run()
    for i, shape in enumerate(SHAPES):
        for weighted in (False, True):
            k = f"{i}{weighted}"
            assert np.array_equal(got[k + "n"], ref[k + "n"]), (shape, weighted)
            for f in "zd":
                scale = np.abs(ref[k + f]).max()
                np.testing.assert_allclose(got[k + f], ref[k + f], rtol=0, atol=3e-5 * scale, err_msg=str((shape, f)))
            diff = np.sqrt(((got[k + "c"].astype(np.float64) - ref[k + "c"]) ** 2).reshape(2, -1).sum(1))
            bound = np.sqrt(2 * np.maximum(got[k + "g"], 0)) + np.sqrt(2 * np.maximum(ref[k + "g"], 0))
            assert (diff <= bound).all(), (shape, weighted, diff, bound)


if __name__ == "__main__":
    sys.path.insert(0, str(ROOT))
    np.savez(sys.argv[1], **_run())
