"""Edges of zero weight in the fibre passes by pieces, against the untiled passes (one
thread per fibre, which scans the parts between two cuts one after another;
FASTPROX_B200_AN_FIB=0 FASTPROX_B200_TILES=0, in a child process: the library reads
its hints once): the same scan part by part, so the same iterates up to the order of
the restart test's sums. Cuts at random, in lines across the image, at the first and
last edge of every fibre, everywhere, and every other edge; fibres at the edges of
pieces and warps; steps small and so large that radii are clamped between the cuts;
weights whose product with the step underflows, which are no cuts."""

import os
import pathlib
import subprocess
import sys

import numpy as np
import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
SIZES = [(3, 2, 3), (2, 20, 21), (40, 33, 32), (2, 97, 481), (1, 480, 130), (1, 3, 5000)]
CUTS = ("random", "lines", "ends", "all", "every other", "tiny")


def _weights(kind, shape, seed):
    rng = np.random.default_rng(seed)
    w = rng.uniform(0.5, 1.5, (2,) + shape)
    H, W = shape
    if kind == "random":
        w[rng.random(w.shape) < 0.05] = 0.0
    elif kind == "lines":
        w[0, H // 3] = w[1, :, W // 4] = 0.0
        w[1, H // 2] = 0.0
    elif kind == "ends":
        w[0, 0] = w[0, max(H - 2, 0)] = w[1, :, 0] = w[1, :, max(W - 2, 0)] = 0.0
    elif kind == "all":
        w[1] = 0.0
        w[0, :, : W // 2] = 0.0
    elif kind == "every other":
        w[0, ::2] = w[1, :, 1::2] = 0.0
    else:
        w[rng.random(w.shape) < 0.1] = 1e-300
        w[rng.random(w.shape) < 0.02] = 0.0
    return w


def _image(i, shape, seed):
    rng = np.random.default_rng(seed)
    n = rng.normal(size=shape)
    if i % 3 == 0:
        return n
    if i % 3 == 1:
        return np.round(2 * n)
    r = np.arange(shape[1])[None, :, None] * 1e-3 + np.arange(shape[2])[None, None, :] * 1e-2
    return r + 0.01 * n


def _cases():
    for s, shape in enumerate(SIZES):
        for i, kind in enumerate(CUTS):
            for dtype in (np.float32, np.float64):
                for big in (False, True):
                    yield shape, kind, dtype, big, i + s, 100 * s + i


def _run():
    import torch
    from fastprox_b200 import TVAniso
    out = []
    for shape, kind, dtype, big, i, seed in _cases():
        x = _image(i, shape, seed).astype(dtype)
        steps = np.array([(0.1, 0.5, 2.0)[b % 3] for b in range(shape[0])]) * (50.0 if big else 1.0)
        z, _ = TVAniso(2, edge_weights=_weights(kind, shape[1:], seed)).solve(
            torch.as_tensor(x, device="cuda"), torch.as_tensor(steps, device="cuda"), tol=0.0, max_iter=3,
            with_dual=False)
        out.append(z.cpu().numpy())
    return out


@pytest.mark.gpu
def test_cuts_match_one_thread_per_fibre(cuda, tmp_path):
    out = tmp_path / "untiled.npz"
    env = dict(os.environ, FASTPROX_B200_AN_FIB="0", FASTPROX_B200_TILES="0")
    r = subprocess.run([sys.executable, str(pathlib.Path(__file__)), str(out)], cwd=ROOT, env=env,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    ref = np.load(out)
    for i, (z, (shape, kind, dtype, big, _, _)) in enumerate(zip(_run(), _cases())):
        zu = ref[f"z{i}"]
        # the same arithmetic: equal up to the order of the restart test's sums
        tol = 1e-13 if dtype == np.float64 else 1e-6
        err = np.abs(z - zu).max()
        assert err <= tol * (1.0 + np.abs(zu).max()), (shape, kind, dtype, big, err)


if __name__ == "__main__":
    sys.path.insert(0, str(ROOT))
    np.savez(sys.argv[1], **{f"z{i}": z for i, z in enumerate(_run())})
