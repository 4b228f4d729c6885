"""Float64 quads and float32 3D pairs that stop on their check form the final iterate
again (the third of four, the first of two). Solves that stop so, against single
steps (FASTPROX_B200_QUADS=0 FASTPROX_B200_PAIRS=0, in a child process: the library
reads its hints once): the same number of iterations, more than the nine that run
singly, and the same z and dual up to the two paths' roundings (an iteration at most
triples a difference through the momentum's two terms and adds a few roundings:
ITERS x 3 x 4 x 2^-24 or 2^-53 of the largest value, with at most 80 iterations
1e-4 and 1e-12), where the iterates before and after it differ by 5e-3 to 7e-2 (the
oracle's, at these tolerances). The reported gap is that of the returned dual, formed in float64 by
NumPy, up to the rounding of its terms (32 units r max |x| per pixel)."""

import os
import pathlib
import subprocess
import sys

import numpy as np
import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
GAMMA = 0.2
# dtype, shape (copies of 16 and 8 bytes; 16 and 4), tolerance
CASES = [(np.float64, (40, 64), 3e-3), (np.float64, (33, 57), 3e-3), (np.float64, (70, 129), 1e-3),
         (np.float32, (18, 24, 32), 3e-3), (np.float32, (9, 31, 61), 3e-3), (np.float32, (20, 40, 90), 1e-3)]


def _cases():
    for i, (dtype, shape, tol) in enumerate(CASES):
        for weighted in (False, True):
            rng = np.random.default_rng(i)
            x = np.zeros((2,) + shape)
            x[(slice(None),) + tuple(slice(n // 3, None) for n in shape)] = 1.0
            x = (x + 0.2 * rng.standard_normal(x.shape)).astype(dtype)
            alpha = rng.uniform(0.5, 1.5, shape).astype(dtype) if weighted else None
            yield f"{i}{weighted}", x, alpha, tol


def _run():
    import torch
    from fastprox_b200 import TVIso
    out = {}
    for k, x, alpha, tol in _cases():
        z, info = TVIso(x.ndim - 1, pixel_weights=alpha).solve(torch.as_tensor(x, device="cuda"), GAMMA, tol=tol)
        assert info.converged
        out[k + "z"], out[k + "d"] = z.cpu().numpy(), info.dual.cpu().numpy()
        out[k + "n"], out[k + "g"] = info.image_iters, info.gaps
    return out


def _gap(x, u, r):
    z, g = x.astype(np.float64), np.zeros(u.shape)
    for a in range(x.ndim):
        z += u[a]
        np.moveaxis(z, a, 0)[1:] -= np.moveaxis(u[a], a, 0)[:-1]
    for a in range(x.ndim):
        np.moveaxis(g[a], a, 0)[:-1] = np.diff(np.moveaxis(z, a, 0), axis=0)
    return float(np.sum(r * np.sqrt((g * g).sum(0)) - (g * u).sum(0)))


@pytest.mark.gpu
def test_final_iterate_formed_again(cuda, tmp_path):
    out = tmp_path / "single.npz"
    env = dict(os.environ, FASTPROX_B200_PAIRS="0", FASTPROX_B200_QUADS="0")
    r = subprocess.run([sys.executable, str(pathlib.Path(__file__)), str(out)], cwd=ROOT, env=env,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    ref, got = np.load(out), _run()
    for k, x, alpha, tol in _cases():
        assert np.array_equal(got[k + "n"], ref[k + "n"]), (k, got[k + "n"], ref[k + "n"])
        assert (got[k + "n"] > 9).all() and (got[k + "n"] <= 80).all(), (k, got[k + "n"])
        f64 = x.dtype == np.float64
        for f in "zd":
            scale = np.abs(ref[k + f]).max()
            np.testing.assert_allclose(got[k + f], ref[k + f], rtol=0, atol=(1e-12 if f64 else 1e-4) * scale, err_msg=k + f)
        rad = GAMMA * (np.ones(x.shape[1:]) if alpha is None else alpha.astype(np.float64))
        for b in range(2):
            gap = _gap(x[b], got[k + "d"][:, b].astype(np.float64), rad)
            slack = 32 * (2.0 ** -53 if f64 else 2.0 ** -24) * rad.sum() * np.abs(x).max()
            assert abs(gap - got[k + "g"][b]) <= slack, (k, gap, got[k + "g"][b], slack)


if __name__ == "__main__":
    sys.path.insert(0, str(ROOT))
    np.savez(sys.argv[1], **_run())
