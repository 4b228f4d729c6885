"""Anisotropic TV of volumes along two of the three axes, on the piece passes, against
the untiled passes (one thread per fibre, FASTPROX_B200_AN_FIB=0
FASTPROX_B200_TILES=0, in a child process: the library reads its hints once): the
same arithmetic per fibre, so the same iterates up to the order of the restart
test's sums. Each axis left out in turn, extents at the edges of pieces and warps,
and a volume whose second pass has more blocks (4160 of 8 fibres) than any other
kernel of the call has partial sums (4096): it runs the pieces as well, a launch
less per round than the untiled passes, which copy y after a restart."""

import os
import pathlib
import subprocess
import sys

import numpy as np
import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
AXES = [(0.0, 1.0, 1.0), (1.0, 0.0, 0.7), (0.5, 1.0, 0.0)]
SHAPES = [(3, 20, 21), (33, 5, 64), (21, 65, 4), (130, 31, 33)]
LARGE = (320, 480, 104)


def _cases():
    for i, shape in enumerate(SHAPES):
        for w in AXES:
            for dtype in (np.float32, np.float64):
                for edge in (False, True):
                    yield i, shape, w, dtype, edge
    yield 99, LARGE, AXES[0], np.float32, True


def _run():
    import ctypes as C

    import torch
    from fastprox_b200 import TVAniso, capi
    out = {}
    for n, (i, shape, w, dtype, edge) in enumerate(_cases()):
        rng = np.random.default_rng(i)
        x = rng.normal(size=(1 if shape == LARGE else 2,) + shape).astype(dtype)
        beta = rng.uniform(0.5, 1.5, (3,) + shape) if edge else None
        x = torch.as_tensor(x, device="cuda")
        op = TVAniso(3, weights=w, edge_weights=beta)
        z, _ = op.solve(x, 0.4, tol=0.0, max_iter=3, with_dual=False)
        launches, rounds = C.c_int64(), C.c_int64()
        capi.check(capi.lib().fp_b200_workspace_stats(op.workspace(x), C.byref(launches), C.byref(rounds)), "stats")
        out[f"z{n}"] = z.cpu().numpy()
        out[f"n{n}"] = np.array([launches.value, rounds.value])
    return out


@pytest.mark.gpu
def test_two_axes_of_a_volume(cuda, tmp_path):
    out = tmp_path / "untiled.npz"
    env = dict(os.environ, FASTPROX_B200_AN_FIB="0", FASTPROX_B200_TILES="0")
    r = subprocess.run([sys.executable, str(pathlib.Path(__file__)), str(out)], cwd=ROOT, env=env,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    ref, got = np.load(out), _run()
    for n, (i, shape, w, dtype, edge) in enumerate(_cases()):
        z, zu = got[f"z{n}"], ref[f"z{n}"]
        tol = 1e-13 if dtype == np.float64 else 1e-6
        err = np.abs(z - zu).max()
        assert err <= tol * (1.0 + np.abs(zu).max()), (shape, w, dtype, edge, err)
        if shape == LARGE:
            (launches, rounds), (untiled, rounds_u) = got[f"n{n}"], ref[f"n{n}"]
            assert rounds == rounds_u and untiled - launches == rounds, (launches, untiled, rounds)


if __name__ == "__main__":
    sys.path.insert(0, str(ROOT))
    np.savez(sys.argv[1], **_run())
