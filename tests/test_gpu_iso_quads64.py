"""Float64 quad launches (one column per lane; 16- and 8-byte copies for rows of
an even and an odd width) against single steps (FASTPROX_B200_QUADS=0, in a child
process: the library reads its hints once). Both do the same IEEE float64
operations per pixel, but the compiler may fuse a product into a sum in one and
not in the other, so u and z differ by roundings: a projected step is not
expansive and the momentum at most triples a difference per iteration's two
terms, which over the 60 iterations run here leaves 60 x 3 x 2^-53 of the largest
value, about 2e-14; 1e-12 is asked. The iteration counts are those asked for."""

import os
import pathlib
import subprocess
import sys

import numpy as np
import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
# one window, its last column, two windows, the last window's overlap; heights below and above a band
SHAPES = [(2, 32), (3, 33), (40, 34), (9, 35), (8, 55), (17, 56), (33, 57), (7, 80), (61, 81), (12, 104), (31, 105),
          (70, 129)]
ITERS = 61  # not a multiple of four: a single step follows the quads


def _run():
    import torch
    from fastprox_b200 import TVIso, synth
    out = {}
    for i, (H, W) in enumerate(SHAPES):
        for weighted in (False, True):
            x = torch.as_tensor(synth.phantom(2, H, W, seed=i).astype(np.float64), device="cuda")
            alpha = synth.pixel_weights((H, W), seed=50 + i).astype(np.float64) if weighted else None
            z, info = TVIso(2, pixel_weights=alpha).solve(x, 0.1, tol=0.0, max_iter=ITERS)
            out[f"{i}{weighted}z"], out[f"{i}{weighted}d"] = z.cpu().numpy(), info.dual.cpu().numpy()
            out[f"{i}{weighted}n"], out[f"{i}{weighted}g"] = info.image_iters, info.gaps
    return out


@pytest.mark.gpu
def test_float64_quads_match_single_steps(cuda, tmp_path):
    out = tmp_path / "single.npz"
    env = dict(os.environ, FASTPROX_B200_QUADS="0")
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
                np.testing.assert_allclose(got[k + f], ref[k + f], rtol=0, atol=1e-12 * scale, err_msg=str((shape, f)))
            # sums of at most 2 H W terms that cancel down to the gap from about |x|^2 H W
            np.testing.assert_allclose(got[k + "g"], ref[k + "g"], rtol=1e-9, atol=1e-12 * shape[0] * shape[1])


if __name__ == "__main__":
    sys.path.insert(0, str(ROOT))
    np.savez(sys.argv[1], **_run())
