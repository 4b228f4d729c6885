"""The fibre passes by pieces (several lanes scan one fibre) against the untiled
passes (one thread per fibre, FASTPROX_B200_AN_FIB=0 FASTPROX_B200_TILES=0, in
a child process: the library reads its hints once): the same scan for any
input, so the same iterates up to the order of the restart test's sums. Sizes
at the edges of the pieces and blocks (fibres of 2, 3, 20 and 21 entries, 480
and 481, rows that are and are not a multiple of the vector width, fibres
longer than a block's usual share of shared memory, more images than one
block's fibres) and inputs whose segments are short (noise), long (clean
steps), tied (small integers) and curved (a ramp: many rescans)."""

import os
import pathlib
import subprocess
import sys

import numpy as np
import pytest

ROOT = pathlib.Path(__file__).resolve().parents[1]
SIZES = [(3, 2, 3), (2, 20, 21), (70, 33, 32), (2, 97, 481), (1, 480, 130), (1, 3, 9000), (1, 5000, 4)]
KINDS = ("noise", "steps", "integers", "ramp")


def _image(kind, shape, seed):
    rng = np.random.default_rng(seed)
    n = rng.normal(size=shape)
    if kind == "noise":
        return n
    if kind == "integers":
        return np.round(2 * n)
    B, H, W = shape
    i, j = np.arange(H)[:, None], np.arange(W)[None, :]
    if kind == "steps":
        return np.broadcast_to((i // 37 % 3) * 0.4 + (j // 53 % 2) * 0.7, shape) + 0.0 * n
    return np.broadcast_to(1e-3 * (i * i) / max(H, 1) + 0.01 * j, shape) + 0.01 * n


def _cases():
    for s, shape in enumerate(SIZES):
        for kind in KINDS:
            for dtype in (np.float32, np.float64):
                for edge in (False, True):
                    yield shape, kind, dtype, edge, 100 * s


def _run():
    import torch
    from fastprox_b200 import TVAniso, synth
    out = []
    for shape, kind, dtype, edge, seed in _cases():
        x = _image(kind, shape, seed).astype(dtype)
        beta = synth.pixel_weights((2,) + shape[1:], seed=seed + 1) if edge else None
        steps = np.array([(0.1, 0.5, 2.0)[b % 3] for b in range(shape[0])])
        z, _ = TVAniso(2, edge_weights=beta).solve(torch.as_tensor(x, device="cuda"),
                                                   torch.as_tensor(steps, device="cuda"), tol=0.0, max_iter=3,
                                                   with_dual=False)
        out.append(z.cpu().numpy())
    return out


@pytest.mark.gpu
def test_pieces_match_one_thread_per_fibre(cuda, tmp_path):
    out = tmp_path / "untiled.npz"
    env = dict(os.environ, FASTPROX_B200_AN_FIB="0", FASTPROX_B200_TILES="0")
    r = subprocess.run([sys.executable, str(pathlib.Path(__file__)), str(out)], cwd=ROOT, env=env,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    ref = np.load(out)
    for i, (z, (shape, kind, dtype, edge, _)) in enumerate(zip(_run(), _cases())):
        zu = ref[f"z{i}"]
        # the same arithmetic: equal up to the order of the restart test's sums
        tol = 1e-13 if dtype == np.float64 else 1e-6
        err = np.abs(z - zu).max()
        assert err <= tol * (1.0 + np.abs(zu).max()), (shape, kind, dtype, edge, err)


if __name__ == "__main__":
    sys.path.insert(0, str(ROOT))
    np.savez(sys.argv[1], **{f"z{i}": z for i, z in enumerate(_run())})
