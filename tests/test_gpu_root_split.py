"""Node 0 of the radix tree (the reference's root over all keys but the last)
is searched for by a warp in rounds of 32 probes: every place where it can
split, at the edges of the rounds, against the oracle bit for bit."""
import numpy as np
import pytest

from test_gpu_parity import assert_same, run_gpu

pytestmark = pytest.mark.gpu


def points_of(codes, axis_bits):
    """Points whose Morton codes are `codes` (box [0, 1024))."""
    c = np.asarray(codes, np.uint64)
    pts = np.ones((len(c), 4), np.float32)
    for a in range(3):
        v = np.zeros(len(c), np.uint64)
        for b in range(axis_bits):
            v |= ((c >> np.uint64(3 * b + a)) & np.uint64(1)) << np.uint64(b)
        pts[:, a] = v.astype(np.float64) * (1024.0 / (1 << axis_bits))
    return pts


@pytest.mark.parametrize("key_bits", [32, 64])
@pytest.mark.parametrize("n", [3, 4, 33, 34, 35, 1025, 2300])
def test_root_splits_anywhere(rw, oracle, n, key_bits):
    axis = 10 if key_bits == 32 else 21
    # every coordinate has at most 21 bits: exact in float32
    half = np.uint64(1) << np.uint64(3 * axis - 1)
    rng = np.random.default_rng(n)
    for s in sorted({0, 1, 2, 30, 31, 32, 33, 62, 63, 64, n // 2, n - 3, n - 2}):
        if not 0 <= s < n - 1:
            continue
        low = rng.choice(1 << 20, size=n, replace=False).astype(np.uint64)
        codes = np.sort(low[:s + 1])
        codes = np.concatenate([codes, half + np.sort(low[s + 1:])])  # key s + 1 is the first past the split
        pts = points_of(rng.permutation(codes), axis)
        app = rw.AppData(n, key_bits, points=pts, octree_ratio=24.0)
        got = run_gpu(rw, pts, key_bits, app=app)
        want = oracle.run(pts, key_bits=key_bits, capacity=app.oct_capacity)
        assert got["n_unique"] == n
        assert_same(got, want, f"n {n} split {s}")
