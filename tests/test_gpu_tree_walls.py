"""Radix tree and octree rows of the general kernels where a tile's window of
2,048 gaps and a halo of 256 ends at or near the cloud's ends: whole clouds,
low and high codes at the ends, against the oracle bit for bit."""
import numpy as np
import pytest

from test_gpu_parity import assert_same, run_gpu
from test_gpu_root_split import points_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("key_bits", [32, 64])
@pytest.mark.parametrize("n", [3, 32, 34, 255, 257, 2047, 2048, 2049, 2050, 2304, 2305, 2306,
                               4097, 4352, 4353, 6145])
def test_windows_at_the_ends(rw, oracle, n, key_bits):
    axis = 10 if key_bits == 32 else 21
    full = (1 << 3 * axis) - 1
    rng = np.random.default_rng(n)
    codes = {0, full} | {int(c) for c in rng.integers(0, full, size=n)}
    while len(codes) < n:
        codes.add(int(rng.integers(0, full)))
    codes = np.array(sorted(codes)[:n - 1] + [full], np.uint64)
    pts = points_of(rng.permutation(codes), axis)
    app = rw.AppData(n, key_bits, points=pts, octree_ratio=24.0)
    want = oracle.run(pts, key_bits=key_bits, capacity=app.oct_capacity)
    im = rw.ImStorage(n, key_bits)
    other = [v["index"] for v in rw.sort_variants()
             if v["key_bits"] == key_bits and v["radix_bits"] == 8]
    # a variant the caller chose takes the general kernels: with two, at least one is not the default
    for v in other[:2]:
        im.set_sort_variant(v)
        assert_same(run_gpu(rw, pts, key_bits, app=app, im=im), want, f"n {n} variant {v}")
    im = rw.ImStorage(n, key_bits)
    assert_same(run_gpu(rw, pts, key_bits, fused=False, app=app, im=im), want, f"n {n} stages")
