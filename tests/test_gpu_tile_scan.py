"""The one-block scan of tile counts over one and several rounds, full and
ragged: batches of as many tiny clouds as it has tiles (one tile each)."""
import numpy as np
import pytest

from test_gpu_batch import FIELDS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("key_bits", [32, 64])
@pytest.mark.parametrize("clouds", [1, 127, 4095, 4097, 16384, 16387, 20001])
def test_rounds_of_tiles(rw, oracle, clouds, key_bits):
    rng = np.random.default_rng(clouds)
    sizes = rng.integers(4, 24, size=clouds)
    pts = np.ones((int(sizes.sum()), 4), np.float32)
    pts[:, :3] = rng.integers(0, 1024, size=(len(pts), 3))
    pts[rng.random(len(pts)) < 0.2] = pts[0]  # duplicates within clouds
    ends = np.cumsum(sizes)
    parts = [pts[e - s:e] for s, e in zip(sizes, ends)]
    batch = rw.Batch(parts, key_bits, octree_ratio=24.0)
    batch.run(graph=False)
    want_unique = [len(np.unique(p[:, :3], axis=0)) for p in parts]
    assert list(batch.n_unique) == want_unique
    for c in sorted(set(range(0, clouds, 97)) | {clouds - 1, max(0, clouds - 2), min(16383, clouds - 1)}):
        want = oracle.run(parts[c], key_bits=key_bits, capacity=batch.capacity(c))
        if want.status != 0:
            continue
        got = batch.results(c)
        for k, v in want.trimmed().items():
            if k in FIELDS:
                assert np.ascontiguousarray(got[k]).tobytes() == np.ascontiguousarray(v).tobytes(), (c, k)
