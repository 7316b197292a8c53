"""The end of the 64-bit sort for keys that are dense: segments whose keys mostly
share the bits that the passes sort by (sorted by all digits), long runs among
sparse keys (sorted one by one), and keys sorted in place."""
import numpy as np
import pytest

from test_gpu_parity import FIELDS, assert_same
from test_gpu_root_split import points_of
from test_gpu_sortfix import codes_with_runs, copies, storage

pytestmark = pytest.mark.gpu

FROM, RUN, TILE, SPLIT = 4096, 256, 4096, 1 << 21  # csrc: kDenseFrom, kFixRun, kRestTile, kSplitPoints


def on_gpu(w):
    import torch
    return torch.from_numpy(w.view(np.int32 if w.itemsize == 4 else np.int64)).cuda()


def on_cpu(t):
    a = t.cpu().numpy()
    return a.view(np.uint32 if a.itemsize == 4 else np.uint64)


def dense_keys(kind, n, low):
    """Most keys share the bits above `low` with hundreds of others."""
    rng = np.random.default_rng(n)
    if kind == "one_run":
        return rng.integers(0, 1 << low, size=n, dtype=np.uint64) + (np.uint64(77) << np.uint64(low))
    if kind == "runs":
        return codes_with_runs(rng, [n // 7] * 6 + [n - n // 7 * 6], low)
    if kind == "half_sparse":
        return np.concatenate([dense_keys("runs", n // 2, low),
                               rng.integers(0, 1 << 63, size=n - n // 2, dtype=np.uint64)])
    if kind == "copies":
        return copies(rng, [n // 3, n // 3, n - n // 3 * 2], low)
    return np.full(n, (1 << 64) - 1, np.uint64)  # "equal"


@pytest.mark.parametrize("low", [31, 23])
@pytest.mark.parametrize("n", [FROM, FROM + 1, 2 * TILE + 1, 50021, 300007])
def test_dense(rw, n, low):
    import torch
    im = rw.ImStorage(n if low == 31 else SPLIT + 1, 64)
    for kind in ("one_run", "runs", "half_sparse", "copies", "equal"):
        w = np.random.default_rng(1).permutation(dense_keys(kind, n, low))
        for word in (w, w ^ np.uint64(1 << 63)):  # a caller's keys may have the top bit set
            keys = on_gpu(word)
            out = torch.empty_like(keys)
            rw.sort_keys(keys, out, im)
            assert np.array_equal(on_cpu(out), np.sort(word)), kind


@pytest.mark.parametrize("low", [31, 23])
@pytest.mark.parametrize("lengths", [(RUN, RUN + 1, 300, 512, 1024), (TILE,), (TILE + 1,),
                                     (RUN + 1, 4500)])
def test_long_runs_among_sparse_keys(rw, lengths, low):
    """Few enough that the segment is not dense."""
    import torch
    rng = np.random.default_rng(len(lengths))
    w = rng.integers(0, 1 << 63, size=2000003, dtype=np.uint64)
    w = rng.permutation(np.concatenate([w, codes_with_runs(rng, lengths, low)]))
    keys = on_gpu(w)
    out = torch.empty_like(keys)
    rw.sort_keys(keys, out, rw.ImStorage(len(w) if low == 31 else SPLIT + 1, 64))
    assert np.array_equal(on_cpu(out), np.sort(w))


@pytest.mark.parametrize("low", [31, 23])
def test_pipeline(rw, oracle, low):
    """Head counts of stage 3 with a listed run, and of a dense cloud."""
    rng = np.random.default_rng(low)
    sparse = rng.integers(0, 1 << 63, size=250000, dtype=np.uint64)
    run = codes_with_runs(rng, [1500], low)
    for codes in (np.concatenate([sparse, run, run[::3]]),
                  np.concatenate([dense_keys("runs", 40000, low), sparse[:10000], run[::3]])):
        pts = points_of(rng.permutation(codes), 21)
        want = oracle.run(pts, key_bits=64, capacity=16 * len(pts))
        app = rw.AppData(len(pts), 64, points=pts, octree_ratio=16.0)
        im = storage(rw, len(pts), low, 1)
        for _ in range(2):
            rw.run_pipeline(app, im)
            assert_same(app.results(), want)


def test_batch(rw, oracle):
    rng = np.random.default_rng(9)
    clouds = [points_of(rng.permutation(c), 21) for c in (
        dense_keys("runs", 30000, 31), rng.integers(0, 1 << 63, size=5000, dtype=np.uint64),
        dense_keys("one_run", 9001, 31), dense_keys("one_run", 4001, 31),
        np.concatenate([rng.integers(0, 1 << 63, size=60000, dtype=np.uint64),
                        codes_with_runs(rng, [600], 31)]),
        dense_keys("copies", 8193, 31), rng.integers(0, 1 << 63, size=3, dtype=np.uint64))]
    batch = rw.Batch(clouds, 64, octree_ratio=16.0)
    for _ in range(2):
        batch.run()
        for c, pts in enumerate(clouds):
            want = oracle.run(pts, key_bits=64, capacity=batch.capacity(c)).trimmed()
            got = batch.results(c)
            assert int(batch.status[c]) == 0 or got["n_unique"] < 3
            bad = [k for k in FIELDS
                   if np.ascontiguousarray(got[k]).tobytes() != np.ascontiguousarray(want[k]).tobytes()]
            assert got["n_unique"] == want["n_unique"] and not bad, (c, bad)


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("n", [1, 100, 5000, 200001])
def test_in_place(rw, n, bits):
    w = np.random.default_rng(n).integers(0, 1 << bits, size=n, dtype=np.uint64)
    w = w.astype(np.uint32 if bits == 32 else np.uint64)
    for cap in (n, SPLIT + 1):
        keys = on_gpu(w)
        rw.sort_keys(keys, keys, rw.ImStorage(cap, bits))
        assert np.array_equal(on_cpu(keys), np.sort(w)), cap
