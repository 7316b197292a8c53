"""The one-launch pipeline of small clouds against the oracle and against the
general chain of kernels, bit for bit: one block and several, both key widths,
the options, duplicates, shares and buckets at their edges, and the
digit-by-digit sort that takes over when a bucket overflows."""
import numpy as np
import pytest

from oracle import ORC_OK
from test_gpu_parity import FIELDS, assert_same, cloud, run_gpu
from test_gpu_root_split import points_of

pytestmark = pytest.mark.gpu

SAMPLES, ALONE, SHARE = 32, 4096, 2048  # csrc/k_small.cu


def general(rw, pts, key_bits, options=0):
    """The same cloud through the general kernels (a chosen sort variant keeps
    the one-launch form away)."""
    n = len(pts)
    app, im = rw.AppData(n, key_bits, points=pts, octree_ratio=3.0), rw.ImStorage(n, key_bits)
    im.set_options(options)
    im.set_sort_variant([v["index"] for v in rw.sort_variants()
                         if v["key_bits"] == key_bits and v["radix_bits"] == 8][1])
    rw.run_pipeline(app, im)
    return app.results()


def check(rw, oracle, pts, key_bits, options=0, label=""):
    n = len(pts)
    app, im = rw.AppData(n, key_bits, points=pts, octree_ratio=3.0), rw.ImStorage(n, key_bits)
    im.set_options(options)
    want = oracle.run(pts, key_bits=key_bits, capacity=app.oct_capacity, options=options)
    assert want.status == ORC_OK
    for _ in range(2):  # a second run finds the scratch as the first left it
        rw.run_pipeline(app, im)
        assert_same(app.results(), want, label)
    gen = general(rw, pts, key_bits, options)
    got = app.results()
    assert all(np.ascontiguousarray(got[k]).tobytes() == np.ascontiguousarray(gen[k]).tobytes() for k in FIELDS)


@pytest.mark.parametrize("key_bits", [32, 64])
@pytest.mark.parametrize("kind", ["uniform", "gauss"])
@pytest.mark.parametrize("n", [3, 33, 1023, 1025, ALONE, ALONE + 1, 2 * SHARE + 1, 20001, 65537])
def test_sizes(rw, oracle, n, kind, key_bits):
    check(rw, oracle, cloud(rw, n, kind, n), key_bits, label=f"{n} {kind} {key_bits}")


@pytest.mark.parametrize("key_bits,n", [(32, 148 * SHARE - 1), (32, 148 * SHARE + 1), (32, 879999),
                                        (32, 890000), (32, 1100000), (32, 1100001),
                                        (64, 442000), (64, 550000), (64, 550001)])
def test_largest(rw, oracle, n, key_bits):
    check(rw, oracle, cloud(rw, n, "gauss", 3), key_bits, label=f"{n} {key_bits}")


@pytest.mark.parametrize("options", [1, 2, 3])
@pytest.mark.parametrize("n,key_bits", [(3000, 32), (50000, 32), (50000, 64)])
def test_options(rw, oracle, n, key_bits, options):
    check(rw, oracle, cloud(rw, n, "gauss", options), key_bits, options, f"{n} {key_bits} {options}")


@pytest.mark.parametrize("key_bits", [32, 64])
@pytest.mark.parametrize("distinct", [3, 17, 1000])
def test_duplicates(rw, oracle, distinct, key_bits):
    rng = np.random.default_rng(distinct)
    axis = 10 if key_bits == 32 else 21
    values = rng.choice(1 << 30, size=distinct, replace=False).astype(np.uint64)
    weights = 1.0 / np.arange(1, distinct + 1) ** 2  # one value takes most of the keys
    codes = rng.choice(values, size=60000, p=weights / weights.sum())
    codes[:distinct] = values
    check(rw, oracle, points_of(codes, axis), key_bits, label=f"{distinct} distinct")


def sampled_positions(n):
    """Where the kernel takes its samples."""
    blocks = -(-n // SHARE)
    share = -(-n // blocks)
    at = []
    for b in range(blocks):
        p0 = b * share
        mine = min(n - p0, share)
        for t in range(SAMPLES):
            lo, hi = mine * t // SAMPLES, mine * (t + 1) // SAMPLES
            x = (p0 + lo) & 0xffffffff
            x = ((x ^ 61) ^ (x >> 16)) * 9 & 0xffffffff
            x = (x ^ (x >> 4)) * 0x27d4eb2d & 0xffffffff
            at.append(p0 + lo + (x ^ (x >> 15)) % (hi - lo))
    return at


@pytest.mark.parametrize("key_bits", [32, 64])
def test_overflowing_bucket_sorts_by_digits(rw, oracle, key_bits):
    """Every sample is one key and all the others lie above it: they meet in
    the last bucket, which cannot hold them."""
    n, axis = 20480, 10 if key_bits == 32 else 21
    rng = np.random.default_rng(key_bits)
    codes = rng.integers(1 << 10, 1 << 30, size=n).astype(np.uint64)
    codes[sampled_positions(n)] = 5
    check(rw, oracle, points_of(codes, axis), key_bits, label="overflow")


def test_degenerate_and_capacity_errors(rw, oracle):
    for n in (100, 10000):
        pts = np.ones((n, 4), np.float32)
        app, im = rw.AppData(n, 32, points=pts), rw.ImStorage(n, 32)
        with pytest.raises(rw.RwTreeError) as e:
            rw.run_pipeline(app, im)
        assert e.value.code == rw.RW_ERR_DEGENERATE and app.get_n_unique() == 1
        pts = cloud(rw, n, "uniform", 1)
        tight = rw.AppData(n, 32, points=pts, octree_ratio=0.05)
        with pytest.raises(rw.RwTreeError) as e:
            rw.run_pipeline(tight, im)
        assert e.value.code == rw.RW_ERR_CAPACITY
        # the offsets are made all the same, and the scratch serves the next run
        want = oracle.run(pts, capacity=3 * n)
        b = want.n_brt_nodes
        assert (tight.u_edge_offset[:b].cpu().numpy() == want.edge_offset[:b]).all()
        assert_same(run_gpu(rw, pts, app=rw.AppData(n, 32, points=pts, octree_ratio=3.0), im=im), want)


def test_one_scratch_serves_many_sizes_and_a_graph(rw, oracle):
    import torch
    im = rw.ImStorage(2_000_000, 32)
    sizes = (40000, 5, 1_500_000, 4097, 300000, 100)
    for n in sizes:
        pts = cloud(rw, n, "uniform", n)
        app = rw.AppData(n, 32, points=pts, octree_ratio=3.0)
        assert_same(run_gpu(rw, pts, app=app, im=im), oracle.run(pts, capacity=3 * n), str(n))
    pts = cloud(rw, 50000, "gauss", 9)
    app = rw.AppData(50000, 32, points=pts, octree_ratio=3.0)
    stream = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        rw.pipeline_enqueue(app, im, torch.cuda.current_stream())
    for seed in (9, 10):
        pts = cloud(rw, 50000, "gauss", seed)
        app.set_points(pts)
        for _ in range(3):
            g.replay()
        torch.cuda.synchronize()
        rw.pipeline_finish(app, im)
        assert_same(app.results(), oracle.run(pts, capacity=150000), f"graph {seed}")
    del g
