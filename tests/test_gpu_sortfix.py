"""The end of the 64-bit sort: keys that share the bits the passes sort by are
put in order within their run, clouds with longer runs sorted by all digits.
Run lengths and places at their edges, alone, by stages and in a batch, against
the oracle bit for bit."""
import numpy as np
import pytest

from test_gpu_parity import FIELDS, assert_same
from test_gpu_root_split import points_of

pytestmark = pytest.mark.gpu

RUN, TILE, SPLIT = 256, 4096, 1 << 21  # csrc/k_sortfix.cu, csrc/internal.hpp


def codes_with_runs(rng, lengths, low):
    """Distinct 63-bit codes (low bits random), lengths[i] of them sharing their top bits."""
    tops = np.sort(rng.choice(1 << 30, size=len(lengths), replace=False).astype(np.uint64))
    out = []
    for t, n in zip(tops, lengths):
        out.append((t << np.uint64(low)) + rng.integers(0, 1 << low, size=n).astype(np.uint64))
    return np.concatenate(out)


def copies(rng, lengths, low):
    """Codes where lengths[i] copies of one key stand among keys of the same top bits."""
    tops = np.sort(rng.choice(1 << 30, size=len(lengths), replace=False).astype(np.uint64))
    return np.concatenate([np.full(n, (t << np.uint64(low)) + np.uint64(5)) for t, n in zip(tops, lengths)])


def storage(rw, n, low, variant):
    """Scratch of the general chain of kernels (a chosen sort variant), whose
    passes leave `low` bits out."""
    im = rw.ImStorage(n if low == 31 else SPLIT + 1, 64)
    im.set_sort_variant([v["index"] for v in rw.sort_variants()
                         if v["key_bits"] == 64 and v["radix_bits"] == 8][variant])
    return im


SHAPES = {
    "none": [1] * 9000,
    "edges": [TILE - 1, 2, TILE - 3, RUN - 1, 3, RUN, 1, RUN - 2, 1500] ,
    "short_at_tiles": [1] * (TILE - 100) + [RUN] + [1] * (TILE - 300) + [200] + [1] * 50,
    "at_limit": [1] * (TILE - RUN) + [RUN] + [RUN] + [1] * 100,
    "over_limit": [1] * (TILE - RUN) + [RUN + 1] + [1] * 300,
    "over_across": [1] * (TILE - 10) + [RUN + 200] + [1] * (2 * TILE),
    "one_run": [10000],
    "first_and_last": [RUN] + [1] * 5000 + [RUN],
}


@pytest.mark.parametrize("low", [31, 23])
@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_runs(rw, oracle, shape, low):
    rng = np.random.default_rng(len(SHAPES[shape]) + low)
    codes = codes_with_runs(rng, SHAPES[shape], low)
    codes = np.concatenate([codes, codes[::7]])  # some of them twice
    pts = points_of(rng.permutation(codes), 21)
    n = len(pts)
    want = oracle.run(pts, key_bits=64, capacity=16 * n)
    for variant in (1, 2):
        im = storage(rw, n, low, variant)
        for fused in (True, False):
            app = rw.AppData(n, 64, points=pts, octree_ratio=16.0)
            if fused:
                rw.run_pipeline(app, im)
            else:
                for k in range(1, 8):
                    getattr(rw, f"run_stage{k}")(app, im)
            assert_same(app.results(), want, f"{shape} low {low} variant {variant} fused {fused}")


@pytest.mark.parametrize("low", [31, 23])
def test_copies_of_one_key(rw, oracle, low):
    """Long runs of equal keys are in order as they are."""
    rng = np.random.default_rng(low)
    codes = copies(rng, [1] * 3000 + [RUN, 1, RUN + 1, 5000] + [1] * 2000 + [3 * TILE], low)
    pts = points_of(rng.permutation(codes), 21)
    want = oracle.run(pts, key_bits=64, capacity=len(pts))
    app = rw.AppData(len(pts), 64, points=pts, octree_ratio=1.0)
    rw.run_pipeline(app, storage(rw, len(pts), low, 1))
    assert_same(app.results(), want)


def test_batch_sorts_only_the_clouds_that_need_it(rw, oracle):
    rng = np.random.default_rng(5)
    clouds = [points_of(rng.permutation(codes_with_runs(rng, SHAPES[s], 31)), 21)
              for s in ("none", "over_limit", "short_at_tiles", "one_run", "over_across", "at_limit")]
    clouds.insert(2, rw.generate_points(33, rw.GEN_UNIFORM, 4))
    batch = rw.Batch(clouds, 64, octree_ratio=16.0)
    for _ in range(2):
        batch.run()
        assert (batch.status == 0).all()
        for c, pts in enumerate(clouds):
            want = oracle.run(pts, key_bits=64, capacity=batch.capacity(c)).trimmed()
            got = batch.results(c)
            assert got["n_unique"] == want["n_unique"]
            bad = [k for k in FIELDS
                   if np.ascontiguousarray(got[k]).tobytes() != np.ascontiguousarray(want[k]).tobytes()]
            assert not bad, (c, bad)


def test_sort_alone(rw):
    import torch
    rng = np.random.default_rng(6)
    for lengths in ([1] * 700000, [1] * 500000 + [70000] + [3] * 1000):
        codes = rng.permutation(codes_with_runs(rng, lengths, 31)).astype(np.int64)
        keys = torch.from_numpy(codes).cuda()
        out = torch.empty_like(keys)
        rw.sort_keys(keys, out, rw.ImStorage(len(codes), 64))
        torch.cuda.synchronize()
        assert torch.equal(out, torch.sort(keys).values)
