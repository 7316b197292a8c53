"""Stage 4 on a caller's own keys with the top bit of the word set, which Morton
codes leave clear: the tree depends on the keys' differences only, and nothing
is written for gaps that do not exist."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MORE = 64  # entries behind the nodes
NODE_FIELDS = ("brt_prefix_n", "brt_has_leaf_left", "brt_has_leaf_right", "brt_left_child",
               "brt_parents")


def stage4(rw, keys, bits):
    """The tree's arrays, MORE entries behind the last node's included."""
    import torch
    n = len(keys)
    app = rw.AppData(n + MORE, bits, points=np.zeros((n + MORE, 4), np.float32))
    app.u_morton_keys[:n] = torch.from_numpy(keys.view(np.int32 if bits == 32 else np.int64)).cuda()
    for f in NODE_FIELDS:
        getattr(app, f).fill_(77)
    app.c.n_unique = n
    rw.run_stage4(app, rw.ImStorage(n + MORE, bits))
    return {f: getattr(app, f).cpu().numpy() for f in NODE_FIELDS}


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("n", [3, 32, 33, 257, 2048, 2049, 2305, 6145])
def test_top_bit_set_in_every_key(rw, n, bits):
    dtype = np.uint32 if bits == 32 else np.uint64
    rng = np.random.default_rng(n)
    codes = np.unique(rng.integers(0, 1 << (30 if bits == 32 else 63), size=4 * n, dtype=np.uint64))
    codes = np.sort(rng.permutation(codes)[:n]).astype(dtype)
    want = stage4(rw, codes, bits)
    got = stage4(rw, codes | dtype(1 << (bits - 1)), bits)
    for f in NODE_FIELDS:
        assert np.array_equal(got[f], want[f]), f
        assert (got[f][n:] == 77).all(), f


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("n", [33, 2049, 6145])
def test_top_bit_set_in_some_keys(rw, n, bits):
    """Such keys have no tree of the reference's (its delta would be negative);
    nothing behind the nodes is touched."""
    dtype = np.uint32 if bits == 32 else np.uint64
    rng = np.random.default_rng(n)
    keys = np.unique(rng.integers(0, 1 << bits, size=2 * n, dtype=np.uint64))
    got = stage4(rw, np.sort(rng.permutation(keys)[:n]).astype(dtype), bits)
    for f in NODE_FIELDS:
        assert (got[f][n:] == 77).all(), f
