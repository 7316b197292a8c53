"""Sorts of a caller's own keys order them by the whole word: keys with the bits
above a Morton code's set (30 of 32, 63 of 64) are accepted and come out sorted,
through every entry point that takes keys."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SPLIT = 1 << 21  # csrc/internal.hpp: more passes for larger scratch


def words(n, bits, seed, kind="any"):
    rng = np.random.default_rng(seed)
    w = rng.integers(0, 1 << bits, size=n, dtype=np.uint64)
    if kind == "top":  # most differ in nothing but the bits a code leaves clear
        w = (w >> np.uint64(bits - 2) << np.uint64(bits - 2)) | (w & np.uint64(3))
    return w.astype(np.uint32 if bits == 32 else np.uint64)


def on_gpu(w):
    import torch
    return torch.from_numpy(w.view(np.int32 if w.itemsize == 4 else np.int64)).cuda()


def on_cpu(t):
    a = t.cpu().numpy()
    return a.view(np.uint32 if a.itemsize == 4 else np.uint64)


def variants(rw, bits):
    return [v["index"] for v in rw.sort_variants() if v["key_bits"] == bits and v["radix_bits"] == 8]


@pytest.mark.parametrize("kind", ["any", "top"])
@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("n", [1, 33, 4097, 300007])
def test_sort_keys(rw, n, bits, kind):
    import torch
    w = words(n, bits, n, kind)
    keys = on_gpu(w)
    for variant in variants(rw, bits) if n > 33 else variants(rw, bits)[:1]:
        im = rw.ImStorage(n, bits)
        im.set_sort_variant(variant)
        out = torch.empty_like(keys)
        rw.sort_keys(keys, out, im)
        assert np.array_equal(on_cpu(out), np.sort(w)), variant
        assert np.array_equal(on_cpu(keys), w)  # the input stays


@pytest.mark.parametrize("kind", ["any", "top"])
def test_wide_keys_of_large_scratch(rw, kind):
    import torch
    w = words(200001, 64, 7, kind)
    keys = on_gpu(w)
    out = torch.empty_like(keys)
    rw.sort_keys(keys, out, rw.ImStorage(SPLIT + 1, 64))
    assert np.array_equal(on_cpu(out), np.sort(w))


@pytest.mark.parametrize("bits", [32, 64])
def test_stage2_and_profile(rw, bits):
    n = 50021
    w = words(n, bits, 3)
    app, im = rw.AppData(n, bits, points=np.zeros((n, 4), np.float32)), rw.ImStorage(n, bits)
    app.u_morton_keys.copy_(on_gpu(w))
    rw.run_stage2(app, im)
    assert np.array_equal(on_cpu(app.u_morton_keys_alt), np.sort(w))
    app.u_morton_keys_alt.zero_()
    rw.profile_sort(app.u_morton_keys, app.u_morton_keys_alt, im, reps=1)
    assert np.array_equal(on_cpu(app.u_morton_keys_alt), np.sort(w))


@pytest.mark.parametrize("kind", ["any", "top"])
def test_learned_sort(rw, kind):
    """Below 65,536 keys the learned sort is the onesweep sort; a few values with
    most of the keys each overflow its buckets, which is decided on the device.
    Its sample is sorted by the same kernels."""
    learned = rw.Learned(1 << 18)
    for n, few in ((5000, False), (1 << 17, True), (1 << 18, False)):
        w = words(n, 32, n, kind)
        if few:
            w = np.random.default_rng(1).choice(w[:3], size=n)
        im = rw.ImStorage(n, 32)
        out, stats = learned.sort(on_gpu(w), fallback_im=im)
        assert stats["fell_back"] == 1 or (n == 1 << 18 and kind == "any")
        assert np.array_equal(on_cpu(out), np.sort(w))
