"""Small clouds whose samples miss most of the keys: one bucket cannot hold its
keys and the launch sorts digit by digit, with one sample list per block and with
two, which rw_tree_im_storage_digit_sorts tells."""
import numpy as np
import pytest

from test_gpu_parity import assert_same
from test_gpu_root_split import points_of

pytestmark = pytest.mark.gpu

SHARE, SAMPLES, LINE = 2048, 32, {32: 14336, 64: 7168}  # csrc/k_small.cu: kSmShare, kSmSamples, kCap


def sampled(n, key_bits, sms):
    """Where the kernel takes its samples, and the sample lists per block."""
    blocks = min(-(-n // SHARE), sms, 256)
    share = -(-n // blocks)
    cap = min(LINE[key_bits], 3 * share + 512)
    lists = 1 if 12 * share <= 5 * cap else 2
    at = []
    for b in range(blocks):
        p0 = min(b * share, n)
        mine = min(n - p0, share)
        t = np.arange(SAMPLES * lists, dtype=np.int64)
        lo, hi = mine * t // len(t), mine * (t + 1) // len(t)
        x = (p0 + lo) & 0xffffffff
        x = ((x ^ 61) ^ (x >> 16)) * 9 & 0xffffffff
        x = (x ^ (x >> 4)) * 0x27d4eb2d & 0xffffffff
        at.append((p0 + lo + (x ^ (x >> 15)) % np.maximum(hi - lo, 1))[hi > lo])
    return np.concatenate(at), lists


@pytest.mark.parametrize("n,key_bits,lists", [(20480, 32, 1), (20480, 64, 1), (303104, 32, 1),
                                              (1000003, 32, 2), (500009, 64, 2)])
def test_digit_by_digit(rw, oracle, n, key_bits, lists):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    at, of = sampled(n, key_bits, sms)
    assert of == lists
    rng = np.random.default_rng(n)
    codes = rng.integers(1 << 10, 1 << (30 if key_bits == 32 else 63), size=n, dtype=np.uint64)
    plain = points_of(codes, 10 if key_bits == 32 else 21)
    codes[at] = 5
    missed = points_of(codes, 10 if key_bits == 32 else 21)
    im = rw.ImStorage(n, key_bits)
    for sorts, pts in ((0, plain), (1, missed), (1, plain), (2, missed)):
        app = rw.AppData(n, key_bits, points=pts, octree_ratio=4.0)
        assert rw.one_launch(app, im)
        rw.run_pipeline(app, im)
        assert_same(app.results(), oracle.run(pts, key_bits=key_bits, capacity=4 * n))
        assert im.digit_sorts() == sorts
    im.clear()
    assert im.digit_sorts() == 0


def test_which_runs_are_one_launch(rw):
    im, im10 = rw.ImStorage(2000000, 32), rw.ImStorage(2000000, 32, 10)
    small, large = rw.AppData(5000), rw.AppData(1200000)
    assert rw.one_launch(small, im) and not rw.one_launch(large, im)
    assert not rw.one_launch(small, im10)
    im.set_sort_variant([v["index"] for v in rw.sort_variants()
                         if v["key_bits"] == 32 and v["radix_bits"] == 8][1])
    assert not rw.one_launch(small, im)
