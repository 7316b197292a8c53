"""The sort's unordered first pass at tile edges and with crowded digits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("key_bits", [32, 64])
@pytest.mark.parametrize("low", ["random", "one", "two"])
def test_first_pass_edges(rw, low, key_bits):
    import torch
    rng = np.random.default_rng(key_bits)
    bits = 30 if key_bits == 32 else 63
    for v in sort_variants(rw, key_bits):
        tile = v["threads"] * v["keys_per_thread"]
        for n in (1, 31, tile - 1, tile, tile + 1, 3 * tile + 17):
            k = rng.integers(0, 1 << bits, size=n).astype(np.int64)
            if low != "random":  # the first digit takes one value, or two
                shift = 0 if key_bits == 32 else 31
                k &= ~(0xff << shift)
                if low == "two":
                    k |= rng.integers(0, 2, size=n).astype(np.int64) << (shift + 3)
            keys = torch.from_numpy(k.astype(np.int32) if key_bits == 32 else k).cuda()
            out = torch.full((n + 64,), -1, dtype=keys.dtype, device="cuda")
            im = rw.ImStorage(n, key_bits)
            im.set_sort_variant(v["index"])
            rw.sort_keys(keys, out[:n], im)
            torch.cuda.synchronize()
            assert torch.equal(out[:n], torch.sort(keys).values), (v, n)
            assert (out[n:] == -1).all(), (v, n)


def sort_variants(rw, key_bits):
    seen, out = set(), []
    for v in rw.sort_variants():  # one per tile shape: the first pass is the same for all rankings
        shape = (v["threads"], v["keys_per_thread"])
        if v["key_bits"] == key_bits and v["radix_bits"] == 8 and shape not in seen:
            seen.add(shape)
            out.append(v)
    return out
