"""The learned sort refuses scratch of 64-bit keys for its fallback, whose kernels
would read the 32-bit keys as 64-bit ones, before anything is enqueued."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radix_bits", [8, 10, 11])
@pytest.mark.parametrize("n", [5000, 1 << 16])
def test_wide_fallback_is_refused(rw, n, radix_bits):
    import torch
    learned = rw.Learned(1 << 16)
    w = np.random.default_rng(n).integers(0, 1 << 30, size=n, dtype=np.int32)
    keys = torch.from_numpy(w).cuda()
    with pytest.raises(rw.RwTreeError) as e:
        learned.sort(keys, fallback_im=rw.ImStorage(n, 64, radix_bits))
    assert e.value.code == rw.RW_ERR_ARG
    out, _ = learned.sort(keys, fallback_im=rw.ImStorage(n, 32, radix_bits))
    assert np.array_equal(out.cpu().numpy(), np.sort(w))
