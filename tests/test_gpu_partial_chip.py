"""Clouds of the one-launch pipeline, and the other forms, on a stream that owns
16 of the chip's SMs (a green context): a cooperative launch of one block per SM of
the chip is refused there, and the general chain of kernels has to take it."""
import numpy as np
import pytest

from test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def part():
    """A torch stream of a green context of 16 SMs."""
    import torch
    drv = pytest.importorskip("cuda.bindings.driver")
    torch.zeros(1, device="cuda")

    def ok(result):
        if int(result[0]) != 0:
            pytest.skip(f"no green context here: {result[0]}")
        return result[1:]

    (dev,) = ok(drv.cuDeviceGet(torch.cuda.current_device()))
    (sms,) = ok(drv.cuDeviceGetDevResource(dev, drv.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    groups = ok(drv.cuDevSmResourceSplitByCount(1, sms, 0, 16))[0]
    (desc,) = ok(drv.cuDevResourceGenerateDesc([groups[0]], 1))
    flags = drv.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM
    (ctx,) = ok(drv.cuGreenCtxCreate(desc, dev, flags))
    (stream,) = ok(drv.cuGreenCtxStreamCreate(ctx, drv.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    yield torch.cuda.ExternalStream(int(stream))
    torch.cuda.synchronize()
    drv.cuStreamDestroy(stream)
    drv.cuGreenCtxDestroy(ctx)


@pytest.mark.parametrize("key_bits", [32, 64])
@pytest.mark.parametrize("n", [3001, 20011, 300007, 700001])
def test_pipeline(rw, oracle, part, n, key_bits):
    import torch
    pts = rw.generate_points(n, rw.GEN_GAUSSIAN_MIXTURE, n, n_components=9)
    want = oracle.run(pts, key_bits=key_bits, capacity=2 * n)
    app = rw.AppData(n, key_bits, points=pts, octree_ratio=2.0)
    im = rw.ImStorage(n, key_bits)
    torch.cuda.synchronize()
    for _ in range(2):
        rw.run_pipeline(app, im, part)
        assert_same(app.results(), want)
    rw.run_pipeline(app, im)  # the whole chip again
    assert_same(app.results(), want)


def test_sort_of_dense_keys(rw, part):
    import torch
    w = np.random.default_rng(3).integers(0, 1 << 31, size=300007, dtype=np.int64)
    keys = torch.from_numpy(w).cuda()
    out = torch.empty_like(keys)
    im = rw.ImStorage(len(w), 64)
    torch.cuda.synchronize()
    rw.sort_keys(keys, out, im, part)
    part.synchronize()
    assert np.array_equal(out.cpu().numpy(), np.sort(w))
