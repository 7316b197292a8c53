"""The barriers of a small cloud's one launch and the steps of the 64-bit sort of
dense keys give up when what they wait for never comes, without any fault
(rw_tree_wait_probe), and leave the scratch fit for the next run."""
import numpy as np
import pytest

from test_gpu_parity import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("key_bits", [32, 64])
@pytest.mark.parametrize("n", [4097, 50021, 300007])
def test_grid_barrier(rw, oracle, n, key_bits):
    pts = rw.generate_points(n, rw.GEN_UNIFORM, n)
    want = oracle.run(pts, key_bits=key_bits)
    app = rw.AppData(n, key_bits, points=pts)
    im = rw.ImStorage(n, key_bits)
    for limit in (1, 100):
        assert rw.wait_probe(app, im, rw.WAIT_GRID, limit) == rw.RW_ERR_TIMEOUT
        rw.run_pipeline(app, im)
        assert_same(app.results(), want)
    # one nobody waits to hear of
    rw.wait_probe(app, im, rw.WAIT_GRID, 100)
    rw.pipeline_enqueue(app, im)
    rw.pipeline_finish(app, im)
    assert_same(app.results(), want)


@pytest.mark.parametrize("n", [5000, 100003])
def test_jobs(rw, n):
    import torch
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 1 << 31, size=n, dtype=np.int64)
    app = rw.AppData(n, 64, points=np.zeros((n, 4), np.float32))
    im = rw.ImStorage(n, 64)
    app.u_morton_keys.copy_(torch.from_numpy(keys))
    assert rw.wait_probe(app, im, rw.WAIT_JOBS, 100) == rw.RW_ERR_TIMEOUT
    assert np.array_equal(app.u_morton_keys.cpu().numpy(), keys)
    rw.run_stage2(app, im)
    assert np.array_equal(app.u_morton_keys_alt.cpu().numpy(), np.sort(keys))


def test_refused(rw):
    app, im = rw.AppData(4096), rw.ImStorage(4096)
    assert rw.wait_probe(app, im, rw.WAIT_GRID, 100) == rw.RW_ERR_ARG  # one block
    assert rw.wait_probe(app, im, rw.WAIT_JOBS, 100) == rw.RW_ERR_ARG  # 32-bit keys
    app, im = rw.AppData(5000), rw.ImStorage(5000)
    assert rw.wait_probe(app, im, rw.WAIT_GRID, 0) == rw.RW_ERR_ARG
    assert rw.wait_probe(app, im, 2, 100) == rw.RW_ERR_ARG
