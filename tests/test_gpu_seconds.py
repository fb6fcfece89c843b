"""The seconds that gpre_dense and gmoe_qk_rope return for calls that are cut into chunks: the kernels' own time, whatever the host and the link do
meanwhile.  Lower bounds from the operations and bytes of the call; upper bounds from the number of chunks (86 to 256 tokens each) and the largest
time that a chunk's kernel may take: 15 us for the product (2 row blocks of 16 K-blocks at 0.3 us each, start and epilogue 5 us), 6 us for the
norm and rotation (5.8 MB in and out at 2 TB/s, start 3 us).  Pairs of events around the launches gave 225 us and more for each of them."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
I8_OPS, L2_BYTES = 4.57e15, 2e13       # the tensor pipe's measured rate; no kernel reads or writes faster than this


def chunks(nb):
    return min(-(-nb // 86), 9)          # none but the last has fewer than 86 tokens (1 MB of rows); about seven otherwise, of 256 tokens at most


@pytest.fixture(scope="module")
def matrix(gpu):
    rng = np.random.default_rng(8)
    for rows in (2048, 1024):
        gpu.dense_add(41, (rng.integers(0, 3, (rows, 512)) * 0x55).astype(np.uint8), rng.uniform(0.01, 0.05, rows).astype(np.float32), rows, 2048)
    gpu.dense_done(2048)


@pytest.mark.parametrize("nb", [97, 129, 600, 2048])
def test_product_seconds(nb, matrix, gpu):
    x = np.random.default_rng(nb).standard_normal((nb, 2048)).astype(np.float32)
    for _ in range(6):
        t0 = time.perf_counter()
        secs = gpu.dense(41, x, 3072)[1]
        wall = time.perf_counter() - t0
        assert 2 * nb * 3072 * 2048 / I8_OPS < secs < min(wall, 15e-6 * chunks(nb))


@pytest.mark.parametrize("nb", [97, 300, 2048])
def test_rotation_seconds(nb, gpu):
    rng = np.random.default_rng(nb)
    qkv, pos, one = rng.standard_normal((nb, 3072)).astype(np.float32), np.arange(nb, dtype=np.int32), np.ones(128, np.float32)
    for _ in range(6):
        t0 = time.perf_counter()
        secs = gpu.qk_rope(qkv, pos, 1, one, one)[3]
        wall = time.perf_counter() - t0
        assert nb * (3072 * 4 + 2048 * 4 + 2 * 1024) / L2_BYTES < secs < min(wall, 6e-6 * chunks(nb))
