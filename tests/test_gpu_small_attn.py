"""The calls around attention at decode sizes (rows through page-locked memory in place up to 96 tokens, dense tiles of 8 up to 128, above that the
chunked flow) against the reference statements: the same bits."""
import numpy as np
import pytest

from conftest import same_bits
import dense_ref
from test_gpu_attn_head import attention_head_case, bf16_to_f32

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def matrix(gpu):
    rng = np.random.default_rng(61)
    codes = (rng.integers(0, 3, (3, 1024, 512)) * 0x55).astype(np.uint8)
    scales = rng.uniform(0.01, 0.05, (3, 1024)).astype(np.float32)
    for c, s in zip(codes, scales):
        gpu.dense_add(40, c, s, 1024, 2048)
    gpu.dense_done(2048)
    return codes.reshape(3072, 512), scales.reshape(-1)


@pytest.mark.parametrize("keep", [True, False])
@pytest.mark.parametrize("nb", [1, 7, 8, 9, 20, 64, 95, 96, 97, 127, 128, 129])
def test_dense_at_decode_sizes(nb, keep, matrix, gpu):
    codes, scales = matrix
    x = np.random.default_rng(nb).standard_normal((nb, 2048)).astype(np.float32)
    x[nb // 2] = 0.0
    gpu.keep_stages(keep)
    try:
        y, secs = gpu.dense(40, x, 3072)
    finally:
        gpu.keep_stages(True)
    assert secs > 0 and same_bits(y, dense_ref.dense(codes, scales, 3072, 2048, x))


@pytest.mark.parametrize("nb,glob", [(1, 0), (2, 1), (5, 0), (95, 0), (96, 1), (97, 0)])
def test_rope_at_decode_sizes(nb, glob, gpu, oracle):
    q, k, v, qn, kn, pos = attention_head_case(70 + nb, nb)
    angle = np.arange(4096)[:, None] * (10000.0 ** (-np.arange(32) / 32))[None, :]
    cs = np.stack([np.cos(angle), np.sin(angle)], -1).astype(np.float32)
    want_q, _, want_kc, want_vc = oracle.qk_rope(q, k, v, qn, kn, pos, cs, glob)
    gpu.rope_table(cs)
    got_q, got_kc, got_vc, _ = gpu.qk_rope(np.concatenate([q, k, v], 1), pos, glob, bf16_to_f32(qn), bf16_to_f32(kn))
    assert same_bits(got_q, want_q) and np.array_equal(got_kc, want_kc) and np.array_equal(got_vc, want_vc)
