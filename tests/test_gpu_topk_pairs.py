"""Top-8 by two warps per token (csrc/topk.cuh: exact_topk_pair), the sum of the softmax beside the selection: rows whose exponentials tie, differ by a last bit that
the division drops, or vanish, against the oracle, bit for bit, where the number of tokens per CTA changes."""
import numpy as np
import pytest

from conftest import SEED
from test_gpu_group_one import logits

pytestmark = pytest.mark.gpu
KINDS = ["equal", "last bits", "pairs", "tie at the boundary", "vanishing", "ordinary"]


@pytest.mark.parametrize("nb", [1, 65, 296, 297, 511])
def test_kernel_of_its_own(nb, gpu, oracle):
    rows = np.stack([np.roll(logits(KINDS[i % 6]), 37 * i) for i in range(nb)]).astype(np.float32)
    gpu.synth_layer(SEED, 0)
    gpu.poke("logits", rows)
    gpu.stage("topk", 0, nb)
    top, topw = gpu.peek("top", nb).reshape(nb, 8), gpu.peek("topw", nb).reshape(nb, 8)
    for b in range(nb):
        want, w, _ = oracle.topk(rows[b])
        assert np.array_equal(top[b], want) and np.array_equal(topw[b].view(np.uint32), w.view(np.uint32))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("nb", [9, 31, 32, 33, 64])
def test_inside_the_grouping(nb, kind, gpu, oracle):
    gpu.synth_layer(SEED, 0)
    bias = logits(kind)                                       # rows of zeros have no logits of their own
    want, w, _ = oracle.topk(bias)
    gpu.keep_stages(False)
    try:
        gpu.moe(0, np.zeros((nb, 2048), np.float32), bias)
        assert np.array_equal(gpu.peek("top", nb).reshape(nb, 8), np.tile(want, (nb, 1)))
        assert np.array_equal(gpu.peek("topw", nb).reshape(nb, 8).view(np.uint32), np.tile(w.view(np.uint32), (nb, 1)))
    finally:
        gpu.keep_stages(True)
