"""Top-8 by two warps per token (csrc/topk.cuh: exact_topk_pair), the sum of the softmax beside the selection: rows whose exponentials tie, differ by a last bit that
the division drops, or vanish, against the oracle, bit for bit, where the number of tokens per CTA changes."""
import numpy as np
import pytest

from test_gpu_group_one import layer, logits  # noqa: F401

pytestmark = pytest.mark.gpu
KINDS = ["equal", "last bits", "pairs", "tie at the boundary", "vanishing", "ordinary"]


@pytest.mark.parametrize("nb", [1, 65, 296, 297, 511])
def test_kernel_of_its_own(nb, layer, gpu, oracle):
    rows = np.stack([np.roll(logits(KINDS[i % 6]), 37 * i) for i in range(nb)]).astype(np.float32)
    gpu.poke("logits", rows)
    gpu.stage("topk", 0, nb)
    top, topw = gpu.peek("top", nb).reshape(nb, 8), gpu.peek("topw", nb).reshape(nb, 8)
    for b in range(nb):
        want, w, _ = oracle.topk(rows[b])
        assert np.array_equal(top[b], want) and np.array_equal(topw[b].view(np.uint32), w.view(np.uint32))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("nb", [9, 31, 32, 33, 64])
def test_inside_the_grouping(nb, kind, layer, gpu, oracle):
    bias = logits(kind)                                       # rows of zeros have no logits of their own
    want, w, _ = oracle.topk(bias)
    gpu.keep_stages(False)
    try:
        gpu.moe(0, np.zeros((nb, 2048), np.float32), bias)
        assert np.array_equal(gpu.peek("top", nb).reshape(nb, 8), np.tile(want, (nb, 1)))
        assert np.array_equal(gpu.peek("topw", nb).reshape(nb, 8).view(np.uint32), np.tile(w.view(np.uint32), (nb, 1)))
    finally:
        gpu.keep_stages(True)


# The 8th and 9th exponential are equal and others, smaller by last bits, have the same quotient: the reference's first strict maximum takes the lowest index of them all.
@pytest.mark.parametrize("nb", [1, 9, 32, 33, 296, 297, 511])
def test_ties_and_last_bits_at_the_boundary(nb, layer, gpu, oracle):
    rows = np.stack([logits("tie over a last bit" if i % 8 == 0 else "crowded %d" % i) for i in range(nb)])
    gpu.poke("logits", rows)
    gpu.stage("topk", 0, nb)
    top, topw = gpu.peek("top", nb).reshape(nb, 8), gpu.peek("topw", nb).reshape(nb, 8)
    want = [oracle.topk(r) for r in rows]
    assert [b for b in range(nb) if not np.array_equal(top[b], want[b][0])] == []
    assert [b for b in range(nb) if not np.array_equal(topw[b].view(np.uint32), want[b][1].view(np.uint32))] == []


@pytest.mark.parametrize("kind", ["tie over a last bit", "crowded 4", "crowded 8", "crowded 33"])
@pytest.mark.parametrize("nb", [2, 8, 9, 32, 33, 296, 297, 511])
def test_ties_and_last_bits_inside_a_call(nb, kind, layer, gpu, oracle):
    test_inside_the_grouping(nb, kind, layer, gpu, oracle)


@pytest.mark.parametrize("kind", ["tie over a last bit", "crowded 4", "crowded 8", "crowded 33"])
def test_ties_and_last_bits_in_recomputed_tokens(kind, layer, gpu, clib, oracle):
    nb = 512                                                  # every row has the bias for its logits and is recomputed
    bias = logits(kind)
    want, w, _ = oracle.topk(bias)
    gpu.poke("bias", bias)
    gpu.poke("hn", np.zeros((nb, 2048), np.float32))
    gpu.stage("router_tensor_bias", 0, nb)
    assert clib.gmoe_router_flagged() == nb
    assert np.array_equal(gpu.peek("top", nb).reshape(nb, 8), np.tile(want, (nb, 1)))
    assert np.array_equal(gpu.peek("topw", nb).reshape(nb, 8).view(np.uint32), np.tile(w.view(np.uint32), (nb, 1)))
