"""Top-8 and grouping of one token (csrc/k_route.cu: group_one_kernel), which selects by the exponentials while their sum is still being added up: logits whose
exponentials tie, differ by a last bit that the division drops, or vanish, against the oracle's selection by the quotients."""
import numpy as np
import pytest

from conftest import SEED

pytestmark = pytest.mark.gpu


def logits(kind):
    rng = np.random.default_rng(7)
    if kind == "equal":
        return np.zeros(256, np.float32)
    if kind == "last bits":                                  # exponentials 1 - i 2^-24 over a sum of 256: several to a quotient
        return (-rng.permutation(256) * 2.0 ** -24).astype(np.float32)
    if kind == "pairs":
        return (-(rng.permutation(256) // 2) * 2.0 ** -24).astype(np.float32)
    if kind == "tie at the boundary":
        v = np.full(256, -3.0, np.float32)
        v[[200, 13, 77, 5, 250, 9]] = [1.0, 2.0, 0.5, 0.25, 3.0, 0.125]
        return v
    if kind == "tie over a last bit":                        # the 8th and 9th exponential are equal, a smaller one has their quotient and a lower index
        v = np.full(256, -8.0, np.float32)
        v[100:170:10] = np.arange(1.0, 2.75, 0.25)
        v[[200, 210]] = np.uint32(0x3f0075f7).view(np.float32)
        v[50] = np.uint32(0x3f0075f6).view(np.float32)
        return v
    if kind.startswith("crowded"):                           # many ties and many last bits at the boundary
        k = np.random.default_rng([3, int(kind.split()[1])]).integers(0, 60, 256)
        k[0] = 0
        return (-k * 2.0 ** -24).astype(np.float32)
    if kind == "vanishing":                                  # six exponentials above zero
        v = np.full(256, -200.0, np.float32)
        v[[31, 7, 255, 128, 64, 63]] = [0, -1, -2, -3, -4, -87]
        return v
    return rng.standard_normal(256).astype(np.float32)


@pytest.fixture(scope="module")
def layer(gpu):                                               # once: every generation takes a region id
    gpu.synth_layer(SEED, 0)


@pytest.mark.parametrize("kind", ["equal", "last bits", "pairs", "tie at the boundary", "vanishing", "ordinary", "tie over a last bit", "crowded 4", "crowded 8", "crowded 33"])
def test_one_token(kind, layer, gpu, oracle):
    g = gpu
    bias = logits(kind)
    top, topw, _ = oracle.topk(bias)                          # a row of zeros has no logits of its own
    nu, ue, ustart, utok, uw, tp = oracle.group(top[None, :], topw[None, :])
    g.keep_stages(False)
    try:
        for _ in range(3):                                    # plainly, while captured, as a replay
            g.moe(0, np.zeros((1, 2048), np.float32), bias)
            assert np.array_equal(g.peek("top", 1).ravel(), top) and np.array_equal(g.peek("topw", 1).ravel().view(np.uint32), topw.view(np.uint32))
            assert int(g.peek("nu", 1)[0]) == nu == 8
            assert np.array_equal(g.peek("ue", 1)[:8], ue[:8]) and np.array_equal(g.peek("ustart", 1)[:9], ustart[:9])
            assert np.array_equal(g.peek("utok", 1).ravel(), utok.ravel()) and np.array_equal(g.peek("tp", 1).ravel(), tp.ravel())
            assert np.array_equal(g.peek("uw", 1).ravel().view(np.uint32), uw.ravel().view(np.uint32))
    finally:
        g.keep_stages(True)
