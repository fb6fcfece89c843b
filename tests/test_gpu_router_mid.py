"""The router of a few hundred tokens (csrc/k_router_tile.cu: router_mid_kernel) against the oracle, where its choice of 12 or 16 tokens per CTA changes and
where the last CTA holds one token or all of them."""
import numpy as np
import pytest

from conftest import SEED

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def layer(gpu):
    gpu.synth_layer(SEED, 2)


@pytest.mark.parametrize("nb", [145, 156, 157, 216, 217, 272, 288, 289, 301, 444, 445, 592])
def test_mid_router_equals_oracle(nb, layer, gpu, oracle, weights):
    router, _, _ = weights.layer(2)
    hn = weights.hidden(700, nb)
    bias = np.linspace(-1.0, 1.0, 256).astype(np.float32)
    want = oracle.router_logits(router, hn)
    gpu.poke("hn", hn)
    gpu.stage("router", 2, nb)
    assert np.array_equal(gpu.peek("logits", nb).reshape(nb, 256).view(np.uint32), want.view(np.uint32))
    gpu.poke("bias", bias)
    gpu.stage("router_bias", 2, nb)
    assert np.array_equal(gpu.peek("logits", nb).reshape(nb, 256).view(np.uint32), (want + bias[None, :]).view(np.uint32))


@pytest.mark.parametrize("nb", [217, 296, 297])
def test_where_eight_tokens_per_cta_begin_and_end(nb, layer, gpu, oracle, weights):
    router, _, _ = weights.layer(2)
    hn = weights.hidden(701, nb)
    gpu.poke("hn", hn)
    gpu.stage("router", 2, nb)
    assert np.array_equal(gpu.peek("logits", nb).reshape(nb, 256).view(np.uint32), oracle.router_logits(router, hn).view(np.uint32))


@pytest.mark.parametrize("nb", [298, 360, 361, 446, 504, 505])
def test_where_two_kinds_of_ctas_begin_and_end(nb, layer, gpu, oracle, weights):
    """One token past the last all-small (or all-big) grid, the last token of the mixed grids and the one after it."""
    router, _, _ = weights.layer(2)
    hn = weights.hidden(702, nb)
    gpu.poke("hn", hn)
    gpu.stage("router", 2, nb)
    assert np.array_equal(gpu.peek("logits", nb).reshape(nb, 256).view(np.uint32), oracle.router_logits(router, hn).view(np.uint32))
