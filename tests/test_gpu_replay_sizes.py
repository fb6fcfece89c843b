"""Layer calls of many batch sizes in turn, as a server makes them whose number of conversations moves: every one a replay from its third sight on,
with the bits of its first, plain run."""
import numpy as np
import pytest

from conftest import SEED, same_bits

pytestmark = pytest.mark.gpu


def test_layer_calls_of_many_batch_sizes(gpu, weights, clib):
    from maple_runtime_b200 import lib as ml
    g = gpu
    for L in (3, 4):
        g.synth_layer(SEED, L)
    x = weights.hidden(3100, 96)
    calls = [(nb, L, bias) for nb in range(1, 97) for L in (3, 4) for bias in (None, ml.synth_zipf_bias(clib, 7))]
    g.keep_stages(False)
    try:
        first = [g.moe(L, x[:nb], bias)[0] for nb, L, bias in calls]
        for cycle in range(3):
            before = clib.gmoe_graph_launches()
            for (nb, L, bias), want in zip(calls, first):
                y, _ = g.moe(L, x[:nb], bias)
                assert same_bits(y, want), (cycle, nb, L)
            assert clib.gmoe_graph_launches() - before == len(calls)      # a captured call is launched as a graph too
    finally:
        g.keep_stages(True)
