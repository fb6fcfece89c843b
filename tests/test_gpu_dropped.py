"""Calls without kept stages give up gate, up and the compact down rows of the tcgen05 kernels once they are read (csrc/launch.cuh: l2_discard): what lies there afterwards is
undefined, so that asking for it, or for a stage that starts from it, is refused until something has written it again."""
import numpy as np
import pytest

from conftest import SEED, same_bits

pytestmark = pytest.mark.gpu
WHAT = {"gate": lambda g, nb: g.peek("gate", nb), "up": lambda g, nb: g.peek("up", nb), "actq": lambda g, nb: g.stage("actq", 0, nb),
        "combine_x": lambda g, nb: g.stage("combine_x", 0, nb), "combine_y": lambda g, nb: g.stage("combine_y", 0, nb)}


@pytest.fixture(scope="module")
def layer(gpu):
    gpu.synth_layer(SEED, 0)
    gpu.synth_layer(SEED, 1)


def calls(g, nb, x):
    """every way into the layers, the last one three times: plainly, while captured, as a replay"""
    yield lambda: g.moe(0, x)[0]
    for nl in (1, 2, 2, 2):
        yield lambda: g.forward(x.copy(), 0, nl)


@pytest.mark.parametrize("nb", [161, 301, 600])
def test_what_a_call_has_given_up_is_refused(nb, layer, gpu, weights):
    g = gpu
    x = weights.hidden(1200 + nb, nb)
    g.keep_stages(False)
    try:
        for call in calls(g, nb, x):
            for stage in ("gateup", "down"):
                g.stage(stage, 0, nb)
            for ask in WHAT.values():
                ask(g, nb)
            call()
            for name, ask in WHAT.items():
                with pytest.raises(RuntimeError, match="gave up"):
                    ask(g, nb)
    finally:
        g.keep_stages(True)


@pytest.mark.parametrize("nb", [161, 301, 600])
def test_stages_run_again_after_a_call(nb, layer, gpu, weights):
    g = gpu
    x = weights.hidden(1200 + nb, nb)
    g.keep_stages(False)
    try:
        y, _ = g.moe(0, x)
        want = {k: g.peek(k, nb).copy() for k in ("aq", "aqs", "aqsum")}
        g.stage("gateup", 0, nb)
        gate = g.peek("gate", nb).copy()
        g.stage("actq", 0, nb); g.stage("down", 0, nb); g.stage("combine_y", 0, nb)
        assert all(same_bits(g.peek(k, nb), want[k]) for k in want) and same_bits(g.peek("y", nb).reshape(nb, 2048), y)
        g.moe(0, x)
        g.poke("gate", gate)                                  # a caller's own rows are as good
        assert same_bits(g.peek("gate", nb), gate)
        with pytest.raises(RuntimeError, match="gave up"):
            g.peek("up", nb)
    finally:
        g.keep_stages(True)
    g.moe(0, x)                                               # kept stages: everything there
    assert same_bits(g.peek("gate", nb), gate)
    for ask in WHAT.values():
        ask(g, nb)


def test_smaller_calls_give_up_nothing(layer, gpu, weights):
    g, nb = gpu, 160
    x = weights.hidden(1360, nb)
    g.moe(0, x)
    gate = g.peek("gate", nb).copy()
    g.keep_stages(False)
    try:
        y, _ = g.moe(0, x)
        assert same_bits(g.peek("gate", nb), gate)
        g.stage("actq", 0, nb); g.stage("combine_y", 0, nb)
        assert same_bits(g.peek("y", nb).reshape(nb, 2048), y)
    finally:
        g.keep_stages(True)
