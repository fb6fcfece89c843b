"""The grouping of 33 and more tokens as one cluster of CTAs (csrc/k_route.cu: group_cluster_kernel) against the oracle, at the sizes where its
split changes: one token past a word, eight and sixteen CTAs, CTAs without tokens, skewed and identical rows, arrays that are not 16-byte aligned."""
import numpy as np
import pytest

from conftest import SEED
from test_zz_no_alloc import routing

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb,kind", [(33, "even"), (64, "same"), (97, "skew"), (256, "even"), (257, "even"), (288, "skew"), (511, "even"), (512, "same"), (513, "even"), (777, "skew"), (2047, "even"), (2048, "same")])
@pytest.mark.parametrize("shift", [0, 1])
def test_cluster_grouping_equals_oracle(nb, kind, shift, gpu, clib, oracle):
    torch = pytest.importorskip("torch")   # only to own device buffers for the caller's side of the call
    rng = np.random.default_rng(nb)
    top, tw = routing(rng, nb, kind == "skew")
    if kind == "same":
        top[:] = top[0]
    o_nu, o_ue, o_ustart, o_utok, o_uw, o_tp = oracle.group(top, tw)
    dev = torch.device("cuda:0")

    def buf(n, dt, src=None):              # shift: one word past a 16-byte boundary
        b = torch.zeros(n + 4, dtype=dt, device=dev)[shift:shift + n]
        if src is not None:
            b.copy_(torch.from_numpy(src.ravel()))
        return b
    i32, f32 = torch.int32, torch.float32
    t_top, t_w = buf(nb * 8, i32, top), buf(nb * 8, f32, tw)
    nu, ue, ustart, utok, uw, tp = buf(1, i32), buf(256, i32), buf(257, i32), buf(nb * 8, i32), buf(nb * 8, f32), buf(nb * 8, i32)
    torch.cuda.synchronize()
    assert clib.gmoe_group_noalloc(*(t.data_ptr() for t in (t_top, t_w)), nb, *(t.data_ptr() for t in (nu, ue, ustart, utok, uw, tp)), None) == 0
    torch.cuda.synchronize()
    assert int(nu[0]) == o_nu
    assert np.array_equal(ue.cpu().numpy()[:o_nu], o_ue[:o_nu]) and np.array_equal(ustart.cpu().numpy()[:o_nu + 1], o_ustart[:o_nu + 1])
    assert np.array_equal(utok.cpu().numpy(), o_utok.ravel()) and np.array_equal(tp.cpu().numpy(), o_tp.ravel())
    assert np.array_equal(uw.cpu().numpy().view(np.uint32), o_uw.ravel().view(np.uint32))


@pytest.fixture(scope="module")
def layer(gpu):                                               # once: every generation takes a region id
    gpu.synth_layer(SEED, 0)


@pytest.mark.parametrize("nb,kind", [(161, "even"), (256, "even"), (257, "even"), (257, "same"), (288, "skew"), (289, "even"), (512, "same"), (513, "skew"), (2047, "even"), (2048, "skew")])
def test_grouping_of_a_layer_equals_oracle(nb, kind, layer, gpu, oracle):
    """As a layer runs it (the stage "group"): up to 256 tokens the cluster places the pairs, from 257 the kernel that moves their rows does (k_expert_umma.cu: place_rows_kernel)."""
    rng = np.random.default_rng(nb)
    top, tw = routing(rng, nb, kind == "skew")
    if kind == "same":
        top[:] = top[0]
    o_nu, o_ue, o_ustart, o_utok, o_uw, o_tp = oracle.group(top, tw)
    gpu.poke("top", top.ravel())
    gpu.poke("topw", tw.ravel())
    gpu.poke("utok", np.full(nb * 8, -1, np.int32))
    gpu.poke("tp", np.full(nb * 8, -1, np.int32))
    gpu.stage("group", 0, nb)
    assert int(gpu.peek("nu", nb)[0]) == o_nu
    assert np.array_equal(gpu.peek("ue", nb)[:o_nu], o_ue[:o_nu]) and np.array_equal(gpu.peek("ustart", nb)[:o_nu + 1], o_ustart[:o_nu + 1])
    assert np.array_equal(gpu.peek("utok", nb).ravel(), o_utok.ravel()) and np.array_equal(gpu.peek("tp", nb).ravel(), o_tp.ravel())
    assert np.array_equal(gpu.peek("uw", nb).ravel().view(np.uint32), o_uw.ravel().view(np.uint32))
