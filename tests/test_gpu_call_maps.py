"""The tensor maps that gpre_moe keeps on the card by expert (csrc/gpre_api.c: map_slot): a call that fails after its experts were first seen, then the
first good call, then calls that find the maps; and two arrangements of the same codes."""
import numpy as np
import pytest

from conftest import same_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [209, 600])
def test_maps_of_host_supplied_groupings(nb, gpu, oracle, weights):
    from maple_runtime_b200 import lib as ml
    g = gpu
    router, post_ln, experts = weights.layer(1)
    span = ml.page_aligned(experts.nbytes)
    span[:experts.nbytes] = experts.reshape(-1)
    rid = g.region(span)                                     # a region no call has named
    hn = weights.hidden(640 + nb, nb)
    _, d = oracle.moe(router, post_ln, experts, hn, 0, dots=True)
    nu = int(d["nu"][0])
    regs = np.array([-1, rid, -1, -1], np.int32)
    loc = np.ascontiguousarray(ml.gloc_for_contiguous(0, slot=1)[d["ue"][:nu]])
    args = (d["ustart"], d["utok"], d["uw"], d["tp"])
    bad = d["utok"].copy()
    bad.reshape(-1)[nb * 8 - 1] = nb
    with pytest.raises(RuntimeError, match="ptok"):
        g.gpre_moe(hn, nu, loc, regs, d["ustart"], bad, d["uw"], d["tp"])
    g.set_path(1)
    try:
        want, _ = g.gpre_moe(hn, nu, loc, regs, *args)      # the mma.sync kernels, which need no maps
    finally:
        g.set_path(0)
    for _ in range(3):
        y, _ = g.gpre_moe(hn, nu, loc, regs, *args)
        assert same_bits(y, want)
    same = loc.copy()
    same.reshape(nu, 12)[:, 4:8] = same.reshape(nu, 12)[:, 0:4]      # the gate matrix in both places: known gate codes beside other up codes
    g.set_path(1)
    try:
        want, _ = g.gpre_moe(hn, nu, same, regs, *args)
    finally:
        g.set_path(0)
    y, _ = g.gpre_moe(hn, nu, same, regs, *args)
    assert same_bits(y, want)
