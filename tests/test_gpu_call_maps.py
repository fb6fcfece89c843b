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


def test_slots_that_start_over(gpu):
    """More experts than the table has slots: it starts over, and the addresses on the card get other maps.  256 experts per call, each a window of its own
    of one long run of ternary codes; every call against the mma.sync kernels, which need no maps."""
    from maple_runtime_b200 import lib as ml
    g, c = gpu, ml.CONST
    nb, nu, calls = 256, 256, 66                             # 66 x 256 > 16384 slots
    rng = np.random.default_rng(5)
    run = c.GU_CODES + 16 * nu * calls
    span = ml.page_aligned(-(-(run + 8192) // 4096) * 4096)
    span[:run] = rng.choice(np.array([a | b << 2 | d << 4 | e << 6 for a in range(3) for b in range(3) for d in range(3) for e in range(3)], np.uint8), run)
    scales = -(-run // 16) * 16
    span[scales:scales + 8192].view(np.float32)[:] = rng.uniform(0.01, 0.05, 2048)
    rid = g.region(span)
    regs = np.array([rid, -1, -1, -1], np.int32)
    x = rng.standard_normal((nb, 2048)).astype(np.float32)
    pair = np.arange(nb * 8, dtype=np.int32)
    tables = (np.arange(0, nb * 8 + 1, 8, dtype=np.int32), pair % nb, rng.uniform(0.05, 0.2, nb * 8).astype(np.float32), np.ascontiguousarray(pair.reshape(8, nb).T))

    def loc(call):
        l = np.zeros((nu, 6, 2), np.uint32)
        l[:, ::2, 1] = (16 * (call * nu + np.arange(nu)))[:, None]
        l[:, 1::2, 1] = scales
        return l.reshape(nu, 12)
    for call in list(range(calls)) + [0, calls - 1]:
        y, _ = g.gpre_moe(x, nu, loc(call), regs, *tables)
        if call % 16 == 0 or call >= 62:
            g.set_path(1)
            try:
                want, _ = g.gpre_moe(x, nu, loc(call), regs, *tables)
            finally:
                g.set_path(0)
            assert same_bits(y, want), call
