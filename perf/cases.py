"""Timed cases of this library: what a host program has it do, through its public entry points, from one token to long prompts.

kinds of call
  stack   the residual stream through all 24 layers, page-locked host buffers in and out: gmoe_forward_submit / gmoe_forward_wait with
          two chunks outstanding.  One token = a lone conversation's next token; up to 64 = the --multi batches; more = a prompt.
  layer   one gmoe_moe call per layer, pageable host buffers: a host that keeps attention on its own side of the boundary and so comes
          back for every layer of a decode step.
  plugin  gpre_moe, the reference-shaped call: the host's own routing tables and pageable arrays, as an unmodified host calls it per layer.
  attn    the projections around attention, per layer: q,k,v (gpre_dense), norm + rotary embedding + fp16 cache rows (gmoe_qk_rope),
          o (gpre_dense); pageable host buffers.
  group   gmoe_group_noalloc on device tables: the grouping inside another runtime's pool.
All layers are resident, their weights generated once per process; what is made from the seed is what changes from call to call.
"""
import functools
import math

import numpy as np
import torch

from maple_runtime_b200 import lib as ml

LAYERS, H, NEXP, TOPK = 24, 2048, 256, 8
MAXTOK = 16384                       # one library set-up serves every size, as in a server
WEIGHT_SEED = 20261125
POSITIONS = 16384                    # rows of the rotary table
STREAM_CHUNK = 2048                  # the chunk a long prompt is cut into


def listed():
    return [
        # generation: one conversation, a few, and the 64 that --multi runs at most
        {"name": "stack 1 token", "kind": "stack", "tokens": 1, "chunk": MAXTOK, "skew": False},
        {"name": "stack 13 tokens", "kind": "stack", "tokens": 13, "chunk": MAXTOK, "skew": False},
        {"name": "stack 64 tokens", "kind": "stack", "tokens": 64, "chunk": MAXTOK, "skew": False},
        # prompts: a short ragged one, a page of text, a full chunk whose experts are unequally popular, a long one in streamed chunks
        {"name": "stack 301 tokens", "kind": "stack", "tokens": 301, "chunk": MAXTOK, "skew": False},
        {"name": "stack 843 tokens", "kind": "stack", "tokens": 843, "chunk": MAXTOK, "skew": False},
        {"name": "stack 2048 tokens, skewed", "kind": "stack", "tokens": 2048, "chunk": MAXTOK, "skew": True},
        {"name": "stack 16384 tokens by 2048", "kind": "stack", "tokens": 16384, "chunk": STREAM_CHUNK, "skew": False},
        # a decode step of seven conversations, layer by layer through host buffers
        {"name": "layer calls, 7 tokens", "kind": "layer", "tokens": 7, "layers": 24, "skew": False},
        # a full prompt chunk through the reference-shaped call
        {"name": "plugin calls, 2048 tokens", "kind": "plugin", "tokens": 2048, "layers": 2, "skew": False},
        # the projections around attention: a decode step of 64 conversations, and one layer of a prompt chunk
        {"name": "attention sides, 64 tokens", "kind": "attn", "tokens": 64, "layers": 24},
        {"name": "attention sides, 2048 tokens", "kind": "attn", "tokens": 2048, "layers": 1},
        # the grouping alone
        {"name": "grouping, 1000 tokens", "kind": "group", "tokens": 1000, "skew": True},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["stack", "stack", "stack", "layer", "plugin", "attn", "group"])
    if kind == "stack":
        n = _log_int(rng, 1, 16384)
        return {"kind": kind, "tokens": n, "chunk": rng.choice([STREAM_CHUNK, 4096, MAXTOK]) if n > STREAM_CHUNK else MAXTOK, "skew": rng.random() < 0.3}
    if kind == "layer":
        return {"kind": kind, "tokens": _log_int(rng, 1, 512), "layers": 24, "skew": rng.random() < 0.3}
    if kind == "plugin":
        return {"kind": kind, "tokens": _log_int(rng, 16, 4096), "layers": 2, "skew": rng.random() < 0.3}
    if kind == "attn":
        n = _log_int(rng, 1, 4096)
        return {"kind": kind, "tokens": n, "layers": 24 if n <= 64 else 1}
    return {"kind": kind, "tokens": _log_int(rng, 1, 2048), "skew": rng.random() < 0.5}


# ---- what the process keeps: the library with its resident layers, the host's copies of the router tables ----------------------------
@functools.lru_cache(maxsize=None)
def _moe():
    g = ml.Gpre(MAXTOK)
    for layer in range(LAYERS):
        g.synth_layer(WEIGHT_SEED, layer)
    return g


@functools.lru_cache(maxsize=None)
def _attention():
    """The q,k,v and o matrices of every layer on the card (random ternary codes and row scales), the rotary table, the head norms."""
    g, gen = _moe(), torch.Generator(device="cuda").manual_seed(WEIGHT_SEED)
    rand = functools.partial(torch.rand, generator=gen, device="cuda")
    for layer in range(LAYERS):
        for group, row_counts in ((2 * layer, (2048, 512, 512)), (2 * layer + 1, (2048,))):
            for rows in row_counts:
                u = rand(4, rows, H // 4)
                t = (u > 0.3).to(torch.uint8) + (u > 0.7).to(torch.uint8)
                codes = t[0] | t[1] << 2 | t[2] << 4 | t[3] << 6
                g.dense_add(group, codes.cpu().numpy(), (rand(rows) * 0.04 + 0.01).cpu().numpy(), rows, H)
    g.dense_done(MAXTOK)
    angle = np.arange(POSITIONS)[:, None] * (10000.0 ** (-np.arange(32) / 32))[None, :]
    g.rope_table(np.stack([np.cos(angle), np.sin(angle)], -1))
    qn, kn = (rand(2, 128) + 0.5).cpu().numpy()
    return {"qn": qn, "kn": kn}


@functools.lru_cache(maxsize=None)
def _router(layer):
    bits = ml.synth_router(_moe().lib, WEIGHT_SEED, layer)
    return torch.from_numpy(bits.view(np.int16)).cuda().view(torch.bfloat16).float()


@functools.lru_cache(maxsize=None)
def _zipf_bias():
    return ml.synth_zipf_bias(_moe().lib, WEIGHT_SEED, 1.2)


def _hidden(gen, *shape):
    return torch.randn(*shape, H, generator=gen, device="cuda")


def _route(x, layer, skew):
    """Top-8 of the layer's router with renormalised softmax weights: expert ids and weights [tokens][8]."""
    logits = x @ _router(layer).T
    if skew:
        logits = logits + torch.from_numpy(_zipf_bias()).cuda()
    top = logits.topk(TOPK, dim=1)
    return top.indices.to(torch.int32), torch.softmax(top.values, 1).contiguous()


def _plugin_tables(top, weight, layer):
    """The host's side of gpre_moe: pairs grouped by used expert in token order, and each token's pairs ascending."""
    g, nb = _moe(), top.shape[0]
    flat = top.reshape(-1)
    order = np.argsort(flat, kind="stable")
    used, counts = np.unique(flat, return_counts=True)
    ustart = np.zeros(len(used) + 1, np.int32)
    ustart[1:] = np.cumsum(counts)
    place = np.empty(nb * TOPK, np.int32)
    place[order] = np.arange(nb * TOPK, dtype=np.int32)
    return {"nu": len(used), "loc": np.ascontiguousarray(ml.gloc_for_contiguous()[used]), "regs": np.array([g.layer_region[layer], -1, -1, -1], np.int32),
            "ustart": ustart, "ptok": (order // TOPK).astype(np.int32), "pw": np.ascontiguousarray(weight.reshape(-1)[order]),
            "tp": np.ascontiguousarray(np.sort(place.reshape(nb, TOPK), axis=1))}


# ---- one case --------------------------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, nb = case["kind"], case["tokens"]
    g = _moe()
    state = {"kind": kind, "g": g, "nb": nb}
    if kind == "stack":
        x = torch.empty((nb, H), pin_memory=True)
        x.copy_(_hidden(gen, nb))
        out = torch.empty((nb, H), pin_memory=True)
        state.update(x=x.numpy(), out=out.numpy(), chunk=case["chunk"], bias=_zipf_bias() if case["skew"] else None)
    elif kind == "layer":
        x = _hidden(gen, case["layers"], nb).cpu().numpy()
        state.update(x=x, y=np.zeros_like(x), bias=_zipf_bias() if case["skew"] else None)
    elif kind == "plugin":
        calls = []
        for layer in range(case["layers"]):
            x = _hidden(gen, nb)
            top, weight = _route(x, layer, case["skew"])
            x = x.cpu().numpy()
            calls.append(dict(_plugin_tables(top.cpu().numpy(), weight.cpu().numpy(), layer), x=x, y=np.zeros_like(x)))
        state.update(calls=calls)
    elif kind == "attn":
        pos = torch.randint(0, POSITIONS, (nb,), generator=gen, device="cuda", dtype=torch.int32).cpu().numpy()
        if nb > 64:                                      # a prompt: consecutive positions
            pos = (int(pos[0]) % (POSITIONS - nb + 1) + np.arange(nb)).astype(np.int32)
        x = _hidden(gen, case["layers"], nb).cpu().numpy()
        state.update(_attention(), x=x, pos=pos, o=np.zeros_like(x), qkv=np.zeros((nb, 3072), np.float32), q=np.zeros((nb, H), np.float32),
                     k=np.zeros((nb, 512), np.uint16), v=np.zeros((nb, 512), np.uint16))
    else:
        top, weight = _route(_hidden(gen, nb), 0, case["skew"])
        out = {"nu": torch.zeros(1, dtype=torch.int32, device="cuda"), "ue": torch.zeros(NEXP, dtype=torch.int32, device="cuda"),
               "ustart": torch.zeros(NEXP + 1, dtype=torch.int32, device="cuda"), "utok": torch.zeros(nb * TOPK, dtype=torch.int32, device="cuda"),
               "uw": torch.zeros(nb * TOPK, device="cuda"), "tp": torch.zeros(nb * TOPK, dtype=torch.int32, device="cuda")}
        state.update(top=top, weight=weight, out=out)
    return state


def _run_stack(s):
    g, nb, chunk = s["g"], s["nb"], s["chunk"]
    waiting = 0
    for at in range(0, nb, chunk):
        if waiting == 2:
            g._chk(g.lib.gmoe_forward_wait())
            waiting -= 1
        x, out = s["x"][at:at + chunk], s["out"][at:at + chunk]
        g._chk(g.lib.gmoe_forward_submit(ml._p(x), ml._p(out), x.shape[0], 0, LAYERS, ml._p(s["bias"])))
        waiting += 1
    for _ in range(waiting):
        g._chk(g.lib.gmoe_forward_wait())
    return s["out"]


def _run_group(s):
    g, o = s["g"], s["out"]
    g._chk(g.lib.gmoe_group_noalloc(s["top"].data_ptr(), s["weight"].data_ptr(), s["nb"], o["nu"].data_ptr(), o["ue"].data_ptr(), o["ustart"].data_ptr(),
                                    o["utok"].data_ptr(), o["uw"].data_ptr(), o["tp"].data_ptr(), torch.cuda.current_stream().cuda_stream))
    return o


def _run_layer_calls(s):
    g = s["g"]
    for layer in range(len(s["x"])):
        g._chk(g.lib.gmoe_moe(layer, ml._p(s["x"][layer]), s["nb"], ml._p(s["y"][layer]), ml._p(s["bias"])))
    return s["y"]


def _run_plugin(s):
    for c in s["calls"]:
        s["g"].gpre_moe(c["x"], c["nu"], c["loc"], c["regs"], c["ustart"], c["ptok"], c["pw"], c["tp"], out=c["y"])
    return [c["y"] for c in s["calls"]]


def _run_attention(s):
    g, nb = s["g"], s["nb"]
    qkv, q, k, v, pos, qn, kn = (ml._p(s[name]) for name in ("qkv", "q", "k", "v", "pos", "qn", "kn"))
    for layer in range(len(s["x"])):
        g._chk(g.lib.gpre_dense(2 * layer, ml._p(s["x"][layer]), nb, qkv))
        g._chk(g.lib.gmoe_qk_rope(qkv, pos, nb, int(layer % 4 == 3), qn, kn, q, k, v))
        g._chk(g.lib.gpre_dense(2 * layer + 1, q, nb, ml._p(s["o"][layer])))     # the attended rows have the queries' shape and range
    return [s[name] for name in ("o", "qkv", "q", "k", "v")]


RUN = {"stack": _run_stack, "layer": _run_layer_calls, "plugin": _run_plugin, "attn": _run_attention, "group": _run_group}


def run(state):
    return RUN[state["kind"]](state)


# ---- what a case cannot do without -----------------------------------------------------------------------------------------------------
def _used_experts(pairs_per_expert):
    return sum(1.0 - math.exp(-p) for p in pairs_per_expert)


def _experts_bytes(case):
    """Bytes of one layer's codes and scales that the expected routing touches."""
    nb = case["tokens"]
    if case.get("skew"):
        p = np.exp(_zipf_bias().astype(np.float64))
        pairs = np.minimum(nb, nb * TOPK * p / p.sum())
    else:
        pairs = np.full(NEXP, nb * TOPK / NEXP)
    return _used_experts(pairs) * ml.CONST.EXPERT_BYTES


def work(case):
    nb, kind = case["tokens"], case["kind"]
    rows = nb * H * 4
    expert_ops, router_ops, router_bytes = nb * TOPK * 2 * 3 * 512 * H, nb * NEXP * H * 2, NEXP * H * 2
    if kind == "stack":
        return {"bytes": LAYERS * (_experts_bytes(case) + router_bytes) + 2 * rows, "flops": LAYERS * (expert_ops + router_ops)}
    if kind == "layer":
        return {"bytes": case["layers"] * (_experts_bytes(case) + router_bytes + 2 * rows), "flops": case["layers"] * (expert_ops + router_ops)}
    if kind == "plugin":
        return {"bytes": case["layers"] * (_experts_bytes(case) + 2 * rows + nb * TOPK * 12), "flops": case["layers"] * expert_ops}
    if kind == "attn":       # x, qkv, q, k and v rows, q again, o; codes and scales of 5120 rows
        return {"bytes": case["layers"] * (5120 * (H // 4 + 4) + nb * (5 * H * 4 + 3072 * 4 + 2 * 1024)), "flops": case["layers"] * nb * 5120 * H * 2}
    return {"bytes": nb * TOPK * (4 + 4 + 4 + 4 + 4) + (2 * NEXP + 2) * 4, "flops": 0}


def tolerance(case):
    if case["kind"] == "stack" and min(case["tokens"], case["chunk"]) >= 512:
        # Prompts take their router logits from the tensor cores.  Every layer rounds its activations to 8 bits and routes by comparison,
        # so a last-bit difference of a sum moves a few of them by a whole step, and 24 layers carry that on and spread it.
        return {"rel": 1e-2, "max": 0.9}
    if case["kind"] in ("stack", "layer", "plugin"):
        return {"rel": 1e-5, "max": 1e-3}               # every sum in a stated order: only the last bits of the 32-bit values are open
    return "exact"                                      # integer sums and a fixed order of roundings, or whole numbers
