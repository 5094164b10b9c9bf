"""The work that users of this framework have it do, as cases that can be timed and compared.

A case is a dict of plain values; its "family" says which entry points it goes through:

    decode         decode steps of the LLaMA engine behind a filled KV cache
    prefill        the context phase of an engine: prompts in, logits of the next token out (LLaMA: ragged prompts)
    generate       a short prompt and the decode steps behind it, for the designs whose layers keep a recurrent state
    experts        a mixture-of-experts feed-forward through the kernel interface
    float_context  one decoder layer in float32 over ragged prompts: the launch sequence of the reference's context decoder
    float_decode   one decoder layer and the head in float32, one token per sequence: the sequence of its self decoder

Sizes are the ones of the benchmark and its tests: widths 2048, 4096 and 5120, heads of 128, vocabulary 32000.  A few layers
stand for a model: every layer is the same work.  Input ids of decode steps are given, as they are when a host samples or
scores a text, so that two runs see the same tokens.
"""
import ctypes
import math

import numpy as np
import torch

import onellm_b200 as ob

VOCAB = 32000
SIZES = {
    "w2048": dict(hidden=2048, head_num=16, kv_head_num=4, head_size=128, inter_size=5632),
    "w4096": dict(hidden=4096, head_num=32, kv_head_num=32, head_size=128, inter_size=11008),
    "w5120": dict(hidden=5120, head_num=40, kv_head_num=40, head_size=128, inter_size=13824),
}
# recurrence heads x (key, value) and key/value heads of Finuvik; latents, gla heads and window of Fuposun; experts
FINUVIK = {"w2048": (16, 128, 128, 4), "w4096": (32, 128, 128, 8)}
FUPOSUN = {"w2048": (1536, 512, 1024, 4, 256, 512), "w4096": (1536, 512, 1024, 8, 256, 512)}
EXPERTS, TOP = 32, 4
ROPE_BASE = 10000.0


# ---- the cases ---------------------------------------------------------------------------------------------
def listed():
    return [
        # one user, a small model, a short context: every launch and every wait shows
        dict(name="decode_single", family="decode", size="w2048", layers=4, batch=1, context=127, steps=8),
        # the benchmark's decode workload: batch 8 behind prompts of 512 tokens
        dict(name="decode_batch8", family="decode", size="w4096", layers=4, batch=8, context=515, steps=8),
        # a full serving batch on long contexts: the cache is most of what is read
        dict(name="decode_batch64_long", family="decode", size="w5120", layers=2, batch=64, context=1990, steps=4),
        # a few chat prompts that arrive together, lengths as they come
        dict(name="prefill_short_ragged", family="prefill", design="llama", size="w4096", layers=4, prompts="130,37,71"),
        # documents
        dict(name="prefill_long", family="prefill", design="llama", size="w4096", layers=4, prompts="2040,1777"),
        # one long prompt of the design with a gated recurrence beside biased attention
        dict(name="finuvik_prefill", family="prefill", design="finuvik", size="w2048", layers=4, prompts="2000"),
        # several short conversations of it
        dict(name="finuvik_generate", family="generate", design="finuvik", size="w4096", layers=2, batch=8, prompt=33, steps=16),
        # prompts of the design with latent attention and gated linear attention in turn
        dict(name="fuposun_prefill", family="prefill", design="fuposun", size="w2048", layers=4, prompts="1030,1030"),
        # and conversations of it
        dict(name="fuposun_generate", family="generate", design="fuposun", size="w4096", layers=2, batch=4, prompt=40, steps=16),
        # the experts of a layer on a prompt's tokens
        dict(name="experts_prompt", family="experts", size="w4096", tokens=1000),
        # a caller of the kernel interface in the reference's own type, both phases
        dict(name="float_context", family="float_context", size="w4096", prompts="255,97", history="0,40"),
        dict(name="float_decode", family="float_decode", size="w4096", batch=2, context=255),
    ]


def spread(rng, low, high):
    """A whole number, evenly over the logarithm of the range, odd as often as even."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    family = rng.choice(["decode", "decode", "prefill", "prefill", "generate", "experts", "float_context", "float_decode"])
    if family == "decode":
        size = rng.choice(["w2048", "w4096", "w5120"])
        batch = spread(rng, 1, 64)
        return dict(family=family, size=size, layers=4 if size == "w2048" else 2, batch=batch, context=spread(rng, 16, 1990),
                    steps=rng.randint(3, 8) if batch <= 16 else rng.randint(2, 4))
    if family == "prefill":
        design = rng.choice(["llama", "llama", "finuvik", "fuposun"])
        size = rng.choice(["w2048", "w4096"])
        n = rng.randint(1, 4)
        longest = spread(rng, 16, 2040 // n)
        lens = [longest] * n if design != "llama" else [max(1, int(longest * rng.uniform(0.3, 1.0))) for _ in range(n)]
        return dict(family=family, design=design, size=size, layers=2, prompts=",".join(map(str, lens)))
    if family == "generate":
        return dict(family=family, design=rng.choice(["finuvik", "fuposun"]), size=rng.choice(["w2048", "w4096"]), layers=2,
                    batch=spread(rng, 1, 32), prompt=spread(rng, 2, 60), steps=rng.randint(4, 16))
    if family == "experts":
        return dict(family=family, size=rng.choice(["w2048", "w4096"]), tokens=spread(rng, 1, 1000))
    size = rng.choice(["w2048", "w4096"])
    if family == "float_context":
        n = rng.randint(1, 4)
        longest = spread(rng, 4, 350 // n)
        lens = [max(1, int(longest * rng.uniform(0.3, 1.0))) for _ in range(n)]
        hist = [rng.choice([0, rng.randint(1, 99)]) for _ in range(n)]
        return dict(family=family, size=size, prompts=",".join(map(str, lens)), history=",".join(map(str, hist)))
    return dict(family=family, size=size, batch=spread(rng, 1, 32), context=spread(rng, 8, 1000))


def numbers(text):
    return [int(v) for v in text.split(",")]


# ---- configurations ----------------------------------------------------------------------------------------
def finuvik_config(c, positions):
    s, (rh, rk, rv, kv) = SIZES[c["size"]], FINUVIK[c["size"]]
    layer = {"type": "parallel",
             "mixer": {"left": {"heads": s["head_num"], "kv_heads": kv, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                                "q_temp": {"coef": 0.1, "every": 1024}},
                       "left_scale": 1.0, "right_scale": 1.0, "right": {"heads": rh, "dim": rk, "vdim": rv}},
             "mlp": {"kind": "dense", "ff": s["inter_size"]}}
    return {"architecture": "Finuvik", "vocab": VOCAB, "width": s["hidden"], "max_positions": positions, "norm": {"eps": 1e-6},
            "layers": [layer] * c["layers"]}


def fuposun_config(c):
    """Recurrent and attention layers in turn, dense feed-forwards (experts have a family of their own: which expert a token
    takes is a step function, whole logits behind it cannot be compared)."""
    s, (q_rank, kv_rank, window, gh, gk, gv) = SIZES[c["size"]], FUPOSUN[c["size"]]
    mlp = {"kind": "dense", "ff": s["inter_size"]}
    rec = {"type": "gla", "mixer": {"heads": gh, "dim": gk, "vdim": gv, "tau": 16.0}, "mlp": mlp}
    attn = {"type": "latent_attention", "mixer": {"heads": s["head_num"], "dim": 128, "vdim": 128, "q_rank": q_rank, "kv_rank": kv_rank,
                                                  "scale": 128 ** -0.5, "mask": {"size": window}}, "mlp": mlp}
    return {"architecture": "Fuposun", "vocab": VOCAB, "width": s["hidden"], "norm": {"eps": 1e-6}, "residual_mult": 0.5, "logit_softcap": 30.0,
            "layers": [(rec, attn)[i % 2] for i in range(c["layers"])]}


def engine(c, batch, positions, seed):
    design = c.get("design", "llama")
    if design == "llama":
        m = ob.Llama(num_layers=c["layers"], vocab_size=VOCAB, max_seq_len=positions, max_batch=batch, **SIZES[c["size"]])
    else:
        m = ob.Model(finuvik_config(c, positions) if design == "finuvik" else fuposun_config(c), ob.BF16, batch, positions)
    m.init_random(seed, 0.02)
    m.set_sampling(top_k=1)
    return m


class _Device:
    """Device memory that an engine owns, for torch.as_tensor; the tensor keeps the engine alive."""

    def __init__(self, owner, address, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (address, False), "shape": shape, "typestr": "<f2", "version": 3}


def caches(m, c, batch, positions):
    s = SIZES[c["size"]]
    shape = (batch, s["kv_head_num"], positions, s["head_size"])
    return [tuple(torch.as_tensor(_Device(m, p, shape), device="cuda") for p in m.kv_cache_ptrs(l)) for l in range(c["layers"])]


def token_ids(seed, *shape):
    return np.random.default_rng([seed, 77]).integers(0, VOCAB, shape).astype(np.int32)


def generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


# ---- prepare -----------------------------------------------------------------------------------------------
def positions_of(c):
    """Rows of the cache that a program would set aside for this case."""
    most = {"decode": lambda: c["context"] + c["steps"], "prefill": lambda: max(numbers(c["prompts"])),
            "generate": lambda: c["prompt"] + c["steps"]}[c["family"]]()
    return (most + 63) // 64 * 64


def prepare(case, seed):
    return globals()["prepare_" + case["family"]](case, seed)


def fill_caches(kv, context, seed):
    """Keys and values of `context` positions, as a prompt leaves them: normalised activations times weights."""
    g = generator(seed)
    for pair in kv:
        for t in pair:
            part = t[:, :, :context]
            part.copy_(torch.randn(part.shape, generator=g, device="cuda", dtype=torch.float16))


def prepare_decode(c, seed):
    n = positions_of(c)
    m = engine(c, c["batch"], n, seed)
    kv = caches(m, c, c["batch"], n)
    fill_caches(kv, c["context"], seed)
    torch.cuda.synchronize()
    first, last = c["context"], c["context"] + c["steps"]
    return dict(family="decode", m=m, ids=token_ids(seed, c["steps"], c["batch"]), out=np.zeros(c["batch"], np.int32), context=c["context"],
                rows=[(k[:, :, first:last], v[:, :, first:last]) for k, v in kv])


def prepare_prefill(c, seed):
    lens, n = numbers(c["prompts"]), positions_of(c)
    m = engine(c, len(lens), n, seed)
    ids = token_ids(seed, sum(lens))
    at = np.cumsum([0] + lens)
    if c["design"] != "llama":
        return dict(family="prefill", m=m, prompts=None, ids=ids.reshape(len(lens), lens[0]), kv=[])
    return dict(family="prefill", m=m, prompts=[ids[a:b] for a, b in zip(at, at[1:])], ids=None, kv=caches(m, c, len(lens), n))


def prepare_generate(c, seed):
    m = engine(c, c["batch"], positions_of(c), seed)
    return dict(family="generate", m=m, prompt=token_ids(seed, c["batch"], c["prompt"]), ids=token_ids(seed + 1, c["steps"], c["batch"]),
                out=np.zeros(c["batch"], np.int32))


def prepare_experts(c, seed):
    T, s = c["tokens"], SIZES[c["size"]]
    W, F = s["hidden"], s["inter_size"] // TOP
    g = generator(seed)
    rnd = lambda std, *shape: (std * torch.randn(shape, generator=g, device="cuda")).to(torch.bfloat16)
    h, router = rnd(1.0, T, W), rnd(0.02, W, EXPERTS)
    gate, up, down = (torch.empty(EXPERTS, a, b, device="cuda", dtype=torch.bfloat16) for a, b in ((W, F), (W, F), (F, W)))
    for e in range(EXPERTS):
        for w in (gate, up, down):
            w[e] = rnd(0.02, *w.shape[1:])
    stream = torch.randn(T, W, generator=g, device="cuda")
    i32, f32 = dict(device="cuda", dtype=torch.int32), dict(device="cuda", dtype=torch.float32)
    n, tiles = T * TOP, ob.route_max_tiles(T, EXPERTS, TOP)
    z = torch.zeros(T, EXPERTS, **f32)
    a = {k: torch.zeros(size, **i32) for k, size in (("slot", n), ("slot_token", n), ("off", EXPERTS + 1), ("used", EXPERTS), ("n_used", 1),
                                                     ("tile_group", tiles), ("tile_row", tiles), ("n_tiles", 1), ("choice", n), ("count", EXPERTS))}
    a.update(slot_weight=torch.zeros(n, **f32), choice_weight=torch.zeros(n, **f32))
    p = {k: v.data_ptr() for k, v in a.items()}
    tiled = T > 64  # longer passes copy the rows into expert order, shorter ones pick them in the projection
    xs = torch.zeros(n, W, device="cuda", dtype=torch.bfloat16) if tiled else None
    r = ob.Route(T, EXPERTS, TOP, z.data_ptr(), EXPERTS, dtype=ob.BF16, **p)
    if tiled:
        r.x, r.xs, r.ld_x = h.data_ptr(), xs.data_ptr(), W
    common = dict(n=EXPERTS if tiled else min(EXPERTS, n), used=None if tiled else p["used"], n_used=None if tiled else p["n_used"], off=p["off"],
                  w_stride=W * F, tile_group=p["tile_group"], tile_row=p["tile_row"], n_tiles=p["n_tiles"], max_tiles=tiles, weights=EXPERTS, rows=n)
    into = ob.RowGroups(x_rows=None if tiled else p["slot_token"], row_scale=p["slot_weight"], **common)
    back = ob.RowGroups(**common)
    bf = dict(device="cuda", dtype=torch.bfloat16)
    return dict(family="experts", T=T, W=W, F=F, h=h, router=router, gate=gate, up=up, down=down, stream=stream, x=torch.empty_like(stream), z=z,
                tables=a, route=r, into=into, back=back, xs=xs, act=torch.zeros(n, F, **bf), ys=torch.zeros(n, W, **bf),
                norm=torch.ones(W, **f32), out=torch.zeros(T, W, **bf))


def float_weights(c, seed, head):
    s = SIZES[c["size"]]
    hid, H, G, D, I = (s[k] for k in ("hidden", "head_num", "kv_head_num", "head_size", "inter_size"))
    g = generator(seed)
    rnd = lambda std, *shape: std * torch.randn(shape, generator=g, device="cuda")
    w = dict(table=rnd(1.0, VOCAB, hid), norm1=1 + 0.1 * rnd(1.0, hid), qkv=rnd(0.02, hid, (H + 2 * G) * D), o=rnd(0.02, H * D, hid),
             norm2=1 + 0.1 * rnd(1.0, hid), gate=rnd(0.02, hid, I), up=rnd(0.02, hid, I), down=rnd(0.02, I, hid), last=1 + 0.1 * rnd(1.0, hid))
    if head:
        w["head"] = rnd(0.02, VOCAB, hid)
    return w, rnd, (hid, H, G, D, I)


def prepare_float_context(c, seed):
    lens, hist = numbers(c["prompts"]), numbers(c["history"])
    w, rnd, (hid, H, G, D, I) = float_weights(c, seed, False)
    B, T, Q, ctx = len(lens), sum(lens), max(lens), [a + b for a, b in zip(lens, hist)]
    K = max(ctx)
    S = (K + 63) // 64 * 64
    i32 = lambda v: torch.tensor(v, device="cuda", dtype=torch.int32)
    z = lambda *shape: torch.zeros(shape, device="cuda")
    k, v = rnd(1.0, B, G, S, D), rnd(1.0, B, G, S, D)
    return dict(family="float_context", w=w, dims=(hid, H, G, D, I, B, T, Q, K, S), lens=i32(lens), hist=i32(hist), ctx=i32(ctx), k=k, v=v,
                ids=torch.from_numpy(token_ids(seed, T)).cuda(), offset=torch.zeros(B * Q, device="cuda", dtype=torch.int32),
                cum=torch.zeros(B + 1, device="cuda", dtype=torch.int32), mask=z(B, Q, K), res=z(T, hid), y=z(T, hid), qkv=z(T, (H + 2 * G) * D),
                q=z(B, H, Q, D), kn=z(B, G, Q, D), vn=z(B, G, Q, D), kr=z(B, H, K, D), vr=z(B, H, K, D), score=z(B, H, Q, K), prob=z(B, H, Q, K),
                pv=z(B, H, Q, D), attn=z(T, H * D), pair=z(T, 2, I), act=z(T, I))


def prepare_float_decode(c, seed):
    w, rnd, (hid, H, G, D, I) = float_weights(c, seed, True)
    B, step = c["batch"], c["context"] + 1
    S = (step + 63) // 64 * 64
    z = lambda *shape: torch.zeros(shape, device="cuda")
    k, v = rnd(1.0, B, G, S, D), rnd(1.0, B, G, S, D)
    need = ob.decode_attn_workspace_bytes(B, H, D, step)
    return dict(family="float_decode", w=w, dims=(hid, H, G, D, I, B, S, step), k=k, v=v, ids=torch.from_numpy(token_ids(seed, B)).cuda(),
                res=z(B, hid), y=z(B, hid), qkv=z(B, (H + 2 * G) * D), attn=z(B, H * D), pair=z(B, 2, I), act=z(B, I), logits=z(B, VOCAB),
                ws=torch.zeros(max(16, need), device="cuda", dtype=torch.uint8), need=need)


# ---- run ---------------------------------------------------------------------------------------------------
def run(state):
    return globals()["run_" + state["family"]](state)


def run_decode(s):
    m, ids = s["m"], s["ids"]
    m.seek(ids.shape[1], s["context"], ids[0])
    for t in range(len(ids)):
        m.decode_step(ids[t], s["out"])
    return {"logits": m.logits(ids.shape[1]), "rows": s["rows"]}


def run_prefill(s):
    first = s["m"].prefill(s["ids"]) if s["prompts"] is None else s["m"].prefill_ragged(s["prompts"])
    return {"logits": s["m"].logits(len(first)), "kv": s["kv"]}


def run_generate(s):
    m, ids = s["m"], s["ids"]
    m.prefill(s["prompt"])
    for t in range(len(ids)):
        m.decode_step(ids[t], s["out"])
    return {"logits": m.logits(ids.shape[1])}


def run_experts(s):
    T, W, F, n = s["T"], s["W"], s["F"], s["T"] * TOP
    s["x"].copy_(s["stream"])
    ob.project(ob.BF16, s["h"], s["router"], None, s["z"], T, EXPERTS, W, f32=True)
    ob.route(s["route"])
    ob.project(ob.BF16, s["h"] if s["xs"] is None else s["xs"], s["gate"], s["up"], s["act"], T, F, W, act=ob.GATE_CLAMPED, limit=7.0, groups=s["into"])
    ob.project(ob.BF16, s["act"], s["down"], None, s["ys"], T, W, F, groups=s["back"])
    ob.norm_rows(ob.BF16, s["x"], None, T, s["norm"], None, s["out"], None, 1e-6, W, W, add=s["ys"], add_rows=s["tables"]["slot"], add_n=TOP,
                 add_scale=0.5)
    return {"stream": s["x"], "out": s["out"], "router": s["z"], "off": s["tables"]["off"]}


def float_feed_forward(s, T):
    """Output projection, feed-forward and the two norms, as both decoders have them behind the attention."""
    w, (hid, H, G, D, I) = s["w"], s["dims"][:5]
    F = ob.F32
    ob.gemm(F, s["attn"], w["o"], s["y"], T, hid, H * D)
    ob.add_residual_rmsnorm(F, s["res"], s["y"], None, w["norm2"], 1e-5, T, hid)
    half = s["pair"].data_ptr()
    for name, at in (("gate", half), ("up", half + 4 * I)):
        ob._check(ob.lib().onellm_gemm_ld(ctypes.c_int(F), ob._p(s["y"]), ob._p(w[name]), ob._p(at), ctypes.c_long(2 * I), ctypes.c_int(T),
                                          ctypes.c_int(I), ctypes.c_int(hid), ctypes.c_int(ob.W_KN), ob._stream(None)))
    ob.swiglu(F, s["pair"], s["act"], T, I)
    ob.gemm(F, s["act"], w["down"], s["y"], T, hid, I)
    ob.add_residual_rmsnorm(F, s["res"], s["y"], None, w["last"], 1e-5, T, hid)


def run_float_context(s):
    w, (hid, H, G, D, I, B, T, Q, K, S) = s["w"], s["dims"]
    F = ob.F32
    ob.cal_padding_offset(s["offset"], s["cum"], s["lens"], B, Q, want_token_num=False)
    ob.build_causal_mask(F, s["mask"], s["lens"], s["ctx"], Q, K, B, attend_history=True)
    ob.embedding(F, s["ids"], s["res"], w["table"], T, hid, VOCAB)
    s["y"].copy_(s["res"])
    ob.rmsnorm(F, s["y"], w["norm1"], 1e-5, T, hid)
    ob.gemm(F, s["y"], w["qkv"], s["qkv"], T, (H + 2 * G) * D, hid)
    ob.qkv_bias_rope_transpose(F, s["q"], s["kn"], s["vn"], s["qkv"], None, s["offset"], s["hist"], B, Q, T, H, G, D, D, ROPE_BASE)
    for new, cache, rep in ((s["kn"], s["k"], s["kr"]), (s["vn"], s["v"], s["vr"])):
        ob.append_kv_cache(F, cache, new, s["lens"], s["hist"], B, G, Q, S, D)
        ob.repeat_kv(F, rep, cache, s["ctx"], B, H, G, K, S, D)
    ob.batched_gemm(F, s["q"], s["kr"], s["score"], B * H, Q, K, D, trans_b=True)
    ob.scale_mask_softmax(F, s["prob"], s["score"], s["mask"], B, H, Q, K, D ** -0.5)
    ob.batched_gemm(F, s["prob"], s["vr"], s["pv"], B * H, Q, D, K)
    ob.transpose_remove_padding(F, s["attn"], s["pv"], s["offset"], T, B, Q, H, D)
    float_feed_forward(s, T)
    return {"out": s["y"], "stream": s["res"], "k": s["k"], "v": s["v"]}


def run_float_decode(s):
    w, (hid, H, G, D, I, B, S, step) = s["w"], s["dims"]
    F, row = ob.F32, (H + 2 * G) * D
    ob.embedding(F, s["ids"], s["res"], w["table"], B, hid, VOCAB)
    s["y"].copy_(s["res"])
    ob.rmsnorm(F, s["y"], w["norm1"], 1e-5, B, hid)
    ob.gemm(F, s["y"], w["qkv"], s["qkv"], B, row, hid)
    p = s["qkv"].data_ptr()
    ob.decode_attn(F, p, p + 4 * H * D, p + 4 * (H + G) * D, row, row, row, None, None, None, s["k"], s["v"], G * S * D, S * D, D, B, H, G, D, step,
                   step - 1, D, ROPE_BASE, D ** -0.5, s["attn"], H * D, s["ws"], s["need"])
    float_feed_forward(s, B)
    ob.gemm(F, s["y"], w["head"], s["logits"], B, VOCAB, hid, w_layout=ob.W_NK)
    return {"logits": s["logits"], "stream": s["res"], "k": s["k"], "v": s["v"]}


# ---- what a pass cannot do without ---------------------------------------------------------------------------
def layer_elements(c):
    """(weights of a layer, attention columns of a token's query, columns of its key and value) of a case's design"""
    s = SIZES[c["size"]]
    hid, H, G, D, I = (s[k] for k in ("hidden", "head_num", "kv_head_num", "head_size", "inter_size"))
    design = c.get("design", "llama")
    if design == "finuvik":
        rh, rk, rv, G = FINUVIK[c["size"]]
        return hid * ((H + 2 * G) * D + rh * (2 * rk + rv)) + hid * (H * D + rh * rv) + 3 * hid * I, H * D, 2 * G * D
    return hid * (H + 2 * G) * D + hid * H * D + 3 * hid * I, H * D, 2 * G * D


def fuposun_layers(c):
    """Weights of all layers, (heads, key, value) of the recurrences, number of recurrent and of attention layers."""
    s, (q_rank, kv_rank, window, gh, gk, gv) = SIZES[c["size"]], FUPOSUN[c["size"]]
    hid, H, D, I = s["hidden"], s["head_num"], s["head_size"], s["inter_size"]
    rec = (c["layers"] + 1) // 2
    attn = c["layers"] - rec
    n = rec * hid * (gh * (2 * gk + 3 * gv) + 16) + attn * (hid * (q_rank + kv_rank + H) + q_rank * H * D + 2 * kv_rank * H * D + H * D * hid)
    return n + c["layers"] * 3 * hid * I, rec, attn


def work(case):
    c = case
    s = SIZES[c["size"]]
    hid, H, D, I = s["hidden"], s["head_num"], s["head_size"], s["inter_size"]
    if c["family"] in ("float_context", "float_decode"):
        G = s["kv_head_num"]
        weights = hid * (H + 2 * G) * D + H * D * hid + 3 * hid * I
        if c["family"] == "float_decode":
            B = c["batch"]
            cells = (c["context"] + 1) * B
            return {"bytes": 4.0 * (weights + VOCAB * hid + cells * 2 * G * D + B * (3 * hid + VOCAB)),
                    "flops": 2.0 * B * (weights + VOCAB * hid) + 4.0 * cells * H * D}
        lens, hist = numbers(c["prompts"]), numbers(c["history"])
        T = sum(lens)
        cells = sum(n * h + n * (n + 1) / 2 for n, h in zip(lens, hist))
        return {"bytes": 4.0 * (weights + sum(hist) * 2 * G * D + T * (3 * hid + 2 * G * D)), "flops": 2.0 * T * weights + 4.0 * cells * H * D}
    if c["family"] == "experts":
        T, F = c["tokens"], I // TOP
        reached = EXPERTS * (1 - (1 - TOP / EXPERTS) ** T)
        return {"bytes": 2.0 * (hid * EXPERTS + reached * 3 * hid * F) + T * hid * (2 + 4 + 4 + 2), "flops": 2.0 * T * (hid * EXPERTS + TOP * 3 * hid * F)}
    batch = c["batch"] if "batch" in c else len(numbers(c["prompts"]))
    head = VOCAB * hid
    steps = c.get("steps", 0)
    lens = [c["context"]] * batch if c["family"] == "decode" else [c["prompt"]] * batch if c["family"] == "generate" else numbers(c["prompts"])
    context_pass = c["family"] != "decode"
    T = sum(lens) if context_pass else 0
    design = c.get("design", "llama")
    if design == "fuposun":
        all_weights, rec, attn = fuposun_layers(c)
        q_rank, kv_rank, window, gh, gk, gv = FUPOSUN[c["size"]]
        seen = sum(min(i, window) for n in lens for i in range(1, n + 1))
        later = sum(min(n + t, window) for n in lens for t in range(1, steps + 1))
        cell_flops = 4.0 * attn * H * D * (seen + later)
        rec_flops = 5.0 * rec * gh * gk * gv * (T + steps * batch)
        cell_bytes = 2.0 * attn * kv_rank * (T + later) + 8.0 * rec * gh * gk * gv * batch * (steps + 1)
    else:
        weights, q_cols, kv_cols = layer_elements(c)
        all_weights = weights * c["layers"]
        seen = sum(n * (n + 1) / 2 for n in lens) if context_pass else 0
        later = sum(n + t for n in lens for t in range(1, steps + 1))
        cell_flops = 4.0 * c["layers"] * q_cols * (seen + later)
        cell_bytes = 2.0 * c["layers"] * kv_cols * (T + later)
        rec_flops = 0.0
        if design == "finuvik":
            rh, rk, rv, _ = FINUVIK[c["size"]]
            rec_flops = 5.0 * c["layers"] * rh * rk * rv * (T + steps * batch)
            cell_bytes += 8.0 * c["layers"] * rh * rk * rv * batch * (steps + 1)
    passes = steps + (1 if context_pass else 0)
    return {"bytes": passes * 2.0 * (all_weights + head) + cell_bytes + 4.0 * batch * VOCAB + 2.0 * hid * (T + steps * batch),
            "flops": 2.0 * all_weights * (T + steps * batch) + 2.0 * head * batch * passes + cell_flops + rec_flops}


# Four to five times the error against the sums in 64 bits (0.0021, 0.0046, 0.0047, 0.0024, 2.8e-6): 16-bit activations round at
# every launch of every layer, the float32 layer sums up to 11008 products.
TOLERANCE = {"llama": 1e-2, "finuvik": 2e-2, "fuposun": 2e-2, "experts": 1e-2, "float": 1.2e-5}


def tolerance(case):
    if case["family"].startswith("float"):
        return {"rel": TOLERANCE["float"]}
    if case["family"] == "experts":
        return {"rel": TOLERANCE["experts"]}
    return {"rel": TOLERANCE[case.get("design", "llama")]}


# ---- the same in 64 bits -----------------------------------------------------------------------------------
def init_normal(seed, tag, rows, cols, std, dtype):
    """The engines' random weights: a counter hashed to two uniform numbers, Box-Muller, rounded to the element type."""
    wrap = lambda v: ((v + 2 ** 63) % 2 ** 64) - 2 ** 63
    shift = lambda x, n: (x >> n) & ((1 << (64 - n)) - 1)
    out = torch.empty(rows, cols, device="cuda", dtype=torch.float64)
    part = max(1, (1 << 26) // cols)
    for r in range(0, rows, part):
        n = min(part, rows - r)
        x = torch.arange(r * cols, (r + n) * cols, device="cuda", dtype=torch.int64) + wrap(seed * 0x100000001B3 + tag * 0x9E3779B1)
        x = x + wrap(0x9E3779B97F4A7C15)
        x = (x ^ shift(x, 30)) * wrap(0xBF58476D1CE4E5B9)
        x = (x ^ shift(x, 27)) * wrap(0x94D049BB133111EB)
        x = x ^ shift(x, 31)
        u1 = (shift(x, 40).double() + 1.0) / 16777217.0
        u2 = (shift(x, 8) & 0xFFFFFF).double() / 16777216.0
        z = torch.sqrt(-2.0 * torch.log(u1)) * torch.cos(2.0 * math.pi * u2) * std
        out[r:r + n] = z.float().to(dtype).double().view(n, cols)
    return out


def rms(x, eps, w=1.0):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def rotate(x, pos, D):
    """x [..., H, D] at positions pos [...]: adjacent pairs, angles in single precision as the path defines them."""
    denom = torch.from_numpy(np.power(np.float32(ROPE_BASE), np.arange(0, D, 2, dtype=np.float32) / np.float32(D))).cuda()
    a = (pos.float()[..., None] / denom).double()[..., None, :]
    c, s = torch.cos(a), torch.sin(a)
    x0, x1 = x[..., 0::2], x[..., 1::2]
    return torch.stack((c * x0 - s * x1, c * x1 + s * x0), -1).flatten(-2)


def attend(q, k, v, bias, scale):
    """q [n, H, d] over k, v [m, G, d]; bias [H or 1, n, m] (-inf: not seen), added behind the scale -> [n, H * d]"""
    r = q.shape[1] // k.shape[1]
    out = torch.empty(q.shape[0], q.shape[1], v.shape[2], device="cuda", dtype=torch.float64)
    for h in range(q.shape[1]):
        p = torch.softmax(q[:, h] @ k[:, h // r].T * scale + bias[h % bias.shape[0]], -1)
        out[:, h] = p @ v[:, h // r]
    return out.flatten(1)


def causal(n, m, window=None):
    """Bias of n queries that are the last of m positions."""
    d = torch.arange(m - n, m, device="cuda")[:, None] - torch.arange(m, device="cuda")[None]
    seen = (d >= 0) if window is None else (d >= 0) & (d < window)
    return torch.where(seen, 0.0, float("-inf")).double()[None]


def exact(case, seed):
    if case["family"].startswith("float"):
        return exact_float(case, seed)
    if case["family"] == "experts":
        return exact_experts(case, seed)
    return {"llama": exact_llama, "finuvik": exact_finuvik, "fuposun": exact_fuposun}[case.get("design", "llama")](case, seed)


def exact_llama(c, seed):
    s = SIZES[c["size"]]
    hid, H, G, D, I = (s[k] for k in ("hidden", "head_num", "kv_head_num", "head_size", "inter_size"))
    decode = c["family"] == "decode"
    n = positions_of(c)
    lens = [c["steps"]] * c["batch"] if decode else numbers(c["prompts"])
    hist = c["context"] if decode else 0
    ids = token_ids(seed, c["steps"], c["batch"]).T.reshape(-1) if decode else token_ids(seed, sum(lens))
    B = len(lens)
    W = lambda tag, rows, cols: init_normal(seed, tag, rows, cols, 0.02, torch.float16)
    x = W(1000001, VOCAB, hid)[torch.from_numpy(ids.astype(np.int64)).cuda()]
    at = np.cumsum([0] + lens)
    pos = torch.cat([torch.arange(hist, hist + l, device="cuda") for l in lens])
    g, kv = generator(seed), []
    for l in range(c["layers"]):
        qkv = (rms(x, 1e-5) @ W(16 * l, hid, (H + 2 * G) * D)).view(-1, H + 2 * G, D)
        q, k, v = rotate(qkv[:, :H], pos, D), rotate(qkv[:, H:H + G], pos, D), qkv[:, H + G:]
        if decode:
            old = [torch.randn(B, G, hist, D, generator=g, device="cuda", dtype=torch.float16) for _ in range(2)]
            new = [t.view(B, lens[0], G, D).transpose(1, 2) for t in (k, v)]
        else:
            new = [torch.zeros(B, G, n, D, device="cuda", dtype=torch.float64) for _ in range(2)]
        out = []
        for b in range(B):
            mine = slice(at[b], at[b + 1])
            kk, vv = k[mine], v[mine]
            if decode:
                kk, vv = (torch.cat((o[b].double().transpose(0, 1), t)) for o, t in zip(old, (kk, vv)))
            else:
                for o, t in zip(new, (kk, vv)):
                    o[b, :, :lens[b]] = t.transpose(0, 1)
            out.append(attend(q[mine], kk, vv, causal(lens[b], len(kk)), D ** -0.5))
        kv.append(tuple(new))
        x = x + torch.cat(out) @ W(16 * l + 1, H * D, hid)
        h = rms(x, 1e-5)
        x = x + (torch.nn.functional.silu(h @ W(16 * l + 2, hid, I)) * (h @ W(16 * l + 3, hid, I))) @ W(16 * l + 4, I, hid)
    last = x[torch.from_numpy(at[1:] - 1).cuda()]
    return {"logits": rms(last, 1e-5) @ W(1000002, VOCAB, hid).T, "rows" if decode else "kv": kv}


def tokens_of(c, seed):
    """Ids of every sequence, [batch, prompt and given tokens], and the length of the prompt."""
    if c["family"] == "prefill":
        lens = numbers(c["prompts"])
        return token_ids(seed, sum(lens)).reshape(len(lens), lens[0]), lens[0]
    return np.concatenate((token_ids(seed, c["batch"], c["prompt"]), token_ids(seed + 1, c["steps"], c["batch"]).T), 1), c["prompt"]


def scan(q, f, k, v):
    """state = f * state + k v^T, o = state^T q, from zero; q, f, k [B, n, H, d], v [B, n, H, e]"""
    B, n, H, d = q.shape
    state = torch.zeros(B, H, d, v.shape[3], device="cuda", dtype=torch.float64)
    out = torch.empty_like(v)
    for t in range(n):
        state = torch.addcmul(state * f[:, t, :, :, None], k[:, t, :, :, None], v[:, t, :, None, :])
        out[:, t] = torch.matmul(q[:, t, :, None, :], state)[:, :, 0]
    return out


def exact_finuvik(c, seed):
    s, (rh, rk, rv, G) = SIZES[c["size"]], FINUVIK[c["size"]]
    hid, H, D, I = s["hidden"], s["head_num"], s["head_size"], s["inter_size"]
    ids, _ = tokens_of(c, seed)
    B, n = ids.shape
    W = lambda tag, rows, cols: init_normal(seed, tag, rows, cols, 0.02, torch.bfloat16)
    x = W(1000001, VOCAB, hid)[torch.from_numpy(ids.astype(np.int64)).cuda()] + W(1000003, positions_of(c), hid)[:n]
    cols = [H * D, G * D, G * D, rh * rk, rh * rk, rh * rv]
    dist = (torch.arange(n, device="cuda")[:, None] - torch.arange(n, device="cuda")[None]).double()
    bias = causal(n, n) - torch.log(1.0 + 0.1 * dist.clamp(min=0))[None]
    temp = 1.0 + 0.1 * torch.log(torch.floor((torch.arange(n, device="cuda").double() + 1) / 1024) + 1.0)
    for l in range(c["layers"]):
        h = rms(x, 1e-6)
        q, k, v, rq, rf, rw = (h @ W(16 * l + 32, hid, sum(cols))).split(cols, -1)
        left = torch.stack([attend(q[b].view(n, H, D) * temp[:, None, None], k[b].view(n, G, D), v[b].view(n, G, D), bias, D ** -0.5) for b in range(B)])
        f = (0.5 + 0.5 * torch.sigmoid(rf + 2.0)).view(B, n, rh, rk)
        o = scan(torch.nn.functional.silu(rq).view(B, n, rh, rk), f, 1.0 - f, rw.reshape(B, n, rh, rv))
        ff = torch.relu(h @ W(16 * l + 33, hid, I)) * (h @ W(16 * l + 34, hid, I))
        x = x + torch.cat((left, rms(o, 1e-6).flatten(2), ff), -1) @ W(16 * l + 35, H * D + rh * rv + I, hid)
    return {"logits": rms(x[:, -1], 1e-6) @ W(1000002, hid, VOCAB), **({"kv": []} if c["family"] == "prefill" else {})}


def exact_fuposun(c, seed):
    s, (q_rank, kv_rank, window, gh, gk, gv) = SIZES[c["size"]], FUPOSUN[c["size"]]
    hid, H, D, I = s["hidden"], s["head_num"], s["head_size"], s["inter_size"]
    ids, prompt = tokens_of(c, seed)
    B, n = ids.shape
    tag = iter(range(1, 1 << 20))
    W = lambda rows, cols, dtype=torch.bfloat16: init_normal(seed, next(tag), rows, cols, 0.02, dtype)
    layers = []
    for l in range(c["layers"]):
        if l % 2 == 0:
            w = [W(hid, gh * (2 * gk + 2 * gv) + 16), W(gh * gv, hid), W(gh * gk, 16, torch.float32)]
        else:
            w = [W(hid, q_rank + kv_rank + (H + 15) // 16 * 16), W(H * D, hid), W(q_rank, H * D), W(H * D, kv_rank), W(kv_rank, 2 * H * D)]
        layers.append(w + [W(hid, I), W(hid, I), W(I, hid)])
    x = rms(W(VOCAB, hid)[torch.from_numpy(ids.astype(np.int64)).cuda()], 1e-6)
    head = W(hid, VOCAB)
    in_latent_space = B * prompt <= 64  # keys of the prompt come through the one or the other of two (random) matrices
    for l, w in enumerate(layers):
        z = rms(x, 1e-6) @ w[0]
        if l % 2 == 0:
            q, k, v, g, a = z.split([gh * gk, gh * gk, gh * gv, gh * gv, 16], -1)
            f = torch.exp(torch.nn.functional.logsigmoid(a @ w[2].T + 2.0) / 16.0)
            q, k, f = (t.reshape(B, n, gh, gk) for t in (q * gk ** -0.5, k, f))
            o = rms(scan(q, f, k, v.reshape(B, n, gh, gv)), 1e-6).flatten(2) * torch.nn.functional.silu(g)
        else:
            q, lat = rms(z[..., :q_rank], 1e-6) @ w[2], rms(z[..., q_rank:q_rank + kv_rank], 1e-6)
            gate = torch.sigmoid(z[..., q_rank + kv_rank:q_rank + kv_rank + H])
            bias, o = causal(n, n, window), []
            for b in range(B):
                k_pass, v = (lat[b] @ w[4]).split(H * D, -1)
                k_step = lat[b] @ w[3].T
                qq, v = q[b].view(n, H, D), v.reshape(n, H, D)
                old = attend(qq, (k_step if in_latent_space else k_pass).reshape(n, H, D), v, bias, D ** -0.5)
                if prompt < n:
                    old = torch.cat((old[:prompt], attend(qq, k_step.reshape(n, H, D), v, bias, D ** -0.5)[prompt:]))
                o.append((old.view(n, H, D) * gate[b][:, :, None]).flatten(1))
            o = torch.stack(o)
        x = x + 0.5 * (o @ w[1])
        h = rms(x, 1e-6)
        x = x + 0.5 * ((torch.nn.functional.silu(h @ w[-3]) * (h @ w[-2])) @ w[-1])
    logits = 30.0 * torch.tanh(rms(x[:, -1], 1e-6) @ head / 30.0)
    return {"logits": logits, **({"kv": []} if c["family"] == "prefill" else {})}


def exact_experts(c, seed):
    s = prepare_experts(c, seed)
    z = s["h"].double() @ s["router"].double()
    score, chosen = torch.sigmoid(z).topk(TOP, -1)
    x = s["stream"].double()
    for e in range(EXPERTS):
        token, k = (chosen == e).nonzero(as_tuple=True)
        if len(token):
            h = s["h"][token].double() * score[token, k][:, None]
            g, u = (h @ s["gate"][e].double()).clamp(max=7.0), (h @ s["up"][e].double()).clamp(-7.0, 7.0)
            x.index_add_(0, token, 0.5 * ((g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ s["down"][e].double()))
    return {"stream": x, "out": rms(x, 1e-6), "router": z, "off": None}


def exact_float(c, seed):
    s = (prepare_float_decode if c["family"] == "float_decode" else prepare_float_context)(c, seed)
    w = {k: v.double() for k, v in s["w"].items() if k not in ("table", "head")}
    hid, H, G, D, I, B = s["dims"][:6]
    lens, hist = ([1] * B, [c["context"]] * B) if c["family"] == "float_decode" else (numbers(c["prompts"]), numbers(c["history"]))
    x = s["w"]["table"][s["ids"].long()].double()
    pos = torch.cat([torch.arange(h, h + l, device="cuda") for l, h in zip(lens, hist)])
    qkv = (rms(x, 1e-5, w["norm1"]) @ w["qkv"]).view(-1, H + 2 * G, D)
    q, k, v = rotate(qkv[:, :H], pos, D), rotate(qkv[:, H:H + G], pos, D), qkv[:, H + G:]
    caches, out, at = [s["k"].double(), s["v"].double()], [], 0
    for b, (l, h) in enumerate(zip(lens, hist)):
        for cache, new in zip(caches, (k, v)):
            cache[b, :, h:h + l] = new[at:at + l].transpose(0, 1)
        kk, vv = (cache[b, :, :h + l].transpose(0, 1) for cache in caches)
        out.append(attend(q[at:at + l], kk, vv, causal(l, l + h), D ** -0.5))
        at += l
    x = x + torch.cat(out) @ w["o"]
    h = rms(x, 1e-5, w["norm2"])
    x = x + (torch.nn.functional.silu(h @ w["gate"]) * (h @ w["up"])) @ w["down"]
    y = rms(x, 1e-5, w["last"])
    if c["family"] == "float_decode":
        return {"logits": y @ s["w"]["head"].double().T, "stream": x, "k": caches[0], "v": caches[1]}
    return {"out": y, "stream": x, "k": caches[0], "v": caches[1]}
