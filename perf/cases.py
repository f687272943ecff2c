"""The work a user of this framework has it do, as cases that can be timed and checked.

Families (``kind``):

  lm_decode      one decode step of the decoder stack (engine.LlamaEngine) as the worker serves it: a CUDA-graph replay of plan +
                 forward, one new token per request on a paged cache
  lm_prefill     a prompt step of the same stack, eager, as the worker runs it: plan + forward over ragged prompts
  attn_decode    the attention operator shim on its own (FlashInferDecodeWrapper.plan / run), long ragged contexts
  attn_prefill   FlashInferPrefillWrapper.plan / run: prompt chunks, some of which continue a context
  sample         penalty + filter + draw over a vocabulary of logits (ops.sample)
  snac, mimi     the vocoders on windows of codes (SNAC.decode / MimiDecoder.decode), a CUDA-graph replay as served
  text_prefill   a prompt step of a text LM on the hybrid engine (state space, recurrence beside window attention, attention,
                 experts from a table), eager, as the worker runs it

Shapes are the ones of this repository's models: Orpheus-3B and CSM-1B decoder layers, SNAC 24 kHz, Mimi, Redalix at the width of the
benchmark.  Two decoder layers stand for a stack: every layer does the same work and the head is the benchmark's 32000 rows.
"""
from __future__ import annotations

import math
import random

import torch
import torch.nn.functional as F

BF16, F32, F64, I32 = torch.bfloat16, torch.float32, torch.float64, torch.int32

# hidden, query heads, kv heads, head dim, feed-forward (engine.LlamaDims.orpheus_3b, depth_engine.CsmDims)
STACKS = {"orpheus": (3072, 24, 8, 128, 8192), "csm": (2048, 32, 8, 64, 8192)}
LAYERS, VOCAB, PAGE, MAX_CONTEXT, MAX_PREFILL = 2, 32000, 128, 2304, 1024
ROPE = {"factor": 32.0, "theta": 500000.0, "low": 1.0, "high": 4.0, "original": 8192.0}
EPS = 1e-5
TEXT_WIDTH, TEXT_PAGE = 2048, 64


def _device():
    return torch.device("cuda", torch.cuda.current_device())


# ---- the cases -----------------------------------------------------------------------------------------------------------------
def listed():
    return [
        # a single stream in the middle of a sentence: what bounds time to the first audio chunk after the prompt
        {"name": "lm_decode_one", "kind": "lm_decode", "stack": "orpheus", "batch": 1, "kv_lo": 257, "kv_hi": 257},
        # the benchmark's steady state: 32 streams staggered between one and eight hundred cached tokens
        {"name": "lm_decode_32", "kind": "lm_decode", "stack": "orpheus", "batch": 32, "kv_lo": 193, "kv_hi": 781},
        # a text prompt of the benchmark's length on an idle replica
        {"name": "lm_prefill_one", "kind": "lm_prefill", "stack": "orpheus", "rows": 133, "requests": 1},
        # a full prompt step (the worker's default limit of rows) shared by ragged prompts
        {"name": "lm_prefill_full", "kind": "lm_prefill", "stack": "orpheus", "rows": 1024, "requests": 3},
        # two voice prompts of a multi-codebook model's length
        {"name": "lm_prefill_voice", "kind": "lm_prefill", "stack": "csm", "rows": 901, "requests": 2},
        # 64 streams near the end of long utterances: the cache is the step's largest read
        {"name": "attn_decode_64", "kind": "attn_decode", "stack": "orpheus", "batch": 64, "kv_lo": 301, "kv_hi": 2304},
        # prompts in portions beside fresh ones
        {"name": "attn_prefill_mixed", "kind": "attn_prefill", "stack": "orpheus", "rows": 997, "requests": 4, "context": 1100},
        # the sampler of a step with the default settings of the speech LM
        {"name": "sample_32", "kind": "sample", "batch": 32, "vocab": 156940, "strategy": "top_p"},
        # the vocoder pass of one stream (first audio chunk), of a full batch
        {"name": "snac_one", "kind": "snac", "batch": 1, "frames": 4, "slice": True},
        {"name": "snac_32", "kind": "snac", "batch": 32, "frames": 4, "slice": True},
        # the multi-codebook model's vocoder: ten-frame chunks of 32 streams
        {"name": "mimi_32", "kind": "mimi", "batch": 32, "frames": 10},
        # a text LM's prompt step
        {"name": "text_prefill_full", "kind": "text_prefill", "rows": 1001, "requests": 2},
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random):
    kind = rng.choice(["lm_decode", "lm_prefill", "attn_decode", "attn_prefill", "sample", "snac", "mimi", "text_prefill"])
    stack = rng.choice(sorted(STACKS))
    if kind in ("lm_decode", "attn_decode"):
        lo = _log_int(rng, 17, 800)
        hi = _log_int(rng, lo, 800 if kind == "lm_decode" else MAX_CONTEXT)
        return {"kind": kind, "stack": stack, "batch": _log_int(rng, 1, 32 if kind == "lm_decode" else 64), "kv_lo": lo, "kv_hi": hi}
    if kind in ("lm_prefill", "attn_prefill"):
        rows = _log_int(rng, 24, MAX_PREFILL)
        c = {"kind": kind, "stack": stack, "rows": rows, "requests": rng.randint(1, max(1, min(8, rows // 16)))}
        if kind == "attn_prefill":
            c["context"] = rng.randint(0, 1100)
        return c
    if kind == "sample":
        return {"kind": kind, "batch": _log_int(rng, 1, 32), "vocab": rng.choice([156940, 32000, 3072]),
                "strategy": rng.choice(["top_p", "top_k", "top_k_top_p", "min_p", "greedy"])}
    if kind == "snac":
        return {"kind": kind, "batch": _log_int(rng, 1, 32), "frames": 4, "slice": rng.random() < 0.75}
    if kind == "mimi":
        return {"kind": kind, "batch": _log_int(rng, 1, 32), "frames": rng.randint(3, 10)}
    rows = _log_int(rng, 48, MAX_PREFILL)
    return {"kind": kind, "rows": rows, "requests": rng.randint(1, max(1, min(4, rows // 24)))}


# ---- sizes that follow from a case (the same for prepare, work and exact) --------------------------------------------------------
def _spread(lo: int, hi: int, n: int):
    """n contexts between lo and hi, both ends included, in an order that is not sorted"""
    if n == 1:
        return [hi]
    v = [lo + (hi - lo) * i // (n - 1) for i in range(n)]
    return v[::2] + v[1::2][::-1]


def _ragged(total: int, n: int):
    """total rows in n unequal portions of at least one row"""
    w = [1.0 + 0.7 * ((i * 5) % 7) for i in range(n)]
    cut = [max(1, int(total * x / sum(w))) for x in w]
    cut[-1] += total - sum(cut)
    if cut[-1] < 1:
        cut = [total // n + (1 if i < total % n else 0) for i in range(n)]
    return cut


def _contexts(case):
    """cached tokens in front of every portion of an attn_prefill case: every other portion is a fresh prompt"""
    c = case["context"]
    return [0 if i % 2 == 0 else max(0, c - 37 * i) for i in range(case["requests"])]


# ---- generators of weights and inputs ------------------------------------------------------------------------------------------
def _gen(seed: int):
    return torch.Generator(device=_device()).manual_seed(int(seed))


def _normal(g, *shape, std=1.0, mean=0.0, dtype=BF16):
    return (torch.randn(*shape, generator=g, device=_device()) * std + mean).to(dtype)


def _stack_weights(stack: str, seed: int):
    """bf16 weights under HF Llama names: N(0, 0.02) projections, norms around one, a head whose logits have a spread of a few units"""
    H, hq, hkv, D, inter = STACKS[stack]
    g = _gen(seed * 7919 + 1)
    sd = {"model.embed_tokens.weight": _normal(g, VOCAB, H)}
    for i in range(LAYERS):
        p = f"model.layers.{i}."
        sd[p + "input_layernorm.weight"] = _normal(g, H, std=0.1, mean=1.0)
        sd[p + "post_attention_layernorm.weight"] = _normal(g, H, std=0.1, mean=1.0)
        for n, rows, cols in (("self_attn.q_proj", hq * D, H), ("self_attn.k_proj", hkv * D, H), ("self_attn.v_proj", hkv * D, H),
                              ("self_attn.o_proj", H, hq * D), ("mlp.gate_proj", inter, H), ("mlp.up_proj", inter, H),
                              ("mlp.down_proj", H, inter)):
            sd[p + n + ".weight"] = _normal(g, rows, cols, std=0.02)
    sd["model.norm.weight"] = _normal(g, H, std=0.1, mean=1.0)
    sd["lm_head.weight"] = _normal(g, VOCAB, H, std=0.04)
    return sd


def _page_table(lens, seed: int, page: int):
    """(indptr, indices, pages in all): every request's pages scattered over the pool, as they are after some time of serving"""
    need = [(n + page - 1) // page for n in lens]
    total = sum(need)
    order = list(range(total))
    random.Random(seed * 31 + 5).shuffle(order)
    indptr = [0]
    for n in need:
        indptr.append(indptr[-1] + n)
    return indptr, order, total


def _lm_inputs(case, seed: int):
    H, hq, hkv, D, _ = STACKS[case["stack"]]
    if case["kind"] == "lm_decode":
        lens = _spread(case["kv_lo"], case["kv_hi"], case["batch"])      # cached tokens, the new one included
        rows = [1] * len(lens)
    else:
        lens = rows = _ragged(case["rows"], case["requests"])
    indptr, indices, total = _page_table(lens, seed, PAGE)
    g = _gen(seed * 7919 + 2)
    ids = torch.randint(0, VOCAB, (sum(rows),), generator=g, device=_device()).to(I32)
    kv = torch.zeros(LAYERS, total, 2, PAGE, hkv, D, dtype=BF16, device=_device())
    if case["kind"] == "lm_decode":                                      # the history: keys and values of the size projections give
        kv.copy_(_normal(g, LAYERS, total, 2, PAGE, hkv, D))
    pos = torch.cat([torch.arange(n - r, n) for n, r in zip(lens, rows)]).to(device=_device(), dtype=I32)
    return {"lens": lens, "rows": rows, "indptr": indptr, "indices": indices, "ids": ids, "kv": kv, "pos": pos}


def _attn_inputs(case, seed: int):
    H, hq, hkv, D, _ = STACKS[case["stack"]]
    if case["kind"] == "attn_decode":
        lens = _spread(case["kv_lo"], case["kv_hi"], case["batch"])
        rows = [1] * len(lens)
    else:
        rows = _ragged(case["rows"], case["requests"])
        lens = [r + c for r, c in zip(rows, _contexts(case))]
    indptr, indices, total = _page_table(lens, seed, PAGE)
    g = _gen(seed * 7919 + 3)
    kv = torch.empty(LAYERS, total, 2, PAGE, hkv, D, dtype=BF16, device=_device())
    for i in range(LAYERS):
        kv[i].copy_(_normal(g, total, 2, PAGE, hkv, D))
    q = _normal(g, LAYERS, sum(rows), hq, D)
    return {"lens": lens, "rows": rows, "indptr": indptr, "indices": indices, "kv": kv, "q": q}


def _sample_inputs(case, seed: int):
    """logits with the spread of a trained head, a penalty history of a few hundred tokens per request"""
    g = _gen(seed * 7919 + 4)
    B, V = case["batch"], case["vocab"]
    logits = _normal(g, B, V, std=2.5)
    hist = torch.randint(0, V, (B, 200), generator=g, device=_device())
    cache = torch.zeros(B, 1, 1, V, dtype=torch.bool, device=_device())
    cache.view(B, V).scatter_(1, hist, True)
    return logits, cache


SNAC_RATES, SNAC_STRIDES, SNAC_LATENT, SNAC_DIM, SNAC_CODES = (8, 8, 4, 2), (4, 2, 1), 768, 1024, 4096


def _snac_weights(seed: int):
    """checkpoint names (weight norm: original0 = norms, original1 = directions); scales keep activations of order one"""
    g, sd = _gen(seed * 7919 + 5), {}

    def rnd(*shape, std=1.0, mean=0.0):
        return _normal(g, *shape, std=std, mean=mean, dtype=F32)

    def conv(p, shape, fan, bias=None, gain=1.0):
        jitter = 1.0 + 0.2 * (2.0 * torch.rand(shape[0], *([1] * (len(shape) - 1)), generator=g, device=_device()) - 1.0)
        sd[p + ".parametrizations.weight.original0"] = gain * math.sqrt(math.prod(shape[1:]) / fan) * jitter
        sd[p + ".parametrizations.weight.original1"] = rnd(*shape)
        if bias is not None:
            sd[p + ".bias"] = rnd(bias, std=0.05)

    def alpha(n):
        return 0.5 + torch.rand(1, n, 1, generator=g, device=_device())

    for i in range(3):
        p = f"quantizer.quantizers.{i}"
        sd[p + ".codebook.weight"] = rnd(SNAC_CODES, 8)
        conv(p + ".out_proj", (SNAC_LATENT, 8, 1), 24, SNAC_LATENT)
    conv("decoder.model.0", (SNAC_LATENT, 1, 7), 7, SNAC_LATENT)
    conv("decoder.model.1", (SNAC_DIM, SNAC_LATENT, 1), SNAC_LATENT, SNAC_DIM)
    cin = SNAC_DIM
    for b, s in enumerate(SNAC_RATES):
        p, cout = f"decoder.model.{b + 2}.block.", cin // 2
        sd[p + "0.alpha"] = alpha(cin)
        conv(p + "1", (cin, cout, 2 * s), 2 * cin, cout, gain=0.6)
        conv(p + "2.linear", (cout, cout, 1), cout, None, gain=0.3)
        for j in range(3):
            q = f"{p}{3 + j}.block."
            sd[q + "0.alpha"] = alpha(cout)
            conv(q + "1", (cout, 1, 7), 7, cout)
            sd[q + "2.alpha"] = alpha(cout)
            conv(q + "3", (cout, cout, 1), cout, cout, gain=0.5)
        cin = cout
    n = len(SNAC_RATES) + 2
    sd[f"decoder.model.{n}.alpha"] = alpha(cin)
    conv(f"decoder.model.{n + 1}", (1, cin, 7), 7 * cin, 1, gain=0.25)
    return sd


def _snac_inputs(case, seed: int):
    g, B, T = _gen(seed * 7919 + 6), case["batch"], 4 * case["frames"]
    codes = [torch.randint(0, SNAC_CODES, (B, T // s), generator=g, device=_device()).to(I32) for s in SNAC_STRIDES]
    noises, t = [], T
    for s in SNAC_RATES:
        t *= s
        noises.append(_normal(g, B, 1, t, dtype=F32))
    n = T * math.prod(SNAC_RATES)
    return codes, noises, ((n // 4, n // 2) if case["slice"] else (0, n))


MIMI = {"dim": 512, "filters": 64, "ratios": (8, 6, 5, 4), "books": 32, "bins": 2048, "book_dim": 256, "heads": 8, "layers": 8,
        "ff": 2048, "period": 10000.0}


def _mimi_weights(seed: int):
    """the decode side of the checkpoint, under its names"""
    g, sd, C, D = _gen(seed * 7919 + 7), {}, MIMI["dim"], MIMI["book_dim"]

    def rnd(*shape, std=1.0, mean=0.0):
        return _normal(g, *shape, std=std, mean=mean, dtype=F32)

    for name, n in (("rvq_first", 1), ("rvq_rest", MIMI["books"] - 1)):
        for k in range(n):
            p = f"quantizer.{name}.vq.layers.{k}._codebook."
            sd[p + "cluster_usage"] = torch.rand(MIMI["bins"], generator=g, device=_device()) + 0.5
            sd[p + "embedding_sum"] = rnd(MIMI["bins"], D) * sd[p + "cluster_usage"][:, None]
        sd[f"quantizer.{name}.output_proj.weight"] = rnd(C, D, 1, std=(D * MIMI["books"]) ** -0.5)
    sd["upsample.convtr.convtr.convtr.weight"] = rnd(C, 1, 4, std=0.7)
    for i in range(MIMI["layers"]):
        p = f"decoder_transformer.transformer.layers.{i}."
        sd[p + "self_attn.in_projs.0.weight"], sd[p + "self_attn.out_projs.0.weight"] = rnd(3 * C, C, std=C ** -0.5), rnd(C, C, std=C ** -0.5)
        sd[p + "linear1.weight"], sd[p + "linear2.weight"] = rnd(MIMI["ff"], C, std=C ** -0.5), rnd(C, MIMI["ff"], std=MIMI["ff"] ** -0.5)
        for n in ("norm1", "norm2"):
            sd[p + n + ".weight"], sd[p + n + ".bias"] = rnd(C, std=0.1, mean=1.0), rnd(C, std=0.1)
        for n in ("layer_scale_1", "layer_scale_2"):
            sd[p + n + ".scale"] = rnd(C, std=0.1, mean=0.5)
    ch = MIMI["filters"] * 2 ** len(MIMI["ratios"])
    sd["decoder.model.0.conv.conv.weight"], sd["decoder.model.0.conv.conv.bias"] = rnd(ch, C, 7, std=(C * 7) ** -0.5), rnd(ch, std=0.05)
    for i, r in enumerate(MIMI["ratios"]):
        p, q = f"decoder.model.{3 * i + 2}.convtr.convtr.", f"decoder.model.{3 * i + 3}.block."
        sd[p + "weight"], sd[p + "bias"] = rnd(ch, ch // 2, 2 * r, std=(2 * ch) ** -0.5), rnd(ch // 2, std=0.05)
        ch //= 2
        sd[q + "1.conv.conv.weight"], sd[q + "1.conv.conv.bias"] = rnd(ch // 2, ch, 3, std=(3 * ch) ** -0.5), rnd(ch // 2, std=0.05)
        sd[q + "3.conv.conv.weight"], sd[q + "3.conv.conv.bias"] = rnd(ch, ch // 2, 1, std=0.5 * (ch // 2) ** -0.5), rnd(ch, std=0.05)
    p = f"decoder.model.{3 * len(MIMI['ratios']) + 2}.conv.conv."
    sd[p + "weight"], sd[p + "bias"] = rnd(1, ch, 3, std=0.5 * (3 * ch) ** -0.5), rnd(1, std=0.01)
    return sd


def _mimi_inputs(case, seed: int):
    return torch.randint(0, MIMI["bins"], (case["batch"], MIMI["books"], case["frames"]), generator=_gen(seed * 7919 + 8), device=_device())


def _text_config():
    """the benchmark's stack of one layer of every kind, each with eight experts (two per token) beside a shared one"""
    W, heads = TEXT_WIDTH, TEXT_WIDTH // 128
    att = {"heads": heads, "kv_heads": heads // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5}
    rot = {"dims": 128, "base": 1e6, "scaling": {"factor": 4.0, "original": 8192, "fast": 32.0, "slow": 1.0}}
    pair = {"left": dict(att, mask={"size": 2048, "keep_first": 4}), "right": {"width": W, "blocks": W // 256, "conv": 4}}
    ssm = {"heads": W // 32, "vdim": 64, "state": 128, "groups": 8, "norm_groups": 8, "conv": 4}
    mlp = {"kind": "moe", "router": {"experts": 8, "top": 2}, "expert": {"ff": W}, "shared": {"ff": W}}
    layers = [{"type": "mamba2", "mixer": ssm, "mlp": mlp}, {"type": "parallel", "mixer": pair, "mlp": mlp},
              {"type": "attention", "mixer": dict(att, mask={"size": 4096}, rot=rot), "mlp": mlp}]
    return {"architecture": "Redalix", "width": W, "vocab": VOCAB, "norm": {"eps": 1e-6}, "layers": layers}


def _text_weights(seed: int):
    c, g, sd = _text_config(), _gen(seed * 7919 + 9), {}
    W = c["width"]

    def rnd(*shape, std=1.0, mean=0.0):
        return _normal(g, *shape, std=std, mean=mean)

    def lin(n, k):
        return rnd(n, k, std=k ** -0.5)

    sd["embed"], sd["head"], sd["final.norm"] = rnd(VOCAB, W), lin(VOCAB, W), rnd(W, std=0.1, mean=1.0)
    for i, L in enumerate(c["layers"]):
        p, m = f"l{i}.", L["mixer"]
        x = p + "mix."
        sd[p + "norm1"] = rnd(W, std=0.1, mean=1.0)
        if L["type"] == "mamba2":
            inner, C = m["heads"] * m["vdim"], m["heads"] * m["vdim"] + 2 * m["groups"] * m["state"]
            sd[x + "in"], sd[x + "conv"], sd[x + "conv.b"] = lin(inner + C + m["heads"], W), rnd(C, m["conv"], std=0.5), rnd(C, std=0.1)
            sd[x + "dt_bias"], sd[x + "A_log"], sd[x + "D"] = (rnd(m["heads"], std=0.5, mean=-2.0), rnd(m["heads"], std=0.5),
                                                              rnd(m["heads"], std=0.5))
            sd[x + "norm"], sd[x + "o"] = rnd(inner, std=0.1, mean=1.0), lin(W, inner)
        else:
            pair = L["type"] == "parallel"
            a, q = (m["left"], x + "left.") if pair else (m, x)
            for n, rows in (("q", a["heads"] * a["dim"]), ("k", a["kv_heads"] * a["dim"]), ("v", a["kv_heads"] * a["vdim"])):
                sd[q + n] = lin(rows, W)
                if not pair:
                    sd[q + n + ".b"] = rnd(rows, std=0.1)
            sd[q + "o"] = lin(W, a["heads"] * a["vdim"])
            if pair:
                r, bs, y = m["right"], m["right"]["width"] // m["right"]["blocks"], x + "right."
                sd[q + "sink"] = rnd(a["heads"])
                for n in ("y", "x"):
                    sd[y + n], sd[y + n + ".b"] = lin(r["width"], W), rnd(r["width"], std=0.1)
                sd[y + "conv"], sd[y + "conv.b"] = rnd(r["width"], r["conv"], std=0.5), rnd(r["width"], std=0.1)
                for n in ("ra", "ri"):
                    sd[y + n], sd[y + n + ".b"] = rnd(r["blocks"], bs, bs, std=bs ** -0.5), rnd(r["blocks"], bs, std=0.1)
                sd[y + "lam"], sd[y + "o"] = rnd(r["width"], mean=-4.0), lin(W, r["width"])
                sd[x + "left.out"], sd[x + "right.out"] = rnd(W, std=0.1, mean=1.0), rnd(W, std=0.1, mean=1.0)
            else:
                sd[q + "g"] = lin(a["heads"], W)
        f = L["mlp"]
        for e in range(f["router"]["experts"]):
            sd[p + f"mlp.e{e}.up"], sd[p + f"mlp.e{e}.down"] = lin(f["expert"]["ff"], W), lin(W, f["expert"]["ff"])
        sd[p + "mlp.table"] = torch.argsort(torch.rand(VOCAB, f["router"]["experts"], generator=g, device=_device()), 1)[
            :, :f["router"]["top"]].to(I32).contiguous()
        sd[p + "mlp.shared.up"], sd[p + "mlp.shared.down"], sd[p + "mlp.shared.sg"] = lin(f["shared"]["ff"], W), lin(W, f["shared"]["ff"]), lin(1, W)
    return sd


def _text_ids(case, seed: int):
    return torch.randint(0, VOCAB, (case["rows"],), generator=_gen(seed * 7919 + 10), device=_device()).to(I32)


# ---- what a program has in hand before the call ----------------------------------------------------------------------------------
def _ints(v):
    return torch.tensor(v, dtype=I32, device=_device())


def _captured(body):
    """(graph, outputs) of one call, captured the way the worker captures its steps"""
    from vox_serve_b200.worker.base import capture_graph

    body()                                               # warm: one-time setup of the kernels happens outside the capture
    torch.cuda.synchronize()
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        with capture_graph(graph, stream):
            out = body()
    torch.cuda.current_stream().wait_stream(stream)
    return graph, out


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("lm_decode", "lm_prefill"):
        from vox_serve_b200 import ops
        from vox_serve_b200.engine import LlamaDims, LlamaEngine, LlamaWeights

        H, hq, hkv, D, inter = STACKS[case["stack"]]
        dims = LlamaDims(H, LAYERS, hq, hkv, D, inter, VOCAB)
        x = _lm_inputs(case, seed)
        weights = LlamaWeights.from_state_dict(_stack_weights(case["stack"], seed), dims, _device())
        eng = LlamaEngine(weights, x["kv"], PAGE, max_rows=64 if kind == "lm_decode" else MAX_PREFILL + 64)
        B, T = len(x["rows"]), sum(x["rows"])
        qo = [0]
        for r in x["rows"]:
            qo.append(qo[-1] + r)
        state = {"case": case, "eng": eng, "ids": x["ids"], "pos": x["pos"], "indptr": _ints(x["indptr"]), "indices": _ints(x["indices"]),
                 "last": _ints([(n - 1) % PAGE + 1 for n in x["lens"]]), "qo": _ints(qo), "B": B, "T": T,
                 "last_rows": _ints([q - 1 for q in qo[1:]])}
        if kind == "lm_decode":
            def step():
                ops.plan_rows(eng.plan, None, state["indptr"], state["indices"], state["last"], B, B, PAGE, eng.chunk)
                return eng.forward(state["ids"], state["pos"], B)

            state["graph"], state["logits"] = _captured(step)
        return state
    if kind in ("attn_decode", "attn_prefill"):
        from vox_serve_b200.flashinfer_utils import FlashInferDecodeWrapper, FlashInferPrefillWrapper

        H, hq, hkv, D, _ = STACKS[case["stack"]]
        x = _attn_inputs(case, seed)
        B = len(x["rows"])
        common = dict(attn_buffer=None, n_qo_head=hq, n_kv_head=hkv, n_state=hq * D, page_size=PAGE, device=_device(), max_pages=2048)
        qo = [0]
        for r in x["rows"]:
            qo.append(qo[-1] + r)
        # page tables on the host, as a scheduler builds them
        state = {"case": case, "kv": x["kv"], "q": x["q"], "qo": torch.tensor(qo, dtype=I32), "indptr": torch.tensor(x["indptr"], dtype=I32),
                 "indices": torch.tensor(x["indices"], dtype=I32), "last": torch.tensor([(n - 1) % PAGE + 1 for n in x["lens"]], dtype=I32)}
        if kind == "attn_decode":
            state["wrapper"] = FlashInferDecodeWrapper(batch_size=64, **common)
        else:
            state["wrapper"] = FlashInferPrefillWrapper(batch_size=64, max_seq_len=MAX_PREFILL + 64, **common)
        return state
    if kind == "sample":
        logits, cache = _sample_inputs(case, seed)
        return {"case": case, "logits": logits, "cache": cache, "seed": 1234 + seed}
    if kind == "snac":
        from vox_serve_b200.tokenizer.snac import SNAC

        codes, noises, keep = _snac_inputs(case, seed)
        dec = SNAC(device=_device())
        dec.load_state_dict(_snac_weights(seed))
        graph, wav = _captured(lambda: dec.decode(codes, noises=noises, out_range=keep))
        return {"case": case, "dec": dec, "codes": codes, "noises": noises, "graph": graph, "wav": wav}
    if kind == "mimi":
        from vox_serve_b200.tokenizer.mimi import MimiConfig, MimiDecoder

        codes = _mimi_inputs(case, seed)
        dec = MimiDecoder(mimi_config=MimiConfig(), state_dict=_mimi_weights(seed), device=_device())
        graph, wav = _captured(lambda: dec.decode(codes))
        return {"case": case, "dec": dec, "codes": codes, "graph": graph, "wav": wav}
    assert kind == "text_prefill", kind
    from vox_serve_b200 import ops
    from vox_serve_b200.hybrid_engine import StepInputs
    from vox_serve_b200.model.redalix import RedalixModel

    rows = _ragged(case["rows"], case["requests"])
    B, T = len(rows), sum(rows)
    model = RedalixModel("text", config=_text_config(), state_dict=_text_weights(seed), device=str(_device()))
    indptr, indices, total = _page_table(rows, seed, TEXT_PAGE)
    cache = model.make_cache(total, TEXT_PAGE, B)
    eng = model.make_engine(cache, MAX_PREFILL, 64)
    qo, tile_req, tile_row = [0], [], []
    for b, n in enumerate(rows):
        if n > 1:
            for r in range(0, n, ops.window_attn_tile_rows()):
                tile_req.append(b)
                tile_row.append(qo[-1] + r)
        qo.append(qo[-1] + n)
    single = [qo[b] for b, n in enumerate(rows) if n == 1]
    step = StepInputs(ids=_text_ids(case, seed), pos=_ints([p for n in rows for p in range(n)]),
                      row_req=_ints([b for b, n in enumerate(rows) for _ in range(n)]), qo_indptr=_ints(qo), page_indptr=_ints(indptr),
                      page_indices=_ints(indices), slots=_ints(list(range(B))), out_rows=_ints([q - 1 for q in qo[1:]]), B=B, T=T, n_out=B,
                      multi=bool(tile_req), single=bool(single), tiles=(_ints(tile_req), _ints(tile_row), len(tile_req)) if tile_req else None,
                      single_rows=(_ints(single), len(single)) if (tile_req and single) else None)
    return {"case": case, "model": model, "eng": eng, "cache": cache, "step": step}


# ---- one pass --------------------------------------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "lm_decode":
        state["graph"].replay()
        return {"logits": state["logits"], "kv": state["eng"].kv_cache}
    if kind == "lm_prefill":
        from vox_serve_b200 import ops

        eng = state["eng"]
        ops.plan_rows(eng.plan, state["qo"], state["indptr"], state["indices"], state["last"], state["B"], state["T"], PAGE, eng.chunk)
        logits = eng.forward(state["ids"], state["pos"], state["T"], last_rows=state["last_rows"])
        return {"logits": logits, "kv": eng.kv_cache}
    if kind == "attn_decode":
        w = state["wrapper"]
        w.plan(state["indptr"], state["indices"], state["last"])
        return [w.run(state["q"][i], state["kv"][i]) for i in range(LAYERS)]
    if kind == "attn_prefill":
        w = state["wrapper"]
        w.plan(state["qo"], state["indptr"], state["indices"], state["last"])
        return [w.run(state["q"][i], state["kv"][i]) for i in range(LAYERS)]
    if kind == "sample":
        from vox_serve_b200 import ops

        return ops.sample(state["logits"], case["strategy"], rep_cache=state["cache"], penalty=1.3, top_k=50, top_p=0.8, min_p=0.05,
                          temperature=0.6, seed=state["seed"], offset=7)
    if kind in ("snac", "mimi"):
        state["graph"].replay()
        return state["wav"]
    logits = state["eng"].forward(state["step"])
    c = state["cache"]
    return {"logits": logits, "state0": c.state[0], "state1": c.state[1], "k1": c.k[1], "v1": c.v[1], "k2": c.k[2], "v2": c.v[2]}


# ---- what a pass cannot do without -----------------------------------------------------------------------------------------------
def _pairs(lens, rows):
    """(query, key) pairs of causal attention"""
    return sum(r * n - r * (r - 1) // 2 for n, r in zip(lens, rows))


def work(case):
    kind = case["kind"]
    if kind in ("lm_decode", "lm_prefill"):
        H, hq, hkv, D, inter = STACKS[case["stack"]]
        if kind == "lm_decode":
            lens = _spread(case["kv_lo"], case["kv_hi"], case["batch"])
            rows = [1] * len(lens)
        else:
            lens = rows = _ragged(case["rows"], case["requests"])
        T, B = sum(rows), len(rows)
        layer = (hq + 2 * hkv) * D * H + H * hq * D + 3 * inter * H
        old = sum(n - r for n, r in zip(lens, rows))
        byts = 2 * (LAYERS * layer + VOCAB * H) + LAYERS * 4 * hkv * D * (old + T) + 2 * T * H + 2 * B * VOCAB
        flops = 2 * T * LAYERS * layer + 2 * B * VOCAB * H + LAYERS * 4 * hq * D * _pairs(lens, rows)
        return {"bytes": byts, "flops": flops}
    if kind in ("attn_decode", "attn_prefill"):
        H, hq, hkv, D, _ = STACKS[case["stack"]]
        if kind == "attn_decode":
            lens = _spread(case["kv_lo"], case["kv_hi"], case["batch"])
            rows = [1] * len(lens)
        else:
            rows = _ragged(case["rows"], case["requests"])
            lens = [r + c for r, c in zip(rows, _contexts(case))]
        return {"bytes": LAYERS * (4 * hkv * D * sum(lens) + 4 * hq * D * sum(rows)), "flops": LAYERS * 4 * hq * D * _pairs(lens, rows)}
    if kind == "sample":
        n = case["batch"] * case["vocab"]
        return {"bytes": 3 * n + 8 * case["batch"], "flops": 4 * n}
    if kind == "snac":
        # every layer over the positions that the kept samples depend on, each weight read once, codes and noise in, samples out
        B, T, n = case["batch"], 4 * case["frames"], 4 * case["frames"] * math.prod(SNAC_RATES)
        lo, hi = (n // 4, n // 2) if case["slice"] else (0, n)
        lens = [T]
        for s in SNAC_RATES:
            lens.append(lens[-1] * s)
        kept, ch, flops, params, noise = hi - lo, SNAC_DIM >> len(SNAC_RATES), 0, 0, 0
        flops += 14 * ch * kept
        params += 7 * ch
        lo, hi = max(0, lo - 3), min(n, hi + 3)
        for b in reversed(range(len(SNAC_RATES))):
            s, t = SNAC_RATES[b], lens[b + 1]
            for dil in (9, 3, 1):
                flops += (2 * ch * ch + 14 * ch) * (hi - lo)
                params += ch * ch + 7 * ch
                lo, hi = max(0, lo - 3 * dil), min(t, hi + 3 * dil)
            flops += 2 * ch * ch * (hi - lo) + 8 * ch * ch * (hi - lo)          # the noise block, two taps of 2 ch inputs
            params += ch * ch + 4 * ch * ch * s
            noise += hi - lo
            pad = (s + 1) // 2
            lo, hi = max(0, (lo + pad - (2 * s - 1)) // s), min(lens[b], (hi - 1 + pad) // s + 1)
            ch *= 2
        flops += (2 * SNAC_LATENT * SNAC_DIM + 14 * SNAC_LATENT) * (hi - lo) + 48 * SNAC_LATENT * T
        params += SNAC_LATENT * SNAC_DIM + 31 * SNAC_LATENT
        return {"bytes": 4 * params + 4 * B * (noise + kept + T + T // 2 + T // 4), "flops": B * flops}
    if kind == "mimi":
        B, T, C, D = case["batch"], case["frames"], MIMI["dim"], MIMI["book_dim"]
        flops, params, t = 4 * T * C * D, 2 * C * D, 2 * T
        flops += MIMI["layers"] * (2 * t * (4 * C * C + 2 * C * MIMI["ff"]) + 2 * C * t * (t + 1))
        params += MIMI["layers"] * (4 * C * C + 2 * C * MIMI["ff"])
        ch = MIMI["filters"] * 2 ** len(MIMI["ratios"])
        flops, params = flops + 14 * t * C * ch, params + 7 * C * ch
        for r in MIMI["ratios"]:
            params += ch * (ch // 2) * 2 * r + 2 * ch * ch // 4
            t *= r
            flops += 2 * t * 2 * ch * (ch // 2) + 2 * t * 4 * (ch // 2) * (ch // 4)
            ch //= 2
        books = min(B * T, MIMI["bins"]) * MIMI["books"] * D
        return {"bytes": 4 * (params + books + B * t) + 8 * B * T * MIMI["books"], "flops": B * (flops + 6 * t * ch)}
    rows, W, c = _ragged(case["rows"], case["requests"]), TEXT_WIDTH, _text_config()
    T, B = sum(rows), len(rows)
    ssm, pair, att = (L["mixer"] for L in c["layers"])
    inner, bc = ssm["heads"] * ssm["vdim"], 2 * ssm["groups"] * ssm["state"]
    a = att["heads"] * 128 + 2 * att["kv_heads"] * 128
    proj = W * (2 * inner + bc + ssm["heads"]) + inner * W                    # state space
    proj += W * (a + 2 * W) + 2 * W * W + W * 2 * 256                        # pair
    proj += W * (a + att["heads"]) + W * W                                   # attention
    moe = c["layers"][0]["mlp"]
    expert, E, top = 2 * W * moe["expert"]["ff"], moe["router"]["experts"], moe["router"]["top"]
    params = proj + 3 * (min(E, T * top) + 1) * expert + VOCAB * W
    flops = 2 * T * proj + 2 * T * 3 * (top + 1) * expert + 2 * B * VOCAB * W
    flops += 2 * 4 * att["heads"] * 128 * _pairs(rows, rows) + T * ssm["heads"] * ssm["vdim"] * ssm["state"] * 6
    caches = 2 * 2 * 2 * att["kv_heads"] * 128 * T + 4 * B * (inner * ssm["state"] + W)
    return {"bytes": 2 * params + 2 * T * W + caches + 4 * B * VOCAB, "flops": flops}


# ---- tolerances: about four times what a pass differs from ``exact`` by -----------------------------------------------------------
def tolerance(case):
    kind = case["kind"]
    if kind in ("lm_decode", "lm_prefill"):
        return {"rel": 0.03}              # 0.0076: bf16 stream and activations through two layers and the head
    if kind in ("attn_decode", "attn_prefill"):
        return {"rel": 0.009}             # 0.0022: bf16 outputs (and probabilities)
    if kind == "sample":
        return "exact"                    # token ids
    if kind == "snac":
        return {"rel": 5e-4}              # 1.2e-4: 32-bit sums; the sines of the activations amplify an error layer by layer
    if kind == "mimi":
        return {"rel": 1.7e-4}            # 4.2e-5: 32-bit sums
    return {"rel": 0.016}                 # 0.0040: bf16 activations through three layers and the head


# ---- the same outputs in 64 bits, in plain torch ----------------------------------------------------------------------------------
def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _rope_half(x, pos):
    """x [T, heads, D]: the halves turn together, frequencies with the long-context smoothing"""
    D = x.shape[-1]
    f = ROPE["theta"] ** (-2.0 * torch.arange(D // 2, dtype=F64, device=x.device) / D)
    a = ROPE["original"] / (2 * math.pi * (ROPE["high"] - ROPE["low"]))
    smooth = (f * a - 1.0 / (ROPE["high"] / ROPE["low"] - 1.0)).clamp(0.0, 1.0)
    ang = pos.double()[:, None] * ((1.0 - smooth) * f / ROPE["factor"] + smooth * f)
    c, s = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
    u, v = x[..., :D // 2], x[..., D // 2:]
    return torch.cat((u * c - v * s, v * c + u * s), -1)


def _causal(q, k, v, scale, window=0, keep=0, sink=None):
    """q [R, H, D] the last R positions of k [N, G, D], v [N, G, V] -> [R, H, V]"""
    R, H, _ = q.shape
    N, G, _ = k.shape
    out = torch.empty(R, H, v.shape[2], dtype=F64, device=q.device)
    i, j = torch.arange(N - R, N, device=q.device)[:, None], torch.arange(N, device=q.device)[None]
    seen = j <= i
    if window:
        seen &= (i - j < window) | (j < keep)
    for g in range(G):
        hs = slice(g * (H // G), (g + 1) * (H // G))
        s = torch.einsum("rhd,nd->hrn", q[:, hs], k[:, g]) * scale
        s = s.masked_fill(~seen, -math.inf)
        if sink is not None:
            s = torch.cat((s, sink[hs][:, None, None].expand(-1, R, 1)), -1)
        p = torch.softmax(s, -1)[..., :N]
        out[:, hs] = torch.einsum("hrn,nv->rhv", p, v[:, g])
    return out


def _exact_lm(case, seed):
    H, hq, hkv, D, inter = STACKS[case["stack"]]
    x, sd = _lm_inputs(case, seed), _stack_weights(case["stack"], seed)
    kv = x["kv"].double()
    h = sd["model.embed_tokens.weight"][x["ids"].long()].double()

    def mat(name):
        return sd[name + ".weight"].double()

    starts = [0]
    for r in x["rows"]:
        starts.append(starts[-1] + r)
    pages = [torch.tensor(x["indices"][x["indptr"][b]:x["indptr"][b + 1]], device=h.device) for b in range(len(x["rows"]))]
    for i in range(LAYERS):
        p = f"model.layers.{i}."
        n = _rms(h, mat(p + "input_layernorm"), EPS)
        q, k, v = (n @ mat(p + f"self_attn.{c}_proj").T for c in "qkv")
        q, k = _rope_half(q.view(-1, hq, D), x["pos"]), _rope_half(k.view(-1, hkv, D), x["pos"])
        v, o = v.view(-1, hkv, D), torch.empty_like(q)
        for b, (L, r) in enumerate(zip(x["lens"], x["rows"])):
            at, rows = torch.arange(L - r, L, device=h.device), slice(starts[b], starts[b + 1])
            kv[i, pages[b][at // PAGE], 0, at % PAGE], kv[i, pages[b][at // PAGE], 1, at % PAGE] = k[rows], v[rows]
            old = torch.arange(L, device=h.device)
            o[rows] = _causal(q[rows], kv[i, pages[b][old // PAGE], 0, old % PAGE], kv[i, pages[b][old // PAGE], 1, old % PAGE], D ** -0.5)
        h = h + o.reshape(-1, hq * D) @ mat(p + "self_attn.o_proj").T
        n = _rms(h, mat(p + "post_attention_layernorm"), EPS)
        h = h + (F.silu(n @ mat(p + "mlp.gate_proj").T) * (n @ mat(p + "mlp.up_proj").T)) @ mat(p + "mlp.down_proj").T
    n = _rms(h, mat("model.norm"), EPS)
    if case["kind"] == "lm_prefill":
        n = n[torch.tensor([s - 1 for s in starts[1:]], device=n.device)]
    return {"logits": n @ mat("lm_head").T, "kv": kv}


def _exact_attn(case, seed):
    x, outs = _attn_inputs(case, seed), []
    for i in range(LAYERS):
        at, o = 0, []
        for b, (L, r) in enumerate(zip(x["lens"], x["rows"])):
            pages = torch.tensor(x["indices"][x["indptr"][b]:x["indptr"][b + 1]], device=x["kv"].device)
            old = torch.arange(L, device=pages.device)
            k, v = (x["kv"][i, pages[old // PAGE], j, old % PAGE].double() for j in (0, 1))
            o.append(_causal(x["q"][i, at:at + r].double(), k, v, k.shape[-1] ** -0.5))
            at += r
        outs.append(torch.cat(o))
    return outs


def _taps(x, w, b=None, dil=1, left=0, right=0):
    """x [B, C, T], w [out, C, k]: the convolution as one product per tap"""
    x = F.pad(x, (left, right))
    T = x.shape[-1] - (w.shape[-1] - 1) * dil
    y = sum(torch.einsum("oc,bct->bot", w[:, :, k], x[..., k * dil:k * dil + T]) for k in range(w.shape[-1]))
    return y if b is None else y + b[:, None]


def _taps_transposed(x, w, b, s, left):
    """w [in, out, 2 s], stride s: (T + 1) s positions, of which the first ``left`` go and T s stay"""
    B, _, T = x.shape
    y = torch.zeros(B, w.shape[1], T + 1, s, dtype=F64, device=x.device)
    for k in range(2 * s):
        y[:, :, k // s:k // s + T, k % s] += torch.einsum("co,bct->bot", w[:, :, k], x)
    return y.reshape(B, w.shape[1], (T + 1) * s)[..., left:left + T * s] + b[:, None]


def _exact_snac(case, seed):
    codes, noises, (lo, hi) = _snac_inputs(case, seed)
    sd = {k: v.double() for k, v in _snac_weights(seed).items()}

    def w(p):
        v = sd[p + ".parametrizations.weight.original1"]
        return v * (sd[p + ".parametrizations.weight.original0"] / torch.linalg.vector_norm(v, dim=tuple(range(1, v.dim())), keepdim=True))

    def snake(x, a):
        return x + torch.sin(a * x) ** 2 / (a + 1e-9)

    def depthwise(x, p, dil=1):
        k, T = w(p)[:, 0], x.shape[-1]
        xp = F.pad(x, (3 * dil, 3 * dil))
        return sum(k[:, j, None] * xp[..., j * dil:j * dil + T] for j in range(7)) + sd[p + ".bias"][:, None]

    z = 0.0
    for i, s in enumerate(SNAC_STRIDES):
        p = f"quantizer.quantizers.{i}"
        e = sd[p + ".codebook.weight"][codes[i].long()].transpose(1, 2)
        z = z + _taps(e, w(p + ".out_proj"), sd[p + ".out_proj.bias"]).repeat_interleave(s, -1)
    x = _taps(depthwise(z, "decoder.model.0"), w("decoder.model.1"), sd["decoder.model.1.bias"])
    for b, s in enumerate(SNAC_RATES):
        p = f"decoder.model.{b + 2}.block."
        x = _taps_transposed(snake(x, sd[p + "0.alpha"]), w(p + "1"), sd[p + "1.bias"], s, (s + 1) // 2)
        x = x + noises[b].double() * _taps(x, w(p + "2.linear"))
        for j, dil in enumerate((1, 3, 9)):
            q = f"{p}{3 + j}.block."
            y = snake(depthwise(snake(x, sd[q + "0.alpha"]), q + "1", dil), sd[q + "2.alpha"])
            x = x + _taps(y, w(q + "3"), sd[q + "3.bias"])
    n = len(SNAC_RATES) + 2
    x = snake(x, sd[f"decoder.model.{n}.alpha"])
    return torch.tanh(_taps(x, w(f"decoder.model.{n + 1}"), sd[f"decoder.model.{n + 1}.bias"], left=3, right=3))[..., lo:hi]


def _exact_mimi(case, seed):
    codes = _mimi_inputs(case, seed)
    sd = {k: v.double() for k, v in _mimi_weights(seed).items()}
    x = 0.0
    for name, cols in (("rvq_first", codes[:, :1]), ("rvq_rest", codes[:, 1:])):
        q = 0.0
        for k in range(cols.shape[1]):
            p = f"quantizer.{name}.vq.layers.{k}._codebook."
            q = q + (sd[p + "embedding_sum"] / sd[p + "cluster_usage"].clamp(min=1e-5)[:, None])[cols[:, k]].transpose(1, 2)
        x = x + _taps(q, sd[f"quantizer.{name}.output_proj.weight"])
    B, C, T = x.shape
    up, y = sd["upsample.convtr.convtr.convtr.weight"][:, 0], torch.zeros(B, C, T + 1, 2, dtype=F64, device=x.device)
    for k in range(4):
        y[:, :, k // 2:k // 2 + T, k % 2] += up[:, k, None] * x
    x = y.reshape(B, C, 2 * T + 2)[..., :2 * T].transpose(1, 2)
    T, H = 2 * T, MIMI["heads"]
    D = C // H
    ang = torch.arange(T, dtype=F64, device=x.device)[:, None] * MIMI["period"] ** (-2.0 * torch.arange(D // 2, dtype=F64, device=x.device) / D)
    c, s = torch.cos(ang), torch.sin(ang)

    def turn(u):
        a, b = u[..., 0::2], u[..., 1::2]
        return torch.stack((a * c - b * s, a * s + b * c), -1).flatten(-2)

    def norm(u, p):
        return F.layer_norm(u, (C,), sd[p + ".weight"], sd[p + ".bias"], 1e-5)

    late = torch.ones(T, T, dtype=torch.bool, device=x.device).triu(1)
    for i in range(MIMI["layers"]):
        p = f"decoder_transformer.transformer.layers.{i}."
        q, k, v = (norm(x, p + "norm1") @ sd[p + "self_attn.in_projs.0.weight"].T).view(B, T, 3, H, D).permute(2, 0, 3, 1, 4)
        a = torch.softmax((turn(q) @ turn(k).transpose(-1, -2) * D ** -0.5).masked_fill(late, -math.inf), -1) @ v
        x = x + sd[p + "layer_scale_1.scale"] * (a.transpose(1, 2).reshape(B, T, C) @ sd[p + "self_attn.out_projs.0.weight"].T)
        u = F.gelu(norm(x, p + "norm2") @ sd[p + "linear1.weight"].T) @ sd[p + "linear2.weight"].T
        x = x + sd[p + "layer_scale_2.scale"] * u
    x = _taps(x.transpose(1, 2), sd["decoder.model.0.conv.conv.weight"], sd["decoder.model.0.conv.conv.bias"], left=6)
    for i, r in enumerate(MIMI["ratios"]):
        p, q = f"decoder.model.{3 * i + 2}.convtr.convtr.", f"decoder.model.{3 * i + 3}.block."
        x = _taps_transposed(F.elu(x), sd[p + "weight"], sd[p + "bias"], r, 0)
        y = _taps(F.elu(x), sd[q + "1.conv.conv.weight"], sd[q + "1.conv.conv.bias"], left=2)
        x = x + _taps(F.elu(y), sd[q + "3.conv.conv.weight"], sd[q + "3.conv.conv.bias"])
    p = f"decoder.model.{3 * len(MIMI['ratios']) + 2}.conv.conv."
    return _taps(F.elu(x), sd[p + "weight"], sd[p + "bias"], left=2)


def _short(u, w, b):
    """u [T, C], w [C, taps]: causal, zeros in front"""
    k, up = w.shape[1], F.pad(u, (0, 0, w.shape[1] - 1, 0))
    return sum(w[:, j] * up[j:j + u.shape[0]] for j in range(k)) + b


def _turn_pairs(x, rot):
    """x [T, heads, D]: neighbouring coordinates turn together, slow pairs interpolated, the rest as they are"""
    dims, base, sc = rot["dims"], rot["base"], rot["scaling"]

    def pair_of(turns):
        return dims * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))

    i = torch.arange(dims // 2, dtype=F64, device=x.device)
    f = base ** (-2.0 * i / dims)
    lo, hi = max(math.floor(pair_of(sc["fast"])), 0), min(math.ceil(pair_of(sc["slow"])), dims - 1)
    slow = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    ang = torch.arange(x.shape[0], dtype=F64, device=x.device)[:, None] * (slow * f / sc["factor"] + (1.0 - slow) * f)
    m = 1.0 + 0.1 * math.log(sc["factor"])
    c, s, y = (torch.cos(ang) * m)[:, None], (torch.sin(ang) * m)[:, None], x.clone()
    y[..., 0:dims:2], y[..., 1:dims:2] = x[..., 0:dims:2] * c - x[..., 1:dims:2] * s, x[..., 1:dims:2] * c + x[..., 0:dims:2] * s
    return y


def _exact_text(case, seed):
    cfg, ids, raw = _text_config(), _text_ids(case, seed).long(), _text_weights(seed)
    sd, eps, W = {k: v.double() for k, v in raw.items() if not k.endswith("table")}, cfg["norm"]["eps"], TEXT_WIDTH
    rows = _ragged(case["rows"], case["requests"])
    indptr, indices, total = _page_table(rows, seed, TEXT_PAGE)
    cuts = [0]
    for r in rows:
        cuts.append(cuts[-1] + r)
    x = sd["embed"][ids]
    out = {}
    for i, L in enumerate(cfg["layers"]):
        p, m = f"l{i}.", L["mixer"]
        q_ = p + "mix."
        h, y = _rms(x, sd[p + "norm1"], eps), torch.empty_like(x)
        a = m.get("left", m)
        if L["type"] != "mamba2":
            kc = torch.zeros(total, TEXT_PAGE, a["kv_heads"], a["dim"], dtype=F64, device=x.device)
            vc = torch.zeros(total, TEXT_PAGE, a["kv_heads"], a["vdim"], dtype=F64, device=x.device)
            states = torch.zeros(len(rows), W, dtype=F64, device=x.device)
        else:
            states = torch.zeros(len(rows), m["heads"], m["state"], m["vdim"], dtype=F64, device=x.device)
        for b, T in enumerate(rows):
            hb, sl = h[cuts[b]:cuts[b + 1]], slice(cuts[b], cuts[b + 1])
            if L["type"] == "mamba2":
                H, V, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
                inner = H * V
                z, xbc, dt = (hb @ sd[q_ + "in"].T).split([inner, inner + 2 * G * N, H], 1)
                u, Bm, Cm = F.silu(_short(xbc, sd[q_ + "conv"], sd[q_ + "conv.b"])).split([inner, G * N, G * N], 1)
                u, dt = u.reshape(T, H, V), F.softplus(dt + sd[q_ + "dt_bias"])
                Bm, Cm = (t.reshape(T, G, N).repeat_interleave(H // G, 1) for t in (Bm, Cm))
                decay, ys = torch.exp(-torch.exp(sd[q_ + "A_log"]) * dt), torch.empty_like(u)
                S = states[b]
                du = dt[:, :, None] * u
                for t in range(T):
                    S.mul_(decay[t, :, None, None]).addcmul_(Bm[t, :, :, None], du[t, :, None, :])
                    ys[t] = (Cm[t, :, None, :] @ S)[:, 0]
                o = ((ys + sd[q_ + "D"][:, None] * u).reshape(T, inner) * F.silu(z)).view(T, m["norm_groups"], -1)
                o = (o / torch.sqrt((o * o).mean(-1, keepdim=True) + eps)).reshape(T, inner) * sd[q_ + "norm"]
                y[sl] = o @ sd[q_ + "o"].T
                continue
            pair = L["type"] == "parallel"
            n = q_ + ("left." if pair else "")
            q, k, v = (hb @ sd[n + c].T + (0.0 if pair else sd[n + c + ".b"]) for c in "qkv")
            q, k, v = q.view(T, a["heads"], -1), k.view(T, a["kv_heads"], -1), v.view(T, a["kv_heads"], -1)
            if not pair:
                q, k = _turn_pairs(q, m["rot"]), _turn_pairs(k, m["rot"])
            pages, at = torch.tensor(indices[indptr[b]:indptr[b + 1]], device=x.device), torch.arange(T, device=x.device)
            kc[pages[at // TEXT_PAGE], at % TEXT_PAGE], vc[pages[at // TEXT_PAGE], at % TEXT_PAGE] = k, v
            o = _causal(q, k, v, a["scale"], a["mask"]["size"], a["mask"].get("keep_first", 0), sd[n + "sink"] if pair else None)
            if not pair:
                o = o * torch.sigmoid(hb @ sd[n + "g"].T)[:, :, None]
            left = o.reshape(T, -1) @ sd[n + "o"].T
            if not pair:
                y[sl] = left
                continue
            r, n = m["right"], q_ + "right."
            g = F.gelu(hb @ sd[n + "y"].T + sd[n + "y.b"], approximate="tanh")
            u = _short(hb @ sd[n + "x"].T + sd[n + "x.b"], sd[n + "conv"], sd[n + "conv.b"])
            parts = u.view(T, r["blocks"], -1)
            ra, ri = (torch.sigmoid(torch.einsum("tbi,boi->tbo", parts, sd[n + c]) + sd[n + c + ".b"]).reshape(T, -1) for c in ("ra", "ri"))
            decay = torch.exp(-8.0 * ra * F.softplus(sd[n + "lam"]))
            add, S, ss = torch.sqrt(1.0 - decay * decay) * ri * u, states[b], torch.empty_like(u)
            for t in range(T):
                S.mul_(decay[t]).add_(add[t])
                ss[t] = S
            right = (ss * g) @ sd[n + "o"].T
            y[sl] = 0.5 * (_rms(left, sd[q_ + "left.out"], eps) + _rms(right, sd[q_ + "right.out"], eps))
        f, n = L["mlp"], p + "mlp."
        picked = raw[n + "table"][ids].long()
        ff = torch.sigmoid(h @ sd[n + "shared.sg"].T) * (F.relu(h @ sd[n + "shared.up"].T) ** 2 @ sd[n + "shared.down"].T)
        for e in range(f["router"]["experts"]):
            hit = (picked == e).any(1).nonzero()[:, 0]
            ff[hit] += (F.relu(h[hit] @ sd[n + f"e{e}.up"].T) ** 2 @ sd[n + f"e{e}.down"].T) / f["router"]["top"]
        x = x + y + ff
        if i < 2:
            out[f"state{i}"] = states
        if i > 0:
            out[f"k{i}"], out[f"v{i}"] = kc, vc
    last = _rms(x, sd["final.norm"], eps)[torch.tensor([c - 1 for c in cuts[1:]], device=x.device)]
    return {"logits": last @ sd["head"].T, "state0": out["state0"], "state1": out["state1"], "k1": out["k1"], "v1": out["v1"], "k2": out["k2"],
            "v2": out["v2"]}


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind in ("lm_decode", "lm_prefill"):
            return _exact_lm(case, seed)
        if kind in ("attn_decode", "attn_prefill"):
            return _exact_attn(case, seed)
        if kind == "snac":
            return _exact_snac(case, seed)
        if kind == "mimi":
            return _exact_mimi(case, seed)
        if kind == "text_prefill":
            return _exact_text(case, seed)
    return None                                  # a draw has no value of its own
