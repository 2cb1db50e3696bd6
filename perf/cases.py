"""Timed cases of the framework's main path: what its users have it do, through the entry points they call.

A Q8_0 linear by itself (the C ABI), the Qwen2.5-0.5B-architecture Q8_0 model (prompts and replies of one sequence), the
Llama-3-8B-architecture Q8_0 model (steps of a batch of sequences), and the two designs made of mixer layers with bf16 or
fp32 weights (prompts and replies).  Models are random-initialised once per process, as a program loads a model once;
prompts, continuations and cached contexts come from the seed.

Tokens of a reply are given, not fed back, so that every output has a value that 64-bit arithmetic can confirm.
"""
import ctypes
import math

import numpy as np
import torch

from llamatov_b200 import _lib, archs, measure_layered, synth
from llamatov_b200 import dev_residency as dr
from llamatov_b200.fact_dispatch import Q8Weight
from llamatov_b200.sequences import Sequences
from llamatov_b200.tp import TPDecoder, random_q8

REPLY = 16          # tokens of a reply
STEPS = 4           # steps of a batch
F64 = torch.float64


def listed():
    return [
        # one projection of one token, as a host program drives the C ABI op by op: the smallest call, launch latency
        dict(name="linear-1", kind="linear", tokens=1, rows=4864, cols=896),
        # a projection for a small batch of sequences: 8B-sized matrix, memory bound
        dict(name="linear-24", kind="linear", tokens=24, rows=4096, cols=14336),
        # chat replies of the 0.5B model after a short prompt (the headline workload) and late in a conversation
        dict(name="reply-32", kind="reply", context=32),
        dict(name="reply-1000", kind="reply", context=1000),
        # prompts of the 0.5B model: a long document; three short questions of the same odd length in one pass
        dict(name="prompt-2048", kind="prompt", batch=1, tokens=2048),
        dict(name="prompt-3x333", kind="prompt", batch=3, tokens=333),
        # the 8B model: one sequence at a long context (declared split order of the attention), a served batch
        dict(name="batch-1x4096", kind="batch", batch=1, context=4096, split=16),
        dict(name="batch-32x1024", kind="batch", batch=32, context=1024, split=0),
        # models of mixer layers in bf16: long prompts of both designs, replies of both
        dict(name="nugusun-prompt", kind="mixer", design="nugusun", size="3b", dtype="bfloat16", tokens=2048, reply=0),
        dict(name="nugusun-reply", kind="mixer", design="nugusun", size="3b", dtype="bfloat16", tokens=45, reply=REPLY),
        dict(name="pakalix-prompt", kind="mixer", design="pakalix", size="8b", dtype="bfloat16", tokens=1777, reply=0),
        # the fp32 option, which is what a user compares the bf16 one with
        dict(name="pakalix-f32", kind="mixer", design="pakalix", size="0.5b", dtype="float32", tokens=300, reply=REPLY),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear", "reply", "prompt", "batch", "mixer", "mixer"])
    if kind == "linear":
        return dict(kind=kind, tokens=_log(rng, 1, 600), rows=_log(rng, 128, 16384), cols=128 * _log(rng, 4, 112))
    if kind == "reply":
        return dict(kind=kind, context=_log(rng, 2, 1500))
    if kind == "prompt":
        batch = rng.randint(1, 4)
        return dict(kind=kind, batch=batch, tokens=_log(rng, 2, 2048 // batch))
    if kind == "batch":
        batch = _log(rng, 1, 32)
        return dict(kind=kind, batch=batch, context=_log(rng, 32, 32768 // max(batch, 8)), split=rng.choice([0, 16]) if batch == 1 else 0)
    design, size = rng.choice(["nugusun", "pakalix"]), rng.choice(["0.5b", "3b"])
    dtype = rng.choice(["bfloat16", "bfloat16", "float32"])
    if rng.random() < 0.5:
        return dict(kind=kind, design=design, size=size, dtype=dtype, tokens=_log(rng, 2, 2048 if dtype == "bfloat16" else 512), reply=0)
    return dict(kind=kind, design=design, size=size, dtype=dtype, tokens=_log(rng, 2, 200), reply=rng.randint(2, REPLY))


# --------------------------------------------------------------------------- models, loaded once

_models = {}


def _once(key, make):
    if key not in _models:
        _models[key] = make()
    return _models[key]


def _qwen():
    """(w, cfg): the 0.5B architecture with random Q8_0 weights, matrices as host blocks like a GGUF loader's."""
    a = synth.ARCHS["qwen2.5-0.5b"]
    g = torch.Generator(device="cuda").manual_seed(5)
    E, F, V, nq, nk = a["n_embd"], a["n_ffn"], a["vocab"], a["n_head"] * a["hd"], a["n_head_kv"] * a["hd"]

    def q8(N, K):
        q, d = random_q8(N, K, g, "cuda")
        return Q8Weight(q.cpu().numpy(), d.cpu().numpy(), N, K)

    def vec(n, mean, sigma):
        return (mean + sigma * torch.randn(n, generator=g, device="cuda")).cpu()
    w = {"token_embd.weight": q8(V, E), "output_norm.weight": vec(E, 1.0, 0.1)}
    for i in range(a["n_layers"]):
        p = f"blk.{i}."
        w[p + "attn_norm.weight"], w[p + "ffn_norm.weight"] = vec(E, 1.0, 0.1), vec(E, 1.0, 0.1)
        for n, rows, cols in (("attn_q", nq, E), ("attn_k", nk, E), ("attn_v", nk, E), ("attn_output", E, nq), ("ffn_gate", F, E),
                              ("ffn_up", F, E), ("ffn_down", E, F)):
            w[f"{p}{n}.weight"] = q8(rows, cols)
        for n, rows in (("q", nq), ("k", nk), ("v", nk)):
            w[f"{p}attn_{n}.bias"] = vec(rows, 0.0, 0.02)
    return w, {k: a[k] for k in ("n_layers", "n_head", "n_head_kv", "n_embd", "rope_theta", "norm_eps", "arch")}


def _mixer_model(c):
    make = measure_layered.mixer_model if c["design"] == "nugusun" else measure_layered.pakalix_model
    return _once((c["design"], c["size"], c["dtype"]), lambda: make(measure_layered.SIZES[c["size"]], dtype=c["dtype"], seed=3))


def _tokens(seed, vocab, *shape):
    return torch.from_numpy(np.random.default_rng(seed).integers(0, vocab, shape))


# --------------------------------------------------------------------------- prepare

def prepare(case, seed):
    return {"linear": _prepare_linear, "reply": _prepare_reply, "prompt": _prepare_prompt, "batch": _prepare_batch,
            "mixer": _prepare_mixer}[case["kind"]](case, seed)


def _prepare_linear(c, seed):
    N, K, T = c["rows"], c["cols"], c["tokens"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    q, d = random_q8(N, K, g, "cuda")
    dev = dict(device="cuda")
    return dict(case=c, q=q, d=d.view(torch.int16), x=torch.randn((T, K), generator=g, **dev), y=torch.empty((T, N), **dev),
                xq=torch.empty((T, K), dtype=torch.int8, **dev), xd=torch.empty((T, K // 32), dtype=torch.int16, **dev))


def _prepare_reply(c, seed):
    w, cfg = _once("qwen", _qwen)
    dr.apply_production_profile()
    dr._KV_MAX_SEQ = max(dr._KV_MAX_SEQ, c["context"] + REPLY + 8)
    toks = _tokens(seed, 151936, c["context"] + REPLY)
    kv = [None] * archs.of(cfg).n_slots(cfg)
    runner = dr.GraphRunner(w, cfg, kv)
    n = c["context"]
    runner.seed(toks[:n], torch.arange(n))
    runner.capture(toks[n:n + 1], torch.tensor([n]))
    return dict(case=c, runner=runner, kv=kv, toks=toks, feed=toks[n:].tolist())


def _prepare_prompt(c, seed):
    w, cfg = _once("qwen", _qwen)
    dr.apply_production_profile()
    dr._KV_MAX_SEQ = max(dr._KV_MAX_SEQ, c["tokens"] + 8)
    A = archs.of(cfg)
    kvs = [[A.new_cache(w, cfg, run) for run in A.runs(cfg)] for _ in range(c["batch"])]
    return dict(case=c, w=w, cfg=cfg, kvs=kvs, toks=_tokens(seed, 151936, c["batch"], c["tokens"]))


def _prepare_batch(c, seed):
    cfg = synth.ARCHS["llama-3-8b"]
    dec = TPDecoder(cfg, batch=c["batch"], max_seq=c["context"] + 2 * STEPS, seed=5, attn_split=c["split"])
    toks = _tokens(seed, cfg["vocab"], STEPS, c["batch"])
    dec.fill_cache(c["context"], seed=seed % 1000003)
    dec.set_tokens(toks[0])
    dec.capture()
    return dict(case=c, dec=dec, toks=toks)


def _prepare_mixer(c, seed):
    cfg, w = _mixer_model(c)
    dr.apply_production_profile()
    seqs = Sequences(w, cfg, max_tokens=c["tokens"] + c["reply"] + 8)
    if c["reply"]:      # a server that has answered before: its step is captured
        for _ in range(2):
            seqs.step("warm", [1], want=[0])
        seqs.end("warm")
    toks = _tokens(seed, cfg["vocab"], c["tokens"] + c["reply"]).tolist()
    return dict(case=c, seqs=seqs, prompt=toks[:c["tokens"]], feed=toks[c["tokens"]:])


# --------------------------------------------------------------------------- run

def run(state):
    return {"linear": _run_linear, "reply": _run_reply, "prompt": _run_prompt, "batch": _run_batch,
            "mixer": _run_mixer}[state["case"]["kind"]](state)


def _run_linear(s):
    c = s["case"]
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.call("lt_quant_q8", s["x"].data_ptr(), s["xq"].data_ptr(), s["xd"].data_ptr(), c["cols"], c["tokens"], st)
    _lib.call("lt_q8_gemv", s["q"].data_ptr(), s["d"].data_ptr(), s["xq"].data_ptr(), s["xd"].data_ptr(), None, s["y"].data_ptr(),
              c["rows"], c["cols"], c["tokens"], st)
    return s["y"]


def _run_reply(s):
    r = s["runner"]
    with torch.cuda.stream(r.stream):
        for cache in s["kv"]:       # back to the end of the prompt: another reply to it
            cache.length = s["case"]["context"]
            cache._ensure_len_ptr()
    picks = [r.replay_token(t) for t in s["feed"][:-1]]
    return {"tokens": np.array(picks), "logits": r.replay_logits(s["feed"][-1])}


def _run_prompt(s):
    from llamatov_b200 import prefill
    for kv in s["kvs"]:
        for cache in kv:
            cache.reset()
    if s["case"]["batch"] == 1:
        toks = s["toks"][0]
        logits = dr.forward_pass_resident(s["w"], s["cfg"], toks, torch.arange(len(toks)), s["kvs"][0])
    else:
        B, T = s["toks"].shape
        logits = prefill.prefill_resident(s["w"], s["cfg"], s["toks"], s["kvs"], want_rows=[T * b + T - 1 for b in range(B)])
    first, last = s["kvs"][0][0], s["kvs"][-1][-1]
    return {"logits": logits, "k0": first._k[:first.length * first.width], "v_last": last._v[:last.length * last.width]}


def _run_batch(s):
    dec = s["dec"]
    for length in dec.lens:         # back to the end of the cached context
        length.fill_(s["case"]["context"])
    picks = []
    for t in s["toks"]:
        dec.set_tokens(t)
        picks.append(dec.run(1)[0])
    return {"tokens": np.stack(picks), "logits": dec.logits}


def _run_mixer(s):
    seqs, prompt = s["seqs"], s["prompt"]
    out = [seqs.step("s", prompt, want=[len(prompt) - 1])]
    for t in s["feed"]:
        out.append(seqs.step("s", [t], want=[0]))
    seqs.end("s")
    return torch.cat(out)


# --------------------------------------------------------------------------- work

def _q8_work(a, rows, context, positions):
    """bytes, flops of one pass of the Q8_0 block over `rows` tokens in all, `positions` new ones per sequence behind `context` old ones."""
    E, F, nq, nk = a["n_embd"], a["n_ffn"], a["n_head"] * a["hd"], a["n_head_kv"] * a["hd"]
    params = a["n_layers"] * ((nq + 2 * nk) * E + E * nq + 3 * F * E)
    seqs = rows // positions
    pairs = seqs * (positions * context + positions * (positions + 1) // 2)
    head = a["vocab"] * E
    return {"bytes": (params + head) * 34 / 32 + 8 * nk * a["n_layers"] * seqs * (context + positions) + 4 * seqs * a["vocab"],
            "flops": 2 * params * rows + 2 * head * seqs + 4 * nq * a["n_layers"] * pairs}


def work(case):
    c = case
    if c["kind"] == "linear":
        N, K, T = c["rows"], c["cols"], c["tokens"]
        return {"bytes": N * K // 32 * 34 + 4 * T * (K + N), "flops": 2 * N * K * T}
    if c["kind"] == "reply":
        a = synth.ARCHS["qwen2.5-0.5b"]
        parts = [_q8_work(a, 1, c["context"] + i, 1) for i in range(REPLY)]
    elif c["kind"] == "prompt":
        parts = [_q8_work(synth.ARCHS["qwen2.5-0.5b"], c["batch"] * c["tokens"], 0, c["tokens"])]
    elif c["kind"] == "batch":
        a = synth.ARCHS["llama-3-8b"]
        parts = [_q8_work(a, c["batch"], c["context"] + i, 1) for i in range(STEPS)]
    else:
        s = measure_layered.SIZES[c["size"]]
        E, F, H, hd, V, esize = s["E"], s["F"], s["H"], s["hd"], s["V"], 2 if c["dtype"] == "bfloat16" else 4
        inner = measure_layered.ssd_sizes(s)[0] * measure_layered.ssd_sizes(s)[1]
        per = {"lightning": 5 * E * H * hd, "gla": 5 * E * H * hd,
               "latent_attention": E * (H * (hd + s["rot"]) + s["kv_rank"] + s["rot"] + H * hd) + 2 * s["kv_rank"] * H * hd,
               "attention": E * hd * (2 * H + 2 * s["nkv"]), "mamba2": E * (3 * inner + 256)}
        kinds = measure_layered.KINDS if c["design"] == "nugusun" else measure_layered.PAKALIX_KINDS
        params = sum(per[kinds[i % len(kinds)]] + 3 * E * F for i in range(s["layers"]))
        parts = []
        for i in range(1 + c["reply"]):
            n = c["tokens"] if i == 0 else 1
            parts.append({"bytes": (params + E * V) * esize + 4 * V, "flops": 2 * params * n + 2 * E * V})
    return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}


def tolerance(case):
    """The Q8_0 path has a declared order of every sum: the same bits from any correct implementation.  The mixer models
    are as exact as their element type through their layers: four times the distance from `exact` over sizes and seeds
    (Nugusun 1.5-3e-2 in bf16 and 1e-5 in fp32, Pakalix 3.5e-3 and 2e-6)."""
    if case["kind"] != "mixer":
        return "exact"
    return {"rel": {"nugusun": {"bfloat16": 0.1, "float32": 5e-5}, "pakalix": {"bfloat16": 1.4e-2, "float32": 1e-5}}[case["design"]][case["dtype"]]}


# --------------------------------------------------------------------------- exact: plain torch in 64 bits

def exact(case, seed):
    return {"linear": _exact_linear, "reply": _exact_reply, "prompt": _exact_prompt, "batch": _exact_batch,
            "mixer": _exact_mixer}[case["kind"]](case, seed)


def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _rotate(x, pos, base, dims):
    """x [..., T, heads, d]: component i with component i + dims / 2."""
    half = dims // 2
    ang = pos.to(F64)[:, None, None] * base ** (-2.0 * torch.arange(half, dtype=F64, device=x.device) / dims)
    c, s = torch.cos(ang), torch.sin(ang)
    u, v = x[..., :half], x[..., half:dims]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., dims:]], -1)


def _attend(q, k, v, scale, first, window=None, cap=None):
    """q [T, H, d] at positions first .., k [n, G, d], v [n, G, dv]: causal softmax attention -> [T, H, dv]."""
    T, H, n, G = q.shape[0], q.shape[1], k.shape[0], k.shape[1]
    i, j = torch.arange(first, first + T, device=q.device)[:, None], torch.arange(n, device=q.device)[None]
    hidden = j > i if window is None else (j > i) | (j <= i - window)
    out = []
    for g in range(G):
        s = torch.einsum("thd,jd->htj", q[:, g * H // G:(g + 1) * H // G], k[:, g]) * scale
        s = cap * torch.tanh(s / cap) if cap else s
        out.append(torch.einsum("htj,jv->thv", s.masked_fill(hidden, -math.inf).softmax(-1), v[:, g]))
    return torch.cat(out, 1)


def _q8_linear(x, W):
    """x [T, K] times the transposed Q8_0 matrix W = (quants [N, K], scales [N, K / 32]), x in Q8_0 like the path's."""
    Wq, Wd = W
    b = x.reshape(x.shape[0], -1, 32)
    amax = b.abs().amax(-1, keepdim=True)
    d = torch.where(amax > 0, amax / 127, torch.ones_like(amax)).half().to(F64)
    x = (torch.clamp(torch.round(b / d), -127, 127) * d).reshape(x.shape)
    out = []
    for r in range(0, Wq.shape[0], 32768):
        q, s = Wq[r:r + 32768], Wd[r:r + 32768]
        out.append(x @ (q.to(F64).reshape(len(q), -1, 32) * s.to(F64)[..., None]).reshape(len(q), -1).T)
    return torch.cat(out, 1)


def _q8_model(a, x, first, layer, head, caches=None):
    """Logits of the last position of x [B, T, E] (positions first ..), and the rows' keys of the first and values of the
    last layer.  layer(i): dict of norms, matrices and the bias; caches(i): the keys and values before x, [B, first, nk]."""
    B, T, E = x.shape
    nh, G, hd, F = a["n_head"], a["n_head_kv"], a["hd"], a["n_ffn"]
    nq, nk = nh * hd, G * hd
    pos = torch.arange(first, first + T, device=x.device)
    x = x.reshape(B * T, E)
    keep = []
    for i in range(a["n_layers"]):
        ly = layer(i)
        y = _q8_linear(_rms(x, ly["attn_norm"], a["norm_eps"]), ly["qkv"])
        y = y if ly["bias"] is None else y + ly["bias"]
        q, k, v = y[:, :nq].reshape(B, T, nh, hd), y[:, nq:nq + nk].reshape(B, T, G, hd), y[:, nq + nk:].reshape(B, T, G, hd)
        q, k = _rotate(q, pos, a["rope_theta"], hd), _rotate(k, pos, a["rope_theta"], hd)
        keep.append((k, v))
        if caches is not None:
            ck, cv = caches(i)
            k = torch.cat([ck.to(F64).reshape(B, first, G, hd), k], 1)
            v = torch.cat([cv.to(F64).reshape(B, first, G, hd), v], 1)
        att = torch.stack([_attend(q[b], k[b], v[b], hd ** -0.5, first) for b in range(B)]).reshape(B * T, nq)
        x = x + _q8_linear(att, ly["o"])
        gu = _q8_linear(_rms(x, ly["ffn_norm"], a["norm_eps"]), ly["gateup"])
        x = x + _q8_linear(torch.nn.functional.silu(gu[:, :F]) * gu[:, F:], ly["down"])
    norm, lm = head
    return _q8_linear(_rms(x.reshape(B, T, E)[:, -1], norm, a["norm_eps"]), lm), keep[0][0], keep[-1][1]


def _exact_linear(c, seed):
    s = _prepare_linear(c, seed)
    return _q8_linear(s["x"].to(F64), (s["q"], s["d"].view(torch.float16)))


def _exact_qwen(toks):
    """(logits, k0, v_last) of prompts toks [B, T]."""
    w, _cfg = _once("qwen", _qwen)

    def mat(*names):
        ws = [w[n + ".weight"] for n in names]
        return (torch.cat([torch.from_numpy(m.Wq).cuda().reshape(m.N, m.K) for m in ws]),
                torch.cat([torch.from_numpy(m.Wd).cuda().reshape(m.N, m.K // 32) for m in ws]))

    def vec(*names):
        return torch.cat([w[n] for n in names]).cuda().to(F64)

    def layer(i):
        p = f"blk.{i}."
        qkv = [p + n for n in ("attn_q", "attn_k", "attn_v")]
        return dict(attn_norm=vec(p + "attn_norm.weight"), qkv=mat(*qkv), bias=vec(*[n + ".bias" for n in qkv]), o=mat(p + "attn_output"),
                    ffn_norm=vec(p + "ffn_norm.weight"), gateup=mat(p + "ffn_gate", p + "ffn_up"), down=mat(p + "ffn_down"))
    emb = mat("token_embd")
    ids = toks.reshape(-1).cuda()
    x = (emb[0][ids].to(F64).reshape(len(ids), -1, 32) * emb[1][ids].to(F64)[..., None]).reshape(*toks.shape, -1)
    return _q8_model(synth.ARCHS["qwen2.5-0.5b"], x, 0, layer, (vec("output_norm.weight"), emb))


def _exact_reply(c, seed):
    toks = _tokens(seed, 151936, c["context"] + REPLY)
    return {"tokens": None, "logits": _exact_qwen(toks[None])[0].reshape(1, 1, -1)}


def _exact_prompt(c, seed):
    logits, k0, v_last = _exact_qwen(_tokens(seed, 151936, c["batch"], c["tokens"]))
    if c["batch"] == 1:
        logits = logits.reshape(1, 1, -1)
    return {"logits": logits, "k0": k0[0].reshape(-1), "v_last": v_last[-1].reshape(-1)}


def _exact_batch(c, seed):
    s = _prepare_batch(c, seed)
    dec, a, n = s["dec"], synth.ARCHS["llama-3-8b"], c["context"]

    def mat(m):
        return m.q, m.d.view(torch.float16)

    def layer(i):
        ly = dec.layers[i]
        return dict({k: mat(ly[k]) for k in ("qkv", "o", "gateup", "down")}, bias=None, attn_norm=ly["attn_norm"].to(F64),
                    ffn_norm=ly["ffn_norm"].to(F64))

    def caches(i):
        return [t.view(c["batch"], dec.max_seq, -1)[:, :n] for t in (dec.kc[i], dec.vc[i])]
    emb, ids = mat(dec.embd), s["toks"].T.cuda()
    x = (emb[0][ids].to(F64).reshape(*ids.shape, -1, 32) * emb[1][ids].to(F64)[..., None]).reshape(*ids.shape, -1)
    return {"tokens": None, "logits": _q8_model(a, x, n, layer, (dec.out_norm.to(F64), mat(dec.lm)), caches)[0]}


def _recurrence(q, k, v, alpha):
    """S <- diag(alpha_t) S + k_t v_t^T, o_t = S^T q_t.  q, k, alpha [T, H, d], v [T, H, dv]."""
    S = torch.zeros(q.shape[1], q.shape[2], v.shape[2], dtype=F64, device=q.device)
    o = torch.empty_like(v)
    for t in range(len(q)):
        S.mul_(alpha[t, :, :, None]).addcmul_(k[t, :, :, None], v[t, :, None, :])
        o[t] = torch.bmm(q[t, :, None, :], S)[:, 0]
    return o


def _linear_attention(h, kind, m, w, eps):
    T, H, d, dv = len(h), m["heads"], m["dim"], m["vdim"]
    act = torch.nn.functional.silu if kind == "lightning" else lambda z: z
    q, k, v = [act(h @ w(n).T).reshape(T, H, -1) for n in "qkv"]
    if kind == "gla":
        z = h @ w("a1").T @ w("a2").T + w("a2.b")
        o = _recurrence(q * d ** -0.5, k, v, torch.exp(torch.nn.functional.logsigmoid(z) / m["tau"]).reshape(T, H, d))
        return (_rms(o, w("norm"), eps).reshape(T, H * dv) * torch.nn.functional.silu(h @ w("g").T)) @ w("o").T
    decay = torch.tensor(m["decay"], dtype=F64, device=h.device)[None, :, None].expand(T, H, d)
    o = _recurrence(q, k, v, decay).reshape(T, H * dv)
    return (_rms(o, w("norm"), eps) * torch.sigmoid(h @ w("g").T)) @ w("o").T


def _latent_attention(h, m, w, eps):
    T, H, d, r, rank = len(h), m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
    pos, rot = torch.arange(T, device=h.device), (m["rot"]["base"], m["rot"]["dims"])
    q = (h @ w("q").T).reshape(T, H, d + r)
    q = torch.cat([q[..., :d], _rotate(q[..., d:], pos, *rot)], -1)
    c = h @ w("dkv").T
    shared = _rotate(c[:, None, rank:], pos, *rot).expand(T, H, r)
    c = _rms(c[:, :rank], w("dkv.norm"), eps)
    k = torch.cat([(c @ w("uk").T).reshape(T, H, d), shared], -1)
    return _attend(q, k, (c @ w("uv").T).reshape(T, H, -1), m["scale"], 0, window=m["mask"]["size"]).reshape(T, -1) @ w("o").T


def _mamba2(h, m, w, eps):
    T, H, P, N, G, taps = len(h), m["heads"], m["vdim"], m["state"], m["groups"], m["conv"]
    inner = H * P
    z, u, dt = (h @ w("in").T).split([inner, inner + 2 * G * N, H], 1)
    u = torch.cat([u.new_zeros(taps - 1, u.shape[1]), u])
    u = torch.nn.functional.silu(sum(w("conv")[:, i] * u[i:i + T] for i in range(taps)) + w("conv.b"))
    x, B, C = u.split([inner, G * N, G * N], 1)
    x, per = x.reshape(T, H, P), H // G
    B, C = [t.reshape(T, G, N).repeat_interleave(per, 1) for t in (B, C)]
    dt = torch.nn.functional.softplus(dt + w("dt_bias"))
    alpha = torch.exp(-torch.exp(w("A_log")) * dt)
    o = _recurrence(C, B * dt[..., None], x, alpha[..., None].expand(T, H, N)) + w("D")[:, None] * x
    o = (o.reshape(T, inner) * torch.nn.functional.silu(z)).reshape(T, m["norm_groups"], -1)
    return (_rms(o, 1.0, eps).reshape(T, inner) * w("norm")) @ w("o").T


def _grouped_attention(h, m, w, eps, first):
    T, H, G, d = len(h), m["heads"], m["kv_heads"], m["dim"]
    pos, rot = torch.arange(T, device=h.device), (m["rot"]["base"], m["rot"]["dims"])
    q = _rotate(_rms(h @ w("q").T, w("q.norm"), eps).reshape(T, H, d), pos, *rot)
    k = _rotate(_rms(h @ w("k").T, w("k.norm"), eps).reshape(T, G, d), pos, *rot)
    v = h @ w("v").T
    if "v" in first:
        v = (1 - w("vmix")) * v + w("vmix") * first["v"]
    first.setdefault("v", v)
    o = _attend(q, k, v.reshape(T, G, -1), m["scale"], 0, cap=m["softcap"]) * torch.sigmoid(h @ w("g").T)[..., None]
    return o.reshape(T, -1) @ w("o").T


def _exact_mixer(c, seed):
    cfg, tensors = _mixer_model(c)
    nugusun, eps = c["design"] == "nugusun", cfg["norm_eps"]
    plus = 0.0 if nugusun else 1.0          # norm weights are stored around zero

    def w(n):
        return tensors[n].cuda().to(F64)

    def norm(x, n):
        return _rms(x, plus + w(n), eps)
    ids = _tokens(seed, cfg["vocab"], c["tokens"] + c["reply"])
    x, first = tensors["embed"][ids].cuda().to(F64), {}
    x = x if nugusun else norm(x, "embed.norm")
    for i, ly in enumerate(cfg["layers"]):
        h, m, kind = norm(x, f"l{i}.norm1"), ly["mixer"], ly["type"]
        mix = lambda n, p=f"l{i}.mix.": w(p + n)
        if kind in ("gla", "lightning"):
            y = _linear_attention(h, kind, m, mix, eps)
        elif kind == "latent_attention":
            y = _latent_attention(h, m, mix, eps)
        elif kind == "mamba2":
            y = _mamba2(h, m, mix, eps)
        else:
            y = _grouped_attention(h, m, mix, eps, first)
        p = f"l{i}.mlp."
        if nugusun:
            x = x + y * w(f"l{i}.ls1")
            h = norm(x, f"l{i}.norm2")
            f = (torch.nn.functional.gelu(h @ w(p + "gate").T, approximate="tanh") * (h @ w(p + "up").T)) @ w(p + "down").T
            x = x + f * w(f"l{i}.ls2")
        else:
            lim = ly["mlp"]["limit"]
            g, u = (h @ w(p + "gate").T).clamp(max=lim), (h @ w(p + "up").T).clamp(-lim, lim)
            x = x + cfg["residual_mult"] * (y + (g * torch.sigmoid(1.702 * g) * (u + 1)) @ w(p + "down").T)
    return norm(x[c["tokens"] - 1:], "final.norm") @ w("head").T
