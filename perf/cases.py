"""The work that serving has the model driver do, as cases that can be timed and checked.

A case is one fire of `TorchDriver` - a decode step of a batch (`decode_async`, or `fire_batch` where a model's layers carry a
recurrent state) or the prefill of prompts (`fire_batch` with a raw-logits probe per prompt) - over a stack of layers at a
preset's real widths, or one call of the token sampler. The stacks have fewer layers than the presets (`LAYERS`): a layer's work
is that of the whole model, and several batches with their pages fit one GPU together.

Lengths, page tables and page order follow from the case; weights, pages and tokens from the seed.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from pie_b200 import ops
from pie_b200.driver.executor import CohortStep, TorchDriver
from pie_b200.driver.schema import ForwardRequest, SamplerKind, SamplerSpec
from pie_b200.models.config import preset

PAGE = 16
MAX_REQUESTS = 512
MAX_TOKENS = 16384
LAYERS = {"llama-3.1-8b": 8, "qwen3-32b-fp8": 4, "qwen3-30b-a3b": 4, "gdn-8b": 4}


def listed():
    return [
        # one user's chat with nobody beside: launches and weight reads
        dict(name="decode llama 1", kind="decode", model="llama-3.1-8b", requests=1, shortest=1100, longest=1100),
        # a handful of users at uneven lengths: a small server, or the tail of a batch
        dict(name="decode llama 23", kind="decode", model="llama-3.1-8b", requests=23, shortest=100, longest=2300),
        # the headline benchmark's batch: 512 text completions, prompts of 128 to 2048 tokens and part of the answer
        dict(name="decode llama 512", kind="decode", model="llama-3.1-8b", requests=512, shortest=128, longest=2304),
        # the next turn of a chat: a short prompt behind a context that is already in its pages
        dict(name="prefill llama turn", kind="prefill", model="llama-3.1-8b", requests=1, shortest=61, longest=61, past=709),
        # prompts of a busy server in one fire
        dict(name="prefill llama ragged", kind="prefill", model="llama-3.1-8b", requests=7, shortest=128, longest=2048, past=0),
        # long-context serving of a dense model with block-scaled fp8 weights
        dict(name="decode fp8 48", kind="decode", model="qwen3-32b-fp8", requests=48, shortest=3900, longest=4400),
        dict(name="prefill fp8", kind="prefill", model="qwen3-32b-fp8", requests=2, shortest=1200, longest=1800, past=0),
        # a mixture of experts: a batch that touches every expert with a few rows each, and prompts that fill them
        dict(name="decode moe 200", kind="decode", model="qwen3-30b-a3b", requests=200, shortest=256, longest=1280),
        dict(name="prefill moe", kind="prefill", model="qwen3-30b-a3b", requests=6, shortest=256, longest=1024, past=0),
        # gated delta-rule layers beside attention
        dict(name="decode gdn 40", kind="decode", model="gdn-8b", requests=40, shortest=200, longest=2100),
        dict(name="prefill gdn", kind="prefill", model="gdn-8b", requests=3, shortest=500, longest=1300, past=0),
        # the sampler alone, a batch whose requests ask for different settings
        dict(name="sample mixed 300", kind="sample", sampler="mixed", rows=300, vocab=128256),
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("decode", "decode", "decode", "prefill", "prefill", "prefill", "sample"))
    if kind == "sample":
        return dict(kind=kind, sampler=rng.choice(("greedy", "temperature", "top_p", "top_k", "min_p", "mixed")),
                    rows=_between(rng, 1, 512), vocab=rng.choice((128256, 151936)))
    model = rng.choice(("llama-3.1-8b", "llama-3.1-8b", "qwen3-32b-fp8", "qwen3-30b-a3b", "gdn-8b"))
    if kind == "decode":
        longest = _between(rng, 64, 4400)
        shortest = max(2, int(longest * rng.choice((0.06, 0.4, 1.0))))
        pages = MAX_REQUESTS * 1216 if model == "llama-3.1-8b" else 48 * 4400
        most = max(1, min(256 if model != "llama-3.1-8b" else MAX_REQUESTS, pages // longest))
        return dict(kind=kind, model=model, requests=_between(rng, 1, most), shortest=shortest, longest=longest)
    most = {"llama-3.1-8b": 7500, "gdn-8b": 2600}.get(model, 3500)      # tokens of a fire
    longest = _between(rng, 5, 2048)
    shortest = max(2, int(longest * rng.choice((0.1, 0.5, 1.0))))
    past = 0 if model == "gdn-8b" else rng.choice((0, 0, _between(rng, 16, 2000)))
    return dict(kind=kind, model=model, requests=_between(rng, 1, max(1, min(64, most // longest))), shortest=shortest, longest=longest,
                past=past)


# ------------------------------------------------------------------ what follows from a case
def _config(case):
    return preset(case["model"], num_hidden_layers=LAYERS[case["model"]])


def _shape(case):
    """(new tokens, tokens ahead of them) of every request, and its pages, in one order for every seed."""
    rng = random.Random(case["requests"] * 7919 + case["shortest"] * 31 + case["longest"])
    lens = [rng.randint(case["shortest"], case["longest"]) for _ in range(case["requests"])]
    new = [1] * len(lens) if case["kind"] == "decode" else lens
    old = [n - 1 for n in lens] if case["kind"] == "decode" else [case["past"]] * len(lens)
    counts = [-(-(a + b) // PAGE) for a, b in zip(new, old)]
    order = list(range(sum(counts)))
    rng.shuffle(order)
    return np.array(new, np.int64), np.array(old, np.int64), np.array(counts, np.int64), np.array(order, np.int32)


def _normal(g, *shape, std=None, dtype=torch.bfloat16):
    return torch.empty(*shape, dtype=dtype, device="cuda").normal_(0.0, shape[-1] ** -0.5 if std is None else std, generator=g)


def _weights(cfg, g):
    """Random weights in the layout the driver runs. Their variance is 1 / fan-in and the embedding's is 1, so that every sublayer adds to
    the residual stream about what it adds in a trained model; the router is as decisive as a trained one. An fp8 weight is a pair
    (e4m3, scales)."""
    h, d, hq, hkv, inter = cfg.hidden_size, cfg.head_dim, cfg.num_attention_heads, cfg.num_key_value_heads, cfg.intermediate_size
    ones = lambda n: torch.ones(n, dtype=torch.bfloat16, device="cuda")

    def linear(n, k):
        if cfg.quantization != "fp8_block":
            return _normal(g, n, k)
        scale = torch.empty(n, k // 128, device="cuda").uniform_(0.9, 1.1, generator=g) * (k ** -0.5 / 100)
        return _normal(g, n, k, std=100.0).clamp_(-448, 448).to(torch.float8_e4m3fn), scale

    layers = []
    for li in range(cfg.num_hidden_layers):
        lw = {"ln1": ones(h), "ln2": ones(h)}
        if cfg.is_linear_layer(li):
            hv, dv = cfg.linear_num_value_heads, cfg.linear_value_head_dim
            lw.update(w_gdn_in=_normal(g, cfg.gdn_in_features, h), gdn_conv=_normal(g, cfg.gdn_conv_channels, 4, std=0.3),
                      gdn_A_log=_normal(g, hv, std=0.5, dtype=torch.float32), gdn_dt_bias=_normal(g, hv, std=0.5, dtype=torch.float32),
                      gdn_norm=ones(dv), w_gdn_out=_normal(g, h, hv * dv))
        else:
            lw.update(wqkv=linear((hq + 2 * hkv) * d, h), wo=linear(h, hq * d))
            if cfg.qk_norm:
                lw.update(q_norm=ones(d), k_norm=ones(d))
        if cfg.is_moe:
            e, im = cfg.num_experts, cfg.moe_intermediate_size
            lw.update(router=_normal(g, e, h, std=3 * h ** -0.5), experts_gate_up=_normal(g, e, 2 * im, h), experts_down=_normal(g, e, h, im))
        else:
            lw.update(w_gate_up=linear(2 * inter, h), w_down=linear(h, inter))
        layers.append(lw)
    return {"layers": layers, "embed": _normal(g, cfg.vocab_size, h, std=1.0), "final_norm": ones(h),
            "lm_head": _normal(g, cfg.vocab_size, h, std=2 * h ** -0.5), "lm_head_vocab_start": 0}


def _contents(case, cfg, g):
    """Weights, page contents, recurrent states and tokens of a seed."""
    new, old, counts, order = _shape(case)
    w = _weights(cfg, g)
    kv = _normal(g, cfg.num_hidden_layers, len(order) + 1, 2, cfg.num_key_value_heads, PAGE, cfg.head_dim, std=1.0)
    kv[:, -1] = 0                       # the page that padding points at
    tokens = torch.randint(0, cfg.vocab_size, (int(new.sum()),), generator=g, device="cuda")
    conv = state = None
    if cfg.linear_layers:
        n, r = len(cfg.linear_layers), len(new)
        conv = _normal(g, n, r, cfg.gdn_conv_channels, 3, std=1.0, dtype=torch.float32)
        state = _normal(g, n, r, cfg.linear_num_value_heads, cfg.linear_key_head_dim, cfg.linear_value_head_dim, std=0.1,
                        dtype=torch.float32)
    return w, kv, tokens, conv, state


def _sampler_rows(case, g):
    rows, kind = case["rows"], case["sampler"]
    logits = _normal(g, rows, case["vocab"], std=2.5)
    kinds = ["top_p", "top_k", "temperature", "greedy", "min_p"]
    each = [kinds[i % 5] if kind == "mixed" else kind for i in range(rows)]
    dev = lambda v, dt: torch.tensor(v, dtype=dt, device="cuda")
    return dict(logits=logits, temperature=dev([0.0 if k == "greedy" else 1.0 for k in each], torch.float32),
                top_k=dev([50 if k == "top_k" else 0 for k in each], torch.int32),
                top_p=dev([0.9 if k == "top_p" else 1.0 for k in each], torch.float32),
                min_p=dev([0.05 if k == "min_p" else 0.0 for k in each], torch.float32),
                seeds=torch.randint(1, 2 ** 62, (rows,), generator=g, device="cuda"))


# ------------------------------------------------------------------ what a program has in hand, and one pass
def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "sample":
        return dict(case=case, out=torch.zeros(case["rows"], dtype=torch.int32, device="cuda"), **_sampler_rows(case, g))
    cfg = _config(case)
    new, old, counts, order = _shape(case)
    w, kv, tokens, conv, state = _contents(case, cfg, g)
    for lw in w["layers"]:
        for k, v in lw.items():
            if isinstance(v, tuple):
                lw[k] = ops.Fp8Linear(*v)
    r = len(new)
    driver = TorchDriver(cfg, "cuda", weights=w, num_pages=len(order), page_size=PAGE, max_requests=MAX_REQUESTS, max_tokens=MAX_TOKENS,
                         seed=seed, rs_slots=r)
    driver.kv.data.copy_(kv)
    del kv
    if conv is not None:
        driver.rs.conv_state.copy_(conv)
        driver.rs.rec_state.copy_(state)
    tokens = tokens.cpu().numpy().astype(np.int32)
    bucket = next(b for b in driver.buckets if b >= r)
    indptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    total = (new + old).astype(np.int32)
    st = dict(case=case, driver=driver, bucket=bucket, fired=0, last=None)
    if case["kind"] == "decode":
        driver.precapture_graphs([bucket])
        if conv is None:
            full = lambda v, dt: np.full(r, v, dt)
            st["step"] = CohortStep(r=r, host_tokens=tokens, src_row=full(-1, np.int32), positions=old.astype(np.int32), kv_lens=total,
                                    page_indptr=indptr, page_indices=order, temperature=full(1.0, np.float32), top_k=full(0, np.int32),
                                    top_p=full(0.9, np.float32), min_p=full(0.0, np.float32),
                                    seeds=np.random.default_rng(seed).integers(1, 2 ** 62, r, dtype=np.int64))
            return st
    qo = np.concatenate([[0], np.cumsum(new)]).astype(np.int32)
    positions = np.concatenate([o + np.arange(n) for n, o in zip(new, old)]).astype(np.int32)
    probe = SamplerSpec(SamplerKind.TOP_P, temperature=1.0, top_p=0.9, seed=seed + 1) if case["kind"] == "decode" else \
        SamplerSpec(SamplerKind.RAW_LOGITS)
    st["request"] = ForwardRequest(
        tokens=tokens, positions=positions, qo_indptr=qo, kv_page_indices=order, kv_page_indptr=indptr,
        kv_last_page_lens=((total - 1) % PAGE + 1).astype(np.int32), slot_req=np.arange(r, dtype=np.int32), slot_row=qo[1:] - 1,
        slot_samplers=[probe] * r, rs_slots=np.arange(r, dtype=np.int32) if conv is not None else None,
        rs_reset=np.full(r, int(case["kind"] == "prefill"), np.int32) if conv is not None else None,
        single_token_mode=case["kind"] == "decode")
    return st


def run(state):
    case = state["case"]
    if case["kind"] == "sample":
        return ops.sample(state["logits"], state["temperature"], state["top_k"], state["top_p"], state["min_p"], state["seeds"],
                          out=state["out"])
    driver, r = state["driver"], case["requests"]
    if "step" in state:         # a decode loop: the host reads each step's tokens one step late
        handle = driver.decode_async(state["step"], state["fired"] & 1)
        if state["last"] is not None:
            state["last"].wait()
        state["last"], state["fired"] = handle, state["fired"] + 1
        return {"logits": driver.graphs[state["bucket"]].logits[:r]}
    answer = driver.fire_batch(state["request"])
    if case["kind"] == "decode":
        out = {"logits": driver.graphs[state["bucket"]].logits[:r]}
    else:
        out = {"logits": np.stack([np.frombuffer(s.logits, np.float32) for s in answer.slots]), "kv": driver.kv.data}
    if driver.rs is not None:
        out.update(conv=driver.rs.conv_state, state=driver.rs.rec_state)
    return out


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    if case["kind"] == "sample":
        n = case["rows"] * case["vocab"]
        return {"bytes": 2 * n + 32 * case["rows"], "flops": 4 * n}
    cfg = _config(case)
    new, old, _, _ = _shape(case)
    n, r = int(new.sum()), len(new)
    h, d, hq, hkv = cfg.hidden_size, cfg.head_dim, cfg.num_attention_heads, cfg.num_key_value_heads
    each = 1 + 4 / 128 if cfg.quantization == "fp8_block" else 2         # bytes of a weight
    seen = int((new * old + new * (new + 1) // 2).sum())                 # (query, key) pairs
    total = flops = 0.0
    for li in range(cfg.num_hidden_layers):
        if cfg.is_linear_layer(li):
            hv, dk, dv = cfg.linear_num_value_heads, cfg.linear_key_head_dim, cfg.linear_value_head_dim
            mixer = cfg.gdn_in_features * h + h * hv * dv
            total += r * 8 * (hv * dk * dv + 3 * cfg.gdn_conv_channels)
            flops += n * hv * dk * dv * 6
        else:
            mixer = (2 * hq + 2 * hkv) * d * h
            total += (int(old.sum()) + n) * 2 * hkv * d * 2
            flops += 4.0 * seen * hq * d
        if cfg.is_moe:
            e, k = cfg.num_experts, cfg.num_experts_per_tok
            one = 3 * h * cfg.moe_intermediate_size
            total += each * one * e * (1 - (1 - k / e) ** n) + 2 * e * h
            flops += 2.0 * n * (k * one + e * h)
        else:
            mixer += 3 * h * cfg.intermediate_size
        total += each * mixer
        flops += 2.0 * n * mixer
    total += 2 * cfg.vocab_size * h + 2 * n * h + 2 * r * cfg.vocab_size
    flops += 2.0 * r * cfg.vocab_size * h
    return {"bytes": total, "flops": flops}


def tolerance(case):
    if case["kind"] == "sample":
        return {"rel": 0.0, "differ": 0.005}        # a threshold of sums that falls on another value's edge
    # bf16 results measured 0.7 to 2 % from 64 bits (8-bit activations 5 %); a route or an 8-bit rounding that falls the other way
    # moves single values further
    return {"rel": 0.03, "max": 0.3 if case["model"] in ("llama-3.1-8b", "gdn-8b") else 0.6}


# ------------------------------------------------------------------ the same in 64 bits
def _norm(x, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps)


def _times(x, w):
    """x @ w.T, a weight in 64 bits a block of rows at a time."""
    out = []
    rows = w[0].shape[0] if isinstance(w, tuple) else w.shape[0]
    for a in range(0, rows, 32768):
        part = w[0][a:a + 32768].double() * w[1][a:a + 32768].double().repeat_interleave(128, 1) if isinstance(w, tuple) else \
            w[a:a + 32768].double()
        out.append(x @ part.t())
    return torch.cat(out, -1)


def _rotate(x, pos, theta):
    d = x.shape[-1]
    freq = theta ** (-torch.arange(0, d, 2, dtype=torch.float64, device=x.device) / d)
    a = (pos.double()[:, None] * freq)[:, None]
    x1, x2 = x[..., : d // 2], x[..., d // 2:]
    return torch.cat([x1 * a.cos() - x2 * a.sin(), x2 * a.cos() + x1 * a.sin()], -1)


def _attention(cfg, lw, x, layer, pos, new, old, pages, slots):
    d, hq, hkv = cfg.head_dim, cfg.num_attention_heads, cfg.num_key_value_heads
    n = x.shape[0]
    q, k, v = _times(x, lw["wqkv"]).view(n, -1, d).split([hq, hkv, hkv], 1)
    if cfg.qk_norm:
        q, k = _norm(q, cfg.rms_norm_eps), _norm(k, cfg.rms_norm_eps)
    q, k = _rotate(q, pos, cfg.rope_theta), _rotate(k, pos, cfg.rope_theta)
    layer[slots // PAGE, 0, :, slots % PAGE] = k
    layer[slots // PAGE, 1, :, slots % PAGE] = v
    out, at = [], 0
    for a, b, mine in zip(new.tolist(), old.tolist(), pages):
        kk, vv = layer[mine].permute(1, 2, 0, 3, 4).reshape(2, hkv, -1, d)[:, :, : a + b]
        s = q[at:at + a].view(a, hkv, -1, d).permute(1, 2, 0, 3) @ kk[:, None].transpose(-1, -2) / math.sqrt(d)
        if a > 1:
            s.masked_fill_(torch.ones(a, a + b, dtype=torch.bool, device=x.device).triu(b + 1), -math.inf)
        out.append((s.softmax(-1) @ vv[:, None]).permute(2, 0, 1, 3).reshape(a, hq * d))
        at += a
    return _times(torch.cat(out), lw["wo"])


def _delta_rule(cfg, lw, x, conv, state, new):
    """Gated delta rule of a ragged batch, token by token; `conv` and `state` are advanced in place."""
    hk, hv, dk, dv = cfg.linear_num_key_heads, cfg.linear_num_value_heads, cfg.linear_key_head_dim, cfg.linear_value_head_dim
    c = cfg.gdn_conv_channels
    mix = _times(x, lw["w_gdn_in"])
    z, b, a = mix[:, c:c + hv * dv].view(-1, hv, dv), mix[:, -2 * hv:-hv].sigmoid(), mix[:, -hv:]
    decay = torch.exp(-lw["gdn_A_log"].double().exp() * torch.nn.functional.softplus(a + lw["gdn_dt_bias"].double()))
    taps = lw["gdn_conv"].double()
    mixed, starts = [], np.concatenate([[0], np.cumsum(new)])
    for i in range(len(new)):
        rows = torch.cat([conv[i].t(), mix[starts[i]:starts[i + 1], :c]])
        mixed.append(sum(rows[j:j + int(new[i])] * taps[:, j] for j in range(4)))
        conv[i] = rows[-3:].t()
    y = torch.nn.functional.silu(torch.cat(mixed))
    q, k, v = y.split([hk * dk, hk * dk, hv * dv], 1)
    unit = lambda t: t * torch.rsqrt(t.pow(2).sum(-1, keepdim=True) + 1e-6)
    q = (unit(q.view(-1, hk, dk)) / math.sqrt(dk)).repeat_interleave(hv // hk, 1)
    k, v = unit(k.view(-1, hk, dk)).repeat_interleave(hv // hk, 1), v.view(-1, hv, dv)
    out = torch.empty_like(v)
    first = torch.from_numpy(starts[:-1]).to(x.device)
    by_length = np.argsort(-new, kind="stable")
    for t in range(int(new.max())):
        live = torch.from_numpy(by_length[: int((new > t).sum())]).to(x.device)
        at = first[live] + t
        s = state[live] * decay[at][..., None, None]
        delta = (v[at] - torch.einsum("rhk,rhkv->rhv", k[at], s)) * b[at][..., None]
        s = s + k[at][..., None] * delta[:, :, None]
        out[at] = torch.einsum("rhk,rhkv->rhv", q[at], s)
        state[live] = s
    out = _norm(out, cfg.rms_norm_eps) * torch.nn.functional.silu(z)
    return _times(out.reshape(-1, hv * dv), lw["w_gdn_out"])


def _glu(y):
    return torch.nn.functional.silu(y[:, 0::2]) * y[:, 1::2]


def _experts(cfg, lw, x):
    p, ids = _times(x, lw["router"]).softmax(-1).topk(cfg.num_experts_per_tok)
    p = p / p.sum(-1, keepdim=True)
    out = torch.zeros_like(x)
    for e in range(cfg.num_experts):
        row, col = (ids == e).nonzero(as_tuple=True)
        if len(row):
            out[row] += p[row, col, None] * _times(_glu(_times(x[row], lw["experts_gate_up"][e])), lw["experts_down"][e])
    return out


def exact(case, seed):
    if case["kind"] == "sample":
        return None
    cfg = _config(case)
    new, old, counts, order = _shape(case)
    w, kv, tokens, conv, state = _contents(case, cfg, torch.Generator(device="cuda").manual_seed(seed))
    dev = tokens.device
    pages = [torch.from_numpy(p.astype(np.int64)).to(dev) for p in np.split(order, np.cumsum(counts)[:-1])]
    pos = torch.from_numpy(np.concatenate([o + np.arange(n) for n, o in zip(new, old)])).to(dev)
    slots = torch.cat([p[torch.arange(o, o + n, device=dev) // PAGE] * PAGE + torch.arange(o, o + n, device=dev) % PAGE
                       for p, n, o in zip(pages, new.tolist(), old.tolist())])
    prefill = case["kind"] == "prefill"
    if conv is not None:
        conv, state = (torch.zeros_like(t, dtype=torch.float64) if prefill else t.double() for t in (conv, state))
    kv_out = torch.empty(kv.shape, dtype=torch.float64, device=dev) if prefill else None
    x, linear = w["embed"][tokens].double(), 0
    for li, lw in enumerate(w["layers"]):
        y = _norm(x, cfg.rms_norm_eps)
        if cfg.is_linear_layer(li):
            x = x + _delta_rule(cfg, lw, y, conv[linear], state[linear], new)
            linear += 1
            layer = kv[li].double() if prefill else None
        else:
            layer = kv[li].double()
            x = x + _attention(cfg, lw, y, layer, pos, new, old, pages, slots)
        if prefill:
            kv_out[li] = layer
        y = _norm(x, cfg.rms_norm_eps)
        x = x + (_experts(cfg, lw, y) if cfg.is_moe else _times(_glu(_times(y, lw["w_gate_up"])), lw["w_down"]))
    last = torch.from_numpy(np.cumsum(new) - 1).to(dev)
    out = {"logits": _times(_norm(x[last], cfg.rms_norm_eps), w["lm_head"])}
    if prefill:
        out["kv"] = kv_out
    if conv is not None:
        out.update(conv=conv, state=state)
    return out
