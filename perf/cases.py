"""What is timed: steps of the mixture-of-experts decoders that this framework serves, through the engine calls that its generation API
and its scheduler make (`set_inputs`, then `run`).

Three architectures at the layer sizes of their presets, cut to a few layers so that a model fits the card several times (a whole model
repeats these layers):

  qwen3     grouped-query attention; NVFP4 projections and experts (4-bit weights and activations)
  deepseek  latent attention; FP8 projections with 128 x 128 scales, MXFP4 experts, a shared expert and a dense first layer
  hybrid    gated delta-rule layers and grouped-query attention, bf16 throughout; one decay per head, or one per key channel

and the kinds of steps a server runs: `decode` (one token per sequence, or a few drafted ones to verify, over a filled cache; replayed
from a graph) and `prefill` (prompts, or the next portion of prompts, of any length).  Weights are random in their storage formats; the
rows are large beside what a layer adds to them and the head favours one token, as in a trained model, so that the chosen token is no coin toss."""
import math

import torch

from cuteafd_b200.config import QuantSpec, deepseek_v3_spec, hybrid_gdn_spec, qwen3_235b_spec
from cuteafd_b200.engine.engine import PAGE, StepShape
from cuteafd_b200.engine.mla import mla_weights_random
from cuteafd_b200.engine.registry import build_engine
from cuteafd_b200.models.weights import DeviceWeights

DEV = "cuda"
LAYERS = {"qwen3": 4, "deepseek": 3, "hybrid": 4}
RESIDUAL = 16.0      # of the rows that enter the layers: a layer deep in a trained stack adds a small part of what is there


# ------------------------------------------------------------------ the cases
def listed():
    step = lambda name, model, phase, seqs, rows, context, ragged=False, per_channel=False: {
        "name": name, "model": model, "phase": phase, "seqs": seqs, "rows": rows, "context": context, "ragged": ragged, "per_channel": per_channel}
    return [
        # one user waiting for one answer: the smallest step, bound by latency
        step("qwen3-decode-1", "qwen3", "decode", 1, 1, 1000),
        # the benchmark's step: 16 sequences at 4k
        step("qwen3-decode-16", "qwen3", "decode", 16, 1, 4096),
        # a busy server: sequences of all ages
        step("qwen3-decode-48-ragged", "qwen3", "decode", 48, 1, 5000, ragged=True),
        # one full portion of a prompt
        step("qwen3-prefill-4096", "qwen3", "prefill", 1, 4096, 0),
        # chat turns that arrive together, on top of earlier turns
        step("qwen3-prefill-ragged", "qwen3", "prefill", 7, 333, 700, ragged=True),
        step("deepseek-decode-1", "deepseek", "decode", 1, 1, 3000),
        step("deepseek-decode-16", "deepseek", "decode", 16, 1, 8192),
        # a later portion of a long prompt: attention over what came before
        step("deepseek-prefill-2048", "deepseek", "prefill", 1, 2048, 6144),
        # three drafted tokens and the one before them, eight sequences
        step("hybrid-verify-8x4", "hybrid", "decode", 8, 4, 2048),
        step("hybrid-prefill-4096", "hybrid", "prefill", 1, 4096, 0),
        step("hybrid-prefill-ragged", "hybrid", "prefill", 5, 600, 0, ragged=True, per_channel=True),
    ]


def draw(rng):
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    model, phase = rng.choice(("qwen3", "qwen3", "deepseek", "hybrid")), rng.choice(("decode", "prefill"))
    case = {"model": model, "phase": phase, "ragged": rng.random() < 0.5, "per_channel": model == "hybrid" and rng.random() < 0.5}
    if phase == "decode":
        rows = rng.randint(2, 6) if model == "hybrid" else rng.choice((1, 1, rng.randint(2, 5)))      # several: drafted tokens to verify
        seqs = log(1, 48 if rows == 1 else 14)
        return dict(case, seqs=seqs, rows=rows, context=log(100, 8192))
    total = log(100, 2048 if model == "deepseek" else 4096)
    seqs = min(log(1, 16), max(1, total // 16))
    context = 0 if model == "hybrid" or rng.random() < 0.4 else log(50, 6144 // seqs + 100)
    return dict(case, seqs=seqs, rows=max(1, total // seqs), context=context)


def lengths(case):
    """Per sequence: rows of this step and rows in the cache before it.  Ragged: sequence i has (2 i + 1) / seqs of the mean."""
    n, rows, context = case["seqs"], case["rows"], case["context"]
    share = [(2 * i + 1) / n if case["ragged"] else 1.0 for i in range(n)]
    prefill = case["phase"] == "prefill"
    return ([max(1, round(rows * f)) for f in share] if prefill else [rows] * n), [round(context * f) for f in share]


# ------------------------------------------------------------------ models
def spec_of(case):
    n = LAYERS[case["model"]]
    if case["model"] == "qwen3":
        return qwen3_235b_spec(n)
    if case["model"] == "hybrid":
        return hybrid_gdn_spec(n, per_channel=case["per_channel"]).replace(quant=QuantSpec(experts="bf16", dense="bf16", kv="bf16"))
    spec = deepseek_v3_spec(n)
    return spec.replace(mtp_layers=0, moe=type(spec.moe)(**{**vars(spec.moe), "first_dense": 1}))


def weights_of(spec, seed):
    w = (mla_weights_random if spec.attn.kind == "mla" else DeviceWeights.random)(spec, torch.device(DEV, 0), seed=seed % 100003)
    gen = torch.Generator(device=DEV).manual_seed(seed)
    w.embed.normal_(0, RESIDUAL, generator=gen)
    w.lm_head.data[0].copy_(w.embed.roll(1, 0)).mul_(spec.init_std / RESIDUAL)      # favours the token after the last one
    return w


def cache_rows(spec, slots, seed):
    """What earlier steps left in the paged cache, layer by layer: normalised keys (rotation changes no norm) or latents, and values."""
    gen = torch.Generator(device=DEV).manual_seed(seed + 1)
    a = spec.attn
    for _ in range(spec.n_layers):
        shape = (slots, a.kv_lora_rank + a.qk_rope_head_dim) if a.kind == "mla" else (slots, 2, a.n_kv_heads, a.head_dim)
        yield torch.empty(shape, dtype=torch.bfloat16, device=DEV).normal_(0, 1, generator=gen)


def states(spec, seqs, seed):
    """Recurrent states and convolution inputs [layers, seqs, ...] of sequences that are being decoded."""
    gen = torch.Generator(device=DEV).manual_seed(seed + 2)
    a = spec.attn
    n, chans = sum(spec.layer_is_linear(i) for i in range(spec.n_layers)), (2 * a.linear_k_heads + a.linear_v_heads) * 128
    return (torch.empty(n, seqs, a.linear_v_heads, 128, 128, device=DEV).normal_(0, 0.1, generator=gen),
            torch.empty(n, seqs, 3, chans, dtype=torch.bfloat16, device=DEV).normal_(0, 1, generator=gen))


def step_inputs(case, spec, seed):
    """The step as a scheduler hands it over, and the number of cache pages; every sequence's pages lie behind each other."""
    q_len, before = lengths(case)
    gen = torch.Generator().manual_seed(seed)
    tokens = torch.randint(0, spec.vocab, (sum(q_len),), generator=gen).tolist()
    positions, slots, q_start, pages, page, logit_rows = [], [], [], [], 0, []
    for n, c in zip(q_len, before):
        q_start.append(len(positions))
        positions += range(c, c + n)
        slots += range(page * PAGE + c, page * PAGE + c + n)
        count = -(-(c + n) // PAGE)
        pages.append(list(range(page, page + count)))
        page += count
        logit_rows += range(len(positions) - n, len(positions)) if case["phase"] == "decode" else [len(positions) - 1]
    return dict(tokens=tokens, positions=positions, slot_map=slots, logit_rows=logit_rows, kv_len=[n + c for n, c in zip(q_len, before)], q_start=q_start, q_len=q_len,
                page_table_rows=pages), page


def prepare(case, seed):
    spec = spec_of(case)
    inputs, pages = step_inputs(case, spec, seed)
    q_len, n = inputs["q_len"], case["seqs"]
    eng = build_engine(spec, weights_of(spec, seed), n_pages=pages, max_seqs=n, max_pages_per_seq=max(len(p) for p in inputs["page_table_rows"]))
    recurrent = case["model"] == "hybrid"
    for li, rows in enumerate(cache_rows(spec, pages * PAGE, seed)):
        eng.kv[li].copy_(rows)
    decode = case["phase"] == "decode"
    if decode and recurrent:
        for t, v in zip((eng.lin_state, eng.lin_carry), states(spec, n, seed)):
            t.copy_(v)
    shape = StepShape(T=len(inputs["tokens"]), n_seq=n, max_q_len=max(q_len), n_logits=len(inputs["logit_rows"]), uniform=decode, defer_state=decode and recurrent,
                      attn_splits=eng.attn_splits_for(n, max(q_len), max(inputs["kv_len"])) if decode else 1)
    written = [eng.kv[:, inputs["slot_map"][s]:inputs["slot_map"][s] + k] for s, k in zip(inputs["q_start"], q_len)]
    if recurrent:      # only the attention layer has keys and values
        written = [r[[i for i in range(spec.n_layers) if not spec.layer_is_linear(i)][0]] for r in written]
    return {"engine": eng, "inputs": inputs, "shape": shape, "decode": decode, "fresh": recurrent and not decode, "written": written}


def run(state):
    eng, shape = state["engine"], state["shape"]
    if state["fresh"]:                                                        # new sequences take over the recurrent-state slots
        eng.reset_state_slots(range(shape.n_seq))
    eng.set_inputs(**state["inputs"])
    lane = eng.run(shape, use_graph=state["decode"])
    out = {"logits": lane.logits[:shape.n_logits], "tokens": lane.next_tok[:shape.n_logits], "cache": state["written"]}
    if state["fresh"]:
        out["recurrent"], out["conv"] = eng.lin_state, eng.lin_carry
    return out


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    spec = spec_of(case)
    a, m, H = spec.attn, spec.moe, spec.hidden
    q_len, before = lengths(case)
    T, logits = sum(q_len), sum(q_len) if case["phase"] == "decode" else case["seqs"]
    pairs = sum(n * c + n * (n + 1) // 2 for n, c in zip(q_len, before))
    keys = sum(n + c for n, c in zip(q_len, before))
    dense = {"nvfp4": 0.5625, "fp8_block128": 1.0, "bf16": 2.0}[spec.quant.dense]
    expert = {"nvfp4": 0.5625, "mxfp4": 0.53125, "bf16": 2.0}[spec.quant.experts]
    used = m.n_experts * (1 - (1 - m.top_k / m.n_experts) ** T)
    nbytes, flops = 2.0 * H * T + 2.0 * spec.vocab * H + 4.0 * spec.vocab * logits, 2.0 * spec.vocab * H * logits
    for i in range(spec.n_layers):
        if a.kind == "mla":
            nh, qk = a.n_heads, a.qk_nope_head_dim + a.qk_rope_head_dim
            row = a.kv_lora_rank + a.qk_rope_head_dim
            mats = a.q_lora_rank * H + nh * qk * a.q_lora_rank + row * H + H * nh * a.v_head_dim
            absorb = nh * a.kv_lora_rank * (a.qk_nope_head_dim + a.v_head_dim)
            nbytes += dense * mats + 2 * absorb + 2.0 * row * (keys + T)
            expanded = 2.0 * keys * absorb + 2.0 * pairs * nh * (qk + a.v_head_dim)       # of the two forms of the attention the one with less to compute
            flops += 2.0 * T * mats + min(expanded, 2.0 * T * absorb + 2.0 * pairs * nh * (row + a.kv_lora_rank))
        elif spec.layer_is_linear(i):
            k, v = a.linear_k_heads, a.linear_v_heads
            mats = H * ((2 * k + 2 * v) * 128 + v + (v * 128 if a.linear_per_channel else v)) + H * v * 128
            nbytes += dense * mats + case["seqs"] * (4.0 * v * 128 * 128 + 6.0 * (2 * k + v) * 128)
            flops += 2.0 * T * (mats + 3 * v * 128 * 128)
        else:
            mats = H * (a.n_heads + 2 * a.n_kv_heads) * a.head_dim + H * a.n_heads * a.head_dim
            nbytes += dense * mats + 4.0 * a.n_kv_heads * a.head_dim * (keys + T)
            flops += 2.0 * T * mats + 4.0 * pairs * a.n_heads * a.head_dim
        if spec.is_moe_layer(i):
            shared = 3 * H * (m.shared_inter or 0)
            nbytes += 2.0 * m.n_experts * H + expert * used * 3 * H * m.intermediate + dense * shared
            flops += 2.0 * T * (m.n_experts * H + m.top_k * 3 * H * m.intermediate + shared)
        else:
            nbytes += dense * 3 * H * m.dense_intermediate
            flops += 2.0 * T * 3 * H * m.dense_intermediate
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """bf16 rounds what passes from product to product (`exact` is 0.005 to 0.008 off); where activations are then rounded to four bits, a
    last place decides between two of them (0.02 to 0.08 off), or between two experts of the next layer."""
    return {"rel": 0.02, "max": 0.5, "differ": 0.01} if case["model"] == "hybrid" else {"rel": 0.03, "max": 0.9, "differ": 0.01}


# ------------------------------------------------------------------ the same in 64 bits
E2M1 = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0)
F64 = torch.float64


def e4m3(bits):
    return bits.view(torch.float8_e4m3fn).to(F64)


def to_e2m1(x):
    """Nearest 4-bit value, ties to the even code, saturating."""
    grid = torch.tensor(E2M1, dtype=F64, device=x.device)
    edge = (grid[1:] + grid[:-1]) / 2
    mag = x.abs().clamp(max=6.0)
    code = torch.bucketize(mag, edge)                                          # a tie takes the lower code
    tie = (mag == edge[code.clamp(max=6)]) & (code < 7) & (code % 2 == 1)
    return grid[code + tie.long()] * x.sign()


def activations(x, fmt):
    """What the product's operand holds of x: the formats' own rounding, which is part of the model, but no other."""
    blocks = lambda n: x.reshape(*x.shape[:-1], -1, n)
    if fmt == "nvfp4":                                                         # 16 values share an E4M3 scale, over a constant of 1 / 64
        b = blocks(16)
        s = (b.abs().amax(-1, keepdim=True) * 64 / 6).clamp(max=448).to(torch.float8_e4m3fn).to(F64) / 64
        return (to_e2m1(torch.where(s > 0, b / s.clamp(min=1e-30), 0.0)) * s).reshape(x.shape)
    if fmt == "mxfp4":                                                         # 32 values share a power of two
        b = blocks(32)
        s = torch.exp2(torch.floor(torch.log2(b.abs().amax(-1, keepdim=True).clamp(min=2.0 ** -120))) - 2)
        return (to_e2m1(b / s) * s).reshape(x.shape)
    if fmt == "fp8_block128":
        b = blocks(128)
        s = b.abs().amax(-1, keepdim=True).clamp(min=1e-4) / 448
        return ((b / s).clamp(-448, 448).to(torch.float8_e4m3fn).to(F64) * s).reshape(x.shape)
    return x


def matrix(w, fmt, g=0):
    """Matrix g of a weight from its stored bytes: E2M1 pairs (low half first) with block scales in tiles of 128 rows x 4 scales,
    E4M3 with a scale per 128 x 128, or bf16."""
    data = w.data[g]
    if fmt == "bf16":
        return data.to(F64)
    if fmt == "fp8_block128":
        return e4m3(data) * w.sf[g].to(F64).repeat_interleave(128, 0)[:w.N].repeat_interleave(128, 1)[:, :w.K]
    n = 16 if fmt == "nvfp4" else 32
    sf = w.sf[g].reshape(-(-w.N // 128), -1, 32, 4, 4).permute(0, 3, 2, 1, 4).reshape(-(-w.N // 128) * 128, -1)[:w.N, :w.K // n]
    scale = e4m3(sf) * float(w.alpha[g]) * 64 if fmt == "nvfp4" else torch.exp2(sf.to(F64) - 127) * float(w.alpha[g])
    table = torch.tensor(E2M1 + tuple(-v for v in E2M1), dtype=F64, device=data.device)
    val = torch.stack([table[(data & 15).long()], table[(data >> 4).long()]], -1).reshape(w.N, w.K // n, n)
    return (val * scale[:, :, None]).reshape(w.N, w.K)


def norm(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def rotate(x, pos, theta, interleaved):
    d = x.shape[-1]
    ang = pos.to(F64)[:, None] / theta ** (torch.arange(0, d, 2, dtype=F64, device=x.device) / d)
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    a, b = (x[..., 0::2], x[..., 1::2]) if interleaved else (x[..., :d // 2], x[..., d // 2:])
    out = a * c - b * s, a * s + b * c
    return torch.stack(out, -1).reshape(x.shape) if interleaved else torch.cat(out, -1)


def attend(q, k, v, scale):
    """q [T, D] of the last T of the keys k [S, D], v [S, Dv]: causal."""
    T, S = q.shape[0], k.shape[0]
    hidden = torch.arange(S, device=q.device)[None] > torch.arange(S - T, S, device=q.device)[:, None]
    return torch.softmax((q @ k.T * scale).masked_fill(hidden, -math.inf), -1) @ v


def swiglu(x, gate, up, down, fmt):
    x = activations(x, fmt)
    return activations(torch.nn.functional.silu(x @ gate.T) * (x @ up.T), fmt) @ down.T


def delta_layer(a, lw, x, q_len, state, carry, eps):
    """Gated delta rule over every sequence's rows; returns the rows and the states and convolution inputs behind them."""
    Hk, Hv = a.linear_k_heads, a.linear_v_heads
    C = (2 * Hk + Hv) * 128
    z, ba, taps = x @ matrix(lw.lin_qkvz, "bf16").T, x @ matrix(lw.lin_ba, "bf16").T, lw.lin_conv.to(F64)
    beta, rate = torch.sigmoid(ba[:, :Hv]), lw.lin_a_log.to(F64).exp()
    soft = torch.nn.functional.softplus
    decay = torch.exp(-rate[:, None] * soft(ba[:, Hv:].reshape(-1, Hv, 128) + lw.lin_dt_bias.to(F64).reshape(Hv, 128))) if a.linear_per_channel else \
        torch.exp(-rate * soft(ba[:, Hv:] + lw.lin_dt_bias.to(F64)))[:, :, None].expand(-1, -1, 128)
    unit = lambda t: t / t.norm(dim=-1, keepdim=True).clamp(min=1e-6)
    rows, ends, hist = torch.empty(x.shape[0], Hv, 128, dtype=F64, device=x.device), [], []
    at, longest = [sum(q_len[:i]) for i in range(len(q_len))], max(q_len)
    q, k, v, d, b = (torch.zeros(longest, len(q_len), Hv, *t, dtype=F64, device=x.device) for t in ((128,), (128,), (128,), (128,), (1,)))
    d += 1
    for i, (s, n) in enumerate(zip(at, q_len)):                                # sequences side by side; a row behind a sequence's end changes nothing
        full = torch.cat([carry[i].to(F64), z[s:s + n, :C]])
        hist.append(full[-3:])
        y = torch.nn.functional.silu(sum(full[j:j + n] * taps[:, j] for j in range(4)))
        q[:n, i] = unit(y[:, :Hk * 128].reshape(n, Hk, 128)).repeat_interleave(Hv // Hk, 1) * 128 ** -0.5
        k[:n, i] = unit(y[:, Hk * 128:2 * Hk * 128].reshape(n, Hk, 128)).repeat_interleave(Hv // Hk, 1)
        v[:n, i], d[:n, i], b[:n, i, :, 0] = y[:, 2 * Hk * 128:].reshape(n, Hv, 128), decay[s:s + n], beta[s:s + n]
    S = state.to(F64).clone()
    o = torch.empty_like(v)
    for t in range(longest):
        S = S * d[t][..., None]
        u = (k[t][..., None, :] @ S)[..., 0, :]
        S = S + k[t][..., None] * (b[t] * (v[t] - u))[..., None, :]
        o[t] = (q[t][..., None, :] @ S)[..., 0, :]
    for i, (s, n) in enumerate(zip(at, q_len)):
        rows[s:s + n] = o[:n, i]
    gate = torch.nn.functional.silu(z[:, C:].reshape(-1, Hv, 128))
    return (norm(rows, eps) * gate).reshape(x.shape[0], -1), S, torch.stack(hist)


def exact(case, seed):
    spec = spec_of(case)
    a, m, eps = spec.attn, spec.moe, spec.rms_eps
    dense, expert = spec.quant.dense, spec.quant.experts
    inputs, pages = step_inputs(case, spec, seed)
    w = weights_of(spec, seed)
    q_len, kv_len, n_seq, decode = inputs["q_len"], inputs["kv_len"], case["seqs"], case["phase"] == "decode"
    on = lambda v: torch.tensor(v, device=DEV)
    pos, slots, seqs = on(inputs["positions"]), on(inputs["slot_map"]), list(zip(inputs["q_start"], q_len, kv_len, (p[0] * PAGE for p in inputs["page_table_rows"])))
    recurrent = case["model"] == "hybrid"
    state, carry = states(spec, n_seq, seed) if recurrent else (None, None)
    if recurrent and not decode:
        state, carry = torch.zeros_like(state), torch.zeros_like(carry)
    x = w.embed[on(inputs["tokens"])].to(F64)
    written, ends, hists = [], [], []
    for i, cache in enumerate(cache_rows(spec, pages * PAGE, seed)):
        lw = w.layer(i)
        xn = norm(x, eps)
        if a.kind == "mla":
            xq, mw, nh, nope = activations(xn, dense), lw.mla, a.n_heads, a.qk_nope_head_dim
            q = (activations(norm(xq @ matrix(mw.wq_a, dense).T, eps), dense) @ matrix(mw.wq_b, dense).T).reshape(-1, nh, nope + a.qk_rope_head_dim)
            q = torch.cat([q[..., :nope], rotate(q[..., nope:], pos, a.rope_theta, a.rope_interleaved)], -1)
            kv = xq @ matrix(mw.wkv_a, dense).T
            rank = a.kv_lora_rank
            new = torch.cat([norm(kv[:, :rank], eps), rotate(kv[:, None, rank:], pos, a.rope_theta, a.rope_interleaved)[:, 0]], -1)
            o = torch.empty(x.shape[0], nh, a.v_head_dim, dtype=F64, device=DEV)
            for s, n, total, base in seqs:
                row = torch.cat([cache[base:base + total - n].to(F64), new[s:s + n]])
                for h in range(nh):
                    k = torch.cat([row[:, :rank] @ mw.w_uk_t.data[h].to(F64), row[:, rank:]], -1)
                    o[s:s + n, h] = attend(q[s:s + n, h], k, row[:, :rank] @ mw.w_uv.data[h].to(F64).T, q.shape[-1] ** -0.5)
        elif spec.layer_is_linear(i):
            j = len(ends)
            o, end, hist = delta_layer(a, lw, xn, q_len, state[j], carry[j], eps)
            ends.append(end), hists.append(hist)
            new = None
        else:
            G, D = a.n_kv_heads, a.head_dim
            q, k, v = (activations(xn, dense) @ matrix(lw.wqkv, dense).T).reshape(-1, a.n_heads + 2 * G, D).split((a.n_heads, G, G), 1)
            q, k = (rotate(norm(t, eps), pos, a.rope_theta, a.rope_interleaved) for t in (q, k))
            new, per = torch.stack([k, v], 1), a.n_heads // G
            o = torch.empty_like(q)
            for s, n, total, base in seqs:
                row = torch.cat([cache[base:base + total - n].to(F64), new[s:s + n]])
                for h in range(a.n_heads):
                    o[s:s + n, h] = attend(q[s:s + n, h], row[:, 0, h // per], row[:, 1, h // per], D ** -0.5)
        x = x + activations(o.reshape(x.shape[0], -1), dense) @ matrix(lw.wo, dense).T
        if new is not None:
            written.append(new)
        xn = norm(x, eps)
        if not spec.is_moe_layer(i):
            x = x + swiglu(xn, *(matrix(t, dense) for t in (lw.ws_gate, lw.ws_up, lw.ws_down)), dense)
            continue
        score = xn @ matrix(lw.router, "bf16").T
        score = torch.softmax(score, -1) if m.scoring == "softmax" else torch.sigmoid(score)
        choice = score
        if m.n_group > 1:
            best = score.reshape(-1, m.n_group, m.n_experts // m.n_group).topk(2, -1).values.sum(-1).topk(m.topk_group, -1).indices
            keep = torch.zeros(x.shape[0], m.n_group, dtype=torch.bool, device=DEV).scatter_(1, best, True)
            choice = score.masked_fill(~keep.repeat_interleave(m.n_experts // m.n_group, 1), -math.inf)
        idx = choice.topk(m.top_k, -1).indices
        weight = score.gather(1, idx)
        weight = weight / weight.sum(-1, keepdim=True) * m.route_scale
        y = torch.zeros_like(x)
        for e in idx.unique().tolist():
            row, col = (idx == e).nonzero(as_tuple=True)
            y.index_add_(0, row, swiglu(xn[row], *(matrix(t, expert, e) for t in (lw.w_gate, lw.w_up, lw.w_down)), expert) * weight[row, col][:, None])
        if lw.ws_gate is not None:
            y = y + swiglu(xn, *(matrix(t, dense) for t in (lw.ws_gate, lw.ws_up, lw.ws_down)), dense)
        x = x + y
    logits = norm(x[on(inputs["logit_rows"])], eps) @ matrix(w.lm_head, "bf16").T
    rows = torch.stack(written)
    out = {"logits": logits, "tokens": None, "cache": [rows[0, s:s + n] if recurrent else rows[:, s:s + n] for s, n, _, _ in seqs]}
    if recurrent and not decode:
        out["recurrent"], out["conv"] = torch.stack(ends), torch.stack(hists)
    return out
