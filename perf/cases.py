"""Workloads of the serving engine: what one step of it does, in the sizes it is used at.

Every case is a step of ``LLM(...).engine`` on a random-init model of a named shape with its layer count cut (embedding and head stay
whole), planned and run as the scheduler and the offline benchmark do it:

* ``decode``   one new token for each of ``batch`` sequences, logits for the sampler;
* ``verify``   ``rows`` rows for each of ``batch`` sequences (the last token and a chain of drafts), greedy tokens and hidden rows;
* ``prefill``  ``batch`` whole prompts, logits of their last rows;
* ``mixed``    a step of the interleaving scheduler: ``batch`` decode rows beside one chunk of ``rows`` prompt tokens that continues a
  prompt of which ``ctx`` tokens are in the cache.

Contexts and prompts are ragged: sequence i has ``ctx`` (or ``rows``) tokens less up to the share ``spread``.  Contexts hold random FP8
keys and values of unit variance (keys are normed per head, and a value row is a product of normed rows with N(0, 0.02) weights).
"""
from __future__ import annotations

import math

import torch

from blaze_b200.config import named_config
from blaze_b200.llm import LLM

PAGE = 16
# layers of each shape: enough for the layers to outweigh the head, few enough to keep three models of a case on the card.  The hybrid
# has one attention layer after three recurrent ones
LAYERS = {"qwen3-8b": 12, "qwen3-32b": 4, "qwen3-30b-a3b": 6, "qwen3-next-80b-a3b": 4}
# standard deviation of the embedding: a trained model's residual outweighs what its layers add to it, and so do these rows (a layer of the
# shape with the widest feed-forwards adds about 2 per element).  On N(0, 0.02) rows random layers would amplify every rounding instead
EMBED_STD = {"qwen3-8b": 32.0, "qwen3-32b": 16.0, "qwen3-30b-a3b": 8.0, "qwen3-next-80b-a3b": 8.0}
BITS = {"nvfp4": 4.5, "mxfp8": 8.25, "fp8_block": 8.0, "bf16": 16.0}


def _case(name, model, weights, kind, batch, ctx, rows, spread=0.0):
    c = {"model": model, "weights": weights, "kind": kind, "batch": batch, "ctx": ctx, "rows": rows, "spread": spread}
    return {"name": name, **c} if name else c


def listed():
    return [
        # one user at a time: every step waits for its token
        _case("8b nvfp4 decode 1", "qwen3-8b", "nvfp4", "decode", 1, 777, 1),
        # the steady state of the throughput benchmark: 256 sequences between 1024 and 1280 tokens
        _case("8b nvfp4 decode 256", "qwen3-8b", "nvfp4", "decode", 256, 1280, 1, 0.2),
        # a few long conversations
        _case("8b nvfp4 decode 6 long", "qwen3-8b", "nvfp4", "decode", 6, 16001, 1, 0.6),
        # speculative decoding: chains of four drafts
        _case("8b nvfp4 verify 16x5", "qwen3-8b", "nvfp4", "verify", 16, 2100, 5, 0.5),
        # the benchmark's prompt steps: eight prompts of 1024 tokens
        _case("8b nvfp4 prefill 8x1024", "qwen3-8b", "nvfp4", "prefill", 8, 0, 1024),
        # decoding goes on while the rest of a prompt comes in
        _case("8b nvfp4 mixed 48+777", "qwen3-8b", "nvfp4", "mixed", 48, 1531, 777, 0.7),
        # an unquantised checkpoint: a few chat prompts of odd lengths
        _case("8b bf16 prefill 3x701", "qwen3-8b", "bf16", "prefill", 3, 0, 701, 0.6),
        # a checkpoint with FP8 block scales, a middling batch
        _case("32b fp8 decode 64", "qwen3-32b", "fp8_block", "decode", 64, 1024, 1, 0.5),
        # experts: the benchmark's decode batch, and a step of prompts
        _case("30b-a3b nvfp4 decode 256", "qwen3-30b-a3b", "nvfp4", "decode", 256, 1280, 1, 0.2),
        _case("30b-a3b nvfp4 prefill 4x1024", "qwen3-30b-a3b", "nvfp4", "prefill", 4, 0, 1024),
        # recurrent layers and many experts: a long prompt, and a small batch
        _case("next-80b mxfp8 prefill 4096", "qwen3-next-80b-a3b", "mxfp8", "prefill", 1, 0, 4096),
        _case("next-80b mxfp8 decode 16", "qwen3-next-80b-a3b", "mxfp8", "decode", 16, 4150, 1, 0.3),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    model, weights = rng.choice([("qwen3-8b", "nvfp4"), ("qwen3-8b", "nvfp4"), ("qwen3-8b", "bf16"), ("qwen3-32b", "fp8_block"),
                                 ("qwen3-30b-a3b", "nvfp4"), ("qwen3-next-80b-a3b", "mxfp8")])
    hybrid = model == "qwen3-next-80b-a3b"
    kind = rng.choice(["decode", "prefill"] if hybrid else ["decode", "decode", "verify", "prefill", "prefill", "mixed"])
    spread = round(rng.uniform(0.0, 0.8), 2)
    if kind == "prefill":
        batch = log(1, 16)
        return _case(None, model, weights, kind, batch, 0, max(log(16, 4096 if model != "qwen3-8b" else 8192) // batch, 5), spread)
    batch = log(1, {"verify": 32, "mixed": 128}.get(kind, 64 if hybrid else 256))
    ctx = log(20, min(16384, (8192 if hybrid else 262144) * (8 if hybrid else 1) // batch))
    return _case(None, model, weights, kind, batch, ctx, {"decode": 1, "verify": rng.randint(2, 8), "mixed": log(20, 2048)}[kind], spread)


def _ragged(n, top, spread):
    """``n`` lengths up to ``top``, the first of them ``top`` itself."""
    return [max(top - int(top * spread * (i * 0.6180339887 % 1.0)), 1) for i in range(n)]


def _lengths(case):
    """(tokens in the cache, new tokens) of each sequence of the step."""
    n = case["batch"]
    if case["kind"] == "prefill":
        return [(0, k) for k in _ragged(n, case["rows"], case["spread"])]
    if case["kind"] == "mixed":
        return [(k, 1) for k in _ragged(n, case["ctx"], case["spread"])] + [(case["ctx"], case["rows"])]
    return [(k, case["rows"]) for k in _ragged(n, case["ctx"], case["spread"])]


def _config(case):
    cfg = named_config(case["model"])
    cfg.num_layers = LAYERS[case["model"]]
    cfg.layer_types = cfg.layer_types[:cfg.num_layers]
    return cfg


def _inputs(case, seed):
    """The engine with its sequences open and their contexts filled, and each step's (sequence, new tokens, rows with logits)."""
    cfg, lens = _config(case), _lengths(case)
    need = [-(-(c + n) // PAGE) for c, n in lens]
    longest = (max(c + n for c, n in lens) + 1023) // 1024 * 1024
    llm = LLM(cfg, weight_format=case["weights"], device="cuda", kv_cache_dtype="fp8", kv_tokens=(sum(need) + 8) * PAGE, max_seqs=len(lens),
              max_model_len=longest, chunk=8192, seed=seed)
    llm.model.embed.mul_(EMBED_STD[case["model"]] / 0.02)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    host = torch.Generator().manual_seed(seed)
    rows = [torch.randint(0, cfg.vocab_size, (n,), generator=host).tolist() for _, n in lens]
    want = {"verify": case["rows"]}.get(case["kind"], 1)
    state = {"kind": case["kind"], "llm": llm, "engine": llm.engine, "rows": rows, "want": want, "lens": lens,
             "seqs": [llm.engine.open_from() for _ in lens]}
    for s, (c, n) in zip(state["seqs"], lens):
        llm.engine.reserve(s, c + n)
        s.length = c
    return state, gen


def _fill(state, gen):
    kv = state["engine"].kv
    for pool in kv.kv.values():
        flat = pool.view(-1)
        for a in range(0, flat.numel(), 1 << 28):
            part = flat[a:a + (1 << 28)]
            part.copy_(torch.randn(part.shape, generator=gen, device="cuda", dtype=torch.float32).to(torch.float8_e4m3fn).view(torch.uint8))
    for t in [*kv.conv_state.values(), *kv.rec_state.values()]:
        t.normal_(0.0, 0.3 if t.dim() == 3 else 0.05, generator=gen)


def prepare(case, seed):
    state, gen = _inputs(case, seed)
    for _ in range(2):          # a server's warm-up: weights in the kernels' layouts, and the captured steps of this shape
        run(state)
    _fill(state, gen)
    return state


def run(state):
    eng = state["engine"]
    for s, (c, _) in zip(state["seqs"], state["lens"]):
        s.length = c            # the step is taken again from the same place
    chunks = eng.plan([(s, r, state["want"]) for s, r in zip(state["seqs"], state["rows"])])
    kv = eng.kv
    cache = {"kv": [p.view(torch.float8_e4m3fn) for p in kv.kv.values()], "state": list(kv.rec_state.values()), "conv": list(kv.conv_state.values())}
    if state["kind"] == "verify":
        tokens, hidden = eng.forward(chunks, "greedy_hidden")
        return {"tokens": tokens, "hidden": hidden, **cache}
    return {"logits": eng.forward(chunks, "logits"), **cache}


# ---------------------------------------------------------------------------------------------- work
def _layer_params(cfg, kind):
    """(weights every row is multiplied by, weights of one expert, weights kept in 16 bits) of a layer."""
    H, D = cfg.hidden_size, cfg.head_dim
    if kind == "full_attention":
        mix = H * D * (cfg.num_heads * (3 if cfg.attn_output_gate else 2) + 2 * cfg.num_kv_heads)
    else:
        hk, hv = cfg.linear_num_key_heads * cfg.linear_key_head_dim, cfg.linear_num_value_heads * cfg.linear_value_head_dim
        mix = H * (2 * hk + 3 * hv + 2 * cfg.linear_num_value_heads)
    if not cfg.is_moe:
        return mix + 3 * H * cfg.intermediate_size, 0, 0
    return mix + 3 * H * cfg.shared_expert_intermediate_size, 3 * H * cfg.moe_intermediate_size, H * (cfg.num_experts + 1)


def work(case):
    cfg, lens = _config(case), _lengths(case)
    T = sum(n for _, n in lens)
    R = sum(n for _, n in lens) if case["kind"] == "verify" else len(lens)
    wb = BITS[case["weights"]] / 8
    H, V = cfg.hidden_size, cfg.vocab_size
    pairs = sum(n * c + n * (n + 1) // 2 for c, n in lens)
    total_bytes = V * H * 2 + T * H * 2 + (R * V * 4 if case["kind"] != "verify" else R * H * 2 + R * 8)
    flops = 2.0 * R * V * H
    for i in range(cfg.num_layers):
        kind = cfg.layer_type(i)
        every, one, dense = _layer_params(cfg, kind)
        total_bytes += every * wb + dense * 2
        flops += 2.0 * T * (every + dense)
        if one:
            k, E = cfg.num_experts_per_tok, cfg.num_experts
            total_bytes += one * wb * E * (1.0 - (1.0 - k / E) ** T)
            flops += 2.0 * T * k * one
        if kind == "full_attention":
            total_bytes += sum(c + n for c, n in lens) * 2 * cfg.num_kv_heads * cfg.head_dim
            flops += 4.0 * pairs * cfg.num_heads * cfg.head_dim
        else:
            hv, dk, dv = cfg.linear_num_value_heads, cfg.linear_key_head_dim, cfg.linear_value_head_dim
            total_bytes += len(lens) * hv * dk * dv * 4 * (1 if case["kind"] == "prefill" else 2)      # a fresh state is not read
            flops += 6.0 * T * hv * dk * dv
    return {"bytes": total_bytes, "flops": flops}


def tolerance(case):
    # about four times what a step differs from the same in 64 bits.  An activation near the edge between two codes of the weight's
    # format moves a whole code when a sum takes another order: 4-bit codes show that most, and a greedy token moves where two logits
    # lie that close (every fifth of the verified rows, at a distance of 0.04 between the logits of random layers)
    rel = {("qwen3-8b", "nvfp4"): 0.2, ("qwen3-8b", "bf16"): 0.035, ("qwen3-32b", "fp8_block"): 0.1, ("qwen3-30b-a3b", "nvfp4"): 0.03,
           ("qwen3-next-80b-a3b", "mxfp8"): 0.03}[case["model"], case["weights"]]
    return {"rel": rel, "differ": 0.3} if case["kind"] == "verify" else {"rel": rel}


# ---------------------------------------------------------------------------------------------- 64 bits
E2M1 = [0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0]


def _weight(lin):
    """A stored weight ``[N, K]`` as numbers."""
    N, K, fmt = lin.N, lin.K, lin.fmt.value
    if fmt == "dense":
        return lin.w.double()
    if fmt == "nvfp4":
        lut = torch.tensor(E2M1 + [-v for v in E2M1], dtype=torch.float64, device=lin.w.device)
        w = torch.stack([lut[(lin.w & 15).int()], lut[(lin.w >> 4).int()]], -1).view(N, K // 16, 16)
        return (w * lin.sf.double()[..., None]).view(N, K) * lin.alpha.double()[:, None]
    if fmt == "mxfp8":
        return (lin.w.double().view(N, K // 32, 32) * torch.exp2(lin.sf.double() - 127)[..., None]).view(N, K)
    s = lin.sf.double().repeat_interleave(128, 0)[:N].repeat_interleave(128, 1)[:, :K]
    return lin.w.double() * s


def _e4m3(x):
    return x.clamp(-448, 448).float().to(torch.float8_e4m3fn).double()


def _rounded(x, lin):
    """Activations as the format of ``lin`` holds them: scales of a row's blocks, codes to the nearest."""
    T, K, fmt = *x.shape, lin.fmt.value
    if not lin.act_quant or fmt == "dense":
        return x
    if fmt == "nvfp4":
        g = (x.abs().amax(1) / (6.0 * 448.0)).clamp_min(1e-30).view(-1, 1, 1)
        b = x.view(T, K // 16, 16)
        s = _e4m3(b.abs().amax(2, keepdim=True) / 6.0 / g) * g
        grid = torch.tensor(E2M1, dtype=torch.float64, device=x.device)
        a = torch.where(s > 0, b.abs() / s.clamp_min(1e-300), 0.0)
        return (grid[torch.bucketize(a, (grid[1:] + grid[:-1]) / 2)] * s * b.sign()).view(T, K)
    if fmt == "mxfp8":
        b = x.view(T, K // 32, 32)
        s = torch.exp2(torch.ceil(torch.log2(b.abs().amax(2, keepdim=True).clamp_min(2.0 ** -127) / 448.0)).clamp(-127, 127))
    else:
        b = x.view(T, K // 128, 128)
        s = (b.abs().amax(2, keepdim=True) / 448.0).clamp_min(1e-12)
    return (_e4m3(b / s) * s).view(T, K)


def _mul(lin, x):
    return _rounded(x, lin) @ _weight(lin).t()


def _norm(x, w, cfg, centred):
    w = w.double() + 1 if centred else w.double()
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + cfg.rms_norm_eps) * w


def _turn(x, pos, cfg):
    n = cfg.rotary_dim // 2
    f = torch.tensor([cfg.rope.theta ** (-i / n) for i in range(n)], dtype=torch.float64, device=x.device)
    a = (pos.double()[:, None] * f)[:, None]
    c, s = torch.cos(a), torch.sin(a)
    u, v = x[..., :n], x[..., n:2 * n]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * n:]], -1)


def _cached(pool, pages, n, D):
    """The first ``n`` keys and values ``[heads, n, D]`` of pages in the kernels' layout."""
    b = pool[pages].view(torch.float8_e4m3fn)
    k = b[:, :, 0].reshape(len(pages), -1, 2, D // 16, 8, 16).double().permute(1, 0, 2, 4, 3, 5)
    v = b[:, :, 1].reshape(len(pages), -1, D, 16).double().permute(1, 0, 3, 2)
    return [t.reshape(t.shape[0], -1, D)[:, :n] for t in (k, v)]


def _attention(A, h, cfg, lens, pos, old):
    D, nh, nk, T = cfg.head_dim, A.heads, A.kv_heads, h.shape[0]
    qkv = _mul(A.qkv, h)
    gated = cfg.attn_output_gate
    q, k, v = qkv.split([nh * D * (2 if gated else 1), nk * D, nk * D], 1)
    q = q.view(T, nh, -1)
    q, gate = (q[..., :D], q[..., D:]) if gated else (q, None)
    q = _turn(_norm(q, A.q_norm, cfg, cfg.zero_centered_norm), pos, cfg)
    k = _e4m3(_turn(_norm(k.view(T, nk, D), A.k_norm, cfg, cfg.zero_centered_norm), pos, cfg))
    v = _e4m3(v.view(T, nk, D))
    o, r = torch.empty(T, nh, D, dtype=torch.float64, device=h.device), 0
    for i, (c, n) in enumerate(lens):
        kk, vv = k[r:r + n].transpose(0, 1), v[r:r + n].transpose(0, 1)
        if c:
            ck, cv = old(i)
            kk, vv = torch.cat([ck, kk], 1), torch.cat([cv, vv], 1)
        later = torch.arange(c + n, device=h.device) > torch.arange(c, c + n, device=h.device)[:, None]
        qq = q[r:r + n].view(n, nk, nh // nk, D)
        for g in range(nk):
            s = torch.einsum("qhd,kd->hqk", qq[:, g], kk[g]) * D ** -0.5
            o[r:r + n].view(n, nk, -1, D)[:, g] = torch.einsum("hqk,kd->qhd", s.masked_fill(later, -math.inf).softmax(-1), vv[g])
        r += n
    if gate is not None:
        o = o * gate.sigmoid()
    return _mul(A.o, o.reshape(T, nh * D))


def _recurrence(G, h, cfg, lens, states, convs):
    dk, dv, hk, hv = cfg.linear_key_head_dim, cfg.linear_value_head_dim, G.k_heads, G.v_heads
    qkv, z, b, a = _mul(G.in_proj, h).split([2 * hk * dk + hv * dv, hv * dv, hv, hv], 1)
    w, taps = G.conv_w.double(), G.conv_w.shape[1]
    o, r, after = [], 0, []
    for i, (c, n) in enumerate(lens):
        before = convs[i].double().t() if c else qkv.new_zeros(taps - 1, qkv.shape[1])
        S = states[i].double().clone() if c else qkv.new_zeros(hv, dk, dv)
        u = torch.cat([before, qkv[r:r + n]])
        u = torch.nn.functional.silu(sum(u[j:j + n] * w[:, j] for j in range(taps)))
        q, k, v = u.split([hk * dk, hk * dk, hv * dv], 1)
        q, k = [torch.nn.functional.normalize(t.view(n, hk, dk), dim=-1, eps=1e-6).repeat_interleave(hv // hk, 1) for t in (q, k)]
        q, v = q * dk ** -0.5, v.view(n, hv, dv)
        keep = torch.exp(-G.A_log.double().exp() * torch.nn.functional.softplus(a[r:r + n] + G.dt_bias.double()))[..., None, None]
        beta = b[r:r + n].sigmoid()[..., None]
        for t in range(n):
            S = S * keep[t]
            S = torch.baddbmm(S, k[t][:, :, None], ((v[t] - (k[t][:, None] @ S)[:, 0]) * beta[t])[:, None])
            o.append((q[t][:, None] @ S)[:, 0])
        after.append(S)
        r += n
    o = torch.stack(o)
    y = o * torch.rsqrt(o.pow(2).mean(-1, keepdim=True) + cfg.rms_norm_eps) * G.norm_w.double() * torch.nn.functional.silu(z.reshape(o.shape))
    return _mul(G.out_proj, y.reshape(len(o), -1)), after


def _glu(up, down, x):
    g, u = _mul(up, x).chunk(2, 1)
    return _mul(down, torch.nn.functional.silu(g) * u)


def _feed(M, x, cfg):
    if not cfg.is_moe:
        return _glu(M.gate_up, M.down, x)
    w, ids = _mul(M.router, x).softmax(-1).topk(M.top_k, -1)
    w = w / w.sum(-1, keepdim=True) if M.renorm else w
    y = torch.zeros_like(x)
    for e in range(cfg.num_experts):
        t, j = (ids == e).nonzero(as_tuple=True)
        if len(t):
            y.index_add_(0, t, _glu(M.experts.gate_up[e], M.experts.down[e], x[t]) * w[t, j, None])
    if M.shared is not None:
        y = y + _glu(M.shared.gate_up, M.shared.down, x) * _mul(M.shared_gate, x).sigmoid()
    return y


def exact(case, seed):
    """The step in 64 bits, with weights, cached keys and values and the inputs of products in the formats that hold them."""
    state, gen = _inputs(case, seed)
    _fill(state, gen)
    model, kv, cfg, lens = state["llm"].model, state["engine"].kv, state["llm"].model.cfg, state["lens"]
    dev = model.embed.device
    pos = torch.cat([torch.arange(c, c + n, device=dev) for c, n in lens])
    x = model.embed[torch.tensor(sum(state["rows"], []), device=dev)].double()
    new_states = []
    for i, L in enumerate(model.layers):
        h = _norm(x, L.input_norm, cfg, cfg.zero_centered_norm)
        if L.attn is not None:
            def old(b, i=i):
                s = state["seqs"][b]
                return _cached(kv.kv[i], torch.tensor(s.pages[:-(-s.length // PAGE)], device=dev), s.length, cfg.head_dim)
            x = x + _attention(L.attn, h, cfg, lens, pos, old)
        else:
            rows = [s.row for s in state["seqs"]]
            y, after = _recurrence(L.gdn, h, cfg, lens, kv.rec_state[i][rows], kv.conv_state[i][rows])
            x = x + y
            new_states.append(kv.rec_state[i].double().index_copy(0, torch.tensor(rows, device=dev), torch.stack(after)))
        x = x + _feed(L.mlp, _norm(x, L.post_norm, cfg, cfg.zero_centered_norm), cfg)
    none = [None] * len(kv.kv)
    if case["kind"] == "verify":
        return {"tokens": None, "hidden": x, "kv": none, "state": new_states, "conv": []}
    last = torch.tensor([n for _, n in lens], device=dev).cumsum(0) - 1
    logits = _mul(model.lm_head, _norm(x[last], model.final_norm, cfg, cfg.zero_centered_norm))
    return {"logits": logits, "kv": none, "state": new_states, "conv": [None] * len(kv.conv_state)}
