"""Kernel forms chosen by a step's sizes, at the sizes where one takes over from another, against the references of the general forms."""
import pytest
import torch

from blaze_b200 import quant
from blaze_b200.batch import SeqChunk, build_batch
from blaze_b200.config import ModelConfig, RopeConfig, inv_freq
from blaze_b200.kv import KVCache
from blaze_b200.linear import Linear
from blaze_b200.ops import ref
from blaze_b200.quant import Format
from test_gpu_kernels import _A, _attention_case, _experts, ops       # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30)).item()


def test_logits_steps_replay_a_captured_step():
    """A decode step with logits: the first of a batch size runs launch by launch, the others replay it; what a step handed out stays as
    it was when the next one runs."""
    from blaze_b200.llm import LLM
    cfg = ModelConfig(vocab_size=2048, hidden_size=512, num_layers=2, num_heads=8, num_kv_heads=2, head_dim=128, intermediate_size=1024,
                      rope=RopeConfig(theta=1e6))
    cfg.layer_types = ["full_attention"] * 2
    eng = LLM(cfg, weight_format="nvfp4", max_seqs=8, max_model_len=256, seed=4).engine
    gen = torch.Generator().manual_seed(1)
    seqs = [eng.open_from() for _ in range(3)]
    eng.forward(eng.plan([(s, torch.randint(0, 2048, (n,), generator=gen).tolist(), 0) for s, n in zip(seqs, (40, 7, 100))]), "none")
    base, outs = [s.length for s in seqs], []
    for tok in (5, 5, 5, 900):
        for s, n in zip(seqs, base):
            s.length = n
        outs.append(eng.forward(eng.plan([(s, [tok], 1) for s in seqs]), "logits"))
        kept = outs[-1].clone() if len(outs) == 3 else kept if len(outs) > 3 else None
    assert any(k[:2] == ("logits", 3) for k in eng._graphs) and outs[0].shape == (3, 2048) and outs[0].dtype == torch.float32
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[1], outs[2]) and not torch.equal(outs[2], outs[3]) and torch.equal(outs[2], kept)
    some = eng.forward(eng.plan([(seqs[0], [1], 1), (seqs[1], [1], 0)]), "logits")
    assert some.shape[0] == 1                      # rows without logits: not a step of that kind


def _steps_engine(kind):
    """A small model of a kind with 40 sequences open, whose contexts (60 to 1400 tokens) are in the cache."""
    from blaze_b200.config import named_config
    from blaze_b200.llm import LLM
    if kind.startswith("tiny-"):
        cfg, fmt = named_config(kind), "bf16"
        for spec in cfg.layer_specs:               # contexts of one key tile would not be cut at all
            if spec.attn is not None and spec.attn.window:
                spec.attn.window = 0
    else:
        fmt = "mxfp8" if kind == "recurrent" else "nvfp4"
        cfg = ModelConfig(vocab_size=2048, hidden_size=512, num_layers=2, num_heads=8, num_kv_heads={"dense": 8, "experts": 4, "recurrent": 1}[kind],
                          head_dim=256 if kind == "recurrent" else 128, intermediate_size=1024, rope=RopeConfig(theta=1e6))
        cfg.layer_types = ["full_attention"] * 2
    if kind == "experts":
        cfg.num_experts, cfg.num_experts_per_tok, cfg.moe_intermediate_size = 16, 4, 256
    if kind == "recurrent":
        cfg.layer_types = ["linear_attention", "full_attention"]
        cfg.linear_num_key_heads, cfg.linear_num_value_heads, cfg.linear_key_head_dim, cfg.linear_value_head_dim = 2, 4, 128, 128
        cfg.linear_conv_kernel_dim = 4
    eng = LLM(cfg, weight_format=fmt, max_seqs=40, max_model_len=4096, kv_tokens=41 * 1536, seed=4).engine
    gen = torch.Generator().manual_seed(1)
    ctxs = [60 + (i * 743) % 1341 for i in range(40)]
    seqs = [eng.open_from() for _ in ctxs]
    for i in range(0, 40, 8):
        eng.forward(eng.plan([(s, torch.randint(0, 1000, (c,), generator=gen).tolist(), 0) for s, c in zip(seqs[i:i + 8], ctxs[i:i + 8])]), "none")
    kv = eng.kv
    states = [t for d in (kv.conv_state, kv.rec_state, kv.qkv_state, kv.input_state) for t in d.values()]
    before = [t.clone() for t in states]

    def step(n, graphs):
        eng.ecfg.use_graphs = graphs
        for t, b in zip(states, before):
            t.copy_(b)
        for s, c in zip(seqs, ctxs):
            s.length = c
        out = eng.forward(eng.plan([(s, [7 * i + 1], 1) for i, s in enumerate(seqs[:n])]), "logits")
        return [out.clone()] + [t.clone() for t in states]
    return eng, step


@pytest.mark.parametrize("kind", ["dense", "experts", "recurrent", "tiny-sevevik", "tiny-niletar", "tiny-rapisun", "tiny-medodra"])
def test_logits_do_not_depend_on_how_a_step_was_launched(kind):
    """Padded and whole batches, replayed (where the design's steps are) and launched one by one: the same bits, and the same states.
    Keys are cut as the sequences' number asks for, not as the padded batch's would, and batches that differ in that alone have captured
    steps of their own."""
    eng, step = _steps_engine(kind)
    bucket, splits = eng._sampled_bucket, eng._key_splits
    padded = [n for n in range(17, 41) if bucket(n) != n]
    apart = [n for n in padded if splits(n) != splits(bucket(n))]
    shared = [n for n in range(17, 40) if (bucket(n), splits(n)) == (bucket(n + 1), splits(n + 1))][0]
    for n in sorted({1, 3, padded[0], *apart, 37, shared, shared + 1}):
        want = step(n, False)
        for _ in range(3):
            assert all(torch.equal(a, b) for a, b in zip(step(n, True), want)), n
    if not kind.startswith("tiny-"):
        assert apart and sum(k == ("logits", bucket(shared), splits(shared)) for k in eng._graphs) == 1


def test_captured_steps_are_there_from_the_start():
    """With ``warm_graphs`` no decode step of any batch size captures anything; the steps with logits share their memory, which holds
    when they are replayed in any order."""
    eng, step = _steps_engine("dense")
    for s in list(eng.seqs.values())[24:]:
        eng.close(s)                               # (16 rows for the scratch sequences)
    want = {n: step(n, False) for n in (16, 3, 11)}
    eng.ecfg.use_graphs = True
    made = eng.capture_decode_graphs()
    keys = set(eng._graphs)
    assert made == len(keys) and keys == {("decode", b) for b in (1, 2, 4, 8, 16)} | {eng._sampled_key(n) for n in range(1, 17)}
    assert len({eng._graphs[k].graph.pool() for k in keys if k[0] == "logits"}) == 1
    for n in (3, 16, 11, 3, 11, 16):
        assert all(torch.equal(a, b) for a, b in zip(step(n, True), want[n])), n
    assert set(eng._graphs) == keys


def test_capture_while_garbage_holds_a_captured_step():
    """A captured step that only a reference cycle keeps is not given back in the middle of another step's capture."""
    import gc
    eng, step = _steps_engine("dense")
    want = step(3, False)
    run, old, lists = eng._run, gc.get_threshold(), []

    def collecting(batch, mode, hidden_in=None):
        gc.set_threshold(1, 1, 1)
        lists.extend([[i] for i in range(4)])      # a collection would come now
        try:
            return run(batch, mode, hidden_in)
        finally:
            gc.set_threshold(1 << 30)
    gc.collect()
    gc.set_threshold(1 << 30)                      # none until the steps run
    try:
        g, x = torch.cuda.CUDAGraph(), torch.zeros(8, device=DEV)
        with torch.cuda.graph(g):
            x += 1
        cycle = [g]
        cycle.append(cycle)
        step(3, True)                              # launched one by one
        del g, cycle
        eng._run = collecting
        got = step(3, True)                        # captured
    finally:
        eng._run = run
        gc.set_threshold(*old)
    assert ("logits", 3, eng._key_splits(3)) in eng._graphs and gc.isenabled()
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("Hq,Hkv,ctxs,q", [
    (32, 8, [1], 1), (32, 8, [129], 1), (32, 8, [5000, 3, 128, 1291], 1),          # fewer items than CTAs: runs of tiles
    (16, 2, [2600, 40, 1025], 1), (32, 4, [700], 2), (32, 8, [900, 260], 5), (32, 4, [1500, 64], 8),      # 8, 16, 20 and 64 rows
    (8, 8, [129, 1500], 1), (16, 8, [700, 40], 1), (24, 8, [900, 260], 3), (40, 8, [1291], 2), (12, 4, [513, 77], 4),      # 1, 2, 9, 10 and 12 rows
    (32, 8, [33 + 7 * i for i in range(40)], 1), (24, 8, [33 + 7 * i for i in range(40)], 3), (64, 8, [200 + i for i in range(19)], 3),                 # more items than CTAs
])
def test_decode_attention_runs_of_tiles(ops, Hq, Hkv, ctxs, q):      # noqa: F811
    got, want = _attention_case(ops, Hq, Hkv, ctxs, [q] * len(ctxs))
    assert torch.isfinite(got.float()).all() and _rel(got, want) < 0.06
    err = (got.float() - want.float()).flatten(1).norm(dim=1) / want.float().flatten(1).norm(dim=1)
    assert err.max().item() < 0.15                 # row by row: an item that got a wrong piece is off by its size


def _raw_decode(ops, kv, q, out, ctxs, Hq, Hkv, splits, po, pm):      # noqa: F811
    """``blz_attn_decode_tree`` for one row per sequence, as another program calls it."""
    from blaze_b200.ops.cuda_ops import VP, _ptr
    B, D, pool = len(ctxs), 128, kv.kv[0]
    slots, q_start, ctx = [torch.tensor(v, dtype=torch.int32, device=DEV) for v in (range(B), range(B + 1), ctxs)]
    rc = ops.lib.blz_attn_decode_tree(_ptr(q), _ptr(out), _ptr(pool), _ptr(kv.block_table), _ptr(slots), _ptr(q_start), _ptr(ctx), B, Hq, Hkv, D,
                                      kv.block_table.stride(0), pool.stride(0), pool.stride(1), D ** -0.5, 1.0, 1.0, 16, 1, 1, Hq // Hkv, splits,
                                      _ptr(po), _ptr(pm), 0, VP(0), VP(0), VP(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert rc == 0 and ops.take_status() == 0


def _decode_inputs(Hq, Hkv, ctxs):
    """A cache with the sequences' keys and values (finite codes) and one query row each."""
    cfg = ModelConfig(hidden_size=Hq * 128, num_heads=Hq, num_kv_heads=Hkv, head_dim=128, num_layers=1, rope=RopeConfig(theta=1e6))
    cfg.layer_types = ["full_attention"]
    g = torch.Generator(device=DEV).manual_seed(3)
    pages = (max(ctxs) + 15) // 16 + 1
    kv = KVCache(cfg, 1 + len(ctxs) * pages, len(ctxs), pages, "fp8", DEV, "umma")
    for b in range(len(ctxs)):
        kv.set_pages(b, list(range(1 + b * pages, 1 + (b + 1) * pages)))
    kv.flush()
    kv.kv[0][1:].copy_(torch.randn(kv.kv[0][1:].shape, generator=g, device=DEV).to(torch.float8_e4m3fn).view(torch.uint8))
    return kv, torch.randn(len(ctxs), Hq, 128, generator=g, device=DEV).bfloat16()


def test_decode_attention_leaves_rows_without_a_key_alone(ops):      # noqa: F811
    """A sequence whose row sees no key, without splits and without scratch: nothing is written for it, nor anywhere else."""
    kv, q = _decode_inputs(8, 2, [300, 16, 1500])
    out, want = [torch.full_like(q, 7.0) for _ in range(2)]
    _raw_decode(ops, kv, q, out, [300, 0, 1500], 8, 2, 1, None, None)
    _raw_decode(ops, kv, q, want, [300, 16, 1500], 8, 2, 1, None, None)
    assert (out[1] == 7).all() and torch.equal(out[[0, 2]], want[[0, 2]]) and not (want == 7).all()


@pytest.mark.parametrize("shift", [1, 2, 3])
def test_decode_attention_merges_runs_at_any_address(ops, shift):      # noqa: F811
    """Scratch and output that lie on their elements' size only."""
    ctxs, splits = [700, 16, 1500], 4
    kv, q = _decode_inputs(8, 2, ctxs)
    n, outs = len(ctxs) * 2 * splits * 16, []
    for s in (0, shift):
        po, pm = [torch.empty(m + s, dtype=torch.float32, device=DEV)[s:] for m in (n * 128, n * 2)]
        out = torch.zeros(q.numel() + s, dtype=torch.bfloat16, device=DEV)[s:].view_as(q)
        _raw_decode(ops, kv, q, out, ctxs, 8, 2, splits, po, pm)
        outs.append(out)
    assert torch.equal(*outs) and outs[0].float().abs().amax(-1).min().item() > 0


def test_decode_attention_runs_that_are_not_a_number(ops):      # noqa: F811
    """Keys that are not a number spoil the run that they lie in: the merged row is that of the other runs."""
    ctxs, splits, Hkv = [512], 4, 2
    kv, q = _decode_inputs(8, Hkv, ctxs)
    n = Hkv * splits * 16
    po, pm = [torch.empty(m, dtype=torch.float32, device=DEV) for m in (n * 128, n * 2)]
    got = torch.zeros_like(q)
    kv.kv[0][kv.block_table[0, 16:24].long(), :, 0] = 0x7F       # the third run's keys
    _raw_decode(ops, kv, q, got, ctxs, 8, Hkv, splits, po, pm)
    ml = pm.view(Hkv, splits, 16, 2)[:, :, :4]
    sums = po.view(Hkv, splits, 16, 128)[:, :, :4].double()
    assert ml[:, 2, :, 1].isnan().all() and (ml[:, [0, 1, 3], :, 1] > 0).all()
    f = torch.exp2(ml[:, [0, 1, 3], :, 0].double() - ml[:, [0, 1, 3], :, 0].amax(1, keepdim=True).double())[..., None]
    want = ((sums[:, [0, 1, 3]] * f).sum(1) / (ml[:, [0, 1, 3], :, 1, None].double() * f).sum(1)).view(1, 8, 128)
    # half a step of bf16; a few roundings of 24 bits per run, of terms that may cancel
    assert ((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-5).all()


@pytest.mark.parametrize("Hq,Hkv,ctxs,qlens,splits", [
    (8, 2, [17], [17], 0), (32, 8, [128, 129, 33], [128, 129, 33], 0), (8, 1, [1100, 40], [300, 40], 1),      # blocks of 128 rows and parts
    (4, 4, [700], [513], 1), (16, 2, [2000, 90], [70, 60], 3), (32, 4, [300], [40], 8),                        # split key ranges, some empty
    # the same with more blocks than SMs: two CTAs of four warps each
    (32, 8, [700, 129, 33], [700, 129, 33], 0), (8, 1, [2600], [2500], 1), (4, 4, [5200], [5000], 0), (16, 2, [2000, 90], [520, 60], 3), (32, 4, [300], [200], 8),
])
def test_prompt_attention(ops, Hq, Hkv, ctxs, qlens, splits):      # noqa: F811
    """Blocks whose rows see no key of a tile, few keys of it, or all; runs of tiles whose maxima grow and do not."""
    got, want = _attention_case(ops, Hq, Hkv, ctxs, qlens, splits=splits)
    assert torch.isfinite(got.float()).all() and _rel(got, want) < 0.06
    err = (got.float() - want.float()).flatten(1).norm(dim=1) / want.float().flatten(1).norm(dim=1)
    assert err.max().item() < 0.15


@pytest.mark.parametrize("D,Hq,Hkv,rot,gated", [(128, 8, 2, 128, False), (128, 16, 8, 128, False), (128, 6, 3, 64, True), (256, 4, 2, 64, True), (256, 2, 1, 256, False)])
@pytest.mark.parametrize("chunks", [[(0, 64)], [(11, 90), (0, 17)], [(5, 1)] * 3 + [(16, 70), (15, 1), (0, 40)], [(3, 20)], [(0, 1100)], [(i % 17, 1) for i in range(170)],
                                    [(3, 15)] * 20, [(5, 300), (0, 3)]])
def test_attention_preparation_writes_pages(ops, D, Hq, Hkv, rot, gated, chunks):      # noqa: F811
    """Queries, keys and values of steps with whole pages, parts of pages and single tokens: every page byte as the reference has
    it, nothing written for rows without a slot."""
    cfg = ModelConfig(hidden_size=Hq * D, num_heads=Hq, num_kv_heads=Hkv, head_dim=D, num_layers=1, attn_output_gate=gated,
                      rope=RopeConfig(theta=1e6, partial_rotary_factor=rot / D))
    cfg.layer_types = ["full_attention"]
    g = torch.Generator(device=DEV).manual_seed(7)
    per = max((c + n + 15) // 16 for c, n in chunks)
    kv = KVCache(cfg, 1 + per * len(chunks), len(chunks), per, "fp8", DEV, "umma")
    order = torch.randperm(per * len(chunks), generator=torch.Generator().manual_seed(2)).tolist()
    for b in range(len(chunks)):
        kv.set_pages(b, [1 + p for p in order[b * per:(b + 1) * per]])
    kv.kv[0].fill_(0x35)
    batch = build_batch([SeqChunk(b, [0] * n, c) for b, (c, n) in enumerate(chunks)], kv.block_table_host, DEV, attn_group=Hq // Hkv)
    T = batch.num_rows
    if T > 20:
        batch.slot_mapping[T - 3] = -1             # a padded row
    model, attn = _A(), _A()
    model.cfg, model.rope_scale, model.kv_rotate = cfg, 1.0, False
    model.inv_freq = torch.tensor(inv_freq(cfg), dtype=torch.float32, device=DEV)
    attn.heads, attn.kv_heads = Hq, Hkv
    attn.q_norm, attn.k_norm = [(1 + 0.1 * torch.randn(D, generator=g, device=DEV)).bfloat16() for _ in range(2)]
    qkv = torch.randn(T, (Hq * (2 if gated else 1) + 2 * Hkv) * D, generator=g, device=DEV).bfloat16()
    q, gate = ops.attn_prep_store(qkv, attn, model, batch, kv, 0, None)
    cos, sin = ref.rope_cos_sin(batch.positions, model.inv_freq)
    qr, kr, vr, gr = ref.attn_prep(qkv, Hq, Hkv, D, attn.q_norm, attn.k_norm, 1e-6, cos, sin, gated=gated)
    torch.cuda.synchronize()
    assert _rel(q, qr) < 4e-3
    if gated:
        assert torch.equal(gate.view(T, Hq, D), gr.reshape(T, Hq, D))
    kl, vl = kv.logical_kv(0)
    slots = batch.slot_mapping.long()
    live = slots >= 0
    page, off = slots[live] // 16, slots[live] % 16
    assert torch.equal(vl[page, :, off].float(), vr[live].to(torch.float8_e4m3fn).float())
    # a key near the edge between two codes may fall on either side (sums of squares in another order)
    assert _rel(kl[page, :, off].float(), kr[live].float()) < 0.04
    touched = torch.zeros(kl.shape[0], 16, dtype=torch.bool, device=DEV)
    touched[page, off] = True
    old = torch.tensor(0x35, dtype=torch.uint8).view(torch.float8_e4m3fn).float().item()
    for pool in (kl, vl):
        assert (pool.float().permute(0, 2, 1, 3)[~touched] == old).all()


@pytest.mark.parametrize("fmt", [Format.NVFP4, Format.MXFP8])
@pytest.mark.parametrize("T,K", [(1, 32), (3, 96), (129, 1056), (5, 1024), (1030, 4128), (2, 12288)])
def test_quantised_rows(ops, fmt, T, K):      # noqa: F811
    """Row quantisers at widths that end inside a tile of scales, against the reference quantisers."""
    if fmt == Format.NVFP4 and K % 64:
        K = (K + 63) // 64 * 64                    # what a product in that format can have
    g = torch.Generator(device=DEV).manual_seed(3)
    x = (torch.randn(T, K, generator=g, device=DEV) * torch.rand(T, 1, generator=g, device=DEV) * 8).bfloat16()
    x[T // 2] = 0
    lin = Linear(fmt, 128, K)
    lin.act_quant = True
    qa = ops.quantize_rows(x, lin)
    per = 16 if fmt == Format.NVFP4 else 32
    sf = quant.unswizzle_sf_128x4(qa.sf, T, K // per)
    if fmt == Format.NVFP4:
        got = quant.nvfp4_dequantize(qa.data, sf.view(torch.float8_e4m3fn), qa.row_scale)
        g_row = x.float().abs().amax(1) / torch.full((T,), 2688.0, device=DEV)      # (by a constant, torch multiplies with its reciprocal)
        want = quant.nvfp4_dequantize(*quant.nvfp4_quantize(x, g_row.clamp_min(1e-30), per_row=True))
    else:
        got = quant.mxfp8_dequantize(qa.data.view(torch.float8_e4m3fn), sf)
        want = quant.mxfp8_dequantize(*quant.mxfp8_quantize(x))
    # The kernel multiplies by a block's reciprocal: a value on the edge between two codes may take the other one.  Quotients of
    # numbers with 8-bit mantissas do lie there, about one in two thousand, and a code is up to a quarter of its value away.
    assert (got != want).float().mean().item() < 1e-3 and _rel(got, want) < 1e-2


@pytest.mark.parametrize("T,H,shift", [(1, 8, 0), (3, 20, 0), (7, 2048, 0), (5, 4096, 1), (1, 33, 3), (300, 5120, 0), (2100, 4096, 0), (2, 12, 4), (3, 20, 4)])
def test_elementwise(ops, T, H, shift):      # noqa: F811
    g = torch.Generator(device=DEV).manual_seed(5)
    a, b = [torch.randn(T * H + shift, generator=g, device=DEV).bfloat16()[shift:].view(T, H) for _ in range(2)]
    gl = torch.randn(T, 1, generator=g, device=DEV).bfloat16()
    assert torch.equal(ops.add(a, b), (a.float() + b.float()).bfloat16())
    want = (a.float() + b.float() * torch.sigmoid(gl.float()).bfloat16().float()).bfloat16()
    assert _rel(ops.add_sigmoid_scaled(a, b, gl), want) < 4e-3
    want = (a.float() * torch.sigmoid(b.float())).bfloat16()
    assert _rel(ops.mul_sigmoid(a.clone(), b), want) < 4e-3


@pytest.mark.parametrize("M", [1, 24, 25, 31, 32, 33, 64, 65])
@pytest.mark.parametrize("N,K", [(128, 128), (200, 384), (512, 25600), (1024, 5120), (2200, 2176), (4100, 3328), (5120, 8192), (6144, 3072), (12288, 4096), (40000, 256)])
def test_fp8_block_product_of_few_rows(ops, M, N, K):      # noqa: F811
    """Rows on the MMA's columns and K over a cluster, against the stored codes and scales in 64 bits."""
    g = torch.Generator(device=DEV).manual_seed(11)
    x = torch.randn(M, K, generator=g, device=DEV).bfloat16()
    lin = Linear.from_dense(torch.randn(N, K, generator=g, device=DEV) * 0.02, Format.FP8_BLOCK)
    lin.bias = torch.randn(N, generator=g, device=DEV).bfloat16()
    q, sc = ops.quantize_fp8_block(x)
    got = ops.linear(lin, x, out_dtype=torch.float32)
    torch.cuda.synchronize()
    assert ops.take_status() == 0
    xd = (q.view(torch.float8_e4m3fn).double().view(M, K // 128, 128) * sc[:, :M].t().double().unsqueeze(-1)).view(M, K)
    assert _rel(got, xd @ lin.dequant().double().t() + lin.bias.double()) < 1e-5
    assert torch.equal(ops.linear(lin, x), got.bfloat16())      # and the same sums when they are rounded


@pytest.mark.parametrize("fmt,T,E,k,H,I", [(Format.NVFP4, 300, 5, 2, 512, 256), (Format.MXFP8, 250, 8, 4, 256, 128), (Format.NVFP4, 128, 3, 3, 256, 384)])
def test_expert_product_of_up_to_a_tile_of_rows(ops, fmt, T, E, k, H, I):      # noqa: F811
    """Experts with no row, a few and more than a tile of 128, around the most rows per expert that the narrow kernel takes: it gives
    what the tiles of the grouped product do."""
    ex = _experts(E, H, I, fmt, 5)
    g = torch.Generator(device=DEV).manual_seed(6)
    x = torch.randn(T, H, generator=g, device=DEV).bfloat16()
    logits = torch.randn(T, E, generator=g, device=DEV) + torch.linspace(3, -3, E, device=DEV)
    if E > k:
        logits[:, -1] = -50                        # nothing for the last one
    outs, old = [], ops.MOE_NARROW_ROWS
    try:
        for ops.MOE_NARROW_ROWS in (1 << 20, 0):
            w, ids = ops.router_topk(logits, k, True, 0, E)
            outs.append(ops.moe(x, w, ids, ex))
    finally:
        ops.MOE_NARROW_ROWS = old
    torch.cuda.synchronize()
    assert ops.take_status() == 0
    assert _rel(outs[0], outs[1]) < 2e-3           # one may round a sum to the neighbouring bf16
    assert _rel(outs[0], ref.moe_forward(x, w, ids, ex.forward_one, E)) < 0.08


@pytest.mark.parametrize("kind,E,N,k,most", [(2, 512, 1024, 10, 6553), (2, 128, 2048, 8, 2048), (2, 127, 2048, 8, 762), (2, 8, 6144, 2, 192), (1, 512, 1024, 10, 2457)])
def test_which_steps_take_the_narrow_expert_kernel(ops, kind, E, N, k, most):      # noqa: F811
    """48 routed rows per expert, 128 where MXFP8 experts have 2048 feature tiles together."""
    ex = _A()
    ex.count, ex.cuda_pack = E, {"gate_up": {"kind": kind, "N": N}}
    assert ops.moe_narrow_tokens(ex, k) == most


@pytest.mark.parametrize("E,T,k", [(1, 5, 1), (33, 300, 4), (512, 700, 10)])
def test_expert_plan(ops, E, T, k):      # noqa: F811
    """Offsets of the experts' rows in tiles of 128 and each tile's expert and live rows."""
    from blaze_b200.ops.cuda_ops import VP, _ptr
    counts = torch.bincount(torch.randint(0, E, (T * k,), generator=torch.Generator().manual_seed(1)), minlength=E).to(torch.int32)
    tiles = (T * k + 127) // 128 + E
    dev = counts.to(DEV)
    off, fill, te, tr = [torch.full((n,), -7, dtype=torch.int32, device=DEV) for n in (E, E, tiles, tiles)]
    assert ops.lib.blz_moe_plan(_ptr(dev), _ptr(off), _ptr(fill), _ptr(te), _ptr(tr), E, tiles, VP(0)) == 0
    torch.cuda.synchronize()
    want_te, want_tr, at = [], [], []
    for e, n in enumerate(counts.tolist()):
        at.append(len(want_te) * 128)
        for r in range(0, n, 128):
            want_te.append(e)
            want_tr.append(min(128, n - r))
    pad = tiles - len(want_te)
    assert te.tolist() == want_te + [-1] * pad and tr.tolist() == want_tr + [0] * pad
    assert off.tolist() == at and fill.tolist() == [0] * E


@pytest.mark.parametrize("T,Hv,DV", [(1, 1, 4), (7, 3, 64), (33, 2, 132), (300, 32, 128), (5, 2, 129)])
@pytest.mark.parametrize("flags", [0, 1, 2, 3])
def test_gated_norm(ops, T, Hv, DV, flags):      # noqa: F811
    """Single elements and runs of four give the same bits, and both what 64 bits give, rounded: also for gates whose sigmoid lies
    near the end of the range (1 + e^-z beyond 2^126)."""
    from blaze_b200.ops.cuda_ops import VP, _ptr
    g = torch.Generator(device=DEV).manual_seed(9)
    o, z = [torch.randn(T, Hv * DV, generator=g, device=DEV).mul(s).bfloat16() for s in (1.0, 3.0)]
    z[:, ::7] = torch.tensor([-87.0, -87.5, -88.0, 88.0, -40.0, 0.0], device=DEV).repeat(-(-z[:, ::7].numel() // 6))[:z[:, ::7].numel()].view_as(z[:, ::7])
    w = (0.3 * torch.randn(DV, generator=g, device=DEV)).bfloat16()
    outs = []
    for shift in (0, 1):                           # rows on 8 bytes, and one element off
        a, b, c = [torch.empty(t.numel() + 1, dtype=torch.bfloat16, device=DEV)[shift:shift + t.numel()].view_as(t).copy_(t) for t in (o, z, w)]
        y = torch.empty_like(o)
        assert ops.lib.blz_gated_rmsnorm(_ptr(a), _ptr(b), b.stride(0), _ptr(c), _ptr(y), T, Hv, DV, 1e-6, flags, VP(0)) == 0
        outs.append(y)
    torch.cuda.synchronize()
    assert torch.equal(outs[0], outs[1])
    x, zd = o.double().view(T, Hv, DV), z.double().view(T, Hv, DV)
    want = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6) * (w.double() + (flags & 1)) * zd.sigmoid() * (1 if flags & 2 else zd)
    # half a step of bf16 (8 bits: up to 2^-8 of the value), and the fast exponential: 2 ulp and, of its argument, 88 * 2^-24
    err = (outs[0].double().view_as(want) - want).abs()
    assert (err <= want.abs() * (2.0 ** -8 + 2e-5) + 1e-40).all()


def test_silu_of_every_gate(ops):      # noqa: F811
    """The activation's quotient over all 16-bit gates: rounded as the division is, up to where e^-x overflows, with its infinities."""
    x = torch.arange(1 << 16, device=DEV, dtype=torch.int32).to(torch.int16).view(torch.bfloat16).view(16, 4096)
    got = ops.silu_mul(torch.cat([x, torch.ones_like(x)], 1)).double()
    xd = x.double()
    want = torch.where(xd < -88.72, 0.0, xd * xd.sigmoid())       # e^-x is infinite there: x / inf
    assert torch.equal(got.isnan(), xd.isnan() | (xd == -torch.inf)) and (got[xd == torch.inf] == torch.inf).all()
    ok = xd.isfinite()
    step = torch.exp2(torch.frexp(want.abs().clamp_min(2.0 ** -126))[1].double() - 8)      # of bf16 (8 bits) at that size
    # half a step, and in front of the rounding the fast exponential: 2 ulp and, of its argument, 88 * 2^-24, of 2^8 steps
    assert ((got - want).abs()[ok] <= step[ok] * (0.5 + 256 * (88 + 4) * 2.0 ** -24)).all()


@pytest.mark.parametrize("mode", [Format.NVFP4, Format.MXFP8])
@pytest.mark.parametrize("W", [32, 96, 480, 1024, 1056, 4096, 4128, 12288, 12320, 24576, 24608])
def test_quantised_rows_of_sixteen_elements_per_thread(ops, mode, W):      # noqa: F811
    """Rows of the quantisers with 16 elements per thread (part of a warp, whole chunks, one block more, the widest, and the kernel
    behind it) against those with 8: activations, gated rows of 511 and 512 tokens, norms whose sums are exact; the same codes, scales
    and row scales, also in rows with infinities and values that are not numbers."""
    g = torch.Generator(device=DEV).manual_seed(4)
    lin = Linear(mode, 128, W)
    lin.act_quant = True
    per = 16 if mode == Format.NVFP4 else 32

    def same(a, b, n):
        sf = [quant.unswizzle_sf_128x4(q.sf, q.rows, W // per)[:n] for q in (a, b)]
        rs = a.row_scale is None or torch.equal(a.row_scale[:n].view(torch.int32), b.row_scale[:n].view(torch.int32))
        return torch.equal(a.data[:n], b.data[:n]) and torch.equal(*sf) and rs
    gu = torch.randn(512, 2 * W, generator=g, device=DEV).bfloat16()
    gu[3, 5], gu[4, 7], gu[5, W + 9], gu[6, :] = float("nan"), float("inf"), float("-inf"), 0.0
    wide = W <= 24576                              # beyond, one kernel takes all of them
    few, many = ops.silu_mul(gu[:511], lin), ops.silu_mul(gu, lin)
    assert same(few, many, 511)
    if wide:
        assert same(ops.quantize_rows(ops.silu_mul(gu[:511]), lin), few, 511)
    x = torch.randint(-4, 5, (33, W), generator=g, device=DEV).bfloat16() / 2
    r = torch.randint(-4, 5, (33, W), generator=g, device=DEV).bfloat16() / 4
    w = (1 + 0.1 * torch.randn(W, generator=g, device=DEV)).bfloat16()
    for zero in (False, True):
        r1, r2, x1 = r.clone(), r.clone(), x.clone()
        plain, _ = ops.norm(x.clone(), r1, w, 1e-6, zero_centered=zero)
        q, _ = ops.norm(x1, r2, w, 1e-6, zero_centered=zero, quant_for=lin, zero_src=True)
        assert torch.equal(r1, r2) and not x1.any()
        if wide:
            assert same(q, ops.quantize_rows(plain, lin), 33)
    torch.cuda.synchronize()
    assert ops.take_status() == 0


@pytest.mark.parametrize("fmt", [Format.NVFP4, Format.MXFP8])
@pytest.mark.parametrize("T,E,k,H,I", [(5, 3, 1, 256, 128), (300, 4, 2, 512, 256), (130, 8, 4, 256, 192)])
def test_experts_with_the_activation_in_the_product(ops, fmt, T, E, k, H, I):      # noqa: F811
    """Interleaved gate and up rows: the pairs', the narrow and the 128-column product give the rounded gate and up sums' activation."""
    g = torch.Generator(device=DEV).manual_seed(8)
    x = torch.randn(T, H, generator=g, device=DEV).bfloat16()
    logits = torch.randn(T, E, generator=g, device=DEV)
    outs, old = [], ops.MOE_NARROW_ROWS
    try:
        for rows in (48, 1 << 20, 0):
            ex = _experts(E, H, I, fmt, 9)
            ops.MOE_NARROW_ROWS = rows
            w, ids = ops.router_topk(logits, k, True, 0, E)
            outs.append(ops.moe(x, w, ids, ex))
            assert ex.cuda_pack["gate_up"]["swiglu"]
    finally:
        ops.MOE_NARROW_ROWS = old
    torch.cuda.synchronize()
    assert ops.take_status() == 0
    for o in outs:
        assert _rel(o, outs[0]) < 2e-3             # one may round a sum to the neighbouring bf16
        assert _rel(o, ref.moe_forward(x, w, ids, ex.forward_one, E)) < 0.08


@pytest.mark.parametrize("M,N,K", [(1, 128, 128), (64, 200, 384), (65, 131, 256), (129, 640, 1152), (300, 1000, 640), (20000, 384, 256)])
def test_fp8_block_product_on_cta_pairs(ops, M, N, K):      # noqa: F811
    """Both tile widths, K whole and split over 2 to 4 pairs, odd numbers of blocks, features that are no whole tiles: against the kernel of
    one CTA per tile, which adds the blocks in the same order, so the same bits where K is not split."""
    from blaze_b200.ops.cuda_ops import VP, _ptr
    g = torch.Generator(device=DEV).manual_seed(12)
    x = torch.randn(M, K, generator=g, device=DEV).bfloat16()
    lin = Linear.from_dense(torch.randn(N, K, generator=g, device=DEV) * 0.02, Format.FP8_BLOCK)
    lin.bias = torch.randn(N, generator=g, device=DEV).bfloat16()
    pk = ops.pack(lin)
    q, sc = ops.quantize_fp8_block(x)
    odd = torch.zeros(K // 128, M + 1 - M % 2, dtype=torch.float32, device=DEV)        # rows off 16 bytes: the other kernel
    odd[:, :M] = sc[:, :M]
    for dt in (torch.float32, torch.bfloat16):
        want, out = torch.empty(M, N, dtype=dt, device=DEV), torch.empty(M, N, dtype=dt, device=DEV)
        shape = (_ptr(q), K, _ptr(pk["w"]), K)
        rest = (_ptr(pk["sf"]), _ptr(pk["bias"]), int(dt == torch.float32))
        assert ops.lib.blz_gemm_fp8_block(*shape, _ptr(want), N, M, N, K, _ptr(odd), odd.stride(0), *rest, VP(0)) == 0
        for cn in (64, 128):
            for ks in range(1, min(4, (K + 255) // 256) + 1):
                if ks > 1 and M > 1000:
                    continue
                out.fill_(float("nan"))
                assert ops.lib.blz_gemm_fp8_pair(*shape, _ptr(out), N, M, N, K, _ptr(sc), sc.stride(0), *rest, cn, ks, VP(0)) == 0
                torch.cuda.synchronize()
                assert ops.take_status() == 0
                # parts of K add in another order: up to 2^-24 of the terms' size per addition
                assert torch.equal(out, want) if ks == 1 else _rel(out, want) < (1e-6 if dt == torch.float32 else 2e-3), (cn, ks)


@pytest.mark.parametrize("T,K", [(1, 128), (7, 384), (8, 512), (9, 640), (65, 1152), (300, 25600)])
def test_fp8_groups_with_and_without_the_activation(ops, T, K):      # noqa: F811
    """Codes and scales are those of the definition bit for bit; gated rows give those of the activation rounded to bf16; rows that start
    on 8 bytes only, an infinity and a NaN give the same codes as anywhere else."""
    g = torch.Generator(device=DEV).manual_seed(13)
    gu = torch.randn(T, 2 * K, generator=g, device=DEV).bfloat16()
    # (no -0 among the gates: the activation kernel of rows beyond 24576 divides, which keeps the zero's sign, and silu() does not)
    gu[0, :2] = torch.tensor([float("inf"), float("nan")], device=DEV)
    gu[T // 2, 128:256] = 0
    down = Linear.from_dense(torch.randn(128, K, generator=g, device=DEV), Format.FP8_BLOCK)
    act = ops.silu_mul(gu)
    wide = torch.zeros(T, K + 4, dtype=torch.bfloat16, device=DEV)
    wide[:, 4:] = act
    gated, (q, sc), (q8, sc8) = ops.silu_mul(gu, quant_for=down), ops.quantize_fp8_block(act), ops.quantize_fp8_block(wide[:, 4:])
    torch.cuda.synchronize()
    v = act.float().view(T, K // 128, 128)
    most = torch.nan_to_num(v.abs(), nan=0.0, posinf=float("inf")).amax(-1)
    want = (most / torch.full_like(most, 448.0)).clamp_min(1e-12)      # (a division by a number multiplies by its rounded inverse)
    assert torch.equal(sc[:, :T].t(), want)
    codes = (v / want.unsqueeze(-1)).view(T, K)
    ok = codes.isfinite()
    assert torch.equal(q.view(torch.float8_e4m3fn).float()[ok], codes.clamp(-448, 448).to(torch.float8_e4m3fn).float()[ok])
    assert q.view(torch.float8_e4m3fn).float()[~ok].isnan().all()
    for a, b in ((gated.data, gated.sf), (q8, sc8)):
        assert torch.equal(a, q) and torch.equal(b[:, :T], sc[:, :T])


@pytest.mark.parametrize("mode", [Format.NVFP4, Format.MXFP8])
@pytest.mark.parametrize("T,W", [(3, 32), (3, 2016), (1200, 2048), (1200, 2080), (1024, 4096), (1025, 4096), (1025, 2304), (1025, 3840), (40, 4128), (1025, 7168), (40, 12320), (3, 24576)])
def test_quantised_norm_adds_squares_like_the_plain_one(ops, mode, T, W):      # noqa: F811
    """One pass of the plain kernel's threads over a row, several, and both numbers of threads: the same row sums, so the same codes."""
    g = torch.Generator(device=DEV).manual_seed(21)
    lin = Linear(mode, 128, W)
    lin.act_quant = True
    x, r = (torch.randn(T, W, generator=g, device=DEV).bfloat16() for _ in range(2))
    w = (1 + 0.1 * torch.randn(W, generator=g, device=DEV)).bfloat16()
    plain, _ = ops.norm(x.clone(), r.clone(), w, 1e-6)
    got, want = ops.norm(x, r, w, 1e-6, quant_for=lin)[0], ops.quantize_rows(plain, lin)
    per = 16 if mode == Format.NVFP4 else 32
    assert torch.equal(got.data, want.data)
    assert torch.equal(*(quant.unswizzle_sf_128x4(q.sf, T, W // per) for q in (got, want)))
    assert mode != Format.NVFP4 or torch.equal(got.row_scale, want.row_scale)


def test_a_tuned_route_is_taken_where_it_beat_the_rules(ops, tmp_path, monkeypatch):      # noqa: F811
    """An entry of the tuning table counts where its kernel was faster than what the rules pick; one that was measured without the rules'
    time does not count, and is measured anew."""
    from blaze_b200 import tune
    g = torch.Generator(device=DEV).manual_seed(41)
    lin = Linear.from_dense(torch.randn(512, 8192, generator=g, device=DEV) * 0.02)
    x = torch.randn(200, 8192, generator=g, device=DEV).bfloat16()
    rule = ops.linear(lin, x)
    by = {ks: ops.linear(lin, x, sk=ks) for ks in (1, 2, 3, 5, 7)}
    ks = next(k for k in by if not torch.equal(by[k], rule))          # (parts of K add up in another order)
    t = tune.Tuning(str(tmp_path / "t.json"))
    monkeypatch.setattr(ops, "tuning", t)
    for entry, want in (({"ms": 1.0, "rule_ms": 2.0}, by[ks]), ({"ms": 2.0, "rule_ms": 1.0}, rule), ({"ms": 1.0}, rule)):
        t.table = {"gemm0:512x8192x256": {"kernel": "sk", "ks": ks, **entry}}
        assert torch.equal(ops.linear(lin, x), want), entry
    best = tune.tune_linear(ops, lin, 200, t, iters=3)
    assert best["rule_ms"] > 0 and best == t.get("gemm0", 512, 8192, 256) and ops.tuning is t
    t.table["gemm0:512x8192x256"] = {"kernel": "tc", "bn": 256, "ms": 1.0, "rule_ms": 2.0}
    assert torch.equal(ops.linear(lin, x), ops.linear(lin, x, bn=256, wide=False, sk=False))
    torch.cuda.synchronize()
    assert ops.take_status() == 0


@pytest.mark.parametrize("fmt", [Format.NVFP4, Format.MXFP8])
@pytest.mark.parametrize("I", [32, 192, 704, 1056, 4128, 24608])
def test_interleaved_gate_and_up_rows(ops, fmt, I):      # noqa: F811
    """Gate and up values in groups of 16 | 16, as the narrow experts' product stores them, few rows and many: the codes and scales of the
    same values side by side."""
    g = torch.Generator(device=DEV).manual_seed(17)
    lin = Linear(fmt, 128, I)
    lin.act_quant = True
    gu = torch.randn(600, 2 * I, generator=g, device=DEV).bfloat16()
    mixed = gu.view(600, 2, I // 16, 16).transpose(1, 2).reshape(600, 2 * I)
    per = 16 if fmt == Format.NVFP4 else 32
    for n in (40, 600):
        rows = torch.randperm(600, generator=torch.Generator().manual_seed(2))[:n].to(torch.int32).to(DEV)
        a, b = ops._silu_mul_live(gu, lin, rows), ops._silu_mul_live(mixed, lin, rows, 2)
        at = rows.long()
        assert torch.equal(a.data[at], b.data[at]) and (fmt == Format.MXFP8 or torch.equal(a.row_scale[at], b.row_scale[at]))
        assert torch.equal(*(quant.unswizzle_sf_128x4(q.sf, q.rows, I // per)[at] for q in (a, b)))
        assert torch.equal(ops._silu_mul_live(gu, None, rows)[at], ops._silu_mul_live(mixed, None, rows, 2)[at])


def test_narrow_experts_leave_the_activation_to_the_quantiser(ops, monkeypatch):      # noqa: F811
    """Features that are no multiple of 256: the narrow product, whose epilogue is slow at it, stores gate and up sums."""
    acts = []
    real = ops._moe_gemm
    monkeypatch.setattr(ops, "_moe_gemm", lambda *a, **k: (acts.append((list(a[7:]) + [k.get("act", 0)])[0]), real(*a, **k))[1])
    x = torch.randn(40, 256, generator=torch.Generator(device=DEV).manual_seed(3), device=DEV).bfloat16()
    ex = _experts(8, 256, 192, Format.NVFP4, 9)
    w, ids = ops.router_topk(torch.randn(40, 8, device=DEV), 2, True, 0, 8)
    out = ops.moe(x, w, ids, ex)
    assert acts == [0, 0] and _rel(out, ref.moe_forward(x, w, ids, ex.forward_one, 8)) < 0.08


@pytest.mark.parametrize("T,K", [(1535, 512), (191, 4096), (95, 8192), (6143, 128)])
def test_fp8_groups_of_few_elements(ops, T, K):      # noqa: F811
    """The last row counts whose groups are a warp's each, and one row more: the same codes and scales, also of rows that start on 8 bytes,
    and of infinities and values that are not numbers."""
    x = torch.randn(T + 1, K, generator=torch.Generator(device=DEV).manual_seed(14), device=DEV).bfloat16()
    x[0, :3] = torch.tensor([float("inf"), float("nan"), -0.0], device=DEV)
    x[T // 2, :128] = 0
    wide = torch.zeros(T, K + 4, dtype=torch.bfloat16, device=DEV)
    wide[:, 4:] = x[:T]
    (qa, sa), (q, s), (q8, s8) = ops.quantize_fp8_block(x), ops.quantize_fp8_block(x[:T]), ops.quantize_fp8_block(wide[:, 4:])
    assert T * K < 3 << 18 <= (T + 1) * K
    assert torch.equal(q, qa[:T]) and torch.equal(s[:, :T], sa[:, :T]) and torch.equal(q8, q) and torch.equal(s8[:, :T], s[:, :T])


@pytest.mark.parametrize("mode", [Format.NVFP4, Format.MXFP8])
@pytest.mark.parametrize("T,W", [(1024, 768), (768, 1024), (1445, 544), (1536, 512)])
def test_quantised_short_rows_of_few_elements(ops, mode, T, W):      # noqa: F811
    """The last row counts with 8 elements per thread, one row more, and rows of one warp: the same codes and scales."""
    lin = Linear(mode, 128, W)
    lin.act_quant = True
    x = torch.randn(T + 1, W, generator=torch.Generator(device=DEV).manual_seed(15), device=DEV).bfloat16()
    x[0, :3] = torch.tensor([float("inf"), float("nan"), -0.0], device=DEV)
    x[T // 2] = 0
    assert T * W <= 3 << 18 < (T + 1) * W
    few, many = ops.quantize_rows(x[:T], lin), ops.quantize_rows(x, lin)
    per = 16 if mode == Format.NVFP4 else 32
    assert torch.equal(few.data, many.data[:T]) and (mode == Format.MXFP8 or torch.equal(few.row_scale, many.row_scale[:T]))
    assert torch.equal(*(quant.unswizzle_sf_128x4(q.sf, q.rows, W // per)[:T] for q in (few, many)))


@pytest.mark.parametrize("mode", [Format.NVFP4, Format.MXFP8])
@pytest.mark.parametrize("W", [512, 544, 1024, 1056, 4064, 4096, 4128, 5120, 12320, 24576])
def test_quantised_norm_of_few_rows(ops, mode, W):      # noqa: F811
    """The most rows with 8 elements per thread, and one row more: the same residual, codes and scales."""
    g = torch.Generator(device=DEV).manual_seed(16)
    lin = Linear(mode, 128, W)
    lin.act_quant = True
    x, r = (torch.randn(129, W, generator=g, device=DEV).bfloat16() for _ in range(2))
    x[0, 3], x[1, 5], r[2, 7] = float("inf"), float("nan"), float("-inf")
    w, r1, r2 = (1 + 0.1 * torch.randn(W, generator=g, device=DEV)).bfloat16(), r.clone(), r[:128].clone()
    many, few = ops.norm(x, r1, w, 1e-6, quant_for=lin)[0], ops.norm(x[:128].clone(), r2, w, 1e-6, quant_for=lin)[0]
    per = 16 if mode == Format.NVFP4 else 32
    assert torch.equal(r1[:128].view(torch.int16), r2.view(torch.int16)) and torch.equal(few.data, many.data[:128])
    assert torch.equal(*(quant.unswizzle_sf_128x4(q.sf, q.rows, W // per)[:128] for q in (few, many)))
    assert mode == Format.MXFP8 or torch.equal(few.row_scale.view(torch.int32), many.row_scale[:128].view(torch.int32))


@pytest.mark.parametrize("kind,E,N,D,k,want", [
    (1, 128, 1536, 2048, 8, {1536}), (2, 512, 1024, 2048, 10, {4915}), (1, 64, 1408, 2048, 6, {512, 1024}), (0, 128, 1536, 2048, 8, {768, 1536}),
    (1, 64, 1280, 1920, 6, {512, 1024}), (1, 64, 1408, 1920, 6, {512})])
def test_where_experts_change_their_form(ops, kind, E, N, D, k, want):      # noqa: F811
    """A step's experts are computed in one form up to each limit and in another beyond: pairs' rows per tile, and the narrow kernel where
    it is taken."""
    ex = _A()
    ex.count, ex.act, ex.cuda_pack = E, "swiglu", {"gate_up": {"kind": kind, "N": N}, "down": {"kind": kind, "N": D}}
    assert ops.expert_limits(ex, k) == want
    forms = [ops._expert_form(ex, k, T) for T in range(1, 6000)]
    assert {T for T in range(1, 5999) if forms[T - 1] != forms[T]} == want


_PAIRS_OFF = """
import sys
import torch
from blaze_b200.linear import Linear
from blaze_b200.ops.cuda_ops import CudaOps
from blaze_b200.quant import Format
from test_gpu_kernels import _experts
off = sys.argv[2] == "off"
ops = CudaOps("cuda:0")
assert ops._pair_ok == (ops.lib.blz_pair_room(2) > 0) == (not off)
g = torch.Generator(device="cuda:0").manual_seed(51)
rand = lambda *s: torch.randn(*s, generator=g, device="cuda:0")      # noqa: E731
out, launches = {}, ops.launches
for f in (Format.DENSE, Format.NVFP4, Format.MXFP8, Format.FP8_BLOCK):
    lin = Linear.from_dense(rand(768, 1024) * 0.05, f)
    for M in (1, 64, 300):
        out[f"{f} {M}"] = ops.linear(lin, rand(M, 1024).bfloat16())
    gu = Linear.from_dense(rand(512, 1024) * 0.05, f)
    out[f"{f} glu"] = ops.linear_swiglu(gu, rand(100, 1024).bfloat16())
for f in (Format.DENSE, Format.NVFP4, Format.MXFP8):
    for T in (5, 700):
        ex = _experts(8, 256, 256, f, 9)
        w, ids = ops.router_topk(rand(T, 8), 2, True, 0, 8)
        out[f"experts {f} {T}"] = ops.moe(rand(T, 256).bfloat16(), w, ids, ex)
torch.cuda.synchronize()
assert ops.take_status() == 0
torch.save(out, sys.argv[1])
"""


def test_products_without_pairs_of_ctas(tmp_path):
    """BLAZE_GEMM_PAIR=0, or a context without room for a pair: every product, FP8 and experts too, takes the kernels of single CTAs."""
    import os
    import subprocess
    import sys
    here = os.path.dirname(os.path.abspath(__file__))
    for name, env in (("on", {}), ("off", {"BLAZE_GEMM_PAIR": "0"})):
        path = os.pathsep.join([os.path.dirname(here), here])
        subprocess.run([sys.executable, "-c", _PAIRS_OFF, str(tmp_path / name), name], env={**os.environ, "PYTHONPATH": path, **env}, check=True, timeout=300)
    on, off = (torch.load(tmp_path / n) for n in ("on", "off"))
    for k, v in on.items():
        assert _rel(off[k], v) < 2e-3, k           # (K in other parts; a sum may round to the neighbouring bf16)


def test_fp8_rows_without_pairs_of_ctas(tmp_path):
    """The FP8 product of few rows with K over a cluster is what calls take where no pair fits."""
    import os
    import subprocess
    import sys
    run = [sys.executable, "-m", "pytest", "-q", "-x", os.path.abspath(__file__), "-k", "test_fp8_block_product_of_few_rows"]
    got = subprocess.run(run, env={**os.environ, "BLAZE_GEMM_PAIR": "0"}, capture_output=True, text=True, timeout=300)
    assert got.returncode == 0 and " passed" in got.stdout, got.stdout[-2000:]


@pytest.mark.parametrize("T,I", [(5, 256), (300, 256), (40, 192)])
def test_experts_stored_in_fp8_blocks(ops, T, I):      # noqa: F811
    """Experts with 128 x 128 block scales, which are packed as MXFP8, by the pairs and by the narrow product: the stored weights' result,
    within what both formats' 3-bit mantissas leave (2^-4 at most per weight and per activation)."""
    ex = _experts(8, 256, I, Format.FP8_BLOCK, 9)
    g = torch.Generator(device=DEV).manual_seed(18)
    x = torch.randn(T, 256, generator=g, device=DEV).bfloat16()
    w, ids = ops.router_topk(torch.randn(T, 8, generator=g, device=DEV), 2, True, 0, 8)
    out = ops.moe(x, w, ids, ex)
    torch.cuda.synchronize()
    assert ops.take_status() == 0
    assert _rel(out, ref.moe_forward(x, w, ids, ex.forward_one, 8)) < 0.08
