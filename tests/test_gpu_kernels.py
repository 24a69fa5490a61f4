"""Numerics of every CUDA kernel against the plain PyTorch fp32 statement of the same op (deliverance_b200.ops.ref)."""
import math
import time

import pytest
import torch

from deliverance_b200 import ops
from deliverance_b200.ckpt.jq4 import q4_dequantize, q4_quantize
from deliverance_b200.ckpt.safetensors_io import Q4Tensor
from deliverance_b200.ops import LinearWeight, ref

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rel(a, b):
    return ((a.float() - b.float()).norm() / (b.float().norm() + 1e-12)).item()


def _rounded_once(y, want, slack):
    """Whether every bf16 value of ``y`` is ``want`` rounded once: 2^-8 of the value at most (half a step at the low end of its power of two), and on top of it the error
    ``slack`` of what stands in front of the rounding."""
    return bool(((y.double() - want).abs() <= (want.abs() + slack) * 2.0**-8 + slack).all())


def _q4_weight(N, K, seed=0):
    g = torch.Generator().manual_seed(seed)
    w = torch.randn(N, K, generator=g) * 0.05
    p, s = q4_quantize(w)
    return Q4Tensor(p, s, (N, K)), q4_dequantize(p, s)


@pytest.mark.parametrize("M", [1, 2, 3, 4])
@pytest.mark.parametrize("q4", [True, False])
def test_gemv_simt(M, q4):
    N, K = 384, 1024
    qt, wd = _q4_weight(N, K)
    lw = (LinearWeight(qt) if q4 else LinearWeight(wd.to(torch.bfloat16))).to(DEV, torch.bfloat16)
    x = (torch.randn(M, K) * 0.5).to(torch.bfloat16).to(DEV)
    y = ops.linear(x, lw, impl=2)
    wref = wd if q4 else wd.to(torch.bfloat16).float()
    yr = x.float().cpu() @ wref.t()
    assert _rel(y.cpu(), yr) < 1e-2


@pytest.mark.parametrize("M,N,K,splits", [
    (1, 256, 512, 1), (8, 256, 1024, 1), (16, 384, 2560, 0), (17, 128, 256, 1), (64, 512, 2048, 0), (64, 2560, 9728, 0),
    (100, 640, 1216, 1), (128, 256, 4096, 2), (300, 384, 1024, 1), (5, 200, 2560, 4), (33, 1000, 608, 0),
    (64, 256, 4096, 8), (48, 384, 4096, -4), (16, 128, 9728, -16), (7, 256, 2048, 3), (600, 256, 512, 0),
    (64, 19456, 1024, 0), (8, 19712, 1280, 0),  # a few tiles more than SMs: the tail tiles are split over k
])
@pytest.mark.parametrize("q4", [True, False])
def test_gemm_tcgen05(M, N, K, splits, q4):
    qt, wd = _q4_weight(N, K, seed=N + K)
    lw = (LinearWeight(qt) if q4 else LinearWeight(wd.to(torch.bfloat16))).to(DEV, torch.bfloat16)
    x = (torch.randn(M, K) * 0.5).to(torch.bfloat16).to(DEV)
    bias = torch.randn(N, device=DEV) if (M % 2 == 0) else None
    lw.bias = bias
    y = ops.linear(x, lw, impl=1, force_splits=splits)
    torch.cuda.synchronize()
    ops.check_status()
    wref = wd if q4 else wd.to(torch.bfloat16).float()
    yr = x.float().cpu() @ wref.t()
    if bias is not None:
        yr = yr + bias.cpu()
    assert y.shape == (M, N)
    assert _rel(y.cpu(), yr) < 1.5e-2, f"rel err {_rel(y.cpu(), yr)}"
    # fp32 output path
    y32 = ops.linear(x, lw, out_f32=True, impl=1, force_splits=splits)
    assert y32.dtype == torch.float32 and _rel(y32.cpu(), yr) < 1.5e-2
    # repeated launches reuse the split-K scratch and counters
    y2 = ops.linear(x, lw, impl=1, force_splits=splits)
    assert torch.equal(y, y2)


def test_rmsnorm_and_add():
    T, H = 37, 2560
    x = torch.randn(T, H).to(torch.bfloat16).to(DEV)
    w = (torch.randn(H) * 0.1 + 1).to(torch.bfloat16).to(DEV)
    y = ops.rmsnorm(x, w, 1e-6, 0.0)
    assert _rel(y, ref.rmsnorm(x.float(), w.float(), 1e-6)) < 5e-3
    y1 = ops.rmsnorm(x, w, 1e-6, 1.0)
    assert _rel(y1, ref.rmsnorm(x.float(), w.float(), 1e-6, 1.0)) < 5e-3
    res = torch.randn(T, H).to(torch.bfloat16).to(DEV)
    res_ref = res.clone().float()
    y2 = ops.add_rmsnorm(x, res, w, 1e-6, 0.0, 0.5)
    yr = ref.add_rmsnorm(x.float(), res_ref, w.float(), 1e-6, 0.0, 0.5)
    assert _rel(res, res_ref) < 5e-3 and _rel(y2, yr) < 8e-3


def test_layernorm_act_embedding():
    T, H = 19, 768
    x = torch.randn(T, H).to(torch.bfloat16).to(DEV)
    w = torch.randn(H).to(torch.bfloat16).to(DEV)
    b = torch.randn(H).to(torch.bfloat16).to(DEV)
    assert _rel(ops.layernorm(x, w, b, 1e-5), ref.layernorm(x.float(), w.float(), b.float(), 1e-5)) < 5e-3
    gu = torch.randn(T, 2 * 1024).to(torch.bfloat16).to(DEV)
    for act in ("silu", "gelu_pytorch_tanh", "gelu"):
        assert _rel(ops.act_mul(gu, act), ref.act_mul(gu.float(), act)) < 5e-3
    assert _rel(ops.activation(x, "gelu_new"), ref.act_fn("gelu_new")(x.float())) < 5e-3
    table = torch.randn(500, H).to(torch.bfloat16).to(DEV)
    ids = torch.randint(0, 500, (T,), device=DEV)
    assert _rel(ops.embedding(table, ids, 3.0), table[ids].float() * 3.0) < 5e-3
    pos_t = torch.randn(64, H).to(torch.bfloat16).to(DEV)
    pos = torch.randint(0, 64, (T,), device=DEV)
    assert _rel(ops.embedding(table, ids, 1.0, pos_t, pos), table[ids].float() + pos_t[pos].float()) < 5e-3


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("qk_norm", [True, False])
def test_rope_kv(D, qk_norm):
    T, H, KV, page, pages = 45, 8, 2, 32, 16
    qkv = torch.randn(T, (H + 2 * KV) * D).to(torch.bfloat16).to(DEV)
    pos = torch.randint(0, 300, (T,), dtype=torch.int32, device=DEV)
    slots = torch.randperm(pages * page)[:T].to(torch.int64).to(DEV)
    cos, sin = ref.rope_tables(D, 512, 1e6)
    cos, sin = cos.to(DEV), sin.to(DEV)
    qn = (torch.randn(D) * 0.1 + 1).to(torch.bfloat16).to(DEV) if qk_norm else None
    kn = (torch.randn(D) * 0.1 + 1).to(torch.bfloat16).to(DEV) if qk_norm else None
    kc = torch.zeros(pages, KV, page, D, dtype=torch.bfloat16, device=DEV)
    vc = torch.zeros_like(kc)
    kc_r, vc_r = kc.clone().float(), vc.clone().float()
    q_r = ref.qk_prepare_and_cache(qkv.clone().float(), pos.long(), slots, H, KV, D, None if qn is None else qn.float(),
                                   None if kn is None else kn.float(), 1e-6, 0.0, cos, sin, kc_r, vc_r)
    q = ops.rope_kv(qkv, pos, slots, qn, kn, cos, sin, kc, vc, H, KV, D, 1e-6, 0.0)
    assert _rel(q, q_r.reshape(T, H * D)) < 1e-2
    assert _rel(kc, kc_r) < 1e-2 and _rel(vc, vc_r) < 1e-3


def _paged_setup(ctx_lens, KV, D, page=32, seed=0):
    g = torch.Generator().manual_seed(seed)
    n_pages = sum((c + page - 1) // page for c in ctx_lens) + 1
    kc = (torch.randn(n_pages, KV, page, D, generator=g) * 0.5).to(torch.bfloat16)
    vc = (torch.randn(n_pages, KV, page, D, generator=g) * 0.5).to(torch.bfloat16)
    width = max((c + page - 1) // page for c in ctx_lens)
    bt = torch.zeros(len(ctx_lens), width, dtype=torch.int32)
    perm = (torch.randperm(n_pages - 1, generator=g) + 1).tolist()
    for i, c in enumerate(ctx_lens):
        n = (c + page - 1) // page
        bt[i, :n] = torch.tensor([perm.pop() for _ in range(n)], dtype=torch.int32)
    return kc, vc, bt


@pytest.mark.parametrize("impl", [0, 1])
@pytest.mark.parametrize("D,H,KV", [(128, 32, 8), (64, 32, 4), (256, 16, 8), (128, 8, 8), (128, 14, 2), (64, 32, 2)])
@pytest.mark.parametrize("splits", [1, 4])
@pytest.mark.parametrize("softcap,window", [(0.0, 0), (50.0, 0), (0.0, 48)])
def test_decode_attention(D, H, KV, splits, softcap, window, impl):
    """impl 0 = tensor-core kernel (GQA group as MMA rows), impl 1 = CUDA-core kernel; both against the fp32 reference."""
    if impl == 1 and H // KV > 8:
        pytest.skip("the CUDA-core kernel covers groups of up to 8 heads")
    ctx = [1, 31, 32, 33, 100, 257, 700]
    kc, vc, bt = _paged_setup(ctx, KV, D)
    B = len(ctx)
    q = (torch.randn(B, H * D) * 0.5).to(torch.bfloat16)
    scale = 1.0 / math.sqrt(D)
    cl = torch.tensor(ctx, dtype=torch.int32)
    o_ref = ref.paged_attention(q.float().reshape(B, H, D), kc.float(), vc.float(), bt, torch.arange(B), torch.ones(B, dtype=torch.long),
                                cl, scale, softcap, window, True).reshape(B, H * D)
    o = ops.decode_attention(q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), cl.to(DEV), H, scale, softcap, window, splits, impl)
    assert _rel(o.cpu(), o_ref) < 1e-2


@pytest.mark.parametrize("D,H,KV,splits", [(128, 32, 8, 4), (64, 8, 4, 7), (256, 4, 2, 2), (128, 16, 1, 16)])
def test_decode_attention_merges_splits_in_kernel(D, H, KV, splits):
    """Split-KV decode, opt-in form: the CTA that finishes last for a (sequence, KV head) merges the splits itself. Same result as
    the merge in a second launch, bit-identical from launch to launch (the arrival counters return to zero), splits without keys included."""
    ctx = [1, 17, 64, 100, 257, 700, 1500]
    kc, vc, bt = _paged_setup(ctx, KV, D, seed=5)
    B = len(ctx)
    q = (torch.randn(B, H * D) * 0.5).to(torch.bfloat16)
    scale = 1.0 / math.sqrt(D)
    cl = torch.tensor(ctx, dtype=torch.int32)
    o_ref = ref.paged_attention(q.float().reshape(B, H, D), kc.float(), vc.float(), bt, torch.arange(B), torch.ones(B, dtype=torch.long),
                                cl, scale, 0.0, 0, True).reshape(B, H * D)
    args = (q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), cl.to(DEV), H, scale, 0.0, 0, splits, 0)
    o_two = ops.decode_attention(*args)
    ops.set_decode_merge_in_kernel(True)
    try:
        outs = [ops.decode_attention(*args) for _ in range(3)]
        torch.cuda.synchronize()
    finally:
        ops.set_decode_merge_in_kernel(False)
    assert _rel(outs[0].cpu(), o_ref) < 1e-2
    assert _rel(outs[0].cpu().float(), o_two.cpu().float()) < 4e-3
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


@pytest.mark.parametrize("D,H,KV", [(128, 8, 2), (64, 8, 4), (256, 4, 2)])
@pytest.mark.parametrize("softcap,window", [(0.0, 0), (50.0, 0), (0.0, 40)])
def test_prefill_attention(D, H, KV, softcap, window):
    # (q_len, ctx_len): fresh prompts, a chunk continuing a cached prefix, a single-row sequence
    seqs = [(70, 70), (64, 64), (5, 133), (130, 200), (1, 40)]
    ctx = [c for _, c in seqs]
    kc, vc, bt = _paged_setup(ctx, KV, D, seed=3)
    ql = [q for q, _ in seqs]
    T = sum(ql)
    qs = [sum(ql[:i]) for i in range(len(ql))]
    q = (torch.randn(T, H * D) * 0.5).to(torch.bfloat16)
    scale = 1.0 / math.sqrt(D)
    ti = lambda v: torch.tensor(v, dtype=torch.int32)  # noqa: E731
    o_ref = ref.paged_attention(q.float().reshape(T, H, D), kc.float(), vc.float(), bt, ti(qs), ti(ql), ti(ctx), scale, softcap, window,
                                True).reshape(T, H * D)
    o = ops.prefill_attention(q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), ti(qs).to(DEV), ti(ql).to(DEV), ti(ctx).to(DEV), H, scale,
                              softcap, window, True)
    assert _rel(o.cpu(), o_ref) < 1e-2


@pytest.mark.parametrize("D,H,KV,softcap,window", [(128, 8, 2, 0.0, 0), (64, 4, 4, 0.0, 0), (256, 4, 2, 30.0, 0), (128, 4, 1, 0.0, 100), (64, 8, 2, 50.0, 37)])
def test_prefill_attention_tcgen05(D, H, KV, softcap, window):
    """The tcgen05 / TMEM / TMA prefill kernel against the fp32 statement: several key tiles, a chunk continuing a cached prefix,
    ragged tails, GQA, soft-cap and sliding window; pages hold garbage beyond the context end (it must never reach the output)."""
    seqs = [(70, 70), (300, 300), (5, 133), (130, 500), (1, 40), (257, 257)]
    ctx = [c for _, c in seqs]
    kc, vc, bt = _paged_setup(ctx, KV, D, seed=3)
    ql = [q for q, _ in seqs]
    T = sum(ql)
    qs = [sum(ql[:i]) for i in range(len(ql))]
    q = (torch.randn(T, H * D) * 0.5).to(torch.bfloat16)
    scale = 1.0 / math.sqrt(D)
    ti = lambda v: torch.tensor(v, dtype=torch.int32)  # noqa: E731
    o_ref = ref.paged_attention(q.float().reshape(T, H, D), kc.float(), vc.float(), bt, ti(qs), ti(ql), ti(ctx), scale, softcap, window,
                                True).reshape(T, H * D)
    o = ops.prefill_attention(q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), ti(qs).to(DEV), ti(ql).to(DEV), ti(ctx).to(DEV), H, scale,
                              softcap, window, True, impl="tc")
    torch.cuda.synchronize()
    ops.check_status()
    assert _rel(o.cpu(), o_ref) < 1e-2, _rel(o.cpu(), o_ref)
    o2 = ops.prefill_attention(q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), ti(qs).to(DEV), ti(ql).to(DEV), ti(ctx).to(DEV), H, scale,
                               softcap, window, True, impl="mma")
    assert _rel(o.cpu(), o2.cpu()) < 1e-2


def test_argmax_and_logits_post():
    B, V = 5, 151936
    logits = torch.randn(B, V, device=DEV)
    logits[0, 77] = logits[0, 99999] = 50.0  # tie: the first maximum wins
    idx, val = ops.argmax(logits)
    assert idx.tolist() == torch.argmax(logits, dim=-1).tolist() and idx[0].item() == 77
    mask = torch.zeros(B, (V + 31) // 32, dtype=torch.int32, device=DEV)
    allowed = [5, 64, 31, 150000, 1]
    for b, t in enumerate(allowed):
        mask[b, t // 32] = 1 << (t % 32) if t % 32 != 31 else -(1 << 31)
    idx2, _ = ops.argmax(logits, mask)
    assert idx2.tolist() == allowed
    # 64 rows (two-stage path: several CTAs per row) and a short vocabulary (one CTA per row), values included
    for BB, VV in ((64, 151936), (130, 151936), (7, 1000)):
        lg = torch.randn(BB, VV, device=DEV)
        i3, v3 = ops.argmax(lg)
        assert torch.equal(i3, torch.argmax(lg, dim=-1)) and torch.allclose(v3, lg.max(dim=-1).values)
    l2 = logits.clone()
    ops.logits_post(l2, mask, 30.0, 0.5)
    exp = torch.tanh(logits * 0.5 / 30.0) * 30.0
    for b, t in enumerate(allowed):
        assert abs(l2[b, t].item() - exp[b, t].item()) < 1e-4
        assert torch.isinf(l2[b]).sum().item() == V - 1


def test_q4_quantize_bit_exact():
    g = torch.Generator().manual_seed(5)
    w = torch.randn(64, 256, generator=g) * 0.1
    w[3, 32:64] = 0.0
    w[5, 0] = -7.0
    p_ref, s_ref = q4_quantize(w)
    p, s = ops.q4_quantize(w.to(DEV))
    assert torch.equal(p.cpu(), p_ref)
    assert torch.equal(s.cpu().view(torch.int32), s_ref.view(torch.int32))
    wb = w.to(torch.bfloat16)
    p_ref, s_ref = q4_quantize(wb)
    p, s = ops.q4_quantize(wb.to(DEV))
    assert torch.equal(p.cpu(), p_ref) and torch.equal(s.cpu().view(torch.int32), s_ref.view(torch.int32))
    d = ops.require_ext().q4_dequantize(p, s, False)
    assert torch.equal(d.cpu(), q4_dequantize(p_ref, s_ref))


@pytest.mark.parametrize("V,peaked", [(1000, True), (32000, True), (151936, True), (151936, False), (4096, False)])
def test_sample_rows_kernel_matches_sorting_sampler(V, peaked):
    """Histogram-select sampling kernel against the sorting implementation (same uniforms): top-k limits, nucleus, uniform
    picks inside the nucleus, masked (-inf) tokens. Fixed-point weights may move a boundary pick: allow a tiny mismatch rate."""
    from deliverance_b200.engine.sampler import sample_top_k_top_p_batch

    g = torch.Generator().manual_seed(V + int(peaked))
    B = 96
    logits = torch.randn(B, V, generator=g) * (4.0 if peaked else 0.3)
    logits[:, ::7] = float("-inf")  # a guided mask
    logits[3, :] = float("-inf")
    logits[3, 5] = 1.0  # a single allowed token
    temps = torch.tensor([0.5, 0.8, 1.0, 1.3] * (B // 4))
    limits = torch.tensor([V, 50, 1, 1000, V, 7] * (B // 6), dtype=torch.int64).clamp(max=V)
    top_ps = torch.tensor([0.0, 0.1, 0.9, 0.5, 0.99, 0.0, 0.3, 1.0] * (B // 8))
    uniform = torch.tensor([False, False, False, True] * (B // 4))
    us = torch.rand(B, generator=g)
    want = sample_top_k_top_p_batch(logits, temps, limits, top_ps, uniform, us)
    e = ops.require_ext()
    tok, ok = e.sample_rows(logits.to(DEV), (1.0 / temps).to(DEV), limits.to(DEV), top_ps.to(DEV), uniform.to(torch.uint8).to(DEV), us.to(DEV))
    torch.cuda.synchronize()
    tok, ok = tok.cpu(), ok.cpu().bool()
    handled = int(ok.sum())
    assert handled >= (0.6 if peaked else 0.3) * B, handled  # flat rows without top-k may fall into the clamped tail
    agree = (tok[ok] == want[ok]).float().mean().item()
    assert agree >= 0.97, (agree, handled)
    assert tok[3].item() == 5 or not ok[3]
    # every handled pick is an allowed token inside the top-k set of its row
    for i in torch.nonzero(ok).flatten().tolist():
        assert logits[i, tok[i]] != float("-inf")
        kth = torch.topk(logits[i], int(limits[i])).values[-1]
        assert logits[i, tok[i]] >= kth


@pytest.mark.parametrize("M,I,K,q4,act", [(1, 256, 256, True, "silu"), (7, 512, 1024, True, "silu"), (64, 9728, 2560, True, "silu"),
                                           (64, 1216, 2560, True, "silu"), (33, 512, 768, False, "gelu_pytorch_tanh"),
                                           (200, 1024, 512, False, "silu"), (64, 19456, 2560, True, "silu")])
def test_gemm_epilogue_gated_activation(M, I, K, q4, act):
    """linear_act (rows interleaved per 64 outputs, act(gate) * up in the epilogue) against act_mul(linear) in fp32."""
    g = torch.Generator().manual_seed(I + K)
    wg, wu = torch.randn(I, K, generator=g) * 0.05, torch.randn(I, K, generator=g) * 0.05
    if q4:
        pg, sg = q4_quantize(wg)
        pu, su = q4_quantize(wu)
        wg, wu = q4_dequantize(pg, sg), q4_dequantize(pu, su)
        mixed = ops.interleave_gate_up(Q4Tensor(pg, sg, (I, K)), Q4Tensor(pu, su, (I, K)))
    else:
        wg, wu = wg.to(torch.bfloat16).float(), wu.to(torch.bfloat16).float()
        mixed = ops.interleave_gate_up(wg.to(torch.bfloat16), wu.to(torch.bfloat16))
    lw = LinearWeight(mixed).to(DEV, torch.bfloat16)
    x = (torch.randn(M, K, generator=g) * 0.5).to(torch.bfloat16)
    y = ops.linear_act(x.to(DEV), lw, act)
    torch.cuda.synchronize()
    ops.check_status()
    yr = ref.act_fn(act)(x.float() @ wg.t()) * (x.float() @ wu.t())
    assert y.shape == (M, I) and _rel(y.cpu(), yr) < 2e-2, _rel(y.cpu(), yr)
    assert torch.equal(y, ops.linear_act(x.to(DEV), lw, act))


@pytest.mark.parametrize("M,H,KV,K,q4,qk_norm,rot_half,bias", [(1, 4, 2, 256, True, True, 64, False), (7, 32, 8, 2560, True, True, 64, False),
                                                                (64, 32, 8, 2560, True, True, 64, False), (64, 4, 1, 2560, True, False, 64, True),
                                                                (200, 8, 2, 512, False, True, 64, True), (33, 4, 4, 4096, False, False, 64, False),
                                                                (529, 32, 8, 2560, True, True, 64, False), (700, 4, 2, 512, False, True, 64, False)])
def test_gemm_epilogue_rope_kv(M, H, KV, K, q4, qk_norm, rot_half, bias):
    """linear_rope_kv against the two separate kernels (projection, then rope_kv) on the same inputs: query heads and the
    written cache rows must agree up to the bf16 rounding of the intermediate tensor."""
    D, page = 128, 32
    g = torch.Generator().manual_seed(M + H)
    N = (H + 2 * KV) * D
    qt, wd = _q4_weight(N, K, seed=N + K)
    lw = (LinearWeight(qt) if q4 else LinearWeight(wd.to(torch.bfloat16))).to(DEV, torch.bfloat16)
    lw.bias = torch.randn(N, generator=g).to(DEV) * 0.1 if bias else None
    x = (torch.randn(M, K, generator=g) * 0.5).to(torch.bfloat16).to(DEV)
    pos = torch.randint(0, 500, (M,), generator=g).to(torch.int32).to(DEV)
    n_pages = (M + page - 1) // page + 2
    perm = torch.randperm(n_pages * page, generator=g)[:M].to(torch.int64).to(DEV)
    cos, sin = ref.rope_tables(D, 512, 10000.0, 1.0, rot_dim=2 * rot_half)
    cos, sin = cos.to(DEV), sin.to(DEV)
    qn = (1 + 0.1 * torch.randn(D, generator=g)).to(torch.bfloat16).to(DEV) if qk_norm else None
    kn = (1 + 0.1 * torch.randn(D, generator=g)).to(torch.bfloat16).to(DEV) if qk_norm else None
    caches = [torch.zeros(n_pages, KV, page, D, dtype=torch.bfloat16, device=DEV) for _ in range(4)]
    q_ref = ops.rope_kv(ops.linear(x, lw), pos, perm, qn, kn, cos, sin, caches[0], caches[1], H, KV, D, 1e-6, 0.0).clone()
    q = ops.linear_rope_kv(x, lw, pos, perm, qn, kn, cos, sin, caches[2], caches[3], H, KV, D, 1e-6, 0.0)
    torch.cuda.synchronize()
    ops.check_status()
    assert q.shape == (M, H * D) and _rel(q.float().cpu(), q_ref.float().cpu()) < 2e-2
    assert _rel(caches[2].float().cpu(), caches[0].float().cpu()) < 2e-2 and _rel(caches[3].float().cpu(), caches[1].float().cpu()) < 2e-2
    untouched = torch.ones(n_pages * page, dtype=torch.bool)
    untouched[perm.cpu()] = False
    assert caches[2].permute(0, 2, 1, 3).reshape(n_pages * page, -1)[untouched].abs().sum() == 0  # no stray cache rows


def test_bounded_peer_wait_runs_out_and_context_survives():
    """A peer-flag wait that nobody satisfies: the kernel gives up after its limit, records status 2 and returns; nothing
    faults and the same context runs the next kernel normally. The "peer" is a second receive area and flag matrix in this GPU's
    own memory that no kernel ever publishes to (a two-rank layout seen from rank 0 with rank 1 absent)."""
    e = ops.require_ext()
    rows, H, ncta = 4, 256, 256
    slab = rows * H
    recv = [torch.zeros(2 * 2 * slab, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    flags = [torch.zeros(2 * ncta, dtype=torch.int32, device=DEV) for _ in range(2)]
    rounds = torch.zeros(ncta, dtype=torch.int32, device=DEV)
    call = torch.zeros(2, dtype=torch.int32, device=DEV)
    comm = e.TpComm(0, 2, [t.data_ptr() for t in recv], [t.data_ptr() for t in flags], slab, ncta, rounds, call)
    comm.set_wait_limit_ms(2.0)
    ops.check_status()  # clear
    x = torch.randn(rows, H, device=DEV).to(torch.bfloat16)
    out = torch.zeros_like(x)
    t0 = time.perf_counter()
    assert e.oneshot_allreduce(x, comm, out)
    torch.cuda.synchronize()
    assert time.perf_counter() - t0 < 5.0
    with pytest.raises(RuntimeError, match="peer-flag wait"):
        ops.check_status()
    assert out.float().abs().sum().item() == 0.0  # a CTA whose wait ran out writes no result
    assert flags[1][:rows].tolist() == [1] * rows  # rank 0 did publish to the absent peer
    ops.check_status()  # the status word was consumed
    # the context is intact: an ordinary GEMM on the same device gives the right answer
    qt, wd = _q4_weight(256, 512, seed=1)
    lw = LinearWeight(qt).to(DEV, torch.bfloat16)
    xx = (torch.randn(8, 512) * 0.5).to(torch.bfloat16)
    y = ops.linear(xx.to(DEV), lw)
    torch.cuda.synchronize()
    ops.check_status()
    assert _rel(y.float().cpu(), xx.float() @ wd.t()) < 2e-2


@pytest.mark.parametrize("M,H,KV,D,hidden,inter,qk_norm,off,act", [
    (1, 4, 2, 128, 512, 1024, True, 0.0, "silu"), (7, 4, 2, 128, 512, 1024, True, 0.0, "silu"),
    (33, 8, 2, 64, 512, 768, False, 1.0, "gelu_pytorch_tanh"), (64, 16, 4, 64, 1024, 1536, False, 0.0, "silu"),
    (64, 32, 8, 128, 2560, 9728, True, 0.0, "silu"), (8, 32, 8, 128, 2560, 9728, True, 0.0, "silu")])
def test_decode_chain_matches_separate_kernels(M, H, KV, D, hidden, inter, qk_norm, off, act):
    """One persistent launch (o_proj -> add + norm -> gate|up -> act * up -> down -> add + norm -> q|k|v -> norm / rotary / KV write)
    against the same steps as separate kernels; every buffer the chain writes is compared, rows beyond M must stay untouched."""
    e = ops.require_ext()
    g = torch.Generator().manual_seed(M + hidden)
    page, R = 32, 64
    eps = 1e-6

    def lin(N, K, seed, bias=False):
        qt, _ = _q4_weight(N, K, seed=seed)
        lw = LinearWeight(qt).to(DEV, torch.bfloat16)
        lw.bias = (torch.randn(N, generator=g) * 0.1).to(DEV) if bias else None
        return lw

    w_o, w_gu, w_dn, w_qkv = lin(hidden, H * D, 1), lin(2 * inter, hidden, 2), lin(hidden, inter, 3), lin((H + 2 * KV) * D, hidden, 4, bias=not qk_norm)

    def nw(n):
        return (1 + 0.1 * torch.randn(n, generator=g)).to(torch.bfloat16).to(DEV)

    n1, n2 = nw(hidden), nw(hidden)
    qn, kn = (nw(D), nw(D)) if qk_norm else (None, None)
    cos, sin = ref.rope_tables(D, 512, 10000.0, 1.0)
    cos, sin = cos.to(DEV), sin.to(DEV)
    attn = (torch.randn(R, H * D, generator=g) * 0.5).to(torch.bfloat16).to(DEV)
    res0 = (torch.randn(R, hidden, generator=g) * 0.5).to(torch.bfloat16).to(DEV)
    pos = torch.randint(0, 500, (M,), generator=g).to(torch.int32).to(DEV)
    n_pages = 4
    slots = torch.randperm(n_pages * page, generator=g)[:M].to(torch.int64).to(DEV)
    caches = [torch.zeros(n_pages, KV, page, D, dtype=torch.bfloat16, device=DEV) for _ in range(4)]
    # ---- separate kernels ----
    res_ref = res0[:M].clone()
    x1 = ops.add_rmsnorm(ops.linear(attn[:M], w_o), res_ref, n1, eps, off, 1.0)
    res_mid = res_ref.clone()
    hh = ops.act_mul(ops.linear(x1, w_gu), act)
    x2 = ops.add_rmsnorm(ops.linear(hh, w_dn), res_ref, n2, eps, off, 1.0)
    q_ref = ops.rope_kv(ops.linear(x2, w_qkv), pos, slots, qn, kn, cos, sin, caches[0], caches[1], H, KV, D, eps, off).clone()
    # ---- one launch ----
    res = res0.clone()
    bx1, bh, bx2, bq = (torch.full((R, n), 7.0, dtype=torch.bfloat16, device=DEV) for n in (hidden, inter, hidden, H * D))
    poison = [torch.full((n,), float("nan"), device=DEV) for n in (1 << 22, 1 << 21, 1 << 20, 1 << 22)]
    del poison  # the chain's workspaces come from the allocator's cache: a slot that is read but never written shows up as NaN
    ch = e.DecodeChain()
    ch.add_op(w_o.handle(), attn, 1, residual=res, norm_w=n1, out=bx1, eps=eps, offset=off)
    ch.add_op(w_gu.handle(), bx1, 2, dep=True, scale_src=0, out=bh, act=act)
    ch.add_op(w_dn.handle(), bh, 1, dep=True, residual=res, norm_w=n2, out=bx2, eps=eps, offset=off)
    ch.add_op(w_qkv.handle(), bx2, 3, dep=True, scale_src=2, bias=w_qkv.bias, out=bq)
    ch.set_qkv(qn, kn, cos, sin, caches[2], caches[3], H, KV, eps, off)
    for rep in range(2):  # the second launch finds the counters the first one left (zero) and gives the same result
        res.copy_(res0)
        ch.run(M, pos, slots)
        torch.cuda.synchronize()
        ops.check_status()
        assert ch.counters().abs().sum().item() == 0
        # the norm stages hand on residual * weight; the row factor is applied behind the next projection
        x1u = (res_mid.float() * (n1.float() + off)).to(torch.bfloat16)
        x2u = (res_ref.float() * (n2.float() + off)).to(torch.bfloat16)
        rels = {"x1": _rel(bx1[:M], x1u), "h": _rel(bh[:M], hh), "residual": _rel(res[:M], res_ref), "x2": _rel(bx2[:M], x2u),
                "q": _rel(bq[:M], q_ref), "k_cache": _rel(caches[2], caches[0]), "v_cache": _rel(caches[3], caches[1])}
        assert all(v < 2e-2 for v in rels.values()), rels
        if M < R:
            assert (bx1[M:] == 7.0).all() and (bh[M:] == 7.0).all() and (bq[M:] == 7.0).all() and torch.equal(res[M:], res0[M:])
    first = bq[:M].clone()
    res.copy_(res0)
    ch.run(M, pos, slots)
    torch.cuda.synchronize()
    assert torch.equal(first, bq[:M])  # fixed summation order: bit-identical repeats


def test_xtc_and_logprob_kernels_match_torch():
    """xtc_rows against the row-by-row torch statement of exclude-top-choice, logprob_rows against logsumexp / topk."""
    from deliverance_b200.engine.sampler import xtc_pick

    e = ops.require_ext()
    g = torch.Generator().manual_seed(5)
    B, V = 9, 5000
    logits = torch.randn(B, V, generator=g) * 3
    logits[2, 77] = 30.0  # one dominant token: nothing else is above the threshold
    logits[4, :] = float("-inf")
    logits[4, 10:14] = torch.tensor([1.0, 1.0, 0.5, 2.0])  # ties above the threshold: the first index wins
    temps = [1.0, 0.7, 1.0, 1.3, 1.0, 1.0, 0.5, 1.0, 1.0]
    thr = [0.001, 0.01, 0.1, 0.0005, 0.1, 0.002, 0.01, 0.5, 0.001]
    fire = [1, 1, 1, 1, 1, 0, 1, 1, 1]
    special = [int(torch.argmax(logits[8]))]  # row 8: the top token is special and is returned as is
    got = e.xtc_rows(logits.to(DEV), torch.tensor([1 / t for t in temps], device=DEV), torch.tensor(thr, device=DEV),
                     torch.tensor(fire, dtype=torch.uint8, device=DEV), torch.tensor(special, dtype=torch.int32, device=DEV)).cpu().tolist()
    for b in range(B):
        want = xtc_pick(logits[b] / temps[b], thr[b], 1.0 if fire[b] else 0.0, 0.5, frozenset(special))
        assert got[b] == (-1 if want is None else want), (b, got[b], want)
    assert got[8] == special[0] and got[5] == -1 and got[4] == 12
    # log-probabilities
    lg = logits.clone()
    lg[4, :] = torch.randn(V, generator=g)
    chosen = torch.randint(0, V, (B,), generator=g)
    lp, ti, tv = e.logprob_rows(lg.to(DEV), chosen.to(DEV), 5)
    lse = torch.logsumexp(lg, dim=-1)
    assert torch.allclose(lp.cpu(), lg.gather(1, chosen.unsqueeze(1)).squeeze(1) - lse, atol=1e-4)
    wv, wi = torch.topk(lg, 5, dim=-1)
    assert torch.equal(ti.cpu(), wi) and torch.allclose(tv.cpu(), wv - lse.unsqueeze(1), atol=1e-4)
    lp0, ti0, _ = e.logprob_rows(lg.to(DEV), chosen.to(DEV), 0)
    assert torch.allclose(lp0.cpu(), lp.cpu()) and ti0.shape == (B, 0)


def test_lora_pool_softmax_turboquant_kernels():
    """The small device kernels off the hot path against their PyTorch statements."""
    from deliverance_b200.embedding import SentenceTransformersPooling as P
    from deliverance_b200.kv.turboquant import MseTurboQuantCodec

    e = ops.require_ext()
    g = torch.Generator().manual_seed(11)
    # LoRA delta
    M, K, N, r = 37, 512, 768, 16
    x = (torch.randn(M, K, generator=g) * 0.5).to(torch.bfloat16)
    A = (torch.randn(r, K, generator=g) * 0.1).to(torch.bfloat16)
    B = (torch.randn(N, r, generator=g) * 0.1).to(torch.bfloat16)
    y0 = (torch.randn(M, N, generator=g)).to(torch.bfloat16)
    y = y0.clone().to(DEV)
    e.lora_delta(x.to(DEV), A.to(DEV), B.to(DEV), y)
    want = y0.float() + (x.float() @ A.float().t()) @ B.float().t()
    assert _rel(y.cpu(), want) < 1e-2
    # pooling
    H = 384
    lens = [5, 1, 40, 17]
    starts = [0, 5, 6, 46]
    h = (torch.randn(sum(lens), H, generator=g)).to(torch.bfloat16)
    modes = {0: P.MEAN, 1: P.MAX, 3: P.CLS, 4: P.LAST_TOKEN, 5: P.MEAN_SQRT_LEN, 6: P.WEIGHTED_MEAN}
    for mode, pool in modes.items():
        for norm in (False, True):
            got = e.pool_rows(h.to(DEV), torch.tensor(starts, dtype=torch.int32, device=DEV), torch.tensor(lens, dtype=torch.int32, device=DEV), mode, norm).cpu()
            for s, (a, n) in enumerate(zip(starts, lens)):
                w = pool.pool(h[a:a + n].float())
                if norm:
                    w = w / w.norm().clamp_min(1e-12)
                assert torch.allclose(got[s], w, atol=2e-3, rtol=1e-3), (mode, norm, s)
    got = e.pool_rows(h.to(DEV), torch.tensor(starts, dtype=torch.int32, device=DEV), torch.tensor(lens, dtype=torch.int32, device=DEV), 2, False).cpu()
    assert torch.allclose(got[2], h[6:46].float().sum(0), atol=1e-2)
    # softmax
    lg = torch.randn(3, 7, generator=g) * 4
    assert torch.allclose(e.softmax_rows(lg.to(DEV)).cpu(), torch.softmax(lg, -1), atol=1e-6)
    # TurboQuant: device codes against the host codec (a coordinate on a bucket edge may differ by the summation order)
    for dim, bits in ((128, 3), (64, 4), (96, 2), (256, 8)):
        codec = MseTurboQuantCodec(dim, bits)
        rows = (torch.randn(50, dim, generator=g) * 2).to(torch.bfloat16)
        host = codec.encode(rows.float())
        dev_enc = codec.encode(rows.to(DEV))
        assert dev_enc.codes.shape == host.codes.shape and torch.allclose(dev_enc.norms, host.norms, rtol=1e-4)
        assert (dev_enc.codes != host.codes).float().mean().item() < 0.01
        back_host = codec.decode(host)
        back_dev = codec.decode(host, torch.float32, DEV).cpu()
        assert torch.allclose(back_dev, back_host, atol=1e-3, rtol=1e-3)
        assert _rel(codec.decode(dev_enc, torch.bfloat16, DEV).cpu(), rows) < (0.6 if bits <= 2 else 0.25)


def test_outputs_stay_inside_their_guard_areas():
    """Bounds checking: every output sits between two 4 KB guard areas; after a sweep over ragged shapes (token counts around the
    tile sizes, ragged prefill, split decode attention, norms, fused activation) no guard byte has changed. The checker itself
    is shown to see a changed byte (written from the host, no kernel misbehaves)."""
    ext = ops.require_ext()
    ops.set_bounds_check(True)
    try:
        g = torch.Generator().manual_seed(2)
        N, K = 384, 256
        w = torch.randn(N, K, generator=g) * 0.05
        p, s = q4_quantize(w)
        lw_q = LinearWeight(Q4Tensor(p, s, (N, K))).to(DEV)
        lw_d = LinearWeight(w.to(torch.bfloat16).to(DEV))
        for M in (1, 5, 17, 63, 65, 129, 257, 529):
            x = (torch.randn(M, K, generator=g) * 0.5).to(torch.bfloat16).to(DEV)
            ops.linear(x, lw_q)
            ops.linear(x, lw_d)
            ops.linear(x, lw_q, out_f32=True)
            ops.linear_act(x, lw_q, "silu")
            wn = torch.ones(K, dtype=torch.bfloat16, device=DEV)
            ops.rmsnorm(x, wn, 1e-6)
            ops.add_rmsnorm(x, x.clone(), wn, 1e-6)
        D, H, KV = 128, 8, 2
        seqs = [(70, 70), (5, 133), (257, 257)]
        ctx = [c for _, c in seqs]
        kc, vc, bt = _paged_setup(ctx, KV, D, seed=5)
        ql = [q for q, _ in seqs]
        T = sum(ql)
        qs = [sum(ql[:i]) for i in range(len(ql))]
        q = (torch.randn(T, H * D, generator=g) * 0.5).to(torch.bfloat16).to(DEV)
        ti = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
        for impl in ("tc", "mma"):
            ops.prefill_attention(q, kc.to(DEV), vc.to(DEV), bt.to(DEV), ti(qs), ti(ql), ti(ctx), H, 0.09, 0.0, 0, True, impl=impl)
        B = len(ctx)
        qd = (torch.randn(B, H * D, generator=g) * 0.5).to(torch.bfloat16).to(DEV)
        for splits in (1, 4):
            ops.decode_attention(qd, kc.to(DEV), vc.to(DEV), bt.to(DEV), ti(ctx), H, 0.09, 0.0, 0, splits)
        torch.cuda.synchronize()
        ops.check_status()
        ops.check_guards()
        # the checker sees a changed guard byte
        ops.rmsnorm(x, wn, 1e-6)
        ext.poke_last_guard()
        with pytest.raises(RuntimeError, match="wrote outside"):
            ops.check_guards()
    finally:
        ops.set_bounds_check(False)


@pytest.mark.parametrize("bn", [128, 256])
@pytest.mark.parametrize("q4", [True, False])
def test_linear_prefill_token_tiles(bn, q4):
    """Every token tile the prefill-size GEMM can pick (128 / 256 tokens) against the
    fp32 product, with token counts that end inside a tile."""
    ext = ops.require_ext()
    g = torch.Generator().manual_seed(bn)
    N, K = 640, 1152
    w = torch.randn(N, K, generator=g) * 0.05
    if q4:
        p, s = q4_quantize(w)
        lw, wd = LinearWeight(Q4Tensor(p, s, (N, K))).to(DEV), q4_dequantize(p, s)
    else:
        lw, wd = LinearWeight(w.to(torch.bfloat16).to(DEV)), w.to(torch.bfloat16).float()
    ext.gemm_force_bn(bn)
    try:
        for M in (129, 192, 193, 500, 1024):
            x = (torch.randn(M, K, generator=g) * 0.5).to(torch.bfloat16)
            y = ops.linear(x.to(DEV), lw)
            torch.cuda.synchronize()
            ops.check_status()
            assert _rel(y.cpu().float(), x.float() @ wd.t()) < 1e-2, (bn, M)
    finally:
        ext.gemm_force_bn(0)


@pytest.mark.parametrize("split", [0, 4, 8, 16])
@pytest.mark.parametrize("N,K", [(2560, 4096), (384, 256), (200, 1152), (6144, 2560)])
def test_small_batch_gemv_matches_fp32(N, K, split):
    """1..16 token rows of a JQ4 projection on the mma.sync GEMV: plain (bf16 and fp32 output, bias), gated activation epilogue, and
    agreement with the tcgen05 kernel it replaces at these sizes; every number of K-splitting warps per CTA (0: chosen per shape)."""
    ext = ops.require_ext()
    ext.gemv_force_split(split)
    ops.set_gemv_max_rows(16)  # the two-group form (9..16 rows) is covered too; by default it takes up to 8
    try:
        _small_batch_gemv_case(ext, N, K)
    finally:
        ext.gemv_force_split(0)
        ops.set_gemv_max_rows(8)


def _small_batch_gemv_case(ext, N, K):
    g = torch.Generator().manual_seed(N + K)
    w = torch.randn(N, K, generator=g) * 0.05
    p, s = q4_quantize(w)
    wd = q4_dequantize(p, s)
    bias = torch.randn(N, generator=g) * 0.1
    lw = LinearWeight(Q4Tensor(p, s, (N, K))).to(DEV)
    lwb = LinearWeight(Q4Tensor(p, s, (N, K)), bias=bias).to(DEV)
    for M in (1, 2, 5, 8, 9, 13, 16):
        x = (torch.randn(M, K, generator=g) * 0.5).to(torch.bfloat16)
        ref_y = x.float() @ wd.t()
        assert lw.handle().gemv_ok(M, K) and not lw.handle().gemv_ok(17, K)
        y = ops.linear(x.to(DEV), lw)
        y32 = ops.linear(x.to(DEV), lwb, out_f32=True)
        ext.gemv_dense(False)
        try:
            y_tc = ops.linear(x.to(DEV), lw)
        finally:
            ext.gemv_dense(True)
        torch.cuda.synchronize()
        ops.check_status()
        assert y32.dtype == torch.float32 and _rel(y.cpu().float(), ref_y) < 1e-2 and _rel(y32.cpu(), ref_y + bias) < 1e-2
        assert _rel(y.cpu().float(), y_tc.cpu().float()) < 1e-2
        if N % 32 == 0:
            h = ops.linear_gated(x.to(DEV), lw, "silu")
            gu = ref_y.to(torch.bfloat16).float()
            exp = torch.nn.functional.silu(gu[:, : N // 2]) * gu[:, N // 2:]
            assert tuple(h.shape) == (M, N // 2) and _rel(h.cpu().float(), exp) < 2e-2


@pytest.mark.parametrize("N,K,M", [(640, 1024, 500), (384, 512, 257), (2560, 4096, 2048), (200, 512, 1000)])
def test_persistent_prefill_gemm(N, K, M):
    """The persistent JQ4 GEMM (many tiles per CTA, epilogue under the next tile's main loop) against the fp32 product and against
    the one-tile-per-CTA kernel: bf16 and fp32 output, bias, ragged last token tile and last weight tile."""
    ext = ops.require_ext()
    g = torch.Generator().manual_seed(N + M)
    w = torch.randn(N, K, generator=g) * 0.05
    p, s = q4_quantize(w)
    wd = q4_dequantize(p, s)
    bias = torch.randn(N, generator=g) * 0.1
    lw = LinearWeight(Q4Tensor(p, s, (N, K))).to(DEV)
    lwb = LinearWeight(Q4Tensor(p, s, (N, K)), bias=bias).to(DEV)
    x = (torch.randn(M, K, generator=g) * 0.5).to(torch.bfloat16)
    ext.gemm_persist(False)
    try:
        y0 = ops.linear(x.to(DEV), lw)
        ext.gemm_persist(True, True, True)  # issuers in k-block order: repeated launches are bit-identical
        y = ops.linear(x.to(DEV), lw)
        y_again = ops.linear(x.to(DEV), lw)
        y32 = ops.linear(x.to(DEV), lwb, out_f32=True)
        ext.gemm_persist(True, True, False)  # racing issuers: same product up to the accumulation order
        y_race = ops.linear(x.to(DEV), lw)
        torch.cuda.synchronize()
        ops.check_status()
    finally:
        ext.gemm_persist(False)
    assert torch.equal(y, y_again)
    assert _rel(y_race.cpu().float(), y.cpu().float()) < 1e-2
    ref_y = x.float() @ wd.t()
    assert _rel(y.cpu().float(), ref_y) < 1e-2 and _rel(y32.cpu(), ref_y + bias) < 1e-2
    assert _rel(y.cpu().float(), y0.cpu().float()) < 1e-2


# The pair kernel rounds its fp32 sums to bf16 once: 2^-8 of a value at most, about 1.7e-3 in the 2-norm; JQ4 weights are products rounded to
# bf16 twice on top (scale, then nibble times scale): another 1.4e-3. 4e-3 holds both.
@pytest.mark.parametrize("M,N,K", [(1, 256, 64), (255, 264, 64), (257, 520, 192), (300, 512, 2592), (1030, 1096, 416), (2049, 512, 1280)])
@pytest.mark.parametrize("q4", [True, False])
def test_pair_gemm_edges(M, N, K, q4):
    """One row, ragged last token and weight tiles, one k step, k that ends inside a step, more tiles than pairs of SMs; bias; repeatable."""
    qt, wd = _q4_weight(N, K, seed=N + K)
    lw = (LinearWeight(qt) if q4 else LinearWeight(wd.to(torch.bfloat16))).to(DEV, torch.bfloat16)
    lw.bias = torch.randn(N, device=DEV) if M % 2 else None
    x = (torch.randn(M, K) * 0.5).to(torch.bfloat16).to(DEV)
    y, again = ops.linear(x, lw, impl=3), ops.linear(x, lw, impl=3)
    torch.cuda.synchronize()
    ops.check_status()
    yr = x.double().cpu() @ (wd if q4 else wd.to(torch.bfloat16)).double().t() + (lw.bias.double().cpu() if lw.bias is not None else 0.0)
    assert torch.equal(y, again) and _rel(y.cpu(), yr) < 4e-3


@pytest.mark.parametrize("M,N,K", [(255, 264, 64), (257, 520, 192), (300, 1408, 2592)])
def test_pair_gemm_room_is_guarded(M, N, K):
    """The bf16 form of a JQ4 weight lies between guard areas like an output: the newest guarded buffer of a product with an output of the caller's. Ragged
    rows and k of the weight write nothing beside it."""
    ext = ops.require_ext()
    qt, _ = _q4_weight(N, K, seed=N + K)
    lw = LinearWeight(qt).to(DEV, torch.bfloat16)
    x, out = torch.randn(M, K).to(torch.bfloat16).to(DEV), torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    ops.set_bounds_check(True)
    try:
        ops.linear(x, lw, impl=3, out=out)
        torch.cuda.synchronize()
        ops.check_guards()
        ops.linear(x, lw, impl=3, out=out)
        ext.poke_last_guard()
        with pytest.raises(RuntimeError, match=f"{2 * N * K}"):
            ops.check_guards()
        if lw.handle().run_gated(x, 1, 3) is not None:
            ops.check_guards()
    finally:
        ops.set_bounds_check(False)


def test_pair_gemm_without_room():
    """A JQ4 weight whose bf16 form finds no memory: products run as they do without the pair kernel, which needs none. (The allocator's limit is what
    refuses; the GPU has plenty.)"""
    M, N, K, H, KV = 2048, 8192, 4096, 48, 8
    qt, _ = _q4_weight(N, K, seed=3)
    lw = LinearWeight(qt).to(DEV, torch.bfloat16)
    x = (torch.randn(M, K) * 0.5).to(torch.bfloat16).to(DEV)
    pos = torch.arange(M, dtype=torch.int32, device=DEV)
    cos, sin = (t.to(DEV) for t in ref.rope_tables(128, M, 10000.0))
    out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)

    def products(kc, vc):
        ops.linear(x, lw, out=out)
        sums = out.cpu()
        gated = ops.linear_gated(x, lw, "silu").cpu()
        q = ops.linear_rope_kv(x, lw, pos, pos.long(), None, None, cos, sin, kc, vc, H, KV, 128, 1e-6)
        return [sums, gated, q.cpu(), kc.cpu(), vc.cpu()]

    caches = lambda: [torch.zeros(M // 32, KV, 32, 128, dtype=torch.bfloat16, device=DEV) for _ in range(2)]  # noqa: E731
    ops.linear(x[:256], lw)  # (workspaces)
    try:
        ops.set_gemm_pairs(0)
        want = products(*caches())
        ops.set_gemm_pairs(-1)
        kv = caches()
        torch.cuda.empty_cache()
        before = torch.cuda.memory_stats()["num_ooms"]
        # enough for the 32 MB output of a product with its 16 MB activation, not for the 64 MB of the weight
        total = torch.cuda.get_device_properties(0).total_memory
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (56 << 20)) / total)
        got = products(*kv)
        refused = torch.cuda.memory_stats()["num_ooms"] - before
        with pytest.raises(RuntimeError):
            ops.linear(x, lw, impl=3, out=out)
        torch.cuda.synchronize()
        ops.check_status()
    finally:
        ops.set_gemm_pairs(-1)
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert refused >= 3
    for a, b in zip(got, want):
        assert _rel(a, b) < 1e-6  # (the same kernels)


@pytest.mark.parametrize("M,N,K,ldx,ldo", [(300, 520, 192, 200, 528), (1030, 1096, 416, 424, 1104)])
@pytest.mark.parametrize("q4", [True, False])
def test_pair_gemm_strided(M, N, K, ldx, ldo, q4):
    """Rows of x and of the output that are parts of wider ones: what lies between them stays as it was. An output that is not 16-byte aligned is refused
    when the pair kernel is asked for and left to the one-tile kernel otherwise; x that is not aligned is refused by both."""
    qt, wd = _q4_weight(N, K, seed=N + K)
    lw = (LinearWeight(qt) if q4 else LinearWeight(wd.to(torch.bfloat16))).to(DEV, torch.bfloat16)
    wide, room = (torch.randn(M, ldx) * 0.5).to(torch.bfloat16).to(DEV), torch.full((M, ldo), 7.0, dtype=torch.bfloat16, device=DEV)
    x = wide[:, :K]
    yr = x.double().cpu() @ (wd if q4 else wd.to(torch.bfloat16)).double().t()
    ops.linear(x, lw, impl=3, out=room[:, :N])
    odd = torch.full((M, ldo), 7.0, dtype=torch.bfloat16, device=DEV)
    with pytest.raises(RuntimeError):
        ops.linear(x, lw, impl=3, out=odd[:, 4 : 4 + N])
    ops.linear(x, lw, out=odd[:, 4 : 4 + N])
    for impl in (0, 3):
        with pytest.raises(RuntimeError):
            ops.linear(wide[:, 4 : 4 + K], lw, impl=impl)
    torch.cuda.synchronize()
    ops.check_status()
    assert _rel(room[:, :N].cpu(), yr) < 4e-3 and bool((room[:, N:] == 7.0).all())
    assert _rel(odd[:, 4 : 4 + N].cpu(), yr) < 4e-3 and bool((odd[:, :4] == 7.0).all()) and bool((odd[:, 4 + N :] == 7.0).all())


@pytest.mark.parametrize("M,inter,K,act", [(1, 256, 64, "silu"), (255, 264, 128, "silu"), (2048, 256, 128, "silu"), (2100, 1408, 512, "gelu_pytorch_tanh"), (4097, 640, 320, "silu")])
@pytest.mark.parametrize("q4", [True, False])
def test_pair_gemm_gated(M, inter, K, act, q4):
    """One row, ragged last tiles of tokens and outputs, more tiles than pairs of SMs; halves of a JQ4 weight that do not end with a packed tile are refused."""
    qt, wd = _q4_weight(2 * inter, K, seed=inter)
    lw = (LinearWeight(qt) if q4 else LinearWeight(wd.to(torch.bfloat16))).to(DEV, torch.bfloat16)
    x = (torch.randn(M, K) * 0.5).to(torch.bfloat16).to(DEV)
    h = lw.handle().run_gated(x, ops.fused_act_kind(act), 3)
    assert (h is None) == (q4 and inter % 128 != 0)
    if h is None:
        h = ops.linear_gated(x, lw, act)
    torch.cuda.synchronize()
    ops.check_status()
    f = x.double().cpu() @ (wd if q4 else wd.to(torch.bfloat16)).double().t()
    assert _rel(h.cpu(), ref.act_fn(act)(f[:, :inter]) * f[:, inter:]) < 6e-3  # (without the epilogue the projection is rounded once more)


def test_pair_gemm_gated_ragged_rows_cost_no_more():
    """Rows that a last tile does not have cost no more than rows (measured: 1.75 times as long for 300 rows as for 512 when they did)."""
    lw = LinearWeight((torch.randn(11264, 2048) * 0.02).to(torch.bfloat16)).to(DEV, torch.bfloat16)
    h, x = lw.handle(), torch.randn(512, 2048).to(torch.bfloat16).to(DEV)

    def best(M):
        times = []
        for _ in range(12):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            for _ in range(5):
                h.run_gated(x[:M], 1, 3)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    assert best(300) < 1.25 * best(512)


@pytest.mark.parametrize("M", [1, 255, 257, 2310])
@pytest.mark.parametrize("heads,kv,norm,rope,bias", [(4, 1, True, True, False), (6, 3, False, True, True), (3, 1, True, False, True)])
@pytest.mark.parametrize("q4", [True, False])
def test_pair_gemm_heads(M, heads, kv, norm, rope, bias, q4):
    """q | k | v epilogue: an odd number of heads (half a tile at the end), rows without a cache slot, positions behind a prefix, bias; and the one-tile
    kernel on the same call."""
    K, D = 512, 128
    qt, wd = _q4_weight((heads + 2 * kv) * D, K, seed=heads)
    lw = (LinearWeight(qt) if q4 else LinearWeight(wd.to(torch.bfloat16))).to(DEV, torch.bfloat16)
    x = (torch.randn(M, K) * 0.5).to(torch.bfloat16).to(DEV)
    pages = M // 32 + 2
    slots = torch.randperm(pages * 32)[:M]
    slots[M // 3 :: 5] = -1
    used = torch.zeros(pages * 32, dtype=torch.bool)
    used[slots[slots >= 0]] = True
    slots = slots.to(DEV)
    pos = torch.arange(M, dtype=torch.int32, device=DEV) + 37
    cos, sin = (t.to(DEV) for t in ref.rope_tables(D, 4096, 10000.0)) if rope else (None, None)
    qn, kn = ((1 + 0.1 * torch.randn(D)).to(torch.bfloat16).to(DEV) for _ in range(2)) if norm else (None, None)
    b = torch.randn(wd.shape[0], device=DEV) if bias else None
    f = x.float() @ (wd if q4 else wd.to(torch.bfloat16).float()).to(DEV).t() + (b if bias else 0.0)
    k2, v2 = (torch.zeros(pages, kv, 32, D, device=DEV) for _ in range(2))
    scratch = torch.arange(M, device=DEV)  # (the oracle has no rows without a slot)
    qr = ref.qk_prepare_and_cache(f, pos.long(), scratch, heads, kv, D, qn, kn, 1e-6, 0.0, cos, sin, torch.zeros_like(k2), torch.zeros_like(v2))
    live = slots >= 0
    if bool(live.any()):
        ref.qk_prepare_and_cache(f[live], pos[live].long(), slots[live], heads, kv, D, qn, kn, 1e-6, 0.0, cos, sin, k2, v2)
    for impl in (3, 0):
        kc, vc = (torch.zeros(pages, kv, 32, D, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        q = lw.handle().run_qkv(x, pos, slots, qn, kn, cos, sin, kc, vc, heads, kv, 1e-6, 0.0, b, impl)
        torch.cuda.synchronize()
        ops.check_status()
        assert _rel(q, qr.reshape(M, -1)) < 6e-3
        for got, want in ((kc, k2), (vc, v2)):
            rows = got.permute(0, 2, 1, 3).reshape(pages * 32, -1).cpu()
            assert bool((rows[~used] == 0).all()) and (not bool(used.any()) or _rel(got, want) < 6e-3)


@pytest.mark.parametrize("D,T", [(64, 33), (128, 70), (256, 5)])
def test_rope_kv_unaligned_rows(D, T):
    """Rows that start on a 2-byte boundary take the element-wise form: as the wide one does, and nothing beside them changes."""
    H, KV, pages = 4, 2, T // 32 + 1
    n = T * (H + 2 * KV) * D
    base = torch.randn(n).to(torch.bfloat16).to(DEV)
    room = torch.full((n + 2,), 7.0, dtype=torch.bfloat16, device=DEV)
    odd = room[1 : 1 + n].view(T, -1)
    odd.copy_(base.view(T, -1))
    assert odd.data_ptr() % 8 == 2 and odd.is_contiguous()
    slots, pos = torch.randperm(pages * 32)[:T].to(DEV), torch.arange(T, dtype=torch.int32, device=DEV)
    cos, sin = (t.to(DEV) for t in ref.rope_tables(D, 128, 10000.0))
    w = (1 + 0.1 * torch.randn(D)).to(torch.bfloat16).to(DEV)
    got = []
    for t in (base.view(T, -1).clone(), odd):
        kc, vc = (torch.zeros(pages, KV, 32, D, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        ops.rope_kv(t, pos, slots, w, w, cos, sin, kc, vc, H, KV, D, 1e-6)
        got.append((t, kc, vc))
    torch.cuda.synchronize()
    assert all(_rel(a, b) < 1e-3 for a, b in zip(*got))  # (the sum of a head's squares is added in another order: a bf16 step here and there)
    assert room[0].item() == 7.0 and room[-1].item() == 7.0


@pytest.mark.parametrize("E,n,K,T,k", [(4, 512, 256, 700, 2), (3, 768, 1216, 1500, 1), (3, 512, 64, 900, 2), (40, 1280, 160, 9000, 2)])
@pytest.mark.parametrize("q4", [True, False])
def test_pair_gemm_experts(E, n, K, T, k, q4):
    """Work items of 256 rows that end inside a tile, unused ones at the end of the list; plain store and gated activation. K that ends in the
    first half of a packed stage, also with several tiles per pair of SMs and the step ring at every phase."""
    e = ops.require_ext()
    made = [_q4_weight(n, K, seed=i) for i in range(E)]
    g = ops.GroupedLinearWeight([(LinearWeight(qt) if q4 else LinearWeight(wd.to(torch.bfloat16))).to(DEV, torch.bfloat16) for qt, wd in made])
    x = (torch.randn(T, K) * 0.5).to(torch.bfloat16).to(DEV)
    w, idx, counts, offsets, perm, pos = e.moe_route(torch.randn(T, E, device=DEV), k, 0, True)
    items = e.moe_items(offsets, 0, E, 256, (T * k + 255) // 256 + E)
    xs = e.moe_gather(x, perm, k, None, 0, 0)
    y, h = g.run(xs, items, 256), g.run_gated(xs, items, "silu")
    torch.cuda.synchronize()
    ops.check_status()
    off = offsets.tolist()
    for i, (_, wd) in enumerate(made):
        f = xs[off[i]:off[i + 1]].double().cpu() @ (wd if q4 else wd.to(torch.bfloat16)).double().t()
        assert _rel(y[off[i]:off[i + 1]].cpu(), f) < 4e-3
        assert h is not None and _rel(h[off[i]:off[i + 1]].cpu(), torch.nn.functional.silu(f[:, : n // 2]) * f[:, n // 2:]) < 6e-3


@pytest.mark.parametrize("q4", [True, False])
def test_pair_gemm_limits(q4):
    """Products that the pair kernel is preferred for, with no pair (the one-tile kernel takes them all), with three, and with all of the GPU."""
    M, K, I, H, KV, E = 4096, 512, 1024, 16, 8, 3
    gate_up, heads = [_q4_weight(n, K, seed=n) for n in (2 * I, (H + 2 * KV) * 128)]
    a, b = [(LinearWeight(qt) if q4 else LinearWeight(wd.to(torch.bfloat16))).to(DEV, torch.bfloat16) for qt, wd in (gate_up, heads)]
    experts = [_q4_weight(2 * I, K, seed=i) for i in range(E)]
    g = ops.GroupedLinearWeight([(LinearWeight(qt) if q4 else LinearWeight(wd.to(torch.bfloat16))).to(DEV, torch.bfloat16) for qt, wd in experts])
    e = ops.require_ext()
    x = (torch.randn(M, K) * 0.5).to(torch.bfloat16).to(DEV)
    w, idx, counts, offsets, perm, pos = e.moe_route(torch.randn(M, E, device=DEV), 1, 0, True)
    items, xs = e.moe_items(offsets, 0, E, 256, M // 256 + E), e.moe_gather(x, perm, 1, None, 0, 0)
    cos, sin = (t.to(DEV) for t in ref.rope_tables(128, M, 10000.0))
    got = {}
    try:
        for n in (0, 3, -1):
            ops.set_gemm_pairs(n)
            kc, vc = (torch.zeros(M // 32, KV, 32, 128, dtype=torch.bfloat16, device=DEV) for _ in range(2))
            at = torch.arange(M, device=DEV)
            q = ops.linear_rope_kv(x, b, at.int(), at, None, None, cos, sin, kc, vc, H, KV, 128, 1e-6)
            gated, grouped = a.handle().run_gated(x, 1), g.run_gated(xs, items, "silu")
            assert (gated is None) == (grouped is None) == (n == 0)
            got[n] = [ops.linear(x, a), ops.linear_gated(x, a, "silu"), q, kc, vc, g.run(xs, items, 256)] + ([gated, grouped] if n else [])
            if n == 0:
                with pytest.raises(RuntimeError):
                    ops.linear(x, a, impl=3)
        torch.cuda.synchronize()
        ops.check_status()
    finally:
        ops.set_gemm_pairs(-1)
    for u, v in zip(got[3], got[-1]):
        assert torch.equal(u, v)
    for u, v in zip(got[0], got[-1]):  # (sums in another order, rounded to bf16 once or twice: about 1.7e-3 each in the 2-norm)
        assert _rel(u, v) < 6e-3


@pytest.mark.parametrize("B,H,KV,D", [(1, 8, 4, 64), (2, 32, 8, 128), (9, 16, 8, 256), (40, 16, 4, 128), (64, 8, 8, 64)])
@pytest.mark.parametrize("window,cap", [(0, 0.0), (100, 30.0)])
def test_decode_attention_used_splits(B, H, KV, D, window, cap):
    """Contexts around the lengths at which one more split is used (3 and 16 slices of 16 keys), for few and many (sequence, KV head) pairs; a batch
    mixes sequences that write their output alone with ones that are merged. bf16 probabilities and output: about 1.7e-3 each in the 2-norm."""
    lens = [1, 15, 16, 17, 47, 48, 49, 95, 97, 255, 257, 511, 513, 700, 1500]
    ctx = torch.tensor([lens[(7 * i) % len(lens)] for i in range(B)], dtype=torch.int32)
    per = [(int(c) + 31) // 32 for c in ctx]
    bt = torch.zeros(B, max(per), dtype=torch.int32)
    order = torch.randperm(sum(per)) + 1
    for i, n in enumerate(per):
        bt[i, :n] = order[sum(per[:i]):sum(per[:i]) + n]
    kc, vc = (torch.randn(sum(per) + 1, KV, 32, D).to(torch.bfloat16) for _ in range(2))
    q = torch.randn(B, H * D).to(torch.bfloat16)
    r = ref.paged_attention(q.reshape(B, H, D).float(), kc.float(), vc.float(), bt, torch.arange(B), torch.ones(B, dtype=torch.long), ctx, D**-0.5, cap, window)
    for splits in (1, 2, 9, 32):
        o = ops.decode_attention(q.to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), ctx.to(DEV), H, D**-0.5, cap, window, splits)
        torch.cuda.synchronize()
        d = (o.cpu().float() - r.reshape(B, -1)).reshape(B, -1).norm(dim=1) / r.reshape(B, -1).norm(dim=1)
        assert d.max().item() < 6e-3, (splits, d)


def _paged(ctx, KV, D, seed=0):
    """Random paged cache for sequences of these lengths: k, v, block table, context lengths on the GPU (page 0 is nobody's)."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    per = [(c + 31) // 32 for c in ctx]
    bt = torch.zeros(len(ctx), max(per), dtype=torch.int32)
    order = torch.randperm(sum(per), generator=torch.Generator().manual_seed(seed)).to(torch.int32) + 1
    for i, n in enumerate(per):
        bt[i, :n] = order[sum(per[:i]):sum(per[:i]) + n]
    kc, vc = (torch.randn(sum(per) + 1, KV, 32, D, device=DEV, generator=g, dtype=torch.bfloat16) for _ in range(2))
    return kc, vc, bt.to(DEV), torch.tensor(ctx, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("B,H,KV,D,short,long", [(40, 32, 8, 128, 200, 6000), (10, 32, 8, 128, 40, 3000), (130, 8, 4, 64, 64, 9000), (24, 16, 8, 256, 300, 5000)])
@pytest.mark.parametrize("window,cap", [(0, 0.0), (1000, 30.0)])
def test_decode_attention_one_long_sequence(B, H, KV, D, short, long, window, cap):
    """A batch whose pairs occupy the GPU unsplit, or nearly do, with one sequence many times longer than the others, padded sequences of one key among
    them: the long one is cut, whatever the batch. bf16 probabilities and output: about 1.7e-3 each in the 2-norm."""
    ctx = [short + (37 * i) % 50 for i in range(B)]
    ctx[B // 2] = long
    ctx[B - B // 8 :] = [1] * (B // 8)
    kc, vc, bt, cl = _paged(ctx, KV, D)
    q = torch.randn(B, H * D).to(torch.bfloat16).to(DEV)
    r = ref.paged_attention(q.reshape(B, H, D).float().cpu(), kc.float().cpu(), vc.float().cpu(), bt.cpu(), torch.arange(B), torch.ones(B, dtype=torch.long), cl.cpu(),
                            D**-0.5, cap, window)
    for splits, even in ((1, False), (3, False), (32, False), (9, True)):
        o = ops.decode_attention(q, kc, vc, bt, cl, H, D**-0.5, cap, window, splits, even=even)
        torch.cuda.synchronize()
        d = (o.cpu().float() - r.reshape(B, -1)).norm(dim=1) / r.reshape(B, -1).norm(dim=1)
        assert d.max().item() < 6e-3, (splits, even, d)


def test_decode_attention_long_sequence_is_cut():
    """The splits that a caller allows are used for a sequence that is much longer than the rest: its keys do not pass through one CTA per KV head
    (measured: 4.6 times as long at these sizes; two times are asked for)."""
    B, H, KV, D = 32, 32, 8, 128
    kc, vc, bt, cl = _paged([500] * (B - 1) + [24000], KV, D)
    q = torch.randn(B, H * D).to(torch.bfloat16).to(DEV)

    def best(splits):
        times = []
        for _ in range(8):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            ops.decode_attention(q, kc, vc, bt, cl, H, D**-0.5, 0.0, 0, splits)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    assert best(8) * 2 < best(1)


@pytest.mark.parametrize("lo,hi", [(4, 180), (184, 252), (256, 508)])
def test_decode_attention_softcap_error(lo, hi):
    """Probabilities of capped scores against 64 bits where a step of fp32 shows: a cap of 2^20, exact scores of lo / 512 to hi / 512 of it. The tensor-core
    kernel, which has a series for small scores, is no further off than the CUDA-core kernel, which calls tanhf for all."""
    D, n, cap = 64, 64, float(2**20)
    first = torch.arange(lo, hi + 1, 4).float()
    B = len(first)
    q, k = torch.zeros(B, D), torch.zeros(B, n, D)
    q[:, 0], q[:, 1] = 2048.0, 1.0
    k[:, :, 0], k[:, :, 1] = first[:, None], torch.arange(n) / 16.0
    kc, vc = (torch.cat([torch.zeros(1, 1, 32, D), t.reshape(2 * B, 1, 32, D)]).to(torch.bfloat16).to(DEV) for t in (k, torch.eye(D).repeat(B, 1)))
    bt = torch.arange(1, 1 + 2 * B, dtype=torch.int32, device=DEV).view(B, 2)
    cl = torch.full((B,), n, dtype=torch.int32, device=DEV)
    s = 2048.0 * k[:, :, 0].double() + k[:, :, 1].double()
    want = torch.log_softmax(cap * torch.tanh(s / cap), -1)
    err = []
    for impl in (0, 1):
        p = ops.decode_attention(q.to(torch.bfloat16).to(DEV), kc, vc, bt, cl, 1, 1.0, cap, 0, 1, impl)
        d = p.double().cpu().log() - want
        err.append((d - d.mean(1, keepdim=True)).pow(2).mean().sqrt().item())
    # (bf16 probabilities and outputs: about 0.0016 together in the 2-norm, in either kernel; the kernels round them in another order)
    assert err[0] < 1.1 * err[1] + 0.0016, err


@pytest.mark.parametrize("T", [1, 7, 1183, 1185])
@pytest.mark.parametrize("H", [8, 1024, 2048, 2056, 2560, 3584, 4096, 4104, 8192, 8200])
def test_rmsnorm_widths(T, H):
    """Both register forms and the loop behind them at the widths where they take over, with and without the residual."""
    x, res = ((torch.randn(T, H) * s).to(torch.bfloat16) for s in (1.0, 3.0))
    w = (torch.randn(H) * 0.1).to(torch.bfloat16)
    y = ops.rmsnorm(x.to(DEV), w.to(DEV), 1e-6, 1.0)
    got_res = res.to(DEV).clone()
    z = ops.add_rmsnorm(x.to(DEV), got_res, w.to(DEV), 1e-6, 0.0, 0.5)
    torch.cuda.synchronize()
    want_res = (res.float() + 0.5 * x.float()).to(torch.bfloat16)
    assert torch.equal(got_res.cpu(), want_res)
    assert _rel(y.cpu(), ref.rmsnorm(x.double(), w.double(), 1e-6, 1.0)) < 3e-3 and _rel(z.cpu(), ref.rmsnorm(want_res.double(), w.double(), 1e-6)) < 3e-3


@pytest.mark.parametrize("T,H", [(1, 8), (7, 8), (1, 1024), (7, 2056), (3, 4104), (1185, 8), (2, 8200)])
def test_rmsnorm_values(T, H):
    """Value by value: rows in which nothing averages the roundings out."""
    x, res = ((torch.randn(T, H) * s).to(torch.bfloat16) for s in (1.0, 3.0))
    w = (torch.randn(H) * 0.1).to(torch.bfloat16)
    got_res = res.to(DEV).clone()
    y, z = ops.rmsnorm(x.to(DEV), w.to(DEV), 1e-6, 1.0).cpu(), ops.add_rmsnorm(x.to(DEV), got_res, w.to(DEV), 1e-6, 0.0, 0.5).cpu()
    # in front of the rounding, in fp32: at most H / 32 squares added up by a thread and ten sums across threads (the root halves their error), then a division, a
    # reciprocal root, the weight's offset and two products
    slack = (H / 64 + 16) * 2.0**-24
    for got, want in ((y, ref.rmsnorm(x.double(), w.double(), 1e-6, 1.0)), (z, ref.rmsnorm(got_res.cpu().double(), w.double(), 1e-6))):
        assert _rounded_once(got, want, slack * want.abs())


def _row_slack(x, w, bias):
    """Error of the one-row GEMV's fp32 sums: products of bf16 are exact; a lane adds two in a row per 256 elements, two sums of its own follow, five across the warp and the
    bias. Relative to the sum of magnitudes, because a sum may cancel."""
    return (2 * -(-w.shape[1] // 256) + 9) * 2.0**-24 * (x.double().abs() @ w.double().abs().t() + bias.double().abs())


@pytest.mark.parametrize("N,K", [(5, 8), (130, 2040), (64, 2048), (33, 2056), (3, 5632)])
@pytest.mark.parametrize("f32", [True, False])
def test_gemv_bf16_row(N, K, f32):
    w, x = (torch.randn(N, K) * 0.05).to(torch.bfloat16), torch.randn(1, K).to(torch.bfloat16)
    bias = torch.randn(N)
    y = ops.linear(x.to(DEV), LinearWeight(w, bias).to(DEV, torch.bfloat16), out_f32=f32)
    torch.cuda.synchronize()
    assert _rel(y.cpu(), x.double() @ w.double().t() + bias.double()) < (1e-5 if f32 else 4e-3)


@pytest.mark.parametrize("N,K", [(1, 8), (5, 8), (7, 1024), (33, 2056), (300, 3080), (33, 14336), (60000, 1544)])
def test_gemv_bf16_values(N, K):
    """Value by value, with bias: single sums that may cancel."""
    w, x = (torch.randn(N, K) * 0.05).to(torch.bfloat16), torch.randn(1, K).to(torch.bfloat16)
    bias = torch.randn(N)
    lw = LinearWeight(w, bias).to(DEV, torch.bfloat16)
    y, y32 = ops.linear(x.to(DEV), lw).cpu(), ops.linear(x.to(DEV), lw, out_f32=True).cpu()
    want, slack = x.double() @ w.double().t() + bias.double(), _row_slack(x, w, bias)
    assert bool(((y32.double() - want).abs() <= slack).all()) and _rounded_once(y, want, slack)


# As for the pair kernel: fp32 sums rounded to bf16 once, JQ4 products rounded to bf16 twice on top.
@pytest.mark.parametrize("N,K", [(1, 8), (7, 1024), (2500, 1032), (5000, 256), (9, 2056), (2400, 2560), (300, 3080), (33, 14336), (57001, 64), (60000, 1544)])
def test_gemv_bf16_pieces(N, K):
    """Rows of one and several pieces, three to six of them in a warp's ring, fewer rows than warps, several rows per warp, more rows than resident CTAs take, and rows
    wider than a ring. fp32 sums, which bf16 outputs round once."""
    w = LinearWeight((torch.randn(N, K) * 0.05).to(torch.bfloat16)).to(DEV, torch.bfloat16)
    w.bias = torch.randn(N, device=DEV)
    x = torch.randn(1, K).to(torch.bfloat16).to(DEV)
    y, y32, again = ops.linear(x, w), ops.linear(x, w, out_f32=True), ops.linear(x, w)
    f = x.double() @ w.w.double().t() + w.bias.double()
    torch.cuda.synchronize()
    assert _rel(y32, f) < 1e-5 and torch.equal(y, y32.to(torch.bfloat16)) and torch.equal(y, again)


def test_first_product_of_a_fresh_weight():
    """Products directly behind the kernels that make the weight (a cast, a repack, a stack of experts), whose bytes they read ahead of their wait: the same as later."""
    x = torch.randn(1, 2048, device=DEV).to(torch.bfloat16)
    torch.cuda.synchronize()
    for i in range(20):
        w = LinearWeight(torch.randn(11264, 2048, device=DEV))
        q = LinearWeight(Q4Tensor(*q4_quantize(torch.randn(64, 2048)), (64, 2048)))
        first = [ops.linear(x, w), ops.linear(x, q.to(DEV, torch.bfloat16))]
        torch.cuda.synchronize()
        assert torch.equal(first[0], ops.linear(x, w)) and torch.equal(first[1], ops.linear(x, q.to(DEV, torch.bfloat16)))


@pytest.mark.parametrize("M,N,K", [(1, 64, 64), (31, 264, 128), (33, 136, 192), (256, 512, 1280), (257, 2560, 960), (385, 19456, 256), (700, 1000, 2624), (1537, 4104, 512)])
def test_parts_gemm_edges(M, N, K):
    """One row; k that ends inside a packed stage; weight tiles that end inside a tile and inside eight outputs; one and two instructions per tile, several tiles of
    tokens; tiles in equal parts, waves with parts behind them, waves alone; bias; fp32 outputs; repeatable. Rows that are parts of wider ones, with and without 16
    bytes at once: what lies beside them stays."""
    qt, wd = _q4_weight(N, K, seed=N + K)
    lw = LinearWeight(qt).to(DEV, torch.bfloat16)
    lw.bias = torch.randn(N, device=DEV) if M % 2 else None
    wide = (torch.randn(M, K + 8) * 0.5).to(torch.bfloat16).to(DEV)
    x = wide[:, :K]
    yr = x.double().cpu() @ wd.double().t() + (lw.bias.double().cpu() if lw.bias is not None else 0.0)
    y, again, y32 = ops.linear(x, lw, impl=4), ops.linear(x, lw, impl=4), ops.linear(x, lw, impl=4, out_f32=True)
    room = [torch.full((M, N + 24 - N % 8), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(3)]
    for at, t in zip((8, 4, 1), room):
        ops.linear(x, lw, impl=4, out=t[:, at : at + N])
    torch.cuda.synchronize()
    ops.check_status()
    assert torch.equal(y, again) and _rel(y.cpu(), yr) < 4e-3 and _rel(y32.cpu(), yr) < 4e-3
    for at, t in zip((8, 4, 1), room):
        assert torch.equal(t[:, at : at + N], y) and bool((t[:, :at] == 7.0).all()) and bool((t[:, at + N :] == 7.0).all())
    with pytest.raises(RuntimeError):
        ops.linear(wide[:, 4 : 4 + K], lw, impl=4)


def test_parts_gemm_refuses():
    """K that ends inside 64, bf16 weights, no pair of SMs: refused when asked for, left to the other kernels otherwise."""
    for qt, wd in (_q4_weight(512, 96),):
        lw, dense = LinearWeight(qt).to(DEV, torch.bfloat16), LinearWeight(wd.to(torch.bfloat16)).to(DEV, torch.bfloat16)
    ok = LinearWeight(_q4_weight(512, 128)[0]).to(DEV, torch.bfloat16)
    x, x2 = torch.randn(300, 96).to(torch.bfloat16).to(DEV), torch.randn(300, 128).to(torch.bfloat16).to(DEV)
    for w in (lw, dense):
        with pytest.raises(RuntimeError):
            ops.linear(x, w, impl=4)
        assert w.handle().run_gated(x, 1, 4) is None and _rel(ops.linear(x, w).cpu(), x.float().cpu() @ wd.t()) < 1e-2
    try:
        ops.set_gemm_pairs(0)
        with pytest.raises(RuntimeError):
            ops.linear(x2, ok, impl=4)
        one = ops.linear(x2, ok)
        ops.set_gemm_pairs(3)
        few = ops.linear(x2, ok, impl=4)
    finally:
        ops.set_gemm_pairs(-1)
    assert _rel(one, few) < 6e-3


@pytest.mark.parametrize("M,inter,K,act", [(1, 64, 64, "silu"), (65, 192, 128, "gelu_pytorch_tanh"), (333, 9728, 320, "silu"), (513, 4096, 64, "silu"), (1100, 1408, 512, "gelu_pytorch_tanh")])
def test_parts_gemm_gated(M, inter, K, act):
    """Halves of an odd number of 64 rows, tiles in parts, parts behind waves, guard areas around output and sums."""
    qt, wd = _q4_weight(2 * inter, K, seed=inter)
    lw = LinearWeight(qt).to(DEV, torch.bfloat16)
    x = (torch.randn(M, K) * 0.5).to(torch.bfloat16).to(DEV)
    ops.set_bounds_check(True)
    try:
        h = lw.handle().run_gated(x, ops.fused_act_kind(act), 4)
        torch.cuda.synchronize()
        ops.check_guards()
    finally:
        ops.set_bounds_check(False)
    ops.check_status()
    f = x.double().cpu() @ wd.double().t()
    assert _rel(h.cpu(), ref.act_fn(act)(f[:, :inter]) * f[:, inter:]) < 6e-3


@pytest.mark.parametrize("q4", [True, False])
def test_parts_gemm_gated_far_below_zero(q4):
    """SiLU of gates around -88, where 1 + exp(-g) passes 2^126 but is a number still: the activation is small, its product with a large up row is not. As the activation kernel
    has it, one rounding apart."""
    inter, K, M = 128, 64, 4
    w = torch.zeros(2 * inter, K)
    w[:inter, 0], w[inter:, 1] = torch.linspace(-88.5, -86.0, inter).to(torch.bfloat16).float(), 1.0
    x = torch.zeros(M, K)
    x[:, 0], x[:, 1] = 1.0, torch.tensor([2.0**100, -(2.0**115), 2.0**120, 1.0])
    if q4:
        w[:inter, 0] = -88.0  # (one scale per 32: 11 for the gate rows' block)
        p, s = q4_quantize(w)
        lw = LinearWeight(Q4Tensor(p, s, tuple(w.shape))).to(DEV, torch.bfloat16)
    else:
        lw = LinearWeight(w.to(torch.bfloat16)).to(DEV, torch.bfloat16)
    x = x.to(torch.bfloat16).to(DEV)
    h, f = lw.handle().run_gated(x, 1, 4), ops.linear(x, lw, out_f32=True).double().cpu()
    torch.cuda.synchronize()
    ops.check_status()
    want = f[:, :inter] / (1 + torch.exp(-f[:, :inter])) * f[:, inter:]
    # (__expf is 2 ulp and the rounding of its argument, some 2^-17 of the value here)
    assert bool((want[1] != 0).all()) and _rounded_once(h.cpu(), want, 2.0**-16 * want.abs() + 2.0**-130)


@pytest.mark.parametrize("q4,N,K,M,taken", [(True, 19456, 2560, 64, True), (True, 24576, 4096, 96, True), (True, 28672, 4096, 64, False), (True, 11264, 2048, 128, False),
                                            (True, 11264, 2048, 129, True), (False, 28672, 3584, 128, True), (False, 6144, 2560, 100, True), (False, 3072, 1024, 64, False)])
def test_parts_gemm_gated_rule(q4, N, K, M, taken):
    """Where the one kernel takes a gated product and where projection and activation are two launches: a last wave of few one-tile CTAs, a second wave of clusters, narrow and wide
    weights (each choice the faster one by 5 % or more, but for the first, which is so in a decode step)."""
    if q4:
        w = LinearWeight(Q4Tensor(torch.randint(0, 256, (N, K // 2), dtype=torch.uint8), torch.randn(N, K // 32) * 0.01, (N, K))).to(DEV, torch.bfloat16)
    else:
        w = LinearWeight((torch.randn(N, K, device=DEV) * 0.02).to(torch.bfloat16))
    x = torch.randn(M, K, device=DEV).to(torch.bfloat16)
    out = w.handle().run_gated(x, 1)
    torch.cuda.synchronize()
    assert (out is not None) == taken


def test_parts_gemm_gated_huge_gates():
    """Gates of 2^126 and more on either side of zero, and sums that overflow: as they are and nothing, then infinity and not a number, as g / (1 + exp(-g)) has it."""
    inter, K, M = 64, 64, 3
    w, x = torch.zeros(2 * inter, K), torch.zeros(M, K)
    w[:inter, 0], w[inter:, 1] = torch.tensor([2.0**127, -(2.0**127), 2.0**126, -(2.0**126), 1.5 * 2.0**127, -100.0, 0.0, 1.0]).repeat(inter // 8), 2.0**-100
    x[:, 0], x[:, 1] = torch.tensor([1.0, 1.0, 4.0]), torch.tensor([1.0, -(2.0**90), 1.0])
    h = LinearWeight(w.to(torch.bfloat16)).to(DEV, torch.bfloat16).handle().run_gated(x.to(torch.bfloat16).to(DEV), 1, 4).float().cpu()
    ops.check_status()
    for m, up in ((0, 2.0**-100), (1, -(2.0**-10))):
        assert torch.equal(h[m, :5], torch.tensor([2.0**127, 0.0, 2.0**126, 0.0, 1.5 * 2.0**127]) * up) and h[m, 6] == 0 and abs(h[m, 5]) < 2.0**-137
        assert abs(h[m, 7] - 0.7310586 * up) <= abs(up) * 2.0**-8
    assert bool((h[2, [0, 2, 4]] == math.inf).all()) and bool(torch.isnan(h[2, [1, 3]]).all()) and bool((h[2, [5, 6]] == 0).all())


@pytest.mark.parametrize("M", [1, 129, 400, 2310])
@pytest.mark.parametrize("heads,kv,norm,rope,bias", [(4, 1, True, True, False), (6, 3, False, True, True), (3, 1, True, False, True)])
def test_parts_gemm_heads(M, heads, kv, norm, rope, bias):
    """q | k | v heads against the one-tile kernel: an odd number of heads (half a tile at the end), rows without a cache slot, positions behind a prefix, bias."""
    K, D = 512, 128
    qt, wd = _q4_weight((heads + 2 * kv) * D, K, seed=heads)
    lw = LinearWeight(qt).to(DEV, torch.bfloat16)
    x = (torch.randn(M, K) * 0.5).to(torch.bfloat16).to(DEV)
    pages = M // 32 + 2
    slots = torch.randperm(pages * 32)[:M]
    slots[M // 3 :: 5] = -1
    slots, pos = slots.to(DEV), torch.arange(M, dtype=torch.int32, device=DEV) + 37
    cos, sin = (t.to(DEV) for t in ref.rope_tables(D, 4096, 10000.0)) if rope else (None, None)
    qn, kn = ((1 + 0.1 * torch.randn(D)).to(torch.bfloat16).to(DEV) for _ in range(2)) if norm else (None, None)
    b = torch.randn(wd.shape[0], device=DEV) if bias else None
    got = []
    for pairs, impl in ((0, 0), (-1, 4)):
        ops.set_gemm_pairs(pairs)
        kc, vc = (torch.zeros(pages, kv, 32, D, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        q = lw.handle().run_qkv(x, pos, slots, qn, kn, cos, sin, kc, vc, heads, kv, 1e-6, 0.0, b, impl)
        got.append((q, kc, vc))
    torch.cuda.synchronize()
    ops.check_status()
    # (sums in another order, rounded to bf16 up to twice: about 1.7e-3 each in the 2-norm; rows that are not kept stay zeros, whole: a single sum may cancel in one order and not in the other)
    for u, v in zip(*got):
        assert _rel(u, v) < 4e-3 and torch.equal((u == 0).all(-1), (v == 0).all(-1))


@pytest.mark.parametrize("M,N,K", [(1, 256, 64), (70, 272, 192), (200, 136, 64), (257, 1040, 2624), (385, 528, 192), (800, 11264, 192), (2600, 3072, 320), (900, 19200, 128)])
def test_parts_gemm_bf16(M, N, K):
    """bf16 weights: 64-k stages of their own, one and two accumulators, halves of an odd number of eights (gated), rows that end inside a half tile, several waves with
    two accumulators in turn, rows without 16 bytes at once, fp32 outputs; guard areas around output and sums. fp32 sums, rounded once (gated
    products behind the activation): 2^-8 of a value at most, so no more in the 2-norm."""
    wd = (torch.randn(N, K) * 0.05).to(torch.bfloat16)
    lw = LinearWeight(wd).to(DEV, torch.bfloat16)
    x = (torch.randn(M, K + 8) * 0.5).to(torch.bfloat16).to(DEV)[:, :K]
    f = x.double().cpu() @ wd.double().t()
    odd = torch.full((M, N + 1), 7.0, dtype=torch.bfloat16, device=DEV)
    ops.set_bounds_check(True)
    try:
        y, y32 = ops.linear(x, lw, impl=4), ops.linear(x, lw, impl=4, out_f32=True)
        ops.linear(x, lw, impl=4, out=odd[:, :N])
        h = lw.handle().run_gated(x, 1, 4)
        torch.cuda.synchronize()
        ops.check_guards()
    finally:
        ops.set_bounds_check(False)
    ops.check_status()
    assert _rel(y.cpu(), f) < 3e-3 and _rel(y32.cpu(), f) < 2e-5 and torch.equal(odd[:, :N], y) and bool((odd[:, N] == 7.0).all())
    if N % 16 == 0:
        assert _rel(h.cpu(), torch.nn.functional.silu(f[:, : N // 2]) * f[:, N // 2 :]) < 3e-3
    else:
        assert h is None


@pytest.mark.parametrize("M", [1, 129, 900])
def test_parts_gemm_bf16_heads(M):
    """q | k | v heads of bf16 weights against the one-tile kernel, an odd number of heads."""
    heads, kv, K, D = 5, 2, 320, 128
    lw = LinearWeight((torch.randn((heads + 2 * kv) * D, K) * 0.05).to(torch.bfloat16)).to(DEV, torch.bfloat16)
    x = (torch.randn(M, K) * 0.5).to(torch.bfloat16).to(DEV)
    slots, pos = torch.randperm((M // 32 + 2) * 32, device=DEV)[:M], torch.arange(M, dtype=torch.int32, device=DEV) + 37
    cos, sin = (t.to(DEV) for t in ref.rope_tables(D, 4096, 10000.0))
    qn, kn = ((1 + 0.1 * torch.randn(D)).to(torch.bfloat16).to(DEV) for _ in range(2))
    got = []
    for pairs, impl in ((0, 0), (-1, 4)):
        ops.set_gemm_pairs(pairs)
        kc, vc = (torch.zeros(M // 32 + 2, kv, 32, D, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        q = lw.handle().run_qkv(x, pos, slots, qn, kn, cos, sin, kc, vc, heads, kv, 1e-6, 0.0, None, impl)
        got.append((q, kc, vc))
    torch.cuda.synchronize()
    ops.check_status()
    # (sums in another order, rounded to bf16 up to twice: about 1.7e-3 each in the 2-norm; rows that are not kept stay zeros, whole: a single sum may cancel in one order and not in the other)
    for u, v in zip(*got):
        assert _rel(u, v) < 4e-3 and torch.equal((u == 0).all(-1), (v == 0).all(-1))


@pytest.mark.parametrize("E,n,K,T,k", [(4, 512, 256, 900, 2), (3, 384, 1216, 1500, 1), (40, 1280, 128, 9000, 2)])
def test_parts_gemm_experts(E, n, K, T, k):
    """Equal work items of up to 384 rows (one and two instructions, more items than an expert's rows ask for at the end of the list), as the experts of a prompt have them."""
    e = ops.require_ext()
    made = [_q4_weight(n, K, seed=i) for i in range(E)]
    g = ops.GroupedLinearWeight([LinearWeight(qt).to(DEV, torch.bfloat16) for qt, _ in made])
    assert g.prompt_rows() == 384
    x = (torch.randn(T, K) * 0.5).to(torch.bfloat16).to(DEV)
    w, idx, counts, offsets, perm, pos = e.moe_route(torch.randn(T, E, device=DEV), k, 0, True)
    items = e.moe_items(offsets, 0, E, 384, (T * k + 383) // 384 + E)
    xs = e.moe_gather(x, perm, k, None, 0, 0)
    y, h = g.run(xs, items, 384), g.run_gated(xs, items, "silu", 384)
    torch.cuda.synchronize()
    ops.check_status()
    off, it = offsets.tolist(), items.tolist()
    for i, (_, wd) in enumerate(made):
        f = xs[off[i]:off[i + 1]].double().cpu() @ wd.double().t()
        assert _rel(y[off[i]:off[i + 1]].cpu(), f) < 4e-3
        assert _rel(h[off[i]:off[i + 1]].cpu(), torch.nn.functional.silu(f[:, : n // 2]) * f[:, n // 2:]) < 6e-3
        rows = [hi - lo for a, lo, hi, _ in it if a == i]
        assert sum(rows) == off[i + 1] - off[i] and max(rows) <= 384 and max(rows) - min(rows) < len(rows)


@pytest.mark.parametrize("T,E,k", [(1, 3, 3), (33, 8, 2), (70, 128, 8), (128, 129, 16), (50, 256, 8), (40, 257, 9), (20, 1000, 16), (700, 128, 8), (3000, 40, 6), (130, 1024, 16), (129, 8, 2), (442, 8, 2)])
def test_moe_route_choices(T, E, k):
    """Experts and groups of the routing kernels against a sort: equal logits (the lower expert first), both zeros equal, minus infinity chosen last; one launch and
    several, 32 experts per register and their remainders, the pairs grouped chunk by chunk and by one block."""
    e = ops.require_ext()
    z = torch.randint(-4, 5, (T, E)).float() * torch.where(torch.rand(T, E) < 0.5, 1.0, -1.0)  # (minus zeros among them)
    z[::3, : E // 2] = -math.inf
    z[1::4] = torch.randn(z[1::4].shape)
    idx = torch.sort(z + 0.0, dim=-1, descending=True, stable=True).indices[:, :k]
    order = torch.sort(idx.flatten(), stable=True).indices
    for mode in (0, 1):
        routed = [e.moe_route(z.to(DEV), k, mode, True)]
        if T <= 128:
            routed.append(e.moe_route_items(z.to(DEV), k, mode, True, 0, E, 8, T * k))
        for r in routed:
            w, got, counts, offsets, perm, pos = (t.cpu() for t in r[:6])
            wr = torch.softmax(z.gather(1, idx), -1)
            assert torch.equal(got.long(), idx) and torch.allclose(w, wr, rtol=1e-5, atol=1e-7)  # (ratios of __expf, 2 ulp and the rounding of its argument)
            assert torch.equal(counts.long(), torch.bincount(idx.flatten(), minlength=E)) and torch.equal(offsets[1:].long(), counts.long().cumsum(0))
            assert torch.equal(perm.long(), order) and torch.equal(perm[pos.flatten().long()].long(), torch.arange(T * k))


@pytest.mark.parametrize("T,E,k", [(25, 512, 8), (49, 513, 2), (128, 768, 1), (30, 768, 8), (17, 769, 15), (1100, 513, 8), (600, 768, 16)])
def test_moe_route_widths(T, E, k):
    """The numbers of experts at which a lane keeps more scores and a block has fewer warps, and either size of chunk."""
    test_moe_route_choices(T, E, k)


@pytest.mark.parametrize("T,k,H", [(1, 1, 8), (3, 5, 1032), (9, 8, 2048), (2, 70, 128)])
def test_moe_combine_slots(T, k, H):
    """Slots that do not fill a group of four, more of them than are looked up ahead, rows of another rank's experts."""
    e = ops.require_ext()
    ys, w = torch.randn(T * k, H).to(torch.bfloat16), torch.rand(T, k)
    pos = torch.randperm(T * k).view(T, k)
    lo, hi = T * k // 4, T * k - T * k // 3
    for rng in (False, True):
        offsets = torch.tensor([0, lo, hi, T * k], dtype=torch.int32, device=DEV)
        out = e.moe_combine(ys.to(DEV), pos.int().to(DEV), w.to(DEV), T, k, *((offsets, 1, 1) if rng else (None, 0, 0)))
        own = ((pos >= lo) & (pos < hi)).double() if rng else torch.ones(T, k).double()
        r = (ys.double()[pos] * (w.double() * own).unsqueeze(-1)).sum(1)
        assert (out.cpu().double() - r).abs().max() <= 2.0**-8 * max(1e-6, r.abs().max().item())


@pytest.mark.parametrize("D,H,KV", [(64, 32, 8), (64, 16, 1), (64, 32, 4), (64, 12, 12), (64, 9, 1)])
@pytest.mark.parametrize("norm,rope,window,cap,splits", [(True, True, 0, 0.0, 1), (False, True, 0, 0.0, 8), (True, False, 40, 0.0, 3), (False, True, 33, 20.0, 32), (True, True, 0, 0.0, 64)])
def test_decode_attention_rope(D, H, KV, norm, rope, window, cap, splits):
    """Norm, rotation and cache write inside decode attention against the two kernels: one key, the edges of a slice and of a page, contexts cut into several parts (by
    themselves and by a plan), a row that is not kept, positions past the table. The caches bit for bit; the output but for the
    few values whose rounding falls the other way (the rotation's products may be contracted otherwise): less than one rounding of all, 2e-3 in the 2-norm."""
    ctx = [1, 15, 16, 17, 32, 33, 200, 777, 1500]
    B, per = len(ctx), 48
    pages = B * per
    bt = torch.randperm(pages).reshape(B, per).int().to(DEV)
    pos = torch.tensor([c - 1 for c in ctx], dtype=torch.int32)
    slots = torch.tensor([int(bt[i, (c - 1) // 32]) * 32 + (c - 1) % 32 for i, c in enumerate(ctx)])
    slots[4] = -1
    pos[5] = 5000
    qkv = torch.randn(B, (H + 2 * KV) * D).to(torch.bfloat16).to(DEV)
    kc, vc = (torch.randn(pages, KV, 32, D).to(torch.bfloat16).to(DEV) for _ in range(2))
    qn, kn = ((1 + 0.1 * torch.randn(D)).to(torch.bfloat16).to(DEV) for _ in range(2)) if norm else (None, None)
    cos, sin = (t.to(DEV) for t in ref.rope_tables(D, 4096, 10000.0)) if rope else (None, None)
    cl, pos, slots = torch.tensor(ctx, dtype=torch.int32, device=DEV), pos.to(DEV), slots.to(DEV)
    kc2, vc2, raw = kc.clone(), vc.clone(), qkv.clone()
    for even in (True, False):
        q = ops.rope_kv(qkv.clone(), pos, slots, qn, kn, cos, sin, kc2, vc2, H, KV, D, 1e-6, 0.5)
        want = ops.decode_attention(q, kc2, vc2, bt, cl, H, 0.1, cap, window, splits, even=even)
        got = ops.decode_attention_rope(qkv, pos, slots, qn, kn, cos, sin, kc, vc, bt, cl, H, 0.1, cap, window, splits, 1e-6, 0.5, even=even)
        torch.cuda.synchronize()
        keep = [i for i in range(B) if i != 4]  # (what is not kept there is not seen either)
        assert torch.equal(qkv, raw) and torch.equal(kc, kc2) and torch.equal(vc, vc2)
        assert _rel(got[keep], want[keep]) < 2e-3 and bool(torch.isfinite(got).all())


def test_decode_attention_rope_alignment():
    """Rows that start on an odd element are refused; norm weights and tables that start between the kernel's words give what the two kernels give."""
    B, H, KV, D, ctx = 2, 4, 2, 64, 40
    qkv = torch.randn(B, (H + 2 * KV) * D).to(torch.bfloat16).to(DEV)
    kc, vc = (torch.randn(4, KV, 32, D).to(torch.bfloat16).to(DEV) for _ in range(2))
    bt, cl = torch.arange(4, dtype=torch.int32, device=DEV).view(B, 2), torch.full((B,), ctx, dtype=torch.int32, device=DEV)
    pos, slots = cl - 1, torch.tensor([39, 103], device=DEV)
    wide = torch.randn(2 * D + 1, device=DEV).to(torch.bfloat16)
    tables = [torch.cat([torch.zeros(1), t.flatten()]).to(DEV)[1:].view(t.shape) for t in ref.rope_tables(D, 64, 10000.0)]
    odd = torch.empty(qkv.numel() + 1, dtype=torch.bfloat16, device=DEV)[1:].view(qkv.shape).copy_(qkv)
    even = [t.clone() for t in tables]
    with pytest.raises(RuntimeError, match="misaligned"):
        ops.decode_attention_rope(odd, pos, slots, None, None, *even, kc, vc, bt, cl, H, 0.1)
    for qn, kn, cs in ((wide[1 : D + 1], wide[D + 1 :], even), (None, None, tables)):
        c = [t.clone() for t in (kc, vc, kc, vc)]
        q = ops.rope_kv(qkv.clone(), pos, slots, qn, kn, *cs, c[0], c[1], H, KV, D, 1e-6)
        want = ops.decode_attention(q, c[0], c[1], bt, cl, H, 0.1)
        got = ops.decode_attention_rope(qkv.clone(), pos, slots, qn, kn, *cs, c[2], c[3], bt, cl, H, 0.1)
        assert torch.equal(got, want) and torch.equal(c[0], c[2]) and torch.equal(c[1], c[3])
