"""Quantized paged KV cache on the GPU: append is bit-exact against the oracle (codes,
scales, page placement); decode attention is within tolerance of the oracle's fp32
attention over the dequantized cache; full-size cases are covered by properties."""
import numpy as np
import pytest
import torch

from oracle import kv_cache as kc
from oracle import attention as oatt

pytestmark = pytest.mark.gpu
DT = {"fp32": torch.float32, "bf16": torch.bfloat16}
FMTS = ["int8", "fp8", "nvfp4"]
# Decode-attention tolerance, per output element e of head h:
#     |out - oracle| <= C_P * sum_t p_t |V_t,e|  +  C_OUT * |oracle|
# The first term is the element's own error scale (softmax weights applied to |V|, from the oracle): an
# outlier channel (values x20) gets a 20x larger allowance than a normal channel, and no element borrows the
# allowance of another.  C_P covers the relative error of the softmax weights: q and P pass through f16
# (2^-11) or three e4m3 terms (2^-12) in the tensor-core kernels, and the score error of a d=128 dot
# product with outlier channels reaches ~1e-2 before the exponential.  The CUDA-core kernel computes in
# fp32 on the dequantized values.  C_OUT is the rounding of the stored output (bf16: 2^-9).
C_P_TC, C_P_SIMT = 2e-2, 2e-4
C_OUT = {"fp32": 1e-5, "bf16": 4e-3}


def attn_tol(ref, ref_abs, name, simt):
    return (C_P_SIMT if simt else C_P_TC) * ref_abs + C_OUT[name] * np.abs(ref) + 1e-6


def outlier_kv(rng, B, T, Hkv, d, dtype):
    """N(0,1) with 4 outlier channels per head scaled x20 (the config-3 distribution)."""
    k = rng.standard_normal((B, T, Hkv, d)).astype(np.float32)
    v = rng.standard_normal((B, T, Hkv, d)).astype(np.float32)
    for h in range(Hkv):
        ch = rng.choice(d, 4, replace=False)
        k[:, :, h, ch] *= 20
        v[:, :, h, ch] *= 20
    kt, vt = torch.from_numpy(k).to(dtype), torch.from_numpy(v).to(dtype)
    return kt, vt


def make_pair(fmt, B, pages_per_seq, Hkv, d, dev, rng, extra_pages=3):
    npg = B * pages_per_seq + extra_pages
    bt = rng.permutation(npg)[:B * pages_per_seq].reshape(B, pages_per_seq).astype(np.int32)
    from transformer_surgeon_b200 import ops
    o = kc.PagedKV(kc.FMT_NAMES[fmt], npg, Hkv, d, bt, B)
    seq = torch.zeros(B, dtype=torch.int32, device=dev)
    g = ops.PagedKV(fmt, npg, Hkv, d, torch.from_numpy(bt).to(dev), seq, dev)
    return o, g


def sync_scales(o, g, k, v, rope=None):
    if o.fmt == kc.FMT_FP8:
        g.set_fp8_scales(k.to(g.k_pool.device), v.to(g.k_pool.device), rope=rope, pos0=g.seq_lens if rope else None)
        o.k_scale[:] = g.k_scale.cpu().numpy()
        o.v_scale[:] = g.v_scale.cpu().numpy()


@pytest.mark.parametrize("fmt", FMTS)
@pytest.mark.parametrize("name", ["fp32", "bf16"])
@pytest.mark.parametrize("d", [64, 128])
def test_append_bit_exact(cuda, fmt, name, d):
    rng = np.random.default_rng(10)
    B, T, Hkv = 3, 37, 2
    o, g = make_pair(fmt, B, 4, Hkv, d, cuda, rng)
    k, v = outlier_kv(rng, B, T, Hkv, d, DT[name])
    sync_scales(o, g, k, v)
    if fmt == "fp8":   # scale kernel: amax/448 exactly
        ref = kc.fp8_scale_from_amax(k.float().abs().amax(dim=(1, 3)).numpy())
        assert np.array_equal(o.k_scale, ref)
    # prompt in one bulk append, then 5 single-token decode appends
    g.append(k.to(cuda), v.to(cuda))
    g.seq_lens += T
    kc.append_vectorized(o, k.float().numpy(), v.float().numpy())
    for step in range(5):
        k1, v1 = outlier_kv(rng, B, 1, Hkv, d, DT[name])
        g.append(k1.to(cuda), v1.to(cuda))
        g.seq_lens += 1
        o.append(k1.float().numpy(), v1.float().numpy())
    assert np.array_equal(g.k_pool.cpu().numpy(), o.k_pool)
    assert np.array_equal(g.v_pool.cpu().numpy(), o.v_pool)
    assert g.seq_lens.cpu().tolist() == o.seq_lens.tolist()


@pytest.mark.parametrize("fmt", FMTS)
@pytest.mark.parametrize("name", ["fp32", "bf16"])
def test_append_with_fused_rope_and_ragged_lengths(cuda, fmt, name):
    rng = np.random.default_rng(11)
    B, T, Hkv, d = 4, 21, 2, 128
    o, g = make_pair(fmt, B, 3, Hkv, d, cuda, rng)
    cos, sin = oatt.rope_tables(d, 5e5, torch.arange(64))
    k, v = outlier_kv(rng, B, T, Hkv, d, DT[name])
    new_lens = np.array([21, 0, 7, 16], dtype=np.int32)
    start = np.array([3, 0, 16, 5], dtype=np.int32)          # sequences already hold some tokens
    o.seq_lens[:] = start
    g.seq_lens.copy_(torch.from_numpy(start))
    rope = (cos.to(cuda), sin.to(cuda))
    sync_scales(o, g, k, v, rope=rope)
    g.append(k.to(cuda), v.to(cuda), new_lens=torch.from_numpy(new_lens).to(cuda), rope=rope)
    # oracle: rotate with the same rounding points, then append
    pos = torch.from_numpy(start.astype(np.int64))[:, None] + torch.arange(T)[None, :]
    kr = torch.stack([oatt.apply_rope(k[b], cos[pos[b]], sin[pos[b]]) for b in range(B)])
    if fmt == "fp8":
        ref = kc.fp8_scale_from_amax(kr.float().abs().amax(dim=(1, 3)).numpy())
        assert np.array_equal(o.k_scale, ref)
    o.append(kr.float().numpy(), v.float().numpy(), new_lens=new_lens)
    assert np.array_equal(g.k_pool.cpu().numpy(), o.k_pool)
    assert np.array_equal(g.v_pool.cpu().numpy(), o.v_pool)


def test_append_empty_and_overflow(cuda):
    from transformer_surgeon_b200 import ops
    rng = np.random.default_rng(12)
    o, g = make_pair("int8", 2, 1, 2, 64, cuda, rng)
    e = torch.empty((2, 0, 2, 64), device=cuda)
    g.append(e, e)                                             # T == 0: no-op
    k, v = outlier_kv(rng, 2, 20, 2, 64, torch.float32)        # 20 tokens but only one page each
    g.append(k.to(cuda), v.to(cuda))
    o.append(k[:, :16].numpy(), v[:, :16].numpy())             # positions >= 16 are skipped
    assert np.array_equal(g.k_pool.cpu().numpy(), o.k_pool)


@pytest.mark.parametrize("fmt", FMTS + ["fp32", "bf16"])
@pytest.mark.parametrize("d", [64, 128])
def test_gather_dequantizes_bit_exact(cuda, fmt, d):
    """tsb200_kv_gather == the oracle's dequantized cache, element for element (fp32 output), with
    ragged lengths, an empty sequence and zeros beyond each length."""
    from transformer_surgeon_b200 import ops
    rng = np.random.default_rng(21)
    B, Hkv = 4, 2
    lens = np.array([37, 16, 0, 1], dtype=np.int32)
    T = int(lens.max())
    src = torch.bfloat16 if fmt == "bf16" else torch.float32
    if fmt in FMTS:
        o, g = make_pair(fmt, B, 3, Hkv, d, cuda, rng)
        k, v = outlier_kv(rng, B, T, Hkv, d, src)
        sync_scales(o, g, k, v)
        o.append(k.float().numpy(), v.float().numpy(), new_lens=lens)
    else:                                           # unquantized pages: no oracle object needed
        bt = torch.from_numpy(rng.permutation(B * 3 + 2)[:B * 3].reshape(B, 3).astype(np.int32)).to(cuda)
        g = ops.PagedKV(fmt, B * 3 + 2, Hkv, d, bt, torch.zeros(B, dtype=torch.int32, device=cuda), cuda)
        k, v = outlier_kv(rng, B, T, Hkv, d, src)
    nl = torch.from_numpy(lens).to(cuda)
    g.append(k.to(cuda), v.to(cuda), new_lens=nl)
    g.seq_lens.copy_(nl)
    L = 40
    kd, vd = ops.kv_gather(g, L, dtype=torch.float32)
    kd, vd = kd.cpu().numpy(), vd.cpu().numpy()
    for b in range(B):
        if fmt in FMTS:
            Kr, Vr = o.gather(b)
        else:                                       # unquantized pages hold the appended values themselves
            Kr, Vr = k[b, :lens[b]].float().numpy(), v[b, :lens[b]].float().numpy()
        assert np.array_equal(kd[b, :lens[b]], Kr) and np.array_equal(vd[b, :lens[b]], Vr)
        assert not kd[b, lens[b]:].any() and not vd[b, lens[b]:].any()


@pytest.mark.parametrize("fmt", FMTS)
@pytest.mark.parametrize("name", ["fp32", "bf16"])
@pytest.mark.parametrize("H,Hkv,d", [(8, 2, 128), (14, 2, 64), (4, 4, 128), (32, 8, 128)])
@pytest.mark.parametrize("simt", [True, False])
def test_decode_attention_against_oracle(cuda, fmt, name, H, Hkv, d, simt):
    from transformer_surgeon_b200 import ops
    rng = np.random.default_rng(13)
    B = 5
    lens = np.array([1, 16, 17, 130, 0], dtype=np.int32)       # single token, exact page, ragged, multi-split, empty
    o, g = make_pair(fmt, B, 9, Hkv, d, cuda, rng)
    T = int(lens.max())
    k, v = outlier_kv(rng, B, T, Hkv, d, DT[name])
    sync_scales(o, g, k, v)
    nl = torch.from_numpy(lens).to(cuda)
    g.append(k.to(cuda), v.to(cuda), new_lens=nl)
    g.seq_lens.copy_(nl)
    o.append(k.float().numpy(), v.float().numpy(), new_lens=lens)
    assert np.array_equal(g.k_pool.cpu().numpy(), o.k_pool)
    q = torch.from_numpy(rng.standard_normal((B, H, d)).astype(np.float32)).to(DT[name])
    ref, ref_abs = oatt.paged_decode_attention(o, q.float().numpy(), with_abs=True)
    out = ops.paged_decode_attention(g, q.to(cuda), max_seq_len=144, simt=simt).float().cpu().numpy()
    assert np.all(out[4] == 0)
    tol = attn_tol(ref, ref_abs, name, simt)
    assert np.all(np.abs(out - ref) <= tol), (np.abs(out - ref) / tol).max()


@pytest.mark.parametrize("fmt", FMTS)
@pytest.mark.parametrize("name", ["fp32", "bf16"])
@pytest.mark.parametrize("H,Hkv,d,cap,qpad", [(7, 1, 128, 576, 0), (7, 1, 128, 640, 3), (14, 2, 64, 3968, 8), (4, 1, 128, 4400, 0), (9, 1, 128, 520, 0)])
def test_decode_attention_split_merges(cuda, fmt, name, H, Hkv, d, cap, qpad):
    """Eight to 62 splits (the FP8 kernel of up to four heads: eleven) of full, short and empty sequences, one and two head chunks, put together
    by a cluster or the chained reduction; queries off a 16-byte boundary and strided."""
    from transformer_surgeon_b200 import ops
    rng = np.random.default_rng(29)
    B = 3
    lens = np.array([cap, 17, 0], dtype=np.int32)
    o, g = make_pair(fmt, B, (cap + 15) // 16, Hkv, d, cuda, rng)
    k, v = outlier_kv(rng, B, cap, Hkv, d, DT[name])
    sync_scales(o, g, k, v)
    nl = torch.from_numpy(lens).to(cuda)
    g.append(k.to(cuda), v.to(cuda), new_lens=nl)
    g.seq_lens.copy_(nl)
    kc.append_vectorized(o, k.float().numpy(), v.float().numpy())      # tokens beyond a length are never read
    o.seq_lens[:] = lens
    q = torch.from_numpy(rng.standard_normal((B, H, d)).astype(np.float32)).to(DT[name])
    buf = torch.zeros((B, H * d + qpad), dtype=DT[name], device=cuda)
    qv = buf[:, qpad:].unflatten(1, (H, d))
    qv.copy_(q)
    ref, ref_abs = oatt.paged_decode_attention(o, q.float().numpy(), with_abs=True)
    out = ops.paged_decode_attention(g, qv, max_seq_len=cap)
    assert torch.equal(out, ops.paged_decode_attention(g, qv, max_seq_len=cap))
    out = out.float().cpu().numpy()
    assert np.all(out[2] == 0)
    tol = attn_tol(ref, ref_abs, name, False)
    assert np.all(np.abs(out - ref) <= tol), (np.abs(out - ref) / tol).max()


@pytest.mark.parametrize("fmt", ["fp32", "bf16"])
@pytest.mark.parametrize("H,Hkv,d", [(14, 2, 64), (9, 1, 128), (4, 4, 128)])
@pytest.mark.parametrize("lens", [(1, 16, 17), (0, 129, 150), (700, 2049, 33)])
def test_decode_attention_unquantized_pages(cuda, fmt, H, Hkv, d, lens):
    """Unquantized pages: one split and several, empty and one-token sequences, a second chunk of query heads, stale slots; against
    the one-lane-per-element cross-check kernel."""
    from transformer_surgeon_b200 import ops
    B, cap = len(lens), 2064
    g = torch.Generator(device=cuda).manual_seed(3)
    pages = cap // 16
    bt = torch.randperm(B * pages, generator=g, device=cuda).to(torch.int32).reshape(B, pages)
    seq = torch.zeros(B, dtype=torch.int32, device=cuda)
    kv = ops.PagedKV(fmt, B * pages, Hkv, d, bt, seq, cuda)
    k, v = (torch.randn((B, cap, Hkv, d), generator=g, device=cuda).to(DT[fmt]) for _ in range(2))
    kv.append(k, v)
    seq.copy_(torch.tensor(lens, dtype=torch.int32))
    q = torch.randn((B, H, d), generator=g, device=cuda).to(DT[fmt])
    out, ref = ops.paged_decode_attention(kv, q, max(lens)), ops.paged_decode_attention(kv, q, max(lens), simt=True)
    torch.testing.assert_close(out, ref, rtol=1e-5 if fmt == "fp32" else 1e-2, atol=1e-5 if fmt == "fp32" else 1e-2)


@pytest.mark.parametrize("fmt", FMTS)
def test_decode_attention_config3_shape(cuda, fmt):
    """Llama-3-8B layout (32 q heads / 8 kv heads / d 128), batch 8, context 4096, seeded random
    block table: kernel vs oracle on every sequence, and tensor-core vs CUDA-core kernel."""
    from transformer_surgeon_b200 import ops
    rng = np.random.default_rng(14)
    B, L, H, Hkv, d = 8, 4096, 32, 8, 128
    o, g = make_pair(fmt, B, L // 16, Hkv, d, cuda, rng, extra_pages=5)
    k, v = outlier_kv(rng, B, L, Hkv, d, torch.bfloat16)
    sync_scales(o, g, k, v)
    g.append(k.to(cuda), v.to(cuda))
    g.seq_lens += L
    kc.append_vectorized(o, k.float().numpy(), v.float().numpy())
    assert np.array_equal(g.k_pool.cpu().numpy(), o.k_pool)
    assert np.array_equal(g.v_pool.cpu().numpy(), o.v_pool)
    q = torch.from_numpy(rng.standard_normal((B, H, d)).astype(np.float32)).bfloat16()
    ref, ref_abs = oatt.paged_decode_attention(o, q.float().numpy(), with_abs=True)
    out = ops.paged_decode_attention(g, q.to(cuda), max_seq_len=L).float().cpu().numpy()
    out_simt = ops.paged_decode_attention(g, q.to(cuda), max_seq_len=L, simt=True).float().cpu().numpy()
    tol, tol_simt = attn_tol(ref, ref_abs, "bf16", False), attn_tol(ref, ref_abs, "bf16", True)
    assert np.all(np.abs(out - ref) <= tol), (np.abs(out - ref) / tol).max()
    assert np.all(np.abs(out_simt - ref) <= tol_simt), (np.abs(out_simt - ref) / tol_simt).max()


@pytest.mark.parametrize("fmt", FMTS)
def test_full_size_properties(cuda, fmt):
    """Batch 64, context 32768 (the largest config-3 case, ~4.3 GB of pages), checked through
    size-independent properties:
      * V == 1 everywhere -> softmax weights sum to 1 -> output == 1 (exactly representable codes);
      * K == 0 -> uniform weights -> output == mean of V over the context;
      * run-to-run determinism of the split reduction."""
    from transformer_surgeon_b200 import ops
    B, L, H, Hkv, d = 64, 32768, 32, 8, 128
    npg = B * L // 16
    gen = torch.Generator(device=cuda).manual_seed(15)
    bt = torch.randperm(npg, generator=gen, device=cuda).to(torch.int32).reshape(B, L // 16)
    seq = torch.zeros(B, dtype=torch.int32, device=cuda)
    g = ops.PagedKV(fmt, npg, Hkv, d, bt, seq, cuda)
    chunk = 2048
    vmean = torch.zeros((B, Hkv, d), dtype=torch.float64, device=cuda)
    for t0 in range(0, L, chunk):
        k = torch.zeros((B, chunk, Hkv, d), dtype=torch.bfloat16, device=cuda)
        v = (2 * torch.randint(-1, 2, (B, chunk, Hkv, d), generator=gen, device=cuda)).to(torch.bfloat16)
        if fmt == "fp8" and t0 == 0:
            g.k_scale.fill_(1.0); g.v_scale.fill_(1.0 / 64)
        g.append(k, v)
        seq += chunk
        vmean += v.double().sum(dim=1)
    vmean /= L
    q = torch.randn((B, H, d), generator=gen, device=cuda).bfloat16()
    out = ops.paged_decode_attention(g, q, max_seq_len=L)
    out2 = ops.paged_decode_attention(g, q, max_seq_len=L)
    assert torch.equal(out, out2)
    # values in {-2, 0, 2}: int8 and fp8 (scale 1/64) store them exactly; nvfp4 stores 2 as
    # e2m1(2 / e4m3(2/6)) * e4m3(2/6) = 6 * 0.34375 = 2.0625 in every block that holds a 2
    gain = 1.03125 if fmt == "nvfp4" else 1.0
    ref = gain * vmean.float().repeat_interleave(H // Hkv, dim=1)
    torch.testing.assert_close(out.float(), ref, rtol=2e-2, atol=2e-3)
    # V == 1: overwrite the pools through a second append pass at position 0
    seq.zero_()
    for t0 in range(0, L, chunk):
        k = torch.randn((B, chunk, Hkv, d), generator=gen, device=cuda).bfloat16()
        v = torch.ones((B, chunk, Hkv, d), dtype=torch.bfloat16, device=cuda)
        if fmt == "fp8" and t0 == 0:
            g.k_scale.fill_(6.0 / 448); g.v_scale.fill_(1.0 / 64)
        g.append(k, v)
        seq += chunk
    out = ops.paged_decode_attention(g, q, max_seq_len=L).float()
    one = 1.03125 if fmt == "nvfp4" else 1.0          # 1 -> 6 * e4m3(1/6) = 6 * 0.171875
    torch.testing.assert_close(out, torch.full_like(out, one), rtol=1e-2, atol=1e-2)


def test_argument_errors(cuda):
    from transformer_surgeon_b200 import ops, Tsb200Error
    rng = np.random.default_rng(16)
    o, g = make_pair("int8", 2, 2, 2, 64, cuda, rng)
    q = torch.zeros((2, 5, 64), device=cuda)                    # 5 q heads not divisible by 2 kv heads
    with pytest.raises(Tsb200Error):
        ops.paged_decode_attention(g, q, max_seq_len=32)
    with pytest.raises(ValueError):
        ops.PagedKV("int8", 4, 2, 48, g.block_table, g.seq_lens, cuda)      # head_dim 48 unsupported
    small = torch.empty(16, dtype=torch.uint8, device=cuda)
    with pytest.raises(Tsb200Error):
        ops.paged_decode_attention(g, torch.zeros((2, 4, 64), device=cuda), max_seq_len=32, ws=small)
    # max_seq_len beyond what the block table covers (2 pages = 32 tokens): refused, nothing is launched
    with pytest.raises(Tsb200Error) as ei:
        ops.paged_decode_attention(g, torch.zeros((2, 4, 64), device=cuda), max_seq_len=33)
    assert ei.value.status == -1
    empty = ops.PagedKV("int8", 4, 2, 64, g.block_table, g.seq_lens, cuda)
    empty.num_pages = 0                                         # a descriptor with no pages is refused too
    with pytest.raises(Tsb200Error):
        ops.paged_decode_attention(empty, torch.zeros((2, 4, 64), device=cuda), max_seq_len=32)


@pytest.mark.parametrize("name", ["fp32", "bf16"])
def test_rope_append_fused_equals_separate_calls(cuda, name):
    """tsb200_rope_append on column slices of one fused [B, (H+2Hkv)d] projection buffer gives the
    same q and the same pages as tsb200_rope + tsb200_kv_append on dense copies."""
    from transformer_surgeon_b200 import ops
    rng = np.random.default_rng(17)
    B, H, Hkv, d = 6, 8, 2, 128
    _, g1 = make_pair("int8", B, 2, Hkv, d, cuda, rng)
    rng = np.random.default_rng(17)
    _, g2 = make_pair("int8", B, 2, Hkv, d, cuda, rng)
    start = torch.tensor([0, 3, 15, 16, 20, 31], dtype=torch.int32, device=cuda)
    g1.seq_lens.copy_(start); g2.seq_lens.copy_(start)
    cos, sin = oatt.rope_tables(d, 1e6, torch.arange(64))
    rope = (cos.to(cuda), sin.to(cuda))
    qkv = torch.randn((B, (H + 2 * Hkv) * d), generator=torch.Generator().manual_seed(3)).to(DT[name]).to(cuda)
    q_ref = qkv[:, :H * d].reshape(B, 1, H, d).clone()
    k_ref = qkv[:, H * d:(H + Hkv) * d].reshape(B, 1, Hkv, d).clone()
    v_ref = qkv[:, (H + Hkv) * d:].reshape(B, 1, Hkv, d).clone()
    ops.rope_(q_ref, rope[0], rope[1], start)
    g1.append(k_ref, v_ref, rope=rope)
    q4 = qkv[:, :H * d].unflatten(1, (H, d)).unsqueeze(1)
    k4 = qkv[:, H * d:(H + Hkv) * d].unflatten(1, (Hkv, d)).unsqueeze(1)
    v4 = qkv[:, (H + Hkv) * d:].unflatten(1, (Hkv, d)).unsqueeze(1)
    g2.rope_append(q4, k4, v4, rope)
    assert torch.equal(q4, q_ref)
    assert torch.equal(g1.k_pool, g2.k_pool) and torch.equal(g1.v_pool, g2.v_pool)


@pytest.mark.parametrize("fmt", FMTS)
@pytest.mark.parametrize("name", ["fp32", "bf16"])
@pytest.mark.parametrize("H,Hkv,d", [(14, 2, 64), (9, 9, 128)])
@pytest.mark.parametrize("pad", [0, 3])
def test_bulk_append_of_strided_prompts(cuda, fmt, name, H, Hkv, d, pad):
    """Prompt chunks out of a fused projection buffer (pad: vectors off a 16-byte boundary), rotated with their queries: starts within
    a page, ends within a page, pages covered whole and in part, more heads than warps."""
    from transformer_surgeon_b200 import ops
    rng = np.random.default_rng(19)
    B, T = 4, 53
    o, g = make_pair(fmt, B, 5, Hkv, d, cuda, rng)
    start = np.array([0, 5, 16, 27], dtype=np.int32)
    new_lens = np.array([53, 32, 16, 0], dtype=np.int32)
    o.seq_lens[:] = start
    g.seq_lens.copy_(torch.from_numpy(start))
    cos, sin = oatt.rope_tables(d, 5e5, torch.arange(96))
    rope = (cos.to(cuda), sin.to(cuda))
    k, v = outlier_kv(rng, B, T, Hkv, d, DT[name])
    q = torch.randn((B, T, H, d), generator=torch.Generator().manual_seed(3)).to(DT[name])
    sync_scales(o, g, k, v, rope=rope)
    buf = torch.zeros((B, T, (H + 2 * Hkv) * d + 2 * pad), dtype=DT[name], device=cuda)
    q4 = buf[..., :H * d].unflatten(2, (H, d))
    k4 = buf[..., H * d + pad:(H + Hkv) * d + pad].unflatten(2, (Hkv, d))
    v4 = buf[..., (H + Hkv) * d + pad:(H + 2 * Hkv) * d + pad].unflatten(2, (Hkv, d))
    q4.copy_(q); k4.copy_(k); v4.copy_(v)
    if fmt == "fp8":                              # the scales of the same slices
        dense = g.k_scale.clone(), g.v_scale.clone()
        g.set_fp8_scales(k4, v4, rope=rope, pos0=g.seq_lens)
        assert torch.equal(g.k_scale, dense[0]) and torch.equal(g.v_scale, dense[1])
    g.rope_append(q4, k4, v4, rope, new_lens=torch.from_numpy(new_lens).to(cuda))
    pos = torch.from_numpy(start.astype(np.int64))[:, None] + torch.arange(T)[None, :]
    kr, qr = (torch.stack([oatt.apply_rope(x[b], cos[pos[b]], sin[pos[b]]) for b in range(B)]) for x in (k, q))
    o.append(kr.float().numpy(), v.float().numpy(), new_lens=new_lens)
    assert np.array_equal(g.k_pool.cpu().numpy(), o.k_pool)
    assert np.array_equal(g.v_pool.cpu().numpy(), o.v_pool)
    for b in range(B):
        assert torch.equal(q4[b, :new_lens[b]].cpu(), qr[b, :new_lens[b]])


@pytest.mark.parametrize("name", ["fp32", "bf16"])
@pytest.mark.parametrize("B,Hkv,d", [(40, 3, 128), (20, 3, 64), (2, 3, 128)])
@pytest.mark.parametrize("T", [1, 37, 300])
def test_fp8_scales_of_head_groups(cuda, name, B, Hkv, d, T):
    """Four, two and one heads per CTA (the last group short): amax / 448 of the rotated keys and of the values."""
    from transformer_surgeon_b200 import ops
    rng = np.random.default_rng(23)
    o, g = make_pair("fp8", B, 1, Hkv, d, cuda, rng)
    k, v = outlier_kv(rng, B, T, Hkv, d, DT[name])
    cos, sin = oatt.rope_tables(d, 5e5, torch.arange(T + 8))
    start = torch.arange(B, dtype=torch.int32) % 8
    g.set_fp8_scales(k.to(cuda), v.to(cuda), rope=(cos.to(cuda), sin.to(cuda)), pos0=start.to(cuda))
    pos = start.long()[:, None] + torch.arange(T)[None, :]
    kr = torch.stack([oatt.apply_rope(k[b], cos[pos[b]], sin[pos[b]]) for b in range(B)])
    assert np.array_equal(g.k_scale.cpu().numpy(), kc.fp8_scale_from_amax(kr.float().abs().amax(dim=(1, 3)).numpy()))
    assert np.array_equal(g.v_scale.cpu().numpy(), kc.fp8_scale_from_amax(v.float().abs().amax(dim=(1, 3)).numpy()))


@pytest.mark.parametrize("fmt", FMTS)
@pytest.mark.parametrize("name", ["fp32", "bf16"])
@pytest.mark.parametrize("H,Hkv,d", [(14, 2, 64), (9, 9, 128), (0, 1, 128)])
@pytest.mark.parametrize("pad", [0, 3])
def test_large_chunks_equal_small_ones(cuda, fmt, name, H, Hkv, d, pad):
    """Four ragged sequences appended by themselves (small chunks: a warp per vector) and repeated until the chunk goes by page, its heads
    over one or several CTAs per page: the same records and rotated queries."""
    from transformer_surgeon_b200 import ops
    T, copies = 53, 12 if Hkv * d < 1000 else 2
    gen = torch.Generator(device=cuda).manual_seed(5)
    cos, sin = (x.to(cuda) for x in oatt.rope_tables(d, 5e5, torch.arange(96)))
    small = (torch.randn((4, T, (H + 2 * Hkv) * d + 2 * pad), generator=gen, device=cuda) * 3).to(DT[name])
    start = torch.tensor([0, 5, 16, 27], dtype=torch.int32, device=cuda)
    new_lens = torch.tensor([53, 32, 16, 0], dtype=torch.int32, device=cuda)
    runs = []
    for n in (1, copies, 8 * copies):
        B = 4 * n
        assert n == 1 or B * T * Hkv * d >= 1 << 18 or Hkv == 1
        buf = small.repeat(n, 1, 1)
        table = torch.arange(B * 5, dtype=torch.int32, device=cuda).reshape(B, 5)
        kv = ops.PagedKV(fmt, B * 5, Hkv, d, table, start.repeat(n), cuda)
        if fmt == "fp8":
            kv.fill_fp8_scales(torch.full((1,), 0.03, device=cuda), torch.full((1,), 0.02, device=cuda))
        q4 = buf[..., :H * d].unflatten(2, (H, d)) if H else None
        k4 = buf[..., H * d + pad:(H + Hkv) * d + pad].unflatten(2, (Hkv, d))
        v4 = buf[..., (H + Hkv) * d + pad:(H + 2 * Hkv) * d + pad].unflatten(2, (Hkv, d))
        if H:
            kv.rope_append(q4, k4, v4, (cos, sin), new_lens=new_lens.repeat(n))
        else:
            kv.append(k4, v4, new_lens=new_lens.repeat(n))
        runs.append((kv.k_pool.view(n, -1), kv.v_pool.view(n, -1), buf.view(n, -1)))
    for big in runs[1:]:
        for a, b in zip(big, runs[0]):
            assert torch.equal(a, b.expand_as(a))


@pytest.mark.parametrize("name", ["fp32", "bf16"])
@pytest.mark.parametrize("fmt", FMTS)
@pytest.mark.parametrize("d", [64, 128])
def test_append_of_infinities_and_of_quotients_beyond_the_type(cuda, fmt, name, d):
    """Infinities, NaN, the largest finite values and tiny ones, over FP8 scales fixed beforehand (quotients that overflow fp32): a token's
    codes do not depend on whether it came in a chunk (large enough for the kernel by page) or by itself, and FP8 codes saturate."""
    from transformer_surgeon_b200 import ops
    rng = np.random.default_rng(37)
    B, T, Hkv = 4096 // d, 35, 2
    _, bulk = make_pair(fmt, B, 3, Hkv, d, cuda, rng)
    single = ops.PagedKV(fmt, bulk.k_pool.shape[0], Hkv, d, bulk.block_table, torch.zeros(B, dtype=torch.int32, device=cuda), cuda)
    k, v = (x.float() for x in outlier_kv(rng, B, T, Hkv, d, DT[name]))
    big, inf = torch.finfo(DT[name]).max, float("inf")
    for x in (k, v):
        for i, val in enumerate((inf, -inf, big, -big, float("nan"), 1e-30, -1e-30)):
            x[:, 3 * i + 1, :, 5 * i + 2] = val
            x[:, 22 + i, :, (17 * i + 3) % d] = val
    k, v = k.to(DT[name]).to(cuda), v.to(DT[name]).to(cuda)
    for scales in (((1e-6, 0.25), (3e-18, 1e17), (0.0, inf), (-0.5, float("nan")), (1e-30, 1e30)) if fmt == "fp8" else ((1.0, 1.0),)):
        if fmt == "fp8":
            bulk.fill_fp8_scales(*scales)
            single.fill_fp8_scales(*scales)
        bulk.append(k, v)
        single.seq_lens.zero_()
        for t in range(T):
            single.append(k[:, t:t + 1].contiguous(), v[:, t:t + 1].contiguous())
            single.seq_lens += 1
        assert torch.equal(bulk.k_pool, single.k_pool)
        assert torch.equal(bulk.v_pool, single.v_pool)
    if fmt == "fp8":
        bulk.fill_fp8_scales(1e-6, 0.25)
        bulk.append(k, v)
        rec = bulk.k_pool[bulk.block_table[0, 0].long(), 0].cpu()          # head 0 of the first page: codes [16][d]
        codes = rec[:16 * d].view(16, d)
        assert [int(codes[3 * i + 1, 5 * i + 2]) for i in range(4)] == [0x7e, 0xfe, 0x7e, 0xfe]


@pytest.mark.parametrize("fmt", ["fp32", "bf16"])
@pytest.mark.parametrize("H,Hkv,d", [(4, 4, 128), (32, 8, 128), (6, 2, 64), (28, 4, 128)])
def test_unquantized_pages_of_many_sequences(cuda, fmt, H, Hkv, d):
    """Enough sequences to fill the machine, up to four query heads to a kv head and more: against the CUDA-core kernel (both in fp32)."""
    from transformer_surgeon_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(41)
    B, L = 60, 77
    table = torch.randperm(B * 5, generator=g, device=cuda).to(torch.int32).reshape(B, 5)
    seq = torch.zeros(B, dtype=torch.int32, device=cuda)
    kv = ops.PagedKV(fmt, B * 5, Hkv, d, table, seq, cuda)
    k, v = (torch.randn((B, L, Hkv, d), generator=g, device=cuda).to(DT[fmt]) for _ in range(2))
    kv.append(k, v)
    seq.copy_(torch.arange(B) % (L + 1))
    q = torch.randn((B, H, d), generator=g, device=cuda)
    out, ref = ops.paged_decode_attention(kv, q, L), ops.paged_decode_attention(kv, q, L, simt=True)
    # sums of 77 products of unit size in two orders, __expf against expf: 2e-4 of the values' scale, as for that kernel against the oracle
    assert (out - ref).abs().max() <= C_P_SIMT * v.float().abs().max()


def test_fp8_scales_of_flat_vectors(cuda):
    """Contiguous prompts may come with a token's heads as one vector; what is neither that nor evenly strided is refused."""
    rng = np.random.default_rng(43)
    _, g = make_pair("fp8", 3, 1, 2, 64, cuda, rng)
    k, v = (x.to(cuda) for x in outlier_kv(rng, 3, 7, 2, 64, torch.bfloat16))
    g.set_fp8_scales(k, v)
    ks, vs = g.k_scale.clone(), g.v_scale.clone()
    g.fill_fp8_scales(1.0, 1.0)
    g.set_fp8_scales(k.flatten(2), v.flatten(2))
    assert torch.equal(g.k_scale, ks) and torch.equal(g.v_scale, vs)
    for bad in (k.transpose(2, 3).contiguous().transpose(2, 3), k.cpu()):
        with pytest.raises(ValueError):
            g.set_fp8_scales(bad, v)


def test_fp8_attention_after_append_under_dependent_launch(cuda):
    """One decode step's append -> attention pair with programmatic dependent launch on: the attention may fetch pages
    older than the newest token before the append has finished.  Lengths sit on, before and after page boundaries and
    around the page count at which that early fetch starts; the result equals, bit for bit, the one with the setting
    off, and the oracle's within the attention tolerance."""
    from transformer_surgeon_b200 import ops
    rng = np.random.default_rng(29)
    B, H, Hkv, d = 32, 16, 4, 128                            # 128 (sequence, kv head) pairs: one split
    lens = np.array([0, 1, 15, 16, 17, 31, 32, 33, 95, 96, 97, 111, 112, 113, 127, 128, 129, 191, 192, 193, 207, 208, 209,
                     223, 224, 225, 239, 240, 241, 300, 400, 430], dtype=np.int32)
    o, g = make_pair("fp8", B, 28, Hkv, d, cuda, rng)
    T = int(lens.max())
    k, v = outlier_kv(rng, B, T + 1, Hkv, d, torch.bfloat16)
    sync_scales(o, g, k, v)
    nl = torch.from_numpy(lens).to(cuda)
    g.append(k[:, :T].to(cuda), v[:, :T].to(cuda), new_lens=nl)
    o.append(k[:, :T].float().numpy(), v[:, :T].float().numpy(), new_lens=lens)
    k_new = torch.stack([k[b, lens[b]] for b in range(B)]).unsqueeze(1).to(cuda)      # token at position lens[b]
    v_new = torch.stack([v[b, lens[b]] for b in range(B)]).unsqueeze(1).to(cuda)
    q = torch.from_numpy(rng.standard_normal((B, H, d)).astype(np.float32)).bfloat16().to(cuda)
    write_pos, after = nl.clone(), nl + 1
    outs = []
    for pdl in (False, True):
        old = ops.set_pdl(pdl)
        try:
            for _ in range(3):                               # the same token into the same slot every time
                g.append(k_new, v_new, seq_lens=write_pos)
                out = ops.paged_decode_attention(g, q, max_seq_len=448, seq_lens=after)
            torch.cuda.synchronize()
        finally:
            ops.set_pdl(old)
        outs.append(out.clone())
    assert torch.equal(outs[0], outs[1])
    o.seq_lens[:] = lens
    o.append(k_new.float().cpu().numpy(), v_new.float().cpu().numpy())
    o.seq_lens[:] = lens + 1
    ref, ref_abs = oatt.paged_decode_attention(o, q.float().cpu().numpy(), with_abs=True)
    tol = attn_tol(ref, ref_abs, "bf16", False)
    assert np.all(np.abs(outs[1].float().cpu().numpy() - ref) <= tol)


@pytest.mark.parametrize("fmt,H,Hkv,d", [("int8", 16, 8, 128), ("int8", 28, 4, 64), ("nvfp4", 28, 4, 128), ("nvfp4", 16, 8, 64), ("fp8", 28, 4, 128), ("fp8", 16, 8, 64),
                                          ("fp8", 32, 8, 128)])
@pytest.mark.parametrize("name", ["fp32", "bf16"])
@pytest.mark.parametrize("B", [304, 40])
def test_decode_attention_of_every_length(cuda, fmt, H, Hkv, d, B, name):
    """Every length from 0 to 303: pairs of pages to a warp's round, a single one at the end, warps without pages, splits too short for pairs; many
    sequences (one split, more CTAs than the GPU holds at a time) and few (several), against the one-lane-per-element kernel.  The bound is attn_tol's: keys without outlier channels
    and V's magnitudes through the same weights."""
    from transformer_surgeon_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(51)
    pages = 19
    bt = torch.randperm(B * pages, generator=g, device=cuda).to(torch.int32).reshape(B, pages)
    k, v = (torch.randn((B, pages * 16, Hkv, d), generator=g, device=cuda).to(DT[name]) for _ in range(2))
    q = torch.randn((B, H, d), generator=g, device=cuda).to(DT[name])
    lens = (torch.arange(B, device=cuda) * (304 // B) + (0 if B == 304 else 3)).to(torch.int32)
    refs = []
    for vals in (v.abs(), v):
        kv = ops.PagedKV(fmt, B * pages, Hkv, d, bt, torch.zeros(B, dtype=torch.int32, device=cuda), cuda)
        if fmt == "fp8":
            kv.fill_fp8_scales(6.0 / 448, 6.0 / 448)
        kv.append(k, vals)
        kv.seq_lens = lens
        refs.append(ops.paged_decode_attention(kv, q, pages * 16, simt=True).float())
    out = ops.paged_decode_attention(kv, q, pages * 16)
    assert torch.equal(out, ops.paged_decode_attention(kv, q, pages * 16))
    assert torch.all(out[lens == 0] == 0)
    assert torch.all((out.float() - refs[1]).abs() <= C_P_TC * refs[0] + 2 * C_OUT[name] * refs[1].abs() + 1e-6)


@pytest.mark.parametrize("fmt", FMTS)
@pytest.mark.parametrize("name", ["fp32", "bf16"])
def test_append_of_quotients_at_the_midpoints_of_codes(cuda, fmt, name):
    """bf16 elements of every significand over FP8 scales within a few ulps of the divisors that put one of them on the midpoint of two
    codes (and scales of all ones): by page as by vector, which divides."""
    from transformer_surgeon_b200 import ops
    rng = np.random.default_rng(53)
    B, T, Hkv, d = 64, 16, 2, 128
    _, bulk = make_pair(fmt, B, 1, Hkv, d, cuda, rng)
    single = ops.PagedKV(fmt, bulk.k_pool.shape[0], Hkv, d, bulk.block_table, torch.zeros(B, dtype=torch.int32, device=cuda), cuda)
    k, v = (torch.from_numpy((rng.integers(128, 256, (B, T, Hkv, d)) * 2.0 ** rng.integers(-17, 3, (B, T, Hkv, d)) * rng.choice([-1, 1], (B, T, Hkv, d))).astype(np.float32))
            .to(DT[name]).to(cuda) for _ in range(2))
    if fmt == "fp8":
        scales = []
        for _ in range(2):
            near = (rng.integers(128, 256, (B, Hkv)) / (2 * rng.integers(0, 16, (B, Hkv)) + 1)).astype(np.float32)
            s = (near.view(np.int32) + rng.integers(-4, 5, (B, Hkv))).astype(np.int32).view(np.float32)
            s[::8] = np.nextafter(np.float32(2.0), np.float32(0))
            scales.append(torch.from_numpy(s * np.float32(2.0 ** -6)).to(cuda))
        bulk.fill_fp8_scales(*scales)
        single.fill_fp8_scales(*scales)
    assert B * T * Hkv * d >= 1 << 18
    bulk.append(k, v)
    for t in range(T):
        single.append(k[:, t:t + 1].contiguous(), v[:, t:t + 1].contiguous())
        single.seq_lens += 1
    assert torch.equal(bulk.k_pool, single.k_pool)
    assert torch.equal(bulk.v_pool, single.v_pool)


@pytest.mark.parametrize("fmt,H,Hkv,d", [("int8", 16, 8, 128), ("nvfp4", 56, 8, 64), ("fp8", 64, 8, 128)])
@pytest.mark.parametrize("name", ["fp32", "bf16"])
def test_splits_merge_alike_in_a_cluster_and_in_a_launch(cuda, fmt, H, Hkv, d, name):
    """Four splits of up to 19 pages: 16 sequences merge in clusters, 40 in a launch of their own.  The first 16 of the 40 are the same bits."""
    from transformer_surgeon_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(57)
    B, pages = 40, 19
    bt = torch.randperm(B * pages, generator=g, device=cuda).to(torch.int32).reshape(B, pages)
    kv = ops.PagedKV(fmt, B * pages, Hkv, d, bt, torch.zeros(B, dtype=torch.int32, device=cuda), cuda)
    if fmt == "fp8":
        kv.fill_fp8_scales(6.0 / 448, 6.0 / 448)
    kv.append(*(torch.randn((B, pages * 16, Hkv, d), generator=g, device=cuda).to(DT[name]) for _ in range(2)))
    kv.seq_lens = (torch.arange(B, device=cuda) * 20 % 304).to(torch.int32)
    q = torch.randn((B, H, d), generator=g, device=cuda).to(DT[name])
    every = ops.paged_decode_attention(kv, q, pages * 16)
    few = ops.PagedKV(fmt, B * pages, Hkv, d, bt[:16].contiguous(), kv.seq_lens[:16].contiguous(), cuda)
    few.k_pool, few.v_pool = kv.k_pool, kv.v_pool
    if fmt == "fp8":
        few.fill_fp8_scales(6.0 / 448, 6.0 / 448)
    assert torch.equal(ops.paged_decode_attention(few, q[:16].contiguous(), pages * 16), every[:16])


@pytest.mark.parametrize("name", ["fp32", "bf16"])
def test_long_splits_have_the_bits_of_shorter_ones(cuda, name):
    """NVFP4, four splits: deeper rings from 64 pages a split on (a context limit of 4096), the same bits as below (4080)."""
    from transformer_surgeon_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(58)
    B, H, Hkv, d, pages = 40, 16, 8, 128, 256
    bt = torch.arange(B * pages, device=cuda).flip(0).to(torch.int32).reshape(B, pages)
    kv = ops.PagedKV("nvfp4", B * pages, Hkv, d, bt, torch.zeros(B, dtype=torch.int32, device=cuda), cuda)
    for _ in range(4):
        kv.append(*(torch.randn((B, 1020, Hkv, d), generator=g, device=cuda).to(DT[name]) for _ in range(2)))
        kv.seq_lens += 1020
    kv.seq_lens -= (torch.arange(B, device=cuda) * 97).to(torch.int32)
    q = torch.randn((B, H, d), generator=g, device=cuda).to(DT[name])
    assert torch.equal(ops.paged_decode_attention(kv, q, 4096), ops.paged_decode_attention(kv, q, 4080))


def filled_cache(fmt, B, pages, Hkv, d, name, cuda, g):
    """B sequences of pages * 16 tokens over scattered pages, and a function for the first n of them."""
    from transformer_surgeon_b200 import ops
    bt = torch.randperm(B * pages, generator=g, device=cuda).to(torch.int32).reshape(B, pages)
    kv = ops.PagedKV(fmt, B * pages, Hkv, d, bt, torch.zeros(B, dtype=torch.int32, device=cuda), cuda)
    if fmt == "fp8":
        kv.fill_fp8_scales(6.0 / 448, 6.0 / 448)
    kv.append(*(torch.randn((B, pages * 16, Hkv, d), generator=g, device=cuda).to(DT[name]) for _ in range(2)))

    def first(n):
        few = ops.PagedKV(fmt, B * pages, Hkv, d, bt[:n].contiguous(), kv.seq_lens[:n].contiguous(), cuda)
        few.k_pool, few.v_pool = kv.k_pool, kv.v_pool
        if fmt == "fp8":
            few.fill_fp8_scales(6.0 / 448, 6.0 / 448)
        return few
    return kv, first


@pytest.mark.parametrize("fmt,H,Hkv,B,few,S", [("fp8", 4, 1, 33, 33, 2)] + [("fp8", 4, 1, B, 33, S) for S, B in ((3, 96), (4, 73), (5, 58), (6, 48), (7, 40), (8, 37))]
                         + [(f, 8, 2, 128 if S == 3 else 75, 10, S) for f in ("int8", "nvfp4") for S in (3, 5, 6, 7)] + [("fp8", 10, 2, 75, 10, S) for S in (5, 6, 7)])
@pytest.mark.parametrize("name", ["fp32", "bf16"])
def test_clusters_of_every_size_merge_as_a_launch_does(cuda, fmt, H, Hkv, B, few, S, name):
    """Two to eight splits of a sequence: so many pairs that the clusters would not fit the device at once take the reduction launch, the first few
    of the same sequences clusters, with the same bits.  Both against the one-lane-per-element kernel (bound: attn_tol's)."""
    from transformer_surgeon_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(61)
    pages = 24 * S if fmt == "fp8" and H // Hkv <= 4 else 4 * S + 1          # as many as give S splits
    kv, first = filled_cache(fmt, B, pages, Hkv, 128, name, cuda, g)
    kv.seq_lens = (pages * 16 - torch.arange(B, device=cuda) * 37 % (pages * 16 + 1)).to(torch.int32)
    q = torch.randn((B, H, 128), generator=g, device=cuda).to(DT[name])
    out = ops.paged_decode_attention(kv, q, pages * 16)
    assert torch.equal(ops.paged_decode_attention(first(few), q[:few].contiguous(), pages * 16), out[:few])
    ref = ops.paged_decode_attention(kv, q, pages * 16, simt=True).float()
    scale = 6.0 if fmt == "fp8" else 5.0                                    # |V| of N(0, 1)
    assert torch.all((out.float() - ref).abs() <= C_P_TC * scale + 2 * C_OUT[name] * ref.abs() + 1e-6)


@pytest.mark.parametrize("fmt,d,B,Hkv,pages", [("nvfp4", 64, 90, 12, 7), ("nvfp4", 64, 64, 12, 2), ("fp8", 64, 90, 12, 7), ("fp8", 64, 64, 12, 1),
                                               ("nvfp4", 128, 40, 16, 3), ("nvfp4", 128, 30, 16, 3)])
@pytest.mark.parametrize("name", ["fp32", "bf16"])
def test_attention_of_many_and_of_few_ctas(cuda, fmt, d, B, Hkv, pages, name):
    """The instances for more CTAs than the GPU holds and for fewer (more warps against more registers; rings of four pages where more than two CTAs an SM
    and all of them fit): the first sequences of many are the same bits by themselves."""
    from transformer_surgeon_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(62)
    kv, first = filled_cache(fmt, B, pages, Hkv, d, name, cuda, g)
    kv.seq_lens = (torch.arange(B, device=cuda) * 13 % (pages * 16 + 1)).to(torch.int32)
    q = torch.randn((B, 2 * Hkv, d), generator=g, device=cuda).to(DT[name])
    n = 9                                                       # (fewer than eight pages: one split, however few the sequences)
    out = ops.paged_decode_attention(kv, q, pages * 16)
    assert torch.equal(ops.paged_decode_attention(first(n), q[:n].contiguous(), pages * 16), out[:n])


@pytest.mark.parametrize("fmt,H,Hkv,d", [("int8", 16, 4, 128), ("nvfp4", 16, 4, 128), ("fp8", 20, 4, 128), ("fp8", 8, 4, 64)])
@pytest.mark.parametrize("limit", [48, 448, 4096])
def test_attention_after_append_under_dependent_launch(cuda, fmt, H, Hkv, d, limit):
    """As the test above for the other kernel, which looks lengths and pages up ahead of its wait: the token of the append before it is in the
    result, with one split, a cluster and a reduction launch."""
    from transformer_surgeon_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(63)
    B = 6
    kv, _ = filled_cache(fmt, B, limit // 16, Hkv, d, "bf16", cuda, g)
    lens = torch.tensor([0, 15, 16, limit - 1, limit // 2, 31], dtype=torch.int32, device=cuda)
    k, v = (torch.randn((B, 1, Hkv, d), generator=g, device=cuda).bfloat16() for _ in range(2))
    q = torch.randn((B, H, d), generator=g, device=cuda).bfloat16()
    after, outs = lens + 1, []
    for pdl in (False, True):
        old = ops.set_pdl(pdl)
        try:
            for sign in (-1, 1):                                 # another token into the same slot first
                kv.append(sign * k, sign * v, seq_lens=lens)
                out = ops.paged_decode_attention(kv, q, limit, seq_lens=after)
            torch.cuda.synchronize()
        finally:
            ops.set_pdl(old)
        outs.append(out.clone())
    assert torch.equal(outs[0], outs[1])
    ref = ops.paged_decode_attention(kv, q, limit, seq_lens=lens + 1, simt=True)
    assert torch.all((outs[1].float() - ref.float()).abs() <= C_P_TC * 6.0 + 2 * C_OUT["bf16"] * ref.float().abs() + 1e-6)
