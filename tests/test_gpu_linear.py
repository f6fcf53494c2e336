"""LinearCompressed.forward on the GPU against the oracle and the reference's outputs."""
import numpy as np
import pytest
import torch

from oracle import linear as olin
from oracle import weight_quant as wq

pytestmark = pytest.mark.gpu
DT = {"fp32": torch.float32, "bf16": torch.bfloat16}
# stated tolerance: bf16 max-rel-err <= 1e-2 (relative to the largest |y|); fp32 1e-4
TOL = {"fp32": 1e-4, "bf16": 1e-2}


def rel_err(y, ref):
    return ((y.float() - ref.float()).abs().max() / ref.float().abs().max()).item()


@pytest.mark.parametrize("name", ["fp32", "bf16"])
@pytest.mark.parametrize("simt", [True, False])
def test_reference_fixture(cuda, golden, name, simt):
    from transformer_surgeon_b200 import ops
    g = golden("linear.npz")
    dt = DT[name]
    x = g[f"x_{name}"].to(cuda)
    lin = ops.PackedLinear(ops.Factor.dense(g["W"].to(dt).to(cuda)), None, g["bias"].to(dt).to(cuda), dt)
    lin.force_simt = simt
    y = lin(x)
    assert y.shape == (2, 5, 192)
    assert rel_err(y.cpu(), g[f"y_full_{name}"]) < TOL[name]
    lin = ops.PackedLinear(ops.Factor.dense(g[f"US_{name}"].to(cuda)), ops.Factor.dense(g[f"V_{name}"].to(cuda)), None, dt)
    lin.force_simt = simt
    assert rel_err(lin(x).cpu(), g[f"y_lrd_{name}"]) < TOL[name]
    for p in (8, 4, "binary"):
        fu = ops.Factor.from_codes(g[f"qu_{p}_{name}"].to(cuda), g[f"su_{p}_{name}"].to(cuda), p)
        fv = ops.Factor.from_codes(g[f"qv_{p}_{name}"].to(cuda), g[f"sv_{p}_{name}"].to(cuda), p)
        lin = ops.PackedLinear(fu, fv, None, dt)
        lin.force_simt = simt
        assert rel_err(lin(x).cpu(), g[f"y_lrd_q{p}_{name}"]) < TOL[name], (p, name)


def _case(M, K, N, r, p, name, seed=0):
    g = torch.Generator().manual_seed(seed)
    dt = DT[name]
    x = torch.randn(M, K, generator=g).to(dt)
    if r:
        U = (torch.randn(N, r, generator=g) * 0.05).to(dt)
        V = (torch.randn(r, K, generator=g) * 0.05).to(dt)
    else:
        U = (torch.randn(N, K, generator=g) * 0.05).to(dt)
        V = None
    b = (torch.randn(N, generator=g) * 0.1).to(dt)
    return x, U, V, b


@pytest.mark.parametrize("name", ["bf16", "fp32"])
@pytest.mark.parametrize("p", [8, 4, 2, "binary", None])
@pytest.mark.parametrize("M,K,N,r", [(1, 256, 192, 64), (5, 896, 128, 0), (16, 512, 320, 128), (33, 1024, 256, 0),
                                     (128, 1024, 512, 256), (200, 320, 72, 64)])
def test_against_oracle(cuda, name, p, M, K, N, r):
    from transformer_surgeon_b200 import ops
    dt = DT[name]
    x, U, V, b = _case(M, K, N, r, p, name)
    if p is None:
        fu, fv = ops.Factor.dense(U.to(cuda)), (ops.Factor.dense(V.to(cuda)) if r else None)
        Ud, Vd = U, V
    else:
        fu = ops.Factor.quantize(U.to(cuda), p)
        fv = ops.Factor.quantize(V.to(cuda), p) if r else None
        qu, su = wq.quantize_vanilla(U.float().numpy(), p, 1e-6, "per_channel", name)
        assert np.array_equal(fu.codes().cpu().numpy(), qu)
        Ud = torch.from_numpy(wq.dequantize(qu, su, name)).to(dt)
        Vd = None
        if r:
            qv, sv = wq.quantize_vanilla(V.float().numpy(), p, 1e-6, "per_channel", name)
            Vd = torch.from_numpy(wq.dequantize(qv, sv, name)).to(dt)
    ref32 = olin.linear_compressed_fp32(x, Ud, b, Vd)
    for simt in (True, False):
        lin = ops.PackedLinear(fu, fv, b.to(cuda), dt)
        lin.force_simt = simt
        y = lin(x.to(cuda)).cpu()
        assert rel_err(y, ref32) < TOL[name], (simt, rel_err(y, ref32))


@pytest.mark.parametrize("p", [4, 8, "binary"])
@pytest.mark.parametrize("M,K,N,r", [(300, 2048, 1000, 0),      # two 256-token tiles (one ragged), 8-way split-K, ragged row tile
                                     (700, 1024, 2052, 256),    # N not a multiple of 8: outputs leave as single elements
                                     (257, 4096, 136, 1024),    # one token past a tile, 18-way split-K then 4-way
                                     (1024, 512, 4096, 0),      # no split-K, several items per CTA
                                     (129, 832, 264, 0)])       # K not a multiple of the k-block pair
def test_prompt_sized_token_counts(cuda, p, M, K, N, r):
    """More than 128 tokens: the 256-token tile with its transposed 16-byte output stores, every split-K batch
    shape, ragged tiles in both directions; bf16, max-rel-err <= 1e-2 against the fp32 result on the dequantized
    factors, and a second identical call returns the same bits."""
    from transformer_surgeon_b200 import ops
    x, U, V, b = _case(M, K, N, r, p, "bf16", seed=5)
    fu = ops.Factor.quantize(U.to(cuda), p)
    fv = ops.Factor.quantize(V.to(cuda), p) if r else None
    Ud = fu.reconstruct(torch.bfloat16).cpu()
    Vd = fv.reconstruct(torch.bfloat16).cpu() if r else None
    ref32 = olin.linear_compressed_fp32(x, Ud, b, Vd)
    lin = ops.PackedLinear(fu, fv, b.to(cuda), torch.bfloat16)
    y = lin(x.to(cuda))
    assert rel_err(y.cpu(), ref32) < TOL["bf16"], rel_err(y.cpu(), ref32)
    # element-wise: no output may be missing or misplaced (a max-error bound alone would let a zero row through)
    err = (y.cpu().float() - ref32.float()).abs()
    assert (err <= 2e-2 * ref32.float().abs() + 1e-2 * ref32.float().abs().max()).all()
    assert torch.equal(lin(x.to(cuda)), y)


@pytest.mark.parametrize("p", [4, 8, 2, "binary"])
@pytest.mark.parametrize("M,K,N,r", [(1, 72, 37, 0),            # one partial K block per chain pair, rows beyond the last tile
                                     (8, 4096, 256, 0),         # 16 K splits over a cluster, full token tile
                                     (9, 1000, 4100, 136),      # second token tile with one token; K and rank end inside a block; odd block counts
                                     (16, 14336, 520, 0),       # most splits, uneven last split, N not a multiple of 16
                                     (13, 8, 8, 8)])            # smallest
def test_decode_sized_token_counts(cuda, p, M, K, N, r):
    """At most 16 tokens: warp-level kernel with one accumulation chain per warp; every output within 1e-2 of the fp32
    result on the dequantized factors, and a second call returns the same bits."""
    from transformer_surgeon_b200 import ops
    x, U, V, b = _case(M, K, N, r, p, "bf16", seed=9)
    fu = ops.Factor.quantize(U.to(cuda), p)
    fv = ops.Factor.quantize(V.to(cuda), p) if r else None
    ref32 = olin.linear_compressed_fp32(x, fu.reconstruct(torch.bfloat16).cpu(), b, fv.reconstruct(torch.bfloat16).cpu() if r else None)
    lin = ops.PackedLinear(fu, fv, b.to(cuda), torch.bfloat16)
    y = lin(x.to(cuda))
    err = (y.cpu().float() - ref32.float()).abs()
    assert (err <= 2e-2 * ref32.float().abs() + 1e-2 * ref32.float().abs().max()).all()
    assert torch.equal(lin(x.to(cuda)), y)


@pytest.mark.parametrize("p", [None, 8, 4, 2, "binary"])
@pytest.mark.parametrize("M,K,N,r", [(1, 8200, 37, 0),          # one token past a staged K tile, K split over the warps of a CTA
                                     (2, 72, 300, 0), (3, 904, 1000, 40), (5, 2056, 64, 0), (9, 264, 130, 24),
                                     (16, 40, 65, 8), (67, 264, 1000, 136), (130, 512, 4100, 0)])   # 64 x 64 tiles (dense), ragged in both directions
def test_fp32_layers(cuda, p, M, K, N, r):
    """fp32 activations: every token group (1, 2, 4, 8 tokens), ragged rows, pieces that end inside a word of codes; a group of
    layers equals the layers one by one up to the order of summation."""
    from transformer_surgeon_b200 import ops
    x, U, V, b = _case(M, K, N, r, p, "fp32", seed=4)
    mk = (lambda w: ops.Factor.dense(w.to(cuda))) if p is None else (lambda w: ops.Factor.quantize(w.to(cuda), p))
    fu, fv = mk(U), mk(V) if r else None
    ref = olin.linear_compressed_fp32(x, fu.reconstruct(torch.float32).cpu(), b, fv.reconstruct(torch.float32).cpu() if r else None)
    lin = ops.PackedLinear(fu, fv, b.to(cuda), torch.float32)
    y = lin(x.to(cuda))
    assert rel_err(y.cpu(), ref) < 1e-5
    small = ops.PackedLinear(mk(U[:5]), fv, None, torch.float32)
    ya, yb = ops.LinearGroup([lin, small])(x.to(cuda))
    torch.testing.assert_close(ya, y, rtol=1e-5, atol=1e-5)
    torch.testing.assert_close(yb, small(x.to(cuda)), rtol=1e-5, atol=1e-5)


def test_group_follows_its_layers(cuda):
    """A group of layers marked for the CUDA-core kernel runs on it; a decoder layer's group has the layers it has now."""
    from transformer_surgeon_b200 import ops
    from transformer_surgeon_b200.decoder import LayerWeights
    g = torch.Generator(device=cuda).manual_seed(36)
    mk = lambda n: ops.PackedLinear(ops.Factor.dense(torch.randn((n, 512), generator=g, device=cuda)), None, None, torch.float32)
    x = torch.randn((5, 512), generator=g, device=cuda)
    q, k, v = mk(64), mk(32), mk(32)
    L = LayerWeights(None, None, mk(64), mk(64), mk(64), mk(64), q=q, k=k, v=v)
    first = L.qkv_group(x)
    assert L.qkv_group is L.qkv_group
    for l in (q, k, v):
        l.force_simt = True
    for y, l in zip(L.qkv_group(x), (q, k, v)):
        assert torch.equal(y, l(x))
    for l in (q, k, v):
        l.force_simt = False
    L.k = mk(32)
    again = L.qkv_group(x)
    assert torch.equal(again[0], first[0]) and not torch.equal(again[1], first[1])
    torch.testing.assert_close(again[1], L.k(x), rtol=1e-5, atol=1e-4)


def test_config2_shape_sweep(cuda):
    """x [M, 4096], W 4096x4096 factored at r in {256, 1024}, 8/4-bit + binary factors, bf16:
    compared with the dequantized fp32 result (max-rel-err <= 1e-2)."""
    from transformer_surgeon_b200 import ops
    g = torch.Generator().manual_seed(2)
    for r in (256, 1024):
        U = (torch.randn(4096, r, generator=g) * 0.02).bfloat16().to(cuda)
        V = (torch.randn(r, 4096, generator=g) * 0.02).bfloat16().to(cuda)
        for p in (8, 4, "binary"):
            fu, fv = ops.Factor.quantize(U, p), ops.Factor.quantize(V, p)
            Ud, Vd = fu.reconstruct(torch.bfloat16).float(), fv.reconstruct(torch.bfloat16).float()
            lin = ops.PackedLinear(fu, fv, None, torch.bfloat16)
            for M in (1, 16, 128, 2048):
                x = torch.randn(M, 4096, generator=g).bfloat16().to(cuda)
                ref = (x.float() @ Vd.T) @ Ud.T
                y = lin(x)
                assert rel_err(y, ref) < 1e-2, (r, p, M, rel_err(y, ref))


def test_linearity_and_leading_shape(cuda):
    from transformer_surgeon_b200 import ops
    x, U, V, b = _case(6, 512, 128, 64, 4, "fp32")
    lin = ops.PackedLinear(ops.Factor.quantize(U.to(cuda), 4), ops.Factor.quantize(V.to(cuda), 4), None, torch.float32)
    xa = x.to(cuda)
    y1 = lin(xa)
    y2 = lin((2.0 * xa).reshape(2, 3, 512)).reshape(6, 128)
    torch.testing.assert_close(2.0 * y1, y2, rtol=1e-5, atol=1e-5)
    assert lin(xa[:0]).shape == (0, 128)


@pytest.mark.parametrize("name", ["bf16", "fp32"])
@pytest.mark.parametrize("p", [8, 4, None])
@pytest.mark.parametrize("M,K,I,r,N", [(32, 512, 7168, 256, 512), (12, 512, 7168, 0, 384), (32, 256, 640, 64, 256), (5, 256, 640, 64, 256)])
def test_gated_mlp_block(cuda, name, p, M, K, I, r, N):
    """MLPGated.forward (blocks/mlp.py:171-185): fused one-launch path (wide intermediate, bf16, 9<=M<=64)
    and the composed path, against the oracle's silu(gate)*up -> down in fp32 from the dequantized factors."""
    from transformer_surgeon_b200 import ops
    from oracle import attention as oatt
    dt = DT[name]
    g = torch.Generator().manual_seed(7)
    x = torch.randn(M, K, generator=g).to(dt)

    def layer(out, inn, rank, bias):
        U = (torch.randn(out, rank or inn, generator=g) * (0.5 / (rank or inn) ** 0.5)).to(dt)
        V = (torch.randn(rank, inn, generator=g) * (1.0 / inn ** 0.5)).to(dt) if rank else None
        b = (torch.randn(out, generator=g) * 0.1).to(dt) if bias else None
        if p is None:
            fu, fv = ops.Factor.dense(U.to(cuda)), (ops.Factor.dense(V.to(cuda)) if rank else None)
        else:
            fu, fv = ops.Factor.quantize(U.to(cuda), p), (ops.Factor.quantize(V.to(cuda), p) if rank else None)
        lin = ops.PackedLinear(fu, fv, None if b is None else b.to(cuda), dt)
        Ud = fu.reconstruct(dt).float().cpu()
        Vd = fv.reconstruct(dt).float().cpu() if rank else None
        return lin, (Ud, Vd, None if b is None else b.float())

    gate, gw = layer(I, K, r, True)
    up, uw = layer(I, K, r, False)
    down, dw = layer(N, I, r, True)

    def ref_lin(t, w):
        U, V, b = w
        h = t @ V.T if V is not None else t
        y = h @ U.T
        return y + b if b is not None else y

    ref = ref_lin(oatt.swiglu(ref_lin(x.float(), gw), ref_lin(x.float(), uw)), dw)
    mlp = ops.GatedMLP(gate, up, down)
    y = mlp(x.to(cuda))
    y2 = mlp(x.to(cuda))
    if p is None:       # dense factors: the bf16 kernel adds its K splits with fp32 atomics (order varies)
        assert rel_err(y, y2) < 1e-2
    else:               # packed factors: deterministic split-K, workspace left clean
        assert torch.equal(y, y2)
    assert rel_err(y.cpu(), ref) < (2e-2 if name == "bf16" else 1e-4), rel_err(y.cpu(), ref)
    # identical to composing the public pieces
    yc = down(ops.swiglu(gate(x.to(cuda)), up(x.to(cuda))))
    assert rel_err(y, yc) < (1e-2 if name == "bf16" else 1e-5)
    assert ops.PackedLinear.device_status(ws=ops.workspace(cuda, 1, "mlp")) == 0


@pytest.mark.parametrize("p", [8, 4, 2, "binary"])
@pytest.mark.parametrize("M,K,I,r", [(129, 512, 14336, 256), (257, 256, 14344, 0), (300, 512, 7304, 136), (2048, 512, 2048, 128), (2500, 1024, 4104, 0), (200, 512, 640, 64), (350, 4096, 7296, 576)])
def test_gated_mlp_prompt(cuda, p, M, K, I, r):
    """More than 128 tokens: gate's tiles read by up's outputs (one to several items per CTA, ragged tokens and rows, K splits in the
    V phase, items shorter than the ring of stages), or the composed path where up's tiles split K; the same bits as composing the
    pieces."""
    from transformer_surgeon_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(11)
    x = torch.randn(M, K, generator=g, device=cuda).bfloat16()

    def layer(out, inn, rank, bias):
        U = (torch.randn(out, rank or inn, generator=g, device=cuda) * (rank or inn) ** -0.5).bfloat16()
        V = (torch.randn(rank, inn, generator=g, device=cuda) * inn ** -0.5).bfloat16() if rank else None
        return ops.PackedLinear(ops.Factor.quantize(U, p), ops.Factor.quantize(V, p) if rank else None,
                                torch.randn(out, generator=g, device=cuda).bfloat16() if bias else None, torch.bfloat16)

    gate, up, down = layer(I, K, r, True), layer(I, K, r, True), layer(256, I, r, False)
    mlp = ops.GatedMLP(gate, up, down)
    y, y2 = mlp(x), mlp(x)
    assert torch.equal(y, y2)
    a = ops.swiglu(gate(x), up(x))
    assert torch.equal(y, down(a))
    assert ops.PackedLinear.device_status(ws=ops.workspace(cuda, 1, "mlp")) == 0


def test_every_gate_of_a_prompt(cuda):
    """All finite bf16 gates through the block whose up outputs take SiLU(gate) along: the bits of the separate kernels."""
    from transformer_surgeon_b200 import ops
    bits = torch.arange(65536, dtype=torch.int32)
    gates = bits[(bits & 0x7f80) != 0x7f80].to(torch.int16).view(torch.bfloat16).to(cuda)
    g = torch.Generator(device=cuda).manual_seed(37)
    x = torch.zeros((gates.numel(), 64), dtype=torch.bfloat16, device=cuda)
    # up within +-1: a product beyond the type would be infinite, and infinity times the zeros of `down` NaN
    x[:, 0], x[:, 1] = gates, torch.randn(gates.numel(), generator=g, device=cuda).clamp(-1, 1).bfloat16()

    def copies(n, k, column):                                     # n outputs that are column `column` of the input (None: one each)
        codes = torch.zeros((n, k), dtype=torch.int8, device=cuda)
        codes[torch.arange(n), torch.arange(n) if column is None else column] = 1
        return ops.PackedLinear(ops.Factor.from_codes(codes, torch.ones(n, device=cuda), 8), None, None, torch.bfloat16)

    gate, up, down = copies(64, 64, 0), copies(64, 64, 1), copies(64, 64, None)
    y = ops.GatedMLP(gate, up, down)(x)
    assert torch.equal(gate(x)[:, 0], x[:, 0])
    ref = down(ops.swiglu(gate(x), up(x)))
    off = (y != ref).any(1)
    assert not off.any(), (int(off.sum()), gates[off][:8], y[off][:8, 0], ref[off][:8, 0])
    want = torch.nn.functional.silu(gates.double()).bfloat16().double()
    got = ops.swiglu(gates[:, None].expand(-1, 8).contiguous(), torch.ones((gates.numel(), 8), dtype=torch.bfloat16, device=cuda))[:, 0].double()
    assert got.isfinite().all()
    assert ((got - want).abs() <= 2 ** -7 * want.abs() + 2e-36).all()      # one rounding apart at most; exp(-gate) overflows fp32 below -88.7


@pytest.mark.parametrize("p", [8, 4, 2, "binary"])
@pytest.mark.parametrize("M,K,N", [(129, 128, 40000), (256, 64, 19072), (600, 192, 12928), (1000, 320, 9004), (4100, 256, 2560), (777, 1280, 6150),
                                   (300, 1024, 3600), (250, 1024, 4104), (131, 2048, 2200), (1000, 1024, 640)])
def test_many_short_items_per_cta(cuda, p, M, K, N):
    """256-token tiles: items of one to a few stages, widened ahead of the previous item's outputs; ragged tokens, rows and row pitches;
    K ranges shared by two, four, eight and seven CTAs."""
    from transformer_surgeon_b200 import ops
    if p == "binary":
        K = (K + 127) // 128 * 128
    g = torch.Generator(device=cuda).manual_seed(12)
    f = ops.Factor.quantize((torch.randn(N, K, generator=g, device=cuda) * K ** -0.5).bfloat16(), p)
    b = torch.randn(N, generator=g, device=cuda).bfloat16()
    x = torch.randn(M, K, generator=g, device=cuda).bfloat16()
    lin = ops.PackedLinear(f, None, b, torch.bfloat16)
    y = lin(x)
    ref = x.float() @ f.reconstruct(torch.float32).T + b.float()
    assert (y.float() - ref).abs().max() <= 2 ** -8 * ref.abs().max()
    assert torch.equal(y, lin(x))


@pytest.mark.parametrize("p", [4, 8, 2, "binary"])
@pytest.mark.parametrize("M,K,N,r", [(32, 4096, 4096, 0),        # o_proj
                                     (32, 4096, 6144, 0),        # q|k|v
                                     (7, 3584, 4608, 0),         # config-5 q|k|v
                                     (16, 4096, 14336, 1024),    # low-rank pair
                                     (32, 14336, 4096, 1024),    # down_proj: long K
                                     (32, 1792, 200, 0),         # rows not a multiple of 16 / 8
                                     (3, 896, 72, 64)])          # K tail, tiny N
def test_few_tokens_at_model_widths(cuda, p, M, K, N, r):
    """Packed linears at decode token counts and the widths of the benchmark models (split-K over many CTAs, odd
    row counts, K tails): against the fp32 oracle on the dequantized factors (bf16: max-rel-err <= 1e-2); the
    result must not change from run to run (fixed summation order)."""
    from transformer_surgeon_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(31)
    rnd = lambda a, b, s: (torch.randn((a, b), generator=g, device=cuda) * s).bfloat16()
    if r:
        fu, fv = ops.Factor.quantize(rnd(N, r, 0.05), p), ops.Factor.quantize(rnd(r, K, 0.05), p)
    else:
        fu, fv = ops.Factor.quantize(rnd(N, K, 0.05), p), None
    bias = rnd(1, N, 0.1)[0].contiguous()
    lin = ops.PackedLinear(fu, fv, bias, torch.bfloat16)
    x = rnd(M, K, 1.0)
    Ud = fu.reconstruct(torch.bfloat16).float()
    h = x.float() @ fv.reconstruct(torch.bfloat16).float().T if r else x.float()
    ref = h @ Ud.T + bias.float()
    y = lin(x)
    y2 = lin(x)
    assert torch.equal(y, y2)
    assert rel_err(y, ref) < 1e-2, rel_err(y, ref)
    assert ops.PackedLinear.device_status(device=cuda) == 0


@pytest.mark.parametrize("p", [4, 8, 2, "binary"])
@pytest.mark.parametrize("K,N,r", [(4096, 4096, 0), (896, 4864, 0), (3584, 1024, 0), (14336, 4096, 1024), (11008, 6144, 0), (8192, 14336, 0), (640, 200, 0)])
def test_few_tokens_have_the_bits_of_more(cuda, p, K, N, r):
    """Up to 16 tokens run on warp-level MMAs or on the tcgen05 kernel, whichever is modelled to be faster, more always on the latter: the
    same bits, token by token."""
    from transformer_surgeon_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(32)
    def factor(a, b):
        w = (torch.randn((a, b), generator=g, device=cuda) * 0.05).bfloat16()
        return ops.Factor.quantize(torch.where(w == 0, torch.full_like(w, 0.01), w), p)
    lin = ops.PackedLinear(factor(N, r or K), factor(r, K) if r else None, torch.randn(N, generator=g, device=cuda).bfloat16(), torch.bfloat16)
    x = torch.randn((32, K), generator=g, device=cuda).bfloat16()
    y = lin(x)
    for m in (1, 2, 6, 8, 9, 12, 16):
        assert torch.equal(lin(x[:m]), y[:m]), m


@pytest.mark.parametrize("M", [1, 5, 16])
@pytest.mark.parametrize("N", [1, 33, 100, 4099])
@pytest.mark.parametrize("shift", [0, 1])
def test_few_tokens_with_a_bias_of_any_length_and_place(cuda, M, N, shift):
    """A bias of odd length, or that starts within a 32-bit word: its first and last elements share their words with what is not bias."""
    from transformer_surgeon_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(35)
    buf = torch.randn(N + 2, generator=g, device=cuda).bfloat16()
    f = ops.Factor.quantize((torch.randn((N, 512), generator=g, device=cuda) * 0.05).bfloat16(), 4)
    x = torch.randn((M, 512), generator=g, device=cuda).bfloat16()
    bias = buf[shift:shift + N]
    y = ops.PackedLinear(f, None, bias, torch.bfloat16)(x)
    plain = x.float() @ f.reconstruct(torch.float32).T + bias.float()
    assert (y.float() - plain).abs().max() <= 2 ** -8 * plain.abs().max()


@pytest.mark.parametrize("p", [4, 8, 2])
@pytest.mark.parametrize("K,I,r", [(896, 7296, 0), (3584, 18944, 0), (4096, 14336, 1024), (512, 7168, 64)])
def test_few_tokens_of_an_mlp_have_the_bits_of_more(cuda, p, K, I, r):
    """The same for the gated block: chained launches or phases of one, silu(gate) * up rounded alike."""
    from transformer_surgeon_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(34)
    def layer(o, i):
        f = lambda a, b: ops.Factor.quantize((torch.randn((a, b), generator=g, device=cuda) * b ** -0.5).bfloat16(), p)
        return ops.PackedLinear(f(o, r or i), f(r, i) if r else None, torch.randn(o, generator=g, device=cuda).bfloat16(), torch.bfloat16)
    mlp = ops.GatedMLP(layer(I, K), layer(I, K), layer(K, I))
    x = torch.randn((32, K), generator=g, device=cuda).bfloat16()
    y = mlp(x)
    for m in (1, 6, 8, 9, 12, 16):
        assert torch.equal(mlp(x[:m]), y[:m]), m


@pytest.mark.parametrize("M,K,N,r,shift", [(16, 7232, 14336, 0, 0), (8, 14144, 14336, 0, 0), (16, 1024, 14336, 7232, 0), (16, 7232, 14336, 192, 0),
                                           (1, 192, 72, 0, 1), (16, 320, 64, 192, 3), (17, 192, 72, 0, 1)])
def test_binary_rows_of_an_odd_number_of_blocks(cuda, M, K, N, r, shift):
    """1-bit rows that the copy engine does not take (an odd number of 64-column blocks): where the decode-sized kernel has no plan (its
    activations do not fit an SM) or x lies at any alignment (`shift` elements into a buffer), the call runs all the same."""
    from transformer_surgeon_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(33)
    rnd = lambda a, b, s: (torch.randn((a, b), generator=g, device=cuda) * s).bfloat16()
    signs = lambda a, b: rnd(a, b, 0.05).abs().clamp_min(1e-4) * (torch.randint(0, 2, (a, b), generator=g, device=cuda) * 2 - 1).bfloat16()   # no zeros
    fu = ops.Factor.quantize(signs(N, r or K), "binary")
    fv = ops.Factor.quantize(signs(r, K), "binary") if r else None
    assert fu.bits == 1
    bias = rnd(1, N, 0.1)[0].contiguous()
    buf = torch.empty(M * K + shift, dtype=torch.bfloat16, device=cuda)
    x = buf[shift:].view(M, K).copy_(rnd(M, K, 1.0))
    h = (x.float() @ fv.reconstruct(torch.bfloat16).float().T).bfloat16().float() if r else x.float()
    ref = h @ fu.reconstruct(torch.bfloat16).float().T + bias.float()
    y = ops.PackedLinear(fu, fv, bias, torch.bfloat16)(x)
    assert rel_err(y, ref) < 1e-2


@pytest.mark.parametrize("M,K,N", [(1, 512, 1000), (32, 1024, 50257), (100, 256, 4099)])
def test_greedy_head_equals_argmax_of_logits(cuda, M, K, N):
    """tsb200_linear_argmax on a dense bf16 head (reduction in the GEMM epilogue, logits never stored) picks the token
    torch.argmax picks from tsb200_linear's logits - including ties, which go to the first maximum."""
    from transformer_surgeon_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(41)
    W = (torch.randn((N, K), generator=g, device=cuda) * 0.05).bfloat16()
    W[N - 3] = W[7]                                      # duplicated rows: their logits tie exactly
    W[N // 2] = W[7]
    b = (torch.randn(N, generator=g, device=cuda) * 0.1).bfloat16()
    b[N - 3] = b[7]
    b[N // 2] = b[7]
    x = torch.randn((M, K), generator=g, device=cuda).bfloat16()
    x[0] = W[7].float().sign().bfloat16()                # make row 7 (and its copies) the winner for token 0
    lin = ops.PackedLinear(ops.Factor.dense(W), None, b, torch.bfloat16)
    logits = lin(x)
    toks = lin.argmax(x)
    assert torch.equal(toks, torch.argmax(logits, dim=-1))
    assert int(toks[0]) == 7
    assert torch.equal(lin.argmax(x), toks)


def test_greedy_head_general_route(cuda):
    """A packed low-rank head and an fp32 head: logits into the workspace, then the library's own argmax kernel."""
    from transformer_surgeon_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(42)
    U = (torch.randn((3000, 64), generator=g, device=cuda) * 0.05).bfloat16()
    V = (torch.randn((64, 256), generator=g, device=cuda) * 0.05).bfloat16()
    lin = ops.PackedLinear(ops.Factor.quantize(U, 4), ops.Factor.quantize(V, 4), None, torch.bfloat16)
    x = torch.randn((9, 256), generator=g, device=cuda).bfloat16()
    assert torch.equal(lin.argmax(x), torch.argmax(lin(x), dim=-1))
    W = torch.randn((777, 96), generator=g, device=cuda)
    lin32 = ops.PackedLinear(ops.Factor.dense(W), None, None, torch.float32)
    x32 = torch.randn((5, 96), generator=g, device=cuda)
    assert torch.equal(lin32.argmax(x32), torch.argmax(lin32(x32), dim=-1))


def test_split_k_launches_repeat_bit_for_bit(cuda):
    """The split-K exchange (slices in global memory, one fence by the signalling thread, acquire polling, wrap-around
    tile counters) and the grid barriers of the fused MLP under programmatic dependent launch: 600 back-to-back
    launches per shape on cycling weights give the same bits every time, and no bounded wait runs out."""
    from transformer_surgeon_b200 import ops
    dt = torch.bfloat16
    g = torch.Generator().manual_seed(13)

    def lin(out, inn, rank):
        U = (torch.randn(out, rank or inn, generator=g) * 0.05).to(dt).to(cuda)
        V = (torch.randn(rank, inn, generator=g) * 0.05).to(dt).to(cuda) if rank else None
        return ops.PackedLinear(ops.Factor.quantize(U, 4), ops.Factor.quantize(V, 4) if rank else None, None, dt)

    x = torch.randn(32, 4096, generator=g).to(dt).to(cuda)
    qkv = [lin(6144, 4096, 0) for _ in range(3)]                       # 48 tiles x 3 splits
    o = [lin(4096, 4096, 0) for _ in range(3)]                         # 32 tiles x 4 splits
    mlp = [ops.GatedMLP(lin(7168, 4096, 512), lin(7168, 4096, 512), lin(4096, 7168, 512)) for _ in range(2)]   # four phases
    old = ops.set_pdl(True)
    try:
        for layers in (qkv, o, mlp):
            refs = [L(x) for L in layers]
            outs = [torch.empty_like(r) for r in refs]
            bad = torch.zeros((), dtype=torch.int64, device=cuda)
            for it in range(600 // len(layers)):
                for L, out in zip(layers, outs):
                    L(x, out=out)
                if it % 4 == 3:
                    for out, r in zip(outs, refs):
                        bad += (out != r).any()
            torch.cuda.synchronize()
            assert int(bad.item()) == 0
    finally:
        ops.set_pdl(old)
    assert ops.PackedLinear.device_status(device=x.device) == 0


@pytest.mark.parametrize("name", ["fp32", "bf16"])
@pytest.mark.parametrize("M,N", [(1, 1), (3, 7), (2, 4097), (5, 50257), (2, 64)])
def test_argmax_of_rows(cuda, name, M, N):
    """Rows shorter than a cluster, misaligned rows, ties (the first maximum), negative rows, NaN, both zeros."""
    from transformer_surgeon_b200 import ops
    g = torch.Generator().manual_seed(N)
    y = torch.randn(M, N, generator=g).to(DT[name])
    y[0] = -y[0].abs() - 1
    if M > 1:
        y[1, N // 2:] = y[1].max()
    if M > 2:
        y[2] = 0.0
        y[2, 0] = -0.0
        y[2, N - 1] = float("nan") if N > 5 else 0.0
    assert torch.equal(ops.argmax(y.to(cuda)).cpu(), torch.argmax(y.float(), -1))


@pytest.mark.parametrize("M,K,N,r", [(16, 64, 33, 0), (31, 72, 31, 0), (33, 328, 100, 0), (64, 1032, 40, 0),      # one K rank, two, eight (the last two of which have nothing)
                                     (65, 4872, 129, 0), (128, 896, 4864, 128), (130, 136, 9480, 0), (300, 264, 4100, 40)])   # 32 x 32 and 64 x 64 tiles
def test_fp32_prompt_tiles(cuda, M, K, N, r):
    """Dense fp32 layers at prompt sizes: ragged tiles in both directions, K split over a cluster; single layers, a group and the gated pair.
    A sum of K products in fp32 is within about K^0.5 2^-24 of its terms' size of the exact one: 1e-5 of the largest output covers K = 4872."""
    from transformer_surgeon_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(52)
    def layer(o, i):
        f = lambda a, b: ops.Factor.dense(torch.randn((a, b), generator=g, device=cuda) * b ** -0.5)
        return ops.PackedLinear(f(o, r or i), f(r, i) if r else None, torch.randn(o, generator=g, device=cuda), torch.float32)
    def exact(l, x):
        h = x.double() @ l.v.data.double().T if l.v is not None else x.double()
        return h @ l.u.data.double().T + l.bias.double()
    a, b = layer(N, K), layer(N, K)
    x = torch.randn((M, K), generator=g, device=cuda)
    y = a(x)
    assert rel_err(y.cpu(), exact(a, x).cpu()) < 1e-5
    assert torch.equal(y, a(x))
    for o, l in zip(ops.LinearGroup([a, layer(7, K), b])(x), (a, None, b)):
        if l is not None:
            assert rel_err(o.cpu(), exact(l, x).cpu()) < 1e-5
    I = (N + 7) // 8 * 8                                     # (the down projection reads whole 16-byte pieces)
    gate, up, down = layer(I, K), layer(I, K), layer(K, I)
    ref = exact(down, torch.nn.functional.silu(exact(gate, x)) * exact(up, x))
    assert rel_err(ops.GatedMLP(gate, up, down)(x).cpu(), ref.cpu()) < 2e-5


@pytest.mark.parametrize("p", [None, 8, 4, 2, "binary"])
@pytest.mark.parametrize("M,K,I,r", [(1, 896, 4864, 128), (2, 1000, 304, 0), (3, 72, 1024, 40), (4, 2048, 96, 24), (4, 1024, 96, 0), (1, 8192, 64, 8), (1, 4, 40, 0)])
def test_fp32_projections_normalise_their_input(cuda, p, M, K, I, r):
    """Groups and the gated block that take residual + delta: the bits of add_rmsnorm and of the separate calls, the residual included.  Rows
    beyond one staged K tile and more than four tokens are declined."""
    from transformer_surgeon_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(54)
    def layer(o, i):
        f = lambda a, b: (ops.Factor.dense if p is None else lambda w: ops.Factor.quantize(w, p))(torch.randn((a, b), generator=g, device=cuda) * b ** -0.5)
        return ops.PackedLinear(f(o, r or i), f(r, i) if r else None, torch.randn(o, generator=g, device=cuda), torch.float32)
    if p is None and K % 8:
        K = 8
    group = ops.LinearGroup([layer(33, K), layer(8, K), layer(40, K)])
    mlp = ops.GatedMLP(layer(I, K), layer(I, K), layer(K, I))
    residual, delta, w = (torch.randn(s, generator=g, device=cuda) for s in ((M, K), (M, K), (K,)))
    ws = torch.zeros(max(group.workspace_bytes(8), mlp.workspace_bytes(8)), dtype=torch.uint8, device=cuda)
    for d in (delta, None):
        after = residual.clone()
        xn = ops.add_rmsnorm(after, d, w, 1e-6)
        for name in ("group", "mlp"):
            kept = torch.empty_like(residual)
            norm = ops.normalisation(residual, d, w, kept, 1e-6)
            if name == "group":
                outs, ref = [torch.empty((M, l.out_features), device=cuda) for l in group.layers], group(xn)
                assert group.after_norm(norm, M, outs, ws)
            else:
                outs, ref = [torch.empty((M, K), device=cuda)], [mlp(xn)]
                assert mlp.after_norm(norm, M, outs[0], ws)
            assert torch.equal(kept, after)
            assert all(torch.equal(a, b) for a, b in zip(outs, ref))
    big = torch.randn((5, K), generator=g, device=cuda)
    outs = [torch.zeros((5, l.out_features), device=cuda) for l in group.layers]
    assert not group.after_norm(ops.normalisation(big, None, w, torch.empty_like(big), 1e-6), 5, outs, ws)
    assert not any(o.any() for o in outs)
    for l in group.layers:
        l.force_simt = True
    assert not group.after_norm(ops.normalisation(residual, None, w, torch.empty_like(residual), 1e-6), M, outs, ws)


@pytest.mark.parametrize("K", [4096, 4104, 5000, 8192])
def test_long_rows_are_normalised_as_add_rmsnorm_does(cuda, K):
    """One token, rows on both sides of 16 KB, where add_rmsnorm changes the order of its sum: 48 rows each, since two orders of 8192 squares
    often round to the same number."""
    from transformer_surgeon_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(55)
    layer = ops.PackedLinear(ops.Factor.dense(torch.randn((16, K), generator=g, device=cuda) * K ** -0.5), None, None, torch.float32)
    group = ops.LinearGroup([layer])
    ws = torch.zeros(group.workspace_bytes(1), dtype=torch.uint8, device=cuda)
    for _ in range(48):
        residual, delta, w = (torch.randn(s, generator=g, device=cuda) for s in ((1, K), (1, K), (K,)))
        after, kept, out = residual.clone(), torch.empty_like(residual), torch.empty((1, 16), device=cuda)
        xn = ops.add_rmsnorm(after, delta, w, 1e-6)
        assert group.after_norm(ops.normalisation(residual, delta, w, kept, 1e-6), 1, [out], ws)
        assert torch.equal(kept, after)
        assert torch.equal(out, group(xn)[0])


def test_a_residual_over_its_own_terms_is_refused(cuda):
    """residual_out sharing memory with residual or delta, whole or in part: an error from both entry points, nothing written.  Neighbours are fine."""
    from transformer_surgeon_b200 import ops
    M, K = 2, 64
    g = torch.Generator(device=cuda).manual_seed(56)
    dense = lambda o, i: ops.PackedLinear(ops.Factor.dense(torch.randn((o, i), generator=g, device=cuda)), None, None, torch.float32)
    group, mlp = ops.LinearGroup([dense(8, K)]), ops.GatedMLP(dense(32, K), dense(32, K), dense(K, 32))
    ws = torch.zeros(max(group.workspace_bytes(M), mlp.workspace_bytes(M)), dtype=torch.uint8, device=cuda)
    rows = torch.randn((5 * M, K), generator=g, device=cuda)
    w, outs = torch.ones(K, device=cuda), (torch.zeros((M, 8), device=cuda), torch.zeros((M, K), device=cuda))
    before = rows.clone()
    def both(residual, delta, kept):
        norm = ops.normalisation(residual, delta, w, kept, 1e-6)
        return lambda: group.after_norm(norm, M, [outs[0]], ws), lambda: mlp.after_norm(norm, M, outs[1], ws)
    a, b, c = rows[:M], rows[M:2 * M], rows[M + 1:2 * M + 1]
    for residual, delta, kept in ((a, b, a), (a, b, b), (a, b, c), (c, a, b), (a, None, a)):
        for call in both(residual, delta, kept):
            with pytest.raises(ops.Tsb200Error):
                call()
    assert torch.equal(rows, before) and not outs[0].any() and not outs[1].any()
    for call in both(a, b, rows[2 * M:3 * M]):
        assert call()
    assert torch.equal(rows[2 * M:3 * M], a + b)


def test_normalisation_of_other_types_and_sizes_is_refused(cuda):
    from transformer_surgeon_b200 import ops
    r, w = torch.zeros((2, 64), device=cuda), torch.ones(64, device=cuda)
    ops.normalisation(r, r, w, torch.empty_like(r), 1e-6)
    for args in ((r.bfloat16(), None, w, r), (r, r.bfloat16(), w, r), (r, None, w.bfloat16(), r), (r, None, w, r.bfloat16())):
        with pytest.raises(TypeError):
            ops.normalisation(*args, 1e-6)
    for args in ((r, r[:1], w, r), (r, None, w[:32], r), (r, None, w, r[:1]), (r, r.cpu(), w, r), (r, r.t().contiguous().t(), w, r)):
        with pytest.raises(ValueError):
            ops.normalisation(*args, 1e-6)
