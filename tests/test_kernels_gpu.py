"""Kernel-level parity: every C-ABI entry point against the CPU oracle on the same seeded inputs."""
import math

import pytest
import torch

from oracle import ops as O

pytestmark = pytest.mark.gpu


def _gen(seed):
    return torch.Generator().manual_seed(seed)


def _bf(t):
    return t.to(torch.bfloat16)


# ------------------------------------------------------------------------------ ln_modulate
@pytest.mark.parametrize("M,D", [(1, 256), (37, 3072), (130, 5120), (5, 1024), (3, 64), (9, 8192)])
def test_ln_modulate_bf16(dsb, cuda_dev, M, D):
    g = _gen(1)
    x = _bf(torch.randn(M, D, generator=g) * 2 + 0.3)
    shift, scale = torch.randn(D, generator=g) * 0.1, torch.randn(D, generator=g) * 0.1
    ref = O.ln_modulate(x, shift, scale)
    y, _ = dsb.ops.ln_modulate(x.to(cuda_dev), shift.to(cuda_dev), scale.to(cuda_dev))
    assert O.rel_l2(y.float().cpu(), ref) < 3e-3  # bf16 output rounding only


@pytest.mark.parametrize("fmt", ["e4m3", "int8"])
@pytest.mark.parametrize("M,D", [(33, 3072), (7, 5120), (4, 256)])
def test_ln_modulate_quantised(dsb, cuda_dev, fmt, M, D):
    g = _gen(2)
    x = _bf(torch.randn(M, D, generator=g))
    shift, scale = torch.randn(D, generator=g) * 0.1, torch.randn(D, generator=g) * 0.1
    ref = O.ln_modulate(x, shift, scale)
    code = dsb.ops.FMT_E4M3 if fmt == "e4m3" else dsb.ops.FMT_INT8
    q, s = dsb.ops.ln_modulate(x.to(cuda_dev), shift.to(cuda_dev), scale.to(cuda_dev), out_fmt=code)
    qmax = 448.0 if fmt == "e4m3" else 127.0
    s_ref = ref.abs().amax(dim=1) / qmax
    assert torch.allclose(s.cpu(), s_ref, rtol=1e-5, atol=0)
    deq = q.float().cpu() * s.cpu()[:, None]
    # e4m3 has 3 mantissa bits (relative step 2^-4 half-ulp), int8 an absolute step of s/2
    tol = 0.04 if fmt == "e4m3" else 0.02
    assert O.rel_l2(deq, ref) < tol
    # the payload must be what the oracle quantiser produces from the kernel's own fp32 values, up to
    # values that sit within float rounding of a quantisation boundary
    fn = O.quant_rows_e4m3 if fmt == "e4m3" else O.quant_rows_int8
    q_ref, _ = fn(ref)
    mismatch = (q_ref.float() != q.float().cpu()).float().mean().item()
    assert mismatch < 2e-3


def test_ln_modulate_ragged_and_errors(dsb, cuda_dev):
    x = torch.zeros(0, 3072, dtype=torch.bfloat16, device=cuda_dev)
    sh = torch.zeros(3072, device=cuda_dev)
    y, _ = dsb.ops.ln_modulate(x, sh, sh)
    assert y.shape == (0, 3072)
    with pytest.raises(dsb.DsbError):  # D not a multiple of 8
        dsb.ops.ln_modulate(torch.zeros(2, 100, dtype=torch.bfloat16, device=cuda_dev), sh[:100], sh[:100])
    with pytest.raises(dsb.DsbError):  # CPU tensor: there is no fallback
        dsb.ops.ln_modulate(torch.zeros(2, 64, dtype=torch.bfloat16), torch.zeros(64), torch.zeros(64))
    # strided rows (a column slice of a wider buffer)
    g = _gen(3)
    wide = _bf(torch.randn(16, 4096, generator=g))
    shift, scale = torch.randn(1024, generator=g), torch.randn(1024, generator=g)
    y, _ = dsb.ops.ln_modulate(wide.to(cuda_dev)[:, 1024:2048], shift.to(cuda_dev), scale.to(cuda_dev))
    assert O.rel_l2(y.float().cpu(), O.ln_modulate(wide[:, 1024:2048], shift, scale)) < 3e-3


# ---------------------------------------------------------------------------- gate_residual
@pytest.mark.parametrize("M,D,gated", [(4608, 3072, True), (17, 5120, True), (3, 64, False)])
def test_gate_residual(dsb, cuda_dev, M, D, gated):
    g = _gen(4)
    x, y = _bf(torch.randn(M, D, generator=g)), _bf(torch.randn(M, D, generator=g))
    gate = torch.randn(D, generator=g) if gated else None
    ref = O.gate_residual(x, y, gate).to(torch.bfloat16)
    out = dsb.ops.gate_residual(x.to(cuda_dev), y.to(cuda_dev), None if gate is None else gate.to(cuda_dev))
    # one fp32 fma then one rounding on both sides: at most 1 bf16 ulp apart
    assert O.rel_l2(out.float().cpu(), ref.float()) < 1e-3


# ----------------------------------------------------------------------- rmsnorm + rope
def _flux_ids(S_txt, side):
    ids = torch.zeros(S_txt + side * side, 3)
    r = torch.arange(side)
    ids[S_txt:, 1] = r[:, None].expand(side, side).reshape(-1)
    ids[S_txt:, 2] = r[None, :].expand(side, side).reshape(-1)
    return ids


@pytest.mark.parametrize("S,H", [(96, 24), (1536, 24), (5, 2)])
def test_rmsnorm_rope_heads(dsb, cuda_dev, S, H):
    g = _gen(5)
    D = 128
    qkv = _bf(torch.randn(S, 3 * H * D, generator=g))
    wq, wk = 1 + 0.1 * torch.randn(D, generator=g), 1 + 0.1 * torch.randn(D, generator=g)
    side = int(math.isqrt(S)) if int(math.isqrt(S)) ** 2 == S else None
    ids = _flux_ids(0, side) if side else torch.cat([torch.zeros(S, 1), torch.arange(S)[:, None] % 32,
                                                     torch.arange(S)[:, None] // 32], dim=1).float()
    table = O.flux_rope_table(ids)
    q = qkv[:, : H * D].float().reshape(S, H, D)
    k = qkv[:, H * D: 2 * H * D].float().reshape(S, H, D)
    q_ref = O.apply_rope_pairs(O.rmsnorm(q, wq).transpose(0, 1), table).transpose(0, 1).reshape(S, H * D)
    k_ref = O.apply_rope_pairs(O.rmsnorm(k, wk).transpose(0, 1), table).transpose(0, 1).reshape(S, H * D)
    buf = qkv.to(cuda_dev).clone()
    dsb.ops.rmsnorm_rope_heads(buf, H, wq.to(cuda_dev), wk.to(cuda_dev), table.to(cuda_dev).contiguous())
    out = buf.float().cpu()
    assert O.rel_l2(out[:, : H * D], q_ref) < 3e-3
    assert O.rel_l2(out[:, H * D: 2 * H * D], k_ref) < 3e-3
    assert torch.equal(out[:, 2 * H * D:], qkv[:, 2 * H * D:].float())  # v untouched


@pytest.mark.parametrize("M,H,rope", [(60, 40, True), (33, 40, False), (7, 12, True)])
def test_rmsnorm_full(dsb, cuda_dev, M, H, rope):
    g = _gen(6)
    D = H * 128
    x = _bf(torch.randn(M, D, generator=g))
    w = 1 + 0.1 * torch.randn(D, generator=g)
    table = O.wan_rope_table(3, 4, 5)[:M] if rope else None
    ref = O.rmsnorm(x, w)
    if rope:
        ref = O.apply_rope_pairs(ref.reshape(M, H, 128).transpose(0, 1), table).transpose(0, 1).reshape(M, D)
    buf = x.to(cuda_dev).clone()
    dsb.ops.rmsnorm_full(buf, w.to(cuda_dev), None if table is None else table.to(cuda_dev).contiguous())
    assert O.rel_l2(buf.float().cpu(), ref) < 3e-3


# -------------------------------------------------------------------------- quantisation
@pytest.mark.parametrize("fmt", ["e4m3", "int8"])
@pytest.mark.parametrize("M,K", [(64, 3072), (5, 15360), (3, 128)])
def test_quant_rows_bit_exact(dsb, cuda_dev, fmt, M, K):
    g = _gen(7)
    x = _bf(torch.randn(M, K, generator=g) * 3)
    x[0] = 0  # an all-zero row
    fn = O.quant_rows_e4m3 if fmt == "e4m3" else O.quant_rows_int8
    q_ref, s_ref = fn(x)
    code = dsb.ops.FMT_E4M3 if fmt == "e4m3" else dsb.ops.FMT_INT8
    q, s = dsb.ops.quant_rows(x.to(cuda_dev), out_fmt=code)
    assert torch.equal(s.cpu(), s_ref)
    assert torch.equal(q.cpu().view(torch.uint8), q_ref.view(torch.uint8))


@pytest.mark.parametrize("fmt", ["fp8_tensor", "fp8_channel", "int8_channel"])
@pytest.mark.parametrize("src", [torch.float32, torch.bfloat16])
def test_pack_quant_weight_bit_exact(dsb, cuda_dev, fmt, src):
    g = _gen(8)
    W = (torch.randn(200, 384, generator=g) * 0.02).to(src)
    W[3] = 0
    q_ref, s_ref = O.quant_weight(W, fmt)
    code = dsb.ops.FMT_INT8 if fmt == "int8_channel" else dsb.ops.FMT_E4M3
    q, s = dsb.ops.pack_quant_weight(W.to(cuda_dev), code, per_channel=fmt != "fp8_tensor")
    assert torch.equal(s.cpu(), s_ref)
    assert torch.equal(q.cpu().view(torch.uint8), q_ref.view(torch.uint8))


# ---------------------------------------------------------------------------------- gemv
@pytest.mark.parametrize("wfmt", ["bf16", "e4m3", "int8"])
def test_gemv(dsb, cuda_dev, wfmt):
    g = _gen(9)
    N, K = 1000, 3072
    W = torch.randn(N, K, generator=g) * 0.02
    x = torch.randn(K, generator=g)
    bias = torch.randn(N, generator=g) * 0.02
    if wfmt == "bf16":
        Wd, scale, Wref = _bf(W), None, _bf(W).float()
    else:
        q, s = O.quant_weight(W, "fp8_channel" if wfmt == "e4m3" else "int8_channel")
        Wd, scale, Wref = q, s, q.float() * s[:, None]
    ref = Wref @ torch.nn.functional.silu(x) + bias
    y = dsb.ops.gemv(Wd.to(cuda_dev), x.to(cuda_dev), None if scale is None else scale.to(cuda_dev),
                     bias.to(cuda_dev), act_in=dsb.ops.ACT_SILU)
    assert O.rel_l2(y.cpu(), ref) < 1e-5
    ref2 = torch.nn.functional.silu(Wref @ x + bias)
    y2 = dsb.ops.gemv(Wd.to(cuda_dev), x.to(cuda_dev), None if scale is None else scale.to(cuda_dev),
                      bias.to(cuda_dev), act_out=dsb.ops.ACT_SILU)
    assert O.rel_l2(y2.cpu(), ref2) < 1e-5


# ---------------------------------------------------------------------------- euler step
def test_euler_step(dsb, cuda_dev):
    g = _gen(10)
    lat, mo = torch.randn(1, 4096, 64, generator=g), torch.randn(1, 4096, 64, generator=g)
    sig = torch.linspace(1, 0, 11)
    ref = O.euler_step(lat, mo, sig, 3)
    out = dsb.ops.euler_step(lat.to(cuda_dev), mo.to(cuda_dev), float(sig[4] - sig[3]))
    assert torch.allclose(out.cpu(), ref, rtol=1e-6, atol=1e-6)
    lb, mb = _bf(lat), _bf(mo)
    refb = O.euler_step(lb, mb, sig, 3)
    outb = dsb.ops.euler_step(lb.to(cuda_dev), mb.to(cuda_dev), float(sig[4] - sig[3]))
    assert torch.equal(outb.cpu(), refb)


def test_cfg_euler_step(dsb, cuda_dev):
    """CFG combine + Euler update in one kernel, bit-identical to the reference's two tensor expressions."""
    g = _gen(18)
    lat, pos, neg = (torch.randn(1, 16, 21, 30, 52, generator=g) for _ in range(3))
    sig = torch.linspace(0.999, 0.001, 51)
    for cast in (lambda t: t, _bf):
        l, p, n = cast(lat), cast(pos), cast(neg)
        ref = O.euler_step(l, O.cfg_combine(p, n, 5.0), sig, 7)
        out = dsb.ops.cfg_euler_step(l.to(cuda_dev), p.to(cuda_dev), n.to(cuda_dev), 5.0, float(sig[8] - sig[7]))
        if l.dtype == torch.float32:
            assert torch.allclose(out.cpu(), ref, rtol=1e-6, atol=1e-6)
        else:
            assert torch.equal(out.cpu(), ref)


# ---------------------------------------------------------------------------------- gemm
def _gemm_case(dsb, dev, fmt, M, N, K, per_channel, bias, act, gated, seed=11):
    g = _gen(seed)
    x = _bf(torch.randn(M, K, generator=g))
    W = torch.randn(N, K, generator=g) * 0.02
    b = torch.randn(N, generator=g) * 0.1 if bias else None
    resid = _bf(torch.randn(M, N, generator=g)) if gated else None
    gate = torch.randn(N, generator=g) if gated else None
    if fmt == "bf16":
        a_d, w_d, rs, cs = x, _bf(W), None, None
        acc = x.float() @ _bf(W).float().t()
    elif fmt == "e4m3":
        xq, xs = O.quant_rows_e4m3(x)
        wq, ws = O.quant_weight(W, "fp8_channel" if per_channel else "fp8_tensor")
        a_d, w_d, rs, cs = xq, wq, xs, ws
        acc = O.linear_quant(xq, xs, wq, ws)
    else:
        xq, xs = O.quant_rows_int8(x)
        wq, ws = O.quant_weight(W, "int8_channel")
        a_d, w_d, rs, cs = xq, wq, xs, ws
        acc = O.linear_quant(xq, xs, wq, ws)
    ref = acc if b is None else acc + b
    if act:
        ref = O.gelu_tanh(ref)
    if gated:
        ref = resid.float() + gate * ref
    to = lambda t: None if t is None else t.to(dev)
    out = dsb.ops.gemm(to(a_d), to(w_d), row_scale=to(rs), col_scale=to(cs), bias=to(b),
                       act=dsb.ops.ACT_GELU_TANH if act else dsb.ops.ACT_NONE, gate=to(gate), resid=to(resid))
    return out.float().cpu(), ref


@pytest.mark.parametrize("fmt", ["e4m3", "bf16", "int8"])
@pytest.mark.parametrize("M,N,K", [(128, 256, 128), (256, 512, 3072), (300, 3072, 256), (4095, 1024, 512),
                                   (1, 64, 64), (130, 136, 200 * 8)])
def test_gemm_plain(dsb, cuda_dev, fmt, M, N, K):
    if fmt != "bf16" and K % 16:
        pytest.skip("8-bit operands need K % 16 == 0")
    out, ref = _gemm_case(dsb, cuda_dev, fmt, M, N, K, per_channel=False, bias=False, act=False, gated=False)
    assert O.rel_l2(out, ref) < 3e-3, (fmt, M, N, K)


@pytest.mark.parametrize("fmt,per_channel", [("e4m3", False), ("e4m3", True), ("int8", True), ("bf16", False)])
def test_gemm_epilogues(dsb, cuda_dev, fmt, per_channel):
    for bias, act, gated in [(True, False, False), (True, True, False), (True, False, True), (False, True, True)]:
        out, ref = _gemm_case(dsb, cuda_dev, fmt, 517, 768, 1024, per_channel, bias, act, gated)
        assert O.rel_l2(out, ref) < 4e-3, (fmt, per_channel, bias, act, gated)


def test_gemm_split_output_and_act_range(dsb, cuda_dev):
    """Columns below split_col go to out0, the rest to out1; GELU only from act_col0 on
    (the single-stream block's fused qkv|mlp projection, models/flux/flux_dit.py:311-317)."""
    g = _gen(12)
    M, K, N, split = 200, 512, 1024, 512
    x, W = _bf(torch.randn(M, K, generator=g)), _bf(torch.randn(N, K, generator=g) * 0.05)
    b = torch.randn(N, generator=g) * 0.1
    ref = x.float() @ W.float().t() + b
    ref0, ref1 = ref[:, :split], O.gelu_tanh(ref[:, split:])
    out0 = torch.empty(M, split, dtype=torch.bfloat16, device=cuda_dev)
    wide = torch.zeros(M, 256 + N - split, dtype=torch.bfloat16, device=cuda_dev)
    dsb.ops.gemm(x.to(cuda_dev), W.to(cuda_dev), bias=b.to(cuda_dev), act=dsb.ops.ACT_GELU_TANH, act_col0=split,
                 out=out0, out1=wide[:, 256:], split_col=split)
    assert O.rel_l2(out0.float().cpu(), ref0) < 3e-3
    assert O.rel_l2(wide[:, 256:].float().cpu(), ref1) < 3e-3
    assert float(wide[:, :256].abs().max()) == 0.0  # nothing written left of the routed block


def test_gemm_canary_rows(dsb, cuda_dev):
    """M and N tails must not write outside [M, N]."""
    g = _gen(13)
    M, N, K = 130, 136, 384
    x, W = _bf(torch.randn(M, K, generator=g)), _bf(torch.randn(N, K, generator=g) * 0.05)
    big = torch.full((M + 8, N + 64), 7.0, dtype=torch.bfloat16, device=cuda_dev)
    dsb.ops.gemm(x.to(cuda_dev), W.to(cuda_dev), out=big[:M, :N])
    assert O.rel_l2(big[:M, :N].float().cpu(), x.float() @ W.float().t()) < 3e-3
    assert bool((big[M:, :] == 7.0).all()) and bool((big[:, N:] == 7.0).all())


def test_gemm_run_twice_identical(dsb, cuda_dev):
    g = _gen(14)
    x, W = _bf(torch.randn(1000, 1024, generator=g)).to(cuda_dev), _bf(torch.randn(768, 1024, generator=g)).to(cuda_dev)
    a = dsb.ops.gemm(x, W)
    b = dsb.ops.gemm(x, W)
    assert torch.equal(a, b)


def test_gemm_empty_and_bad_args(dsb, cuda_dev):
    x = torch.zeros(0, 128, dtype=torch.bfloat16, device=cuda_dev)
    W = torch.zeros(64, 128, dtype=torch.bfloat16, device=cuda_dev)
    assert dsb.ops.gemm(x, W).shape == (0, 64)
    with pytest.raises(dsb.DsbError):  # N not a multiple of 8
        dsb.ops.gemm(torch.zeros(4, 128, dtype=torch.bfloat16, device=cuda_dev),
                     torch.zeros(60, 128, dtype=torch.bfloat16, device=cuda_dev))


# ----------------------------------------------------------------------------- attention
@pytest.mark.parametrize("B,H,Sq,Sk", [(1, 2, 256, 256), (1, 24, 1536, 1536), (1, 3, 300, 300), (2, 2, 257, 512),
                                       (1, 2, 1000, 77), (1, 1, 1, 1), (1, 40, 384, 512)])
def test_flash_attn(dsb, cuda_dev, B, H, Sq, Sk):
    g = _gen(15)
    q = _bf(torch.randn(B, Sq, H, 128, generator=g))
    k = _bf(torch.randn(B, Sk, H, 128, generator=g))
    v = _bf(torch.randn(B, Sk, H, 128, generator=g))
    ref = O.attention(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2)).transpose(1, 2)
    out = dsb.ops.flash_attn(q.to(cuda_dev), k.to(cuda_dev), v.to(cuda_dev))
    assert O.rel_l2(out.float().cpu(), ref) < 4e-3, (B, H, Sq, Sk)


def test_flash_attn_peaked_rows(dsb, cuda_dev):
    """Large logits late in the sequence force the lazy running-max refresh and O rescale."""
    g = _gen(16)
    H, S = 2, 1024
    q = _bf(torch.randn(1, S, H, 128, generator=g))
    k = _bf(torch.randn(1, S, H, 128, generator=g))
    v = _bf(torch.randn(1, S, H, 128, generator=g))
    k[:, 700:720] *= 6.0
    k[:, 1000:1003] *= 12.0
    ref = O.attention(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2)).transpose(1, 2)
    out = dsb.ops.flash_attn(q.to(cuda_dev), k.to(cuda_dev), v.to(cuda_dev))
    assert O.rel_l2(out.float().cpu(), ref) < 4e-3


def test_flash_attn_one_key_far_above_the_reference_maximum(dsb, cuda_dev):
    """One key deep in the sequence scores more than 2^100 above everything before it for about half of the rows (and
    as far below for the rest): the tile that meets it lifts the reference of its rows, and the rows it dominates return
    that key's value."""
    g = _gen(19)
    H, S = 2, 2048
    q = _bf(torch.randn(1, S, H, 128, generator=g))
    k = _bf(torch.randn(1, S, H, 128, generator=g))
    v = _bf(torch.randn(1, S, H, 128, generator=g))
    k[:, 1500] *= 300.0
    ref = O.attention(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2)).transpose(1, 2)
    out = dsb.ops.flash_attn(q.to(cuda_dev), k.to(cuda_dev), v.to(cuda_dev)).float().cpu()
    assert torch.isfinite(out).all()
    assert O.rel_l2(out, ref) < 4e-3


def test_flash_attn_strided_views(dsb, cuda_dev):
    """q/k/v as column blocks of one fused projection buffer [S, 3*H*128] (text rows first), and
    [B,H,S,D]-strided tensors as the reference's _attn_func receives them (models/flux/flux_dit.py:166-182)."""
    g = _gen(17)
    H, S = 4, 640
    qkv = _bf(torch.randn(S, 3 * H * 128, generator=g))
    q, k, v = (qkv[:, i * H * 128:(i + 1) * H * 128].reshape(1, S, H, 128) for i in range(3))
    ref = O.attention(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2)).transpose(1, 2)
    d = qkv.to(cuda_dev)
    qd, kd, vd = (d[:, i * H * 128:(i + 1) * H * 128].unflatten(1, (H, 128)).unsqueeze(0) for i in range(3))
    out = dsb.ops.flash_attn(qd, kd, vd)
    assert O.rel_l2(out.float().cpu(), ref) < 4e-3
    # [B,H,S,D] contiguous inputs viewed as [B,S,H,D]
    qh = q.transpose(1, 2).contiguous().to(cuda_dev).transpose(1, 2)
    kh = k.transpose(1, 2).contiguous().to(cuda_dev).transpose(1, 2)
    vh = v.transpose(1, 2).contiguous().to(cuda_dev).transpose(1, 2)
    out2 = dsb.ops.flash_attn(qh, kh, vh)
    assert O.rel_l2(out2.float().cpu(), ref) < 4e-3


@pytest.mark.parametrize("fmt", ["e4m3", "bf16"])
@pytest.mark.parametrize("M,H", [(300, 2), (1000, 4)])
def test_gemm_qkv_fused_norm_rope(dsb, cuda_dev, fmt, M, H):
    """q|k|v|mlp projection whose epilogue applies the per-head RMSNorm + RoPE to q and k, GELU to the mlp
    columns and routes the two column ranges to two buffers (models/flux/flux_dit.py:297-317)."""
    g = _gen(21)
    d, K = H * 128, 512
    N = 7 * d
    x = _bf(torch.randn(M, K, generator=g))
    W = torch.randn(N, K, generator=g) * 0.05
    b = torch.randn(N, generator=g) * 0.1
    wq, wk = 1 + 0.1 * torch.randn(128, generator=g), 1 + 0.1 * torch.randn(128, generator=g)
    ids = torch.stack([torch.zeros(M + 7), torch.arange(M + 7) % 37, torch.arange(M + 7) // 37], dim=1).float()
    table = O.flux_rope_table(ids)
    if fmt == "bf16":
        a_d, w_d, rs, cs = x, _bf(W), None, None
        acc = x.float() @ _bf(W).float().t() + b
    else:
        xq, xs = O.quant_rows_e4m3(x)
        wq8, ws = O.quant_weight(W, "fp8_tensor")
        a_d, w_d, rs, cs = xq, wq8, xs, ws
        acc = O.linear_quant(xq, xs, wq8, ws, b)
    q = O.apply_rope_pairs(O.rmsnorm(acc[:, :d].reshape(M, H, 128), wq).transpose(0, 1), table[7:7 + M]).transpose(0, 1)
    k = O.apply_rope_pairs(O.rmsnorm(acc[:, d:2 * d].reshape(M, H, 128), wk).transpose(0, 1), table[7:7 + M]).transpose(0, 1)
    ref_qkv = torch.cat([q.reshape(M, d), k.reshape(M, d), acc[:, 2 * d:3 * d]], dim=1)
    ref_mlp = O.gelu_tanh(acc[:, 3 * d:])
    to = lambda t: None if t is None else t.to(cuda_dev)
    qkv = torch.empty(M, 3 * d, dtype=torch.bfloat16, device=cuda_dev)
    cat = torch.zeros(M, 5 * d, dtype=torch.bfloat16, device=cuda_dev)
    # the oracle rotates with the fp32 table; the kernel's table is the fp16 rounding of it (2^-12)
    dsb.ops.gemm_qkv(to(a_d), to(w_d), to(wq), to(wk), d, to(table).half().contiguous(), 7, 1e-6, row_scale=to(rs),
                     col_scale=to(cs), bias=to(b), act=dsb.ops.ACT_GELU_TANH, act_col0=3 * d, out=qkv, out1=cat[:, d:],
                     split_col=3 * d)
    assert O.rel_l2(qkv.float().cpu(), ref_qkv) < 4e-3
    assert O.rel_l2(cat[:, d:].float().cpu(), ref_mlp) < 4e-3
    assert float(cat[:, :d].abs().max()) == 0.0


@pytest.mark.parametrize("M,N,K", [(300, 512, 256), (1000, 1280, 384), (129, 264, 128)])
def test_gemm_e4m3_output_is_the_cast_of_the_epilogue_value(dsb, cuda_dev, M, N, K):
    """An e4m3 output range: GELU(acc * scales + bias) cast to e4m3 with unit scale (saturating).  Next to a bf16 first
    range (split output) and alone; N = 264 leaves the second 64-column block of the last warp pair out of range."""
    g = _gen(55)
    x = _bf(torch.randn(M, K, generator=g))
    W = torch.randn(N, K, generator=g) * 0.05
    b = torch.randn(N, generator=g) * 0.1
    xq, xs = O.quant_rows_e4m3(x)
    wq, ws = O.quant_weight(W, "fp8_tensor")
    acc = O.linear_quant(xq, xs, wq, ws, b)
    to = lambda t: t.to(cuda_dev)
    # alone
    out8 = torch.zeros(M, (N + 15) // 16 * 16, dtype=torch.float8_e4m3fn, device=cuda_dev)[:, :N]   # row pitch % 16 == 0
    dsb.ops.gemm_group([dict(a=to(xq), w=to(wq), row_scale=to(xs), col_scale=to(ws), bias=to(b),
                             act=dsb.ops.ACT_GELU_TANH, out=out8)])
    ref = O.gelu_tanh(acc)
    got = out8.float().cpu()
    # e4m3 of nearly equal fp32 values: identical except where the two sides' fp32 values straddle a rounding boundary
    close = (got - ref.clamp(-448, 448).to(torch.float8_e4m3fn).float()).abs() <= 0.0626 * ref.abs() + 2e-3
    assert close.float().mean() > 0.999 and O.rel_l2(got, ref) < 4e-2
    if N % 256 == 0:
        split = (N // 512) * 256
        o0 = torch.zeros(M, split, dtype=torch.bfloat16, device=cuda_dev)
        o1 = torch.zeros(M, N - split, dtype=torch.float8_e4m3fn, device=cuda_dev)
        dsb.ops.gemm_group([dict(a=to(xq), w=to(wq), row_scale=to(xs), col_scale=to(ws), bias=to(b),
                                 act=dsb.ops.ACT_GELU_TANH, act_col0=split, out=o0, out1=o1, split_col=split)])
        assert O.rel_l2(o0.float().cpu(), acc[:, :split]) < 4e-3
        assert torch.equal(o1.view(torch.uint8).cpu(), out8[:, split:].contiguous().view(torch.uint8).cpu())
    dsb.ops.check_status(0)


# ------------------------------------------------------------------------- bounded waits
def test_bounded_wait_runs_out_and_reports_timeout(dsb, cuda_dev):
    """A device wait that nothing ever satisfies gives up after its cycle budget: the CTA's abort flag is raised, the
    other role leaves its own wait because of it, the status word reads DSB_ERR_TIMEOUT, and the context is still
    good for the next launch.  (No trap, no endless loop: the wait is bounded by construction.)"""
    import time
    t0 = time.time()
    status, left = dsb.ops.selftest_wait_timeout(limit_cycles=2_000_000)       # about a millisecond of SM cycles
    assert status == dsb._lib.ERR_TIMEOUT and left == 1
    assert time.time() - t0 < 5.0
    # the context is intact: an ordinary kernel runs and the library's own status word was never touched
    x = torch.randn(4, 256).to(torch.bfloat16).to(cuda_dev)
    y, _ = dsb.ops.ln_modulate(x, torch.zeros(256, device=cuda_dev), torch.zeros(256, device=cuda_dev))
    assert torch.isfinite(y.float()).all()
    dsb.ops.check_status(0)


@pytest.mark.parametrize("limit_cycles", [20_000, 500_000])
def test_a_warp_gives_up_as_a_whole(dsb, cuda_dev, limit_cycles):
    """The self-test's third warp: half of its lanes wait for a barrier that completes, half for one that does not.  All of
    its lanes leave (``left`` needs that), as a warp must whose next instruction names every lane."""
    for _ in range(3):
        assert dsb.ops.selftest_wait_timeout(limit_cycles=limit_cycles) == (dsb._lib.ERR_TIMEOUT, 1)


# ------------------------------------------------------------ attention over row ranges in separate buffers
def test_flash_attn_parts_equals_one_buffer(dsb, cuda_dev):
    """Queries read from three separate buffers (256 rows each, the last one half used) and output rows written to four
    separate buffers of 200 rows (ranges that cut through the 128-row tiles) give bit for bit what the one-buffer
    call gives: only addresses change.  On several GPUs the buffers are the other ranks' memory."""
    H, Sq, Sk = 3, 640, 500
    q = (torch.randn(1, Sq, H, 128) * 1.5).bfloat16().to(cuda_dev)
    k = torch.randn(1, Sk, H, 128).bfloat16().to(cuda_dev)
    v = torch.randn(1, Sk, H, 128).bfloat16().to(cuda_dev)
    want = dsb.ops.flash_attn(q, k, v)
    q_rows, o_rows = 256, 200
    q_parts = [torch.zeros(q_rows, H, 128, dtype=torch.bfloat16, device=cuda_dev) for _ in range(3)]
    for i, part in enumerate(q_parts):                                                 # the last one is half filled
        rows = q[0, i * q_rows:(i + 1) * q_rows]
        part[:rows.shape[0]] = rows
    o_parts = [torch.full((o_rows, H, 128), 7.0, dtype=torch.bfloat16, device=cuda_dev) for _ in range(4)]
    dsb.ops.flash_attn_parts(q_parts, q_rows, (H * 128, 128), k, v, o_parts, o_rows, (H * 128, 128), H, Sq)
    got = torch.cat(o_parts)[:Sq]
    assert torch.equal(got, want[0])
    assert (torch.cat(o_parts)[Sq:] == 7.0).all()                                       # rows past Sq stay untouched
    dsb.ops.check_status(0)
    with pytest.raises(dsb._lib.DsbError):                                              # a 128-row tile may not straddle parts
        dsb.ops.flash_attn_parts(q_parts, 192, (H * 128, 128), k, v, o_parts, o_rows, (H * 128, 128), H, Sq)


def test_rank_barrier_alone_passes_and_absent_rank_times_out(dsb, cuda_dev):
    """One rank alone passes its barrier at once.  With a second rank that never arrives (its flag stays 0) the
    waiter gives up after its cycle budget, reports DSB_ERR_TIMEOUT in the status word it was given, has still
    delivered its own signal, and the context stays usable.  (The wait is bounded; nothing traps.)"""
    import time
    status = torch.zeros(1, dtype=torch.int32, device=cuda_dev)
    mine = torch.zeros(8, dtype=torch.int32, device=cuda_dev)
    for epoch in (1, 2, 3):
        dsb.ops.rank_barrier([mine], 0, epoch, status=status)
    assert status.item() == 0 and mine[0].item() == 3
    other = torch.zeros(8, dtype=torch.int32, device=cuda_dev)
    t0 = time.time()
    dsb.ops.rank_barrier([mine, other], 0, 4, limit_cycles=2_000_000, status=status)
    assert status.item() == dsb._lib.ERR_TIMEOUT
    assert time.time() - t0 < 5.0
    assert other[0].item() == 4 and mine[0].item() == 4 and mine[1].item() == 0
    # a rank that is already ahead does not block: the flag only has to be at least the epoch
    mine[1] = 9
    status.zero_()
    dsb.ops.rank_barrier([mine, other], 0, 5, limit_cycles=2_000_000, status=status)
    assert status.item() == 0


def test_gemm_front_end_rejects_buffers_the_kernel_would_overrun(dsb, cuda_dev):
    """The C entry points take raw pointers, so the tensor front end checks shapes and dtypes: an output that is too
    small or of the wrong type raises instead of being written past its end; an e4m3 output is routed to the
    entry point that can describe it and equals the grouped call."""
    M, N, K = 256, 512, 256
    a = torch.randn(M, K).to(torch.float8_e4m3fn).to(cuda_dev)
    w = torch.randn(N, K).to(torch.float8_e4m3fn).to(cuda_dev)
    rs = (torch.rand(M) * 0.01 + 0.001).to(cuda_dev)
    for bad in (torch.empty(M, N - 8, dtype=torch.bfloat16, device=cuda_dev),
                torch.empty(M - 1, N, dtype=torch.bfloat16, device=cuda_dev),
                torch.empty(M, N, dtype=torch.float16, device=cuda_dev)):
        with pytest.raises(dsb._lib.DsbError):
            dsb.ops.gemm(a, w, row_scale=rs, out=bad)
    with pytest.raises(dsb._lib.DsbError):
        dsb.ops.gemm(a, w, row_scale=rs[:M - 1])
    with pytest.raises(dsb._lib.DsbError):
        dsb.ops.gemm(a, w, bias=torch.zeros(N, dtype=torch.bfloat16, device=cuda_dev))
    o8 = torch.empty(M, N, dtype=torch.float8_e4m3fn, device=cuda_dev)
    o8g = torch.empty_like(o8)
    dsb.ops.gemm(a, w, row_scale=rs, act=dsb.ops.ACT_GELU_TANH, out=o8)
    dsb.ops.gemm_group([dict(a=a, w=w, row_scale=rs, act=dsb.ops.ACT_GELU_TANH, out=o8g)])
    assert torch.equal(o8.view(torch.uint8), o8g.view(torch.uint8))
    ref = torch.nn.functional.gelu((a.float() @ w.float().T) * rs[:, None], approximate="tanh")
    assert O.rel_l2(o8.float(), ref.clamp(-448, 448)) < 4e-2          # e4m3 rounding of the output
    dsb.ops.check_status(0)


# ------------------------------------------------------------------ patch embedding input / output of the head
@pytest.mark.parametrize("C,F,gh,gw", [(16, 3, 5, 7), (36, 2, 4, 6), (16, 1, 12, 10)])
def test_patchify_matches_the_reference_rearrangement(dsb, cuda_dev, C, F, gh, gw):
    """``dsb_patchify`` against the rearrangement the reference's Conv3d / patchify perform
    (models/wan/wan_dit.py:271-273, flux_dit.py:364-367: feature order (c, py, pz), tokens in (f, y, z) raster order):
    bit-exact in bf16; the quantised forms equal ``dsb_quant_rows`` of those rows; a row range that runs past the last
    token is zero-filled."""
    lat = torch.randn(C, F, 2 * gh, 2 * gw).bfloat16()
    want = lat.reshape(C, F, gh, 2, gw, 2).permute(1, 2, 4, 0, 3, 5).reshape(F * gh * gw, C * 4)
    S = F * gh * gw
    got, _ = dsb.ops.patchify(lat.to(cuda_dev))
    assert torch.equal(got.cpu(), want)
    row0, n = 5, S                                              # 5 rows past the end
    got, _ = dsb.ops.patchify(lat.to(cuda_dev), row0, n)
    assert torch.equal(got.cpu()[:S - row0], want[row0:]) and (got.cpu()[S - row0:] == 0).all()
    for fmt, qfn in ((dsb.ops.FMT_E4M3, O.quant_rows_e4m3), (dsb.ops.FMT_INT8, O.quant_rows_int8)):
        wide = torch.zeros(n, C * 4 + 64, dtype=dsb.ops._OUT_DTYPE[fmt], device=cuda_dev)   # a column slice as output
        q, s = dsb.ops.patchify(lat.to(cuda_dev), row0, n, fmt, out=wide[:, :C * 4])
        rows = torch.cat([want[row0:], torch.zeros(row0, C * 4, dtype=torch.bfloat16)])
        q_ref, s_ref = qfn(rows.float())
        assert torch.equal(s.cpu(), s_ref)
        assert torch.equal(q.cpu().view(torch.uint8), q_ref.view(torch.uint8))
        assert (wide[:, C * 4:].view(torch.uint8) == 0).all()


@pytest.mark.parametrize("c_fastest", [True, False])
def test_unpatchify_matches_the_reference_rearrangement(dsb, cuda_dev, c_fastest):
    """``dsb_unpatchify`` against WanDiT.unpatchify ("(x y z c)", wan_dit.py:307-317) and FluxDiT.unpatchify
    ("(c ph pw)", flux_dit.py:369-374) on rows wider than the features they hold."""
    C, F, gh, gw = 16, (3 if c_fastest else 1), 6, 5
    tok = torch.randn(F * gh * gw, C * 4 + 8).bfloat16()
    t = tok[:, :C * 4]
    if c_fastest:
        want = t.reshape(F, gh, gw, 1, 2, 2, C).permute(6, 0, 3, 1, 4, 2, 5).reshape(1, C, F, gh * 2, gw * 2)
    else:
        want = t.reshape(gh, gw, C, 2, 2).permute(2, 0, 3, 1, 4).reshape(1, C, 1, gh * 2, gw * 2)
    got = dsb.ops.unpatchify(tok.to(cuda_dev), C, F, gh, gw, c_fastest)
    assert torch.equal(got.cpu(), want)


def test_flash_attn_e4m3_output_equals_bf16_output_then_cast(dsb, cuda_dev):
    """``dsb_flash_attn_out8`` writes bit for bit what ``dsb_flash_attn`` followed by ``dsb_cast_quant`` (unit scale,
    saturating) writes - into a column slice of a wider e4m3 buffer, as the Flux single block uses it - including
    values beyond the e4m3 range."""
    H, Sq, Sk = 2, 300, 333
    q = (torch.randn(1, Sq, H, 128) * 4).bfloat16().to(cuda_dev)            # peaked rows: the output is close to one value row
    k = torch.randn(1, Sk, H, 128).bfloat16().to(cuda_dev)
    v = (torch.randn(1, Sk, H, 128) * 300).bfloat16().to(cuda_dev)          # values up to a thousand: some outputs saturate
    o = dsb.ops.flash_attn(q, k, v)
    want = torch.empty(Sq, H * 128, dtype=torch.float8_e4m3fn, device=cuda_dev)
    dsb.ops.cast_quant(o[0].reshape(Sq, H * 128), want, dsb.ops.FMT_E4M3)
    wide = torch.zeros(Sq, 5 * H * 128, dtype=torch.float8_e4m3fn, device=cuda_dev)
    got = wide[:, :H * 128].unflatten(1, (H, 128)).unsqueeze(0)
    dsb.ops.flash_attn(q, k, v, out=got)
    assert torch.equal(wide[:, :H * 128].view(torch.uint8), want.view(torch.uint8))
    assert (wide[:, H * 128:].view(torch.uint8) == 0).all()
    assert (want.float().abs() == 448).any()                                 # the case did exercise saturation
    dsb.ops.check_status(0)


def test_flash_attn_parts_with_a_split_last_wave(dsb, cuda_dev):
    """With a workspace, the items of a partly filled last wave (156 items on 74 CTA pairs: 8 of them) are cut along
    the keys into two units each and combined afterwards: the result equals the uncut kernel up to the fp32 summation
    order of the partial outputs (the bf16 probabilities are identical), the ragged key tail stays masked, rows of
    the uncut items are bit-identical, and the partial results of the cut ones are all that the workspace is used for."""
    H, Sq, Sk = 3, 52 * 256, 2250
    g = torch.Generator().manual_seed(11)
    q = (torch.randn(1, Sq, H, 128, generator=g) * 1.5).bfloat16().to(cuda_dev)
    k = torch.randn(1, Sk, H, 128, generator=g).bfloat16().to(cuda_dev)
    v = torch.randn(1, Sk, H, 128, generator=g).bfloat16().to(cuda_dev)
    want = dsb.ops.flash_attn(q, k, v)[0]
    o_rows = Sq // 2
    o_parts = [torch.zeros(o_rows, H, 128, dtype=torch.bfloat16, device=cuda_dev) for _ in range(2)]
    ws = dsb.ops.flash_attn_workspace(cuda_dev).fill_(0xAB)
    dsb.ops.flash_attn_parts([q[0]], Sq, (H * 128, 128), k, v, o_parts, o_rows, (H * 128, 128), H, Sq, workspace=ws)
    got = torch.cat(o_parts)
    dsb.ops.check_status(0)
    assert O.rel_l2(got.float().cpu(), want.float().cpu()) < 1e-3
    pairs = ws.numel() // (4 * 256 * 528) + 1            # items that run at once: the workspace is for one less, cut in four
    items = 52 * H
    tail = items % pairs
    # which rows were cut: the last items, head-major, in two (three ranges of 18 key tiles would be shorter than eight)
    assert items > pairs and 0 < tail and -(-tail * 2 // pairs) / 2 + 0.05 < 1, "sizes that leave a last wave worth cutting"
    same = torch.ones(Sq, H, dtype=torch.bool)
    for it in range(items - tail, items):
        same[(it % 52) * 256:(it % 52 + 1) * 256, it // 52] = False
    assert torch.equal(got.cpu()[same], want.cpu()[same])
    rows = ws.view(-1, 528)
    assert not (rows[:tail * 2 * 256, :520] == 0xAB).all(dim=1).any()        # 128 columns, the reference and the row sum
    assert (rows[tail * 2 * 256:] == 0xAB).all()
    # against the exact restatement of the kernel's rounding, on a sample of the cut rows
    rows = slice(Sq - 256, Sq)
    ref = O.attention_bf16_probs(q[:, rows].transpose(1, 2).float().cpu(), k.transpose(1, 2).float().cpu(),
                                 v.transpose(1, 2).float().cpu())[0].transpose(0, 1)
    assert O.rel_l2(got[rows].float().cpu(), ref) < 3e-3
