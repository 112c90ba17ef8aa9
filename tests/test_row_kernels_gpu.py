"""RMSNorm + RoPE rows and the one-row Linear at the sizes where their work split changes: fewer rows than resident CTAs,
one more than a multiple of them, widths from one vector per thread to eight, in place and chunked; weight rows on both sides
of the rule that picks the rows per warp, and activation vectors that are not 16-byte aligned.

Bounds: RMSNorm rounds once to bf16 (2^-9 relative, 1.7e-3 rms); the GEMV sums in fp32 (K * 2^-24 at most, 1e-5)."""
import pytest
import torch

from oracle import ops as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,D", [(1, 128), (3, 1024), (739, 5120), (741, 5120), (1037, 3072), (2221, 3072), (445, 8192), (1500, 640)])
@pytest.mark.parametrize("rope", [False, True])
def test_rmsnorm_rows(dsb, cuda_dev, M, D, rope):
    g = torch.Generator().manual_seed(M + D)
    x, w = torch.randn(M, D, generator=g).bfloat16(), 1 + 0.1 * torch.randn(D, generator=g)
    ang = torch.rand(M + 5, 64, generator=g) * 6
    table = torch.stack([ang.cos(), ang.sin()], dim=-1).contiguous()
    ref = O.rmsnorm(x, w)
    if rope:
        ref = O.apply_rope_pairs(ref.reshape(M, D // 128, 128), table[5:, None]).reshape(M, D)
    dev = dict(rope=table.to(cuda_dev) if rope else None, rope_row0=5 if rope else 0)
    out = torch.empty_like(x, device=cuda_dev)
    dsb.ops.rmsnorm_full(x.to(cuda_dev), w.to(cuda_dev), out=out, **dev)
    assert O.rel_l2(out.float().cpu(), ref) < 2.5e-3
    buf = x.to(cuda_dev)
    dsb.ops.rmsnorm_full(buf, w.to(cuda_dev), **dev)
    assert torch.equal(buf, out)
    if D % 256 == 0:
        chunked = torch.empty(2, M, D // 2, dtype=torch.bfloat16, device=cuda_dev)
        dsb.ops.rmsnorm_full(x.to(cuda_dev), w.to(cuda_dev), out=chunked, chunks=2, **dev)
        assert torch.equal(torch.cat([chunked[0], chunked[1]], dim=1), out)


@pytest.mark.parametrize("N,K", [(1, 16), (7, 256), (33, 3072), (3072, 4080), (3072, 4096), (5120, 5120), (9000, 4608), (20001, 3072)])
@pytest.mark.parametrize("fmt", ["bf16", "e4m3", "int8"])
def test_one_row(dsb, cuda_dev, N, K, fmt):
    g = torch.Generator(device=cuda_dev).manual_seed(N + K)
    W = torch.randn(N, K, generator=g, device=cuda_dev)
    W = {"bf16": lambda t: t.bfloat16(), "e4m3": lambda t: t.to(torch.float8_e4m3fn),
         "int8": lambda t: (t * 30).round().clamp(-127, 127).to(torch.int8)}[fmt](W)
    xb = torch.randn(K + 1, generator=g, device=cuda_dev)
    bias, scale = torch.randn(N, generator=g, device=cuda_dev), torch.rand(N, generator=g, device=cuda_dev) + 0.5
    for x in (xb[:K], xb[1:]):                                     # 16-byte aligned, and not
        for act in (dsb.ops.ACT_NONE, dsb.ops.ACT_SILU):
            f = torch.nn.functional.silu(x.double()) if act else x.double()
            ref = (W.double() @ f) * scale.double() + bias.double()
            y = dsb.ops.gemv(W, x, scale, bias, act_in=act)
            assert O.rel_l2(y.double(), ref) < 1e-5
            acc = ref.float().clone()
            dsb.ops.gemv(W, x, scale, bias, act_in=act, out=acc, accumulate=True)
            assert O.rel_l2(acc.double(), 2 * ref) < 1e-5


@pytest.mark.parametrize("M", [1, 3, 4, 5, 130])
@pytest.mark.parametrize("fmt", ["bf16", "fp8_tensor", "fp8_channel", "int8_channel"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32, torch.float16])
def test_patched_linear_equals_its_parts(dsb, cuda_dev, M, fmt, dtype):
    """The patched F.linear in every dtype and on both sides of its row limit, on strided and 3-D inputs, is bit for bit the
    conversion, quantiser, product and cast that it stands for."""
    from diffsynth_engine_b200 import quant
    from diffsynth_engine_b200.packed import act_format
    ops = dsb.ops
    torch.manual_seed(M)
    layer = torch.nn.Linear(256, 72).to(cuda_dev, torch.bfloat16)
    quant.enable_b200_linear(layer, fmt)
    w, b = layer.weight, layer.bias.float()
    base = torch.randn(2 * M, 512, device=cuda_dev).to(dtype)
    for x in (base[:M, :256], base[::2, 256:], base[:M, 1:257], base[:M, :256].reshape(1, M, 256)):
        with quant.b200_inference():
            got = layer(x)
        rows = x.reshape(-1, 256)
        if M <= 4:
            want = torch.stack([ops.gemv(w.data, r.float().contiguous(), w.scale, b) for r in rows])
        else:
            xb = rows.to(torch.bfloat16).contiguous()
            if fmt == "bf16":
                want = ops.gemm(xb, w.data, bias=b)
            else:
                q, s = ops.quant_rows(xb, act_format(fmt))
                want = ops.gemm(q, w.data, row_scale=s, col_scale=w.scale, bias=b)
        assert got.dtype == dtype and got.shape == (*x.shape[:-1], 72)
        assert torch.equal(got.reshape(M, 72), want.to(dtype))


@pytest.mark.parametrize("fmt", ["e4m3", "int8"])
def test_linear_rows_of_an_empty_product(dsb, cuda_dev, fmt):
    """No rows or no columns: nothing to launch, and no scratch either (an empty tensor has no address)."""
    code = dsb.ops.FMT_E4M3 if fmt == "e4m3" else dsb.ops.FMT_INT8
    W, scale = dsb.ops.pack_quant_weight(torch.randn(64, 256, device=cuda_dev), code, per_channel=True)
    x = torch.randn(9, 256, device=cuda_dev).bfloat16()
    assert dsb.ops.linear_rows(x[:0], W, scale).shape == (0, 64)
    assert dsb.ops.linear_rows(x, W[:0], scale[:0]).shape == (9, 0)
    assert dsb.ops.linear_rows(x, W, scale).shape == (9, 64)


@pytest.mark.parametrize("M", [1, 3, 4])
@pytest.mark.parametrize("N,K", [(1, 16), (7, 2032), (300, 2048), (33, 2064), (72, 4096), (3072, 3072), (260, 5120), (20001, 4608)])
@pytest.mark.parametrize("fmt", ["bf16", "e4m3", "int8"])
def test_few_rows_in_one_launch(dsb, cuda_dev, M, N, K, fmt):
    """``gemv_rows`` at the widths it is for: more than one trip of the activation staging (K > 2048 from bf16 rows, > 4096
    from fp32 ones), one and four weight rows per warp, several rows, which may be strided and start at any element, and
    both output types.  Nothing outside the output's rows is written."""
    g = torch.Generator(device=cuda_dev).manual_seed(M + N + K)
    W = torch.randn(N, K, generator=g, device=cuda_dev)
    W = {"bf16": lambda t: t.bfloat16(), "e4m3": lambda t: t.to(torch.float8_e4m3fn),
         "int8": lambda t: (t * 30).round().clamp(-127, 127).to(torch.int8)}[fmt](W)
    bias, scale = torch.randn(N, generator=g, device=cuda_dev), torch.rand(N, generator=g, device=cuda_dev) + 0.5
    base = torch.randn(M, K + 24, generator=g, device=cuda_dev)
    for x_dtype in (torch.bfloat16, torch.float32):
        for off in (0, 1, 8, 13):
            x = base.to(x_dtype)[:, off:off + K]
            ref = (x.double() @ W.double().t()) * scale.double() + bias.double()
            outs = [torch.full((M, N + 3), 7.0, dtype=t, device=cuda_dev) for t in (torch.float32, torch.bfloat16)]
            for out in outs:
                dsb.ops.gemv_rows(W, x, scale, bias, out=out[:, 1:N + 1])
                assert (out[:, 0] == 7).all() and (out[:, N + 1:] == 7).all()
            # fp32 sums of up to 5120 products; a bf16 output is the fp32 one rounded once
            assert O.rel_l2(outs[0][:, 1:N + 1].double(), ref) < 1e-5
            assert torch.equal(outs[1], outs[0].bfloat16())
    assert torch.equal(dsb.ops.gemv_rows(W, base.bfloat16()[:, :K], scale, bias),
                       dsb.ops.gemv_rows(W, base.bfloat16()[:, :K].contiguous(), scale, bias))
    rows = base[:1, :K].expand(M, K)                          # one row for all of them
    assert torch.equal(dsb.ops.gemv_rows(W, rows, scale, bias), dsb.ops.gemv_rows(W, rows.contiguous(), scale, bias))
