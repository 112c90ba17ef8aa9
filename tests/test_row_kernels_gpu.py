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
def test_gemv_rows(dsb, cuda_dev, N, K, fmt):
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
