"""RMSNorm + RoPE rows at the sizes where their work split changes: fewer rows than resident CTAs, one more than a multiple
of them, widths from one vector per thread to eight, in place and chunked.

Bound: RMSNorm rounds once to bf16 (2^-9 relative, 1.7e-3 rms)."""
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
