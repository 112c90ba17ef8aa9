"""The GEMM on both sides of the rule that picks its tile width, and of the row count from which CTA pairs take it: ragged last
tiles in both directions, each operand format.

Bound: fp32 sums of at most K products (K * 2^-24) in front of one bf16 rounding (2^-9 relative, 1.7e-3 rms); int8 sums are
exact.  2.5e-3 leaves room for the rounding's sample."""
import pytest
import torch

from oracle import ops as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N", [(1, 136), (128, 264), (200, 21504), (256, 5120), (257, 5120), (300, 12288), (512, 3072),
                                 (512, 9216), (512, 12288), (1030, 3080), (2048, 5128), (4095, 5120)])
@pytest.mark.parametrize("fmt", ["bf16", "e4m3", "int8"])
def test_gemm_tile_widths(dsb, cuda_dev, M, N, fmt):
    K = 256
    g = torch.Generator(device=cuda_dev).manual_seed(M + N)
    a, w = (torch.randn(n, K, generator=g, device=cuda_dev) for n in (M, N))
    conv = {"bf16": lambda t: t.bfloat16(), "e4m3": lambda t: t.to(torch.float8_e4m3fn),
            "int8": lambda t: (t * 30).round().clamp(-127, 127).to(torch.int8)}[fmt]
    a, w = conv(a), conv(w)
    bias, rs, cs = (torch.rand(n, generator=g, device=cuda_dev) + 0.5 for n in (N, M, N))
    kw = {} if fmt == "bf16" else dict(row_scale=rs, col_scale=cs)
    ref = a.double() @ w.double().t()
    ref = (ref if fmt == "bf16" else ref * rs.double()[:, None] * cs.double()) + bias.double()
    out = torch.full((M + 1, N), 7.0, dtype=torch.bfloat16, device=cuda_dev)
    dsb.ops.gemm(a, w, bias=bias, out=out[:M], **kw)
    dsb.ops.check_status(0)
    assert O.rel_l2(out[:M].double(), ref) < 2.5e-3
    assert (out[M] == 7.0).all()
    resid = torch.randn(M, N, generator=g, device=cuda_dev).bfloat16()
    got = dsb.ops.gemm(a, w, bias=bias, gate=bias, resid=resid, **kw)
    assert O.rel_l2(got.double(), resid.double() + bias.double() * ref) < 2.5e-3
