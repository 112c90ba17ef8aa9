"""The CTA-pair attention kernel where its schedule can go wrong: key counts around its 128-key tiles and its three
softmax groups, more items per CTA pair than it has row-sum slots, references that move at every tile, odd batches, and
values that are not finite, and rows whose scores climb beyond the range of a probability.

Bound: the oracle rounds where the kernel rounds (bf16 probabilities against an integer reference), so what is left is
fp32 summation order and ex2 (2^-22) in front of one bf16 rounding of the output: about 1e-4, held to 5e-4."""
import pytest
import torch

from oracle import ops as O

pytestmark = pytest.mark.gpu
TOL = 5e-4


def _case(B, H, Sq, Sk, seed, dev, spread=1.5):
    g = torch.Generator().manual_seed(seed)
    q, k, v = (torch.randn(B, s, H, 128, generator=g).bfloat16() for s in (Sq, Sk, Sk))
    return (q.float() * spread).bfloat16(), k, v


def _ref(q, k, v, sm_scale=None):
    return O.attention_bf16_probs(*(t.transpose(1, 2) for t in (q, k, v)), sm_scale).transpose(1, 2)


def _check(dsb, dev, q, k, v, sm_scale=None):
    out = dsb.ops.flash_attn(q.to(dev), k.to(dev), v.to(dev), sm_scale=sm_scale).float().cpu()
    dsb.ops.check_status(0)
    err = O.rel_l2(out, _ref(q, k, v, sm_scale).bfloat16().float())
    assert torch.isfinite(out).all() and err < TOL, err


@pytest.mark.parametrize("Sk", [1, 63, 64, 65, 127, 128, 129, 255, 256, 257, 383, 384, 385, 512, 513, 769, 1025])
def test_key_counts_around_the_tiles(dsb, cuda_dev, Sk):
    """1 to 9 key tiles: fewer than, as many as and more than the three groups; 300 queries cut through both CTAs' rows."""
    _check(dsb, cuda_dev, *_case(1, 2, 300, Sk, Sk, cuda_dev))


@pytest.mark.parametrize("Sq", [1, 127, 128, 129, 255, 256, 257])
def test_query_counts_around_the_tiles(dsb, cuda_dev, Sq):
    _check(dsb, cuda_dev, *_case(3, 1, Sq, 200, Sq, cuda_dev))


@pytest.mark.parametrize("Sk", [70, 200, 300, 500])
def test_many_short_items_per_pair(dsb, cuda_dev, Sk):
    """800 items of 1 to 4 key tiles on at most 74 pairs: each pair reuses its row-sum slots, both Q buffers and the rings
    across items of which the next has begun before the last is written."""
    _check(dsb, cuda_dev, *_case(1, 40, 20 * 256, Sk, 3, cuda_dev))


@pytest.mark.parametrize("growth", [3.0, 15.0])
def test_reference_moves_at_every_tile(dsb, cuda_dev, growth):
    """Each key tile holds one key that is larger than everything before it, so the reference - which trails by up to
    three tiles - moves again and again and O is rescaled by whichever group comes next.  (The largest exponent here is
    about 2^70 above the first tile's: within the range of a probability.)"""
    q, k, v = _case(1, 2, 256, 12 * 128, 7, cuda_dev)
    for j in range(12):
        k[:, j * 128 + (37 * j) % 128] *= 1.0 + growth * j / 12
    out = dsb.ops.flash_attn(q.to(cuda_dev), k.to(cuda_dev), v.to(cuda_dev)).float().cpu()
    ref = O.attention(*(t.transpose(1, 2) for t in (q, k, v))).transpose(1, 2)
    assert torch.isfinite(out).all()
    assert O.rel_l2(out, ref) < 4e-3        # bf16 probabilities and output against exact: 2^-9 each, as in the other tests


def _exact(q, k, v):
    """softmax in 64 bits on the device; [B, S, H, 128] in and out"""
    q, k, v = (t.double().transpose(1, 2) for t in (q, k, v))
    return (torch.softmax(q @ k.transpose(-1, -2) * 128 ** -0.5, dim=-1) @ v).transpose(1, 2)


def _check_rows(out, ref):
    """Every row by itself: a probability is off by its bf16 rounding (2^-9) and by its score's fp32 error (scores up to 2^10
    in log2 units, 2^-24 of the sum of their products' magnitudes: 2^-12), an output by its rounding (2^-9); 2e-2 leaves a
    factor of four for rows whose values cancel."""
    assert torch.isfinite(out).all()
    err = (out.double() - ref).norm(dim=-1) / ref.norm(dim=-1)
    assert err.max() < 2e-2, err.max()
    assert O.rel_l2(out.double(), ref) < 4e-3


@pytest.mark.parametrize("exponents", [(101, 110), (105, 125), (120, 160), (130, 250), (90, 180), (99.5, 100.5, 101.5)])
@pytest.mark.parametrize("spots", ["neighbours", "one tile", "across chunks", "next item"])
def test_keys_beyond_the_range_of_a_probability(dsb, cuda_dev, exponents, spots):
    """Keys that score 2^100 and more above everything before them, before the reference has had a chance to follow: the
    largest one must win by as much as it should.  Rows see them with a positive, a negative or no weight at all."""
    dev = cuda_dev
    at = {"neighbours": (140, 300, 450), "one tile": (131, 133, 140), "across chunks": (383, 257, 310),
          "next item": (650, 600, 20)}[spots]
    g = torch.Generator(device=dev).manual_seed(17)
    q, k, v = (torch.randn(1, s, 6, 128, generator=g, device=dev) * w for s, w in ((3000, 0.3), (700, 0.3), (700, 1.0)))
    q[..., 0] = 16.0 * (1 - torch.arange(3000, device=dev) % 3)[None, :, None]
    k[..., 0] = 0.0
    for e, j in zip(exponents, at):
        k[:, j, :, 0] = e / (16.0 * 128 ** -0.5 * 1.4426950408889634)
    q, k, v = (t.bfloat16() for t in (q, k, v))
    _check_rows(dsb.ops.flash_attn(q, k, v), _exact(q, k, v))


@pytest.mark.parametrize("B,H,Sq,Sk", [(1, 2, 256, 12 * 128), (2, 40, 700, 500), (1, 3, 300, 257), (1, 2, 200, 4000)])
@pytest.mark.parametrize("std", [6.0, 10.0, 16.0])
def test_queries_and_keys_of_any_spread(dsb, cuda_dev, B, H, Sq, Sk, std):
    """Scores whose spread is a multiple of the range of a probability: references are lifted in most tiles."""
    g = torch.Generator(device=cuda_dev).manual_seed(19)
    q, k = (torch.randn(B, s, H, 128, generator=g, device=cuda_dev).mul(std).bfloat16() for s in (Sq, Sk))
    v = torch.randn(B, Sk, H, 128, generator=g, device=cuda_dev).bfloat16()
    _check_rows(dsb.ops.flash_attn(q, k, v), _exact(q, k, v))


def test_steep_rows_in_a_split_last_wave(dsb, cuda_dev):
    """The same through the launch whose last items are cut along the keys (partial results with references of their own),
    and with an e4m3 output, which is the bf16 one cast."""
    g = torch.Generator(device=cuda_dev).manual_seed(23)
    H, Sq, Sk = 3, 52 * 256, 2250
    q, k = (torch.randn(1, s, H, 128, generator=g, device=cuda_dev).mul(10).bfloat16() for s in (Sq, Sk))
    v = torch.randn(1, Sk, H, 128, generator=g, device=cuda_dev).bfloat16()
    out = torch.zeros(Sq, H, 128, dtype=torch.bfloat16, device=cuda_dev)
    dsb.ops.flash_attn_parts([q[0]], Sq, (H * 128, 128), k, v, [out], Sq, (H * 128, 128), H, Sq,
                             workspace=dsb.ops.flash_attn_workspace(cuda_dev))
    _check_rows(out[None, -2048:], _exact(q[:, -2048:], k, v))
    plain = dsb.ops.flash_attn(q, k, v)
    out8 = torch.empty(1, Sq, H, 128, dtype=torch.float8_e4m3fn, device=cuda_dev)
    dsb.ops.flash_attn(q, k, v, out=out8)
    assert torch.equal(out8.float(), plain.float().clamp(-448, 448).to(torch.float8_e4m3fn).float())


def test_keys_that_score_minus_infinity(dsb, cuda_dev):
    """A whole first key tile of weight zero leaves the row to the others."""
    q, k, v = _case(1, 2, 200, 600, 29, cuda_dev)
    q[..., 0] = 1.0
    k[:, :200, :, 0] = float("-inf")
    q, k, v = (t.to(cuda_dev) for t in (q, k, v))
    _check_rows(dsb.ops.flash_attn(q, k, v), _exact(q, k[:, 200:], v[:, 200:]))


@pytest.mark.parametrize("sm_scale", [-0.08, 0.0, 1.0])
def test_any_scale(dsb, cuda_dev, sm_scale):
    _check(dsb, cuda_dev, *_case(1, 2, 200, 450, 11, cuda_dev, spread=1.0), sm_scale=sm_scale)


def test_a_nan_query_spoils_its_row_only_and_a_nan_key_every_row(dsb, cuda_dev):
    q, k, v = _case(1, 2, 300, 700, 13, cuda_dev)
    clean = dsb.ops.flash_attn(q.to(cuda_dev), k.to(cuda_dev), v.to(cuda_dev)).cpu()
    q2 = q.clone()
    q2[0, 130, 1, 5] = float("nan")
    out = dsb.ops.flash_attn(q2.to(cuda_dev), k.to(cuda_dev), v.to(cuda_dev)).cpu()
    bad = torch.zeros(1, 300, 2, dtype=torch.bool)
    bad[0, 130, 1] = True
    assert out[bad].isnan().all() and torch.equal(out[~bad], clean[~bad])
    for key in (3, 400, 699):               # the first tile, one in the middle, the ragged last one
        k2 = k.clone()
        k2[0, key, 0, 9] = float("nan")
        out = dsb.ops.flash_attn(q.to(cuda_dev), k2.to(cuda_dev), v.to(cuda_dev)).cpu()
        assert out[:, :, 0].isnan().all() and torch.equal(out[:, :, 1], clean[:, :, 1])
    dsb.ops.check_status(0)
