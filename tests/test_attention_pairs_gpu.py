"""The CTA-pair attention kernel where its schedule can go wrong: key counts around its 128-key tiles and its three
softmax groups, more items per CTA pair than it has row-sum slots, references that move at every tile, odd batches, and
values that are not finite.

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
    three tiles - moves again and again and O is rescaled by whichever group comes next.  The largest exponent here is
    about 2^70 above the first tile's: growth beyond 2^100 within three tiles is cut there by contract."""
    q, k, v = _case(1, 2, 256, 12 * 128, 7, cuda_dev)
    for j in range(12):
        k[:, j * 128 + (37 * j) % 128] *= 1.0 + growth * j / 12
    out = dsb.ops.flash_attn(q.to(cuda_dev), k.to(cuda_dev), v.to(cuda_dev)).float().cpu()
    ref = O.attention(*(t.transpose(1, 2) for t in (q, k, v))).transpose(1, 2)
    assert torch.isfinite(out).all()
    assert O.rel_l2(out, ref) < 4e-3        # bf16 probabilities and output against exact: 2^-9 each, as in the other tests


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
