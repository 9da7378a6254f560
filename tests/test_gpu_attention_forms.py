"""The attention kernel's forms at the sizes where they can go wrong: ragged last key tiles, references that rise late,
smaller items behind the last full round, items of different widths on one CTA.  Against the fp32 oracle with the
tolerances of the bf16 path; forms that only deal the same work out differently give the same bits."""
import pytest
import torch

from af3_kernels_b200.dpa import dot_product_attention
from oracle import attention_oracle as O

pytestmark = pytest.mark.gpu


def _inputs(B1, B2, S, D, seed, Sk=None):
    g = torch.Generator().manual_seed(seed)
    Sk = Sk or S
    q = torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16)
    k, v = (torch.randn(B1, B2, Sk, D, generator=g).to(torch.bfloat16) for _ in range(2))
    bias = torch.randn(B2, S, Sk, generator=g).to(torch.bfloat16)
    mask = torch.rand(B1, Sk, generator=g) >= 0.1
    return q, k, v, mask, bias


def _call(dev, q, k, v, mask, bias, **kw):
    return dot_product_attention(*(t.to(dev) for t in (q, k, v, mask, bias)), check_status=True, **kw).cpu()


def _check(out, ref, what):
    st = O.error_stats(out, ref)
    assert st["nan"] == 0 and st["max_abs"] <= 2e-2 and st["mean_abs"] <= 2e-3, (what, st)


@pytest.mark.parametrize("Sk", [1, 31, 32, 33, 64, 65, 96, 97, 127, 129, 159, 161, 193, 224, 225, 257, 389, 513])
def test_ragged_last_key_tile(cuda_device, Sk):
    for B1, B2, Sq, D in [(3, 2, 70, 32), (1, 3, 200, 24)]:
        q, k, v, mask, bias = _inputs(B1, B2, Sq, D, Sk, Sk)
        mask[:, -1] = True
        _check(_call(cuda_device, q, k, v, mask, bias), O.oracle_fp32(q, k, v, mask, bias), (Sk, B1))


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("at", [(32,), (130,), (160,), (250,), (300, 320, 352), (0,)])
def test_reference_rises(cuda_device, at, fp8):
    """Keys from some position on outweigh all before by 2^10 to 2^130; what was accumulated with the lower reference is
    scaled."""
    B1, B2, S, D = 3, 2, 384, 32
    q, k, v, mask, bias = _inputs(B1, B2, S, D, sum(at))
    for n, pos in enumerate(at):
        rows = torch.arange(S) % 4
        bias[:, :, pos:] += torch.tensor([0.0, 7.0, 20.0, 90.0])[rows][None, :, None].to(torch.bfloat16) * (1 if n == 0 else 0.5)
    if not fp8:
        _check(_call(cuda_device, q, k, v, mask, bias), O.oracle_fp32(q, k, v, mask, bias), at)
        return
    q8, qs = O.quantize_e4m3_per_head(q.float())
    k8, ks = O.quantize_e4m3_per_head(k.float())
    ref = O.oracle_fp32(q8, k8, v, mask, bias, qs, ks)
    # no workspace: the softmax threads add the bias, in fp32 (a staged copy rounds bias / scale to bf16, 2^-9 of a logit of 100)
    out = dot_product_attention(q8.to(cuda_device), k8.to(cuda_device), v.to(cuda_device), mask.to(cuda_device), bias.to(cuda_device),
                                q_scale=qs.to(cuda_device), k_scale=ks.to(cuda_device), use_workspace=False, check_status=True).cpu()
    st = O.error_stats(out, ref)
    assert st["nan"] == 0 and st["max_abs"] <= 6e-2, (at, st)


@pytest.mark.parametrize("gone", [40, 128, 160, 300])
@pytest.mark.parametrize("how", ["mask", "lowest"])
def test_leading_keys_out_of_play(cuda_device, gone, how):
    """The first keys masked, or with a bias of the type's lowest value: the reference starts there and rises to real logits."""
    q, k, v, mask, bias = _inputs(3, 2, 390, 32, gone)
    if how == "mask":
        mask[:, :gone] = False
        mask[0] = False
    else:
        bias[:, :, :gone] = torch.finfo(torch.bfloat16).min
    mask[1:, -1] = True
    _check(_call(cuda_device, q, k, v, mask, bias), O.oracle_fp32(q, k, v, mask, bias), (how, gone))


@pytest.mark.parametrize("B1,B2,S,D", [(78, 8, 256, 16), (77, 8, 250, 32), (41, 4, 640, 32), (5, 16, 700, 48), (7, 16, 900, 64), (150, 1, 130, 8)])
def test_smaller_items_behind_the_last_full_round(cuda_device, B1, B2, S, D):
    q, k, v, mask, bias = _inputs(B1, B2, S, D, S + D)
    out = _call(cuda_device, q, k, v, mask, bias)
    assert torch.equal(_call(cuda_device, q, k, v, mask, bias, rows_per_item=1), out)
    rows = [0, B1 // 2, B1 - 1]
    _check(out[rows], O.oracle_fp32(q[rows], k[rows], v[rows], mask[rows], bias), (B1, B2, S, D))


def test_items_of_one_and_two_query_tiles_on_one_cta(cuda_device):
    """Nine query tiles in pairs leave items of one; with five items to a CTA a slot of the Q buffers is skipped and used
    again."""
    q, k, v, mask, bias = _inputs(1, 10, 1100, 32, 3)
    ref = O.oracle_fp32(q, k, v, mask, bias)
    for ctas in (9, 11, 13):
        _check(_call(cuda_device, q, k, v, mask, bias, max_ctas=ctas), ref, ctas)


@pytest.mark.parametrize("D", [32, 40, 48, 56])
@pytest.mark.parametrize("B1,B2,S", [(1, 2, 77), (5, 3, 300), (2, 16, 1100)])
def test_heads_of_33_to_48_channels(cuda_device, B1, B2, S, D):
    """Q and K tiles in two parts (40 and 48 channels) beside the widths around them, channels strided as in [B1, S, B2, D]."""
    q, k, v, mask, bias = _inputs(B1, B2, S, D, S + D)
    q, k = (t.transpose(1, 2).contiguous().transpose(1, 2) for t in (q, k))
    _check(_call(cuda_device, q, k, v, mask, bias), O.oracle_fp32(q, k, v, mask, bias), (B1, B2, S, D))
