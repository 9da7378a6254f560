"""The attention kernel's forms at the sizes where they can go wrong: ragged last key tiles, references that rise late,
smaller items behind the last full round, items of different widths on one CTA.  Against the fp32 oracle with the
tolerances of the bf16 path; forms that only deal the same work out differently give the same bits."""
import pytest
import torch

import af3_kernels_b200 as A
from af3_kernels_b200 import _capi
from af3_kernels_b200.dpa import dot_product_attention, read_status, stage_bias
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
    return dot_product_attention(*(None if t is None else t.to(dev) for t in (q, k, v, mask, bias)), check_status=True, **kw).cpu()


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


_LOWEST = torch.finfo(torch.bfloat16).min


@pytest.mark.parametrize("route", ["scaled_q", "unscaled_q", "f32_bias", "fp8", "fp8_no_workspace"])
@pytest.mark.parametrize("value", [-1e7, -1e9, -2e9, -1e10, -1e12, -1e15, -1e30, -2.2e38, _LOWEST, torch.finfo(torch.float32).min])
def test_keys_far_below_all_others(cuda_device, value, route):
    """A bias far below every logit, down to the type's lowest value: on the first 1 to 300 keys it takes them out, on a
    whole query row it leaves the softmax uniform.  (No mask: whether a masked key lies above such a bias is the caller's
    choice of fill.)"""
    B1, B2, S, D = 3, 2, 392, 32
    if route != "f32_bias":
        value = max(value, _LOWEST)
    q, k, v, _, bias = _inputs(B1, B2, S, D, 7)
    bias = bias.float()
    for first, row in [(1, 3), (40, 10), (128, 11), (160, 150), (300, 260)]:
        bias[:, row::23, :first] = value
    bias[:, 5::7] = value                       # whole rows
    scales, kw, scale = {}, {}, None
    if route == "unscaled_q":
        q, scale = q * D ** -0.5, 1.0           # the producer has applied the softmax scale
    if route.startswith("fp8"):
        (q, qs), (k, ks) = O.quantize_e4m3_per_head(q.float()), O.quantize_e4m3_per_head(k.float())
        scales = {"q_scale": qs, "k_scale": ks}
        kw = {"use_workspace": route == "fp8"}
    if route != "f32_bias":
        bias = bias.to(torch.bfloat16)
    qf = (q.float() * qs.view(1, -1, 1, 1) if scales else q.float()).double() * (D ** -0.5 if scale is None else scale)
    kf = (k.float() * ks.view(1, -1, 1, 1) if scales else k.float()).double()
    # the logits as fp32 holds them: next to 1e9 products of q and k are below half of the last bit
    logits = (qf @ kf.transpose(-1, -2) + bias.double()).float().double()
    ref = torch.softmax(logits, -1) @ v.double()
    out = _call(cuda_device, q, k, v, None, bias, softmax_scale=scale, **{n: t.to(cuda_device) for n, t in scales.items()}, **kw)
    assert torch.isfinite(out.float()).all(), (route, value, torch.isfinite(out.float()).all(-1).sum())
    # rows that keep an ordinary key, and rows that have none above the value.  At 1e7 fp32's last bit is 1, so a row's logits there
    # are rounded to whole numbers, by the oracle in one step and by the kernel in several: such rows are compared from 1e9 on.
    whole = torch.arange(S) % 7 == 5
    limit = (6e-2, 6e-3) if scales else (2e-2, 2e-3)
    for rows in [~whole] + ([whole] if abs(value) >= 1e9 else []):
        st = O.error_stats(out[:, :, rows], ref[:, :, rows].float())
        assert st["max_abs"] <= limit[0] and st["mean_abs"] <= limit[1], (route, value, st)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("Sk,pitch,offset", [(1, 1, 0), (7, 8, 0), (8, 8, 0), (9, 16, 0), (9, 9, 0), (64, 72, 3), (77, 80, 0), (77, 84, 4), (129, 136, 8)])
def test_conversion_of_the_bias(cuda_device, Sk, pitch, offset, dtype):
    """Eight columns a thread: rows that do and do not start on 16-byte boundaries, last columns of every remainder.  The
    same bits as torch's conversion, zeros in the padding; with fp8 scales the quotient is taken first."""
    B2, Sq = 3, 37
    g = torch.Generator().manual_seed(Sk)
    buf = torch.randn(B2 * Sq * pitch + 16, generator=g).to(cuda_device, dtype)
    bias = buf[offset:offset + B2 * Sq * pitch].view(B2, Sq, pitch)[:, :, :Sk]
    scales = (torch.rand(2, B2, generator=g) + 0.5).to(cuda_device)
    plain, scaled = stage_bias(bias, B2, Sq, Sk).data, stage_bias(bias, B2, Sq, Sk, q_scale=scales[0], k_scale=scales[1], softmax_scale=0.25).data
    factor = (1.0 / (0.25 * scales[0] * scales[1])).view(B2, 1, 1)
    for got, want in [(plain, bias.float()), (scaled, bias.float() * factor)]:
        assert torch.equal(got[:, :, :Sk], want.to(torch.bfloat16)) and not got[:, :, Sk:].any()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B1,B2,Sq,Sk,D,pitch,offset", [
    (1, 16, 77, 77, 24, 77, 0), (1, 16, 512, 512, 32, 516, 4), (1, 3, 129, 131, 64, 131, 0), (2, 16, 300, 300, 48, 300, 0), (1, 2, 1, 1, 8, 1, 0),
    (1, 5, 130, 385, 32, 388, 8), (1, 5, 130, 388, 32, 388, 8), (1, 4, 127, 640, 40, 644, 3), (1, 4, 127, 640, 40, 644, 4), (1, 4, 250, 100, 32, 100, 0),
    (1, 300, 100, 260, 16, 260, 0), (1, 300, 100, 99, 16, 99, 0), (1, 16, 1100, 1100, 24, 1100, 0)])
def test_bias_converted_by_the_attention_kernel(cuda_device, B1, B2, Sq, Sk, D, pitch, offset, dtype):
    """Items of one query tile (several to a CTA with 300 heads), rows that start on four keys or a single key tile: one
    launch, the same bits as with a pass of its own over the bias; -inf and the lowest value included.  Otherwise that pass."""
    q, k, v, mask, _ = _inputs(B1, B2, Sq, D, Sk, Sk)
    g = torch.Generator().manual_seed(Sk)
    mask[:, -1] = True
    flat = torch.randn(B2 * Sq * pitch + 16, generator=g)
    bias = flat[offset:offset + B2 * Sq * pitch].view(B2, Sq, pitch)[:, :, :Sk]
    bias[torch.rand(bias.shape, generator=g) < 0.05] = -float("inf")
    bias[:, Sq // 2] = torch.finfo(dtype).min
    bias[..., -1] = 0
    on_dev = flat.to(cuda_device, dtype)
    bias = on_dev[offset:offset + B2 * Sq * pitch].view(B2, Sq, pitch)[:, :, :Sk]
    args = [t.to(cuda_device) for t in (q, k, v, mask)]
    lib = _capi.load()
    out = A.dot_product_attention_cpp(*args, bias)
    in_kernel = Sk <= 128 or (Sk % 4 == 0 and pitch % 4 == 0 and offset % 4 == 0)
    assert lib.af3k_last_launch_count() == (1 if in_kernel else 2)
    staged = dot_product_attention(*args, bias, cache_bias=False, check_status=True)
    assert lib.af3k_last_launch_count() == 2
    assert torch.equal(out, staged)
    _check(out.cpu(), O.oracle_fp32(q, k, v, mask, bias.cpu()), (B1, B2, Sq, Sk, D))


@pytest.mark.parametrize("N", [77, 500, 1300])
def test_single_block_converts_its_bias(cuda_device, N):
    """With the gate: the same bits as with the bf16 bias in rows of 16 bytes, within the kernel's own conversion and beyond."""
    g = torch.Generator().manual_seed(N)
    H, C = 4, 96
    x, w = torch.randn(N, C, generator=g).to(cuda_device, torch.bfloat16), [(torch.randn(C, C, generator=g) * 0.1).to(cuda_device, torch.bfloat16) for _ in range(4)]
    bias = torch.randn(H, N, N, generator=g).to(cuda_device)
    mask = (torch.rand(N, generator=g) >= 0.1).to(cuda_device)
    block = lambda b: A.self_attention_cpp(x, mask, b, w[0], torch.zeros(C, device=cuda_device), *w[1:], H)
    assert torch.equal(block(bias), block(stage_bias(bias, H, N, N).data[:, :, :N]))


@pytest.mark.parametrize("dtype,Sk", [(torch.float32, 392), (torch.bfloat16, 389)])
def test_minus_infinity_in_a_bias_that_is_converted(cuda_device, dtype, Sk):
    """fp32 or ragged rows: keys with a bias of -inf have no weight, a key with +inf has all of it, the keys beside them keep
    theirs; NaN still makes its row NaN and no other."""
    q, k, v, mask, bias = _inputs(3, 2, 200, 32, 8, Sk)
    bias = bias.to(dtype)
    g = torch.Generator().manual_seed(3)
    bias[torch.rand(bias.shape, generator=g) < 0.2] = -float("inf")
    bias[:, 7, :140] = -float("inf")
    mask[:, -1], bias[..., -1] = True, 0
    ref = O.oracle_fp32(q, k, v, mask, bias)
    _check(_call(cuda_device, q, k, v, mask, bias), ref, "-inf")
    bias[:, 20, Sk - 1], bias[:, 21, Sk - 1] = float("inf"), float("nan")
    out = _call(cuda_device, q, k, v, mask, bias)
    assert torch.isnan(out).any(-1).any(0).any(0).nonzero().flatten().tolist() == [21]
    assert torch.equal(out[:, :, 20], v[:, :, Sk - 1])


@pytest.mark.parametrize("value", [0, -38 * 2 ** 12, -152 * 2 ** 14, -152 * 2 ** 16, 152 * 2 ** 16])
def test_reference_rises_under_a_large_bias(cuda_device, value):
    """Logits of 1e7 that differ by a few units, all whole numbers that fp32 holds exactly: what earlier key tiles summed
    up is brought to the later reference without the rounding of the one or the other (half a unit of the exponent here)."""
    B1, B2, S, D = 2, 3, 500, 32
    g = torch.Generator().manual_seed(11)
    k = torch.zeros(B1, B2, S, D)
    k[..., 0] = torch.randint(-60, -40, (B1, B2, S), generator=g).float()
    k[:, :, :128, 0] = 0                                  # 128 keys of weight e^-6 .. e^-9, then one of weight 1
    for n, step in enumerate((6, 7, 9)):
        k[:, n, 200 + 100 * n, 0] = step
    q = torch.zeros(B1, B2, S, D)
    q[..., 0] = 1
    v = torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16)
    v[:, :, :128] += 2
    bias = torch.full((B2, S, S), float(value)) - torch.randint(0, 2, (B2, S, 1), generator=g) * 2.0 ** 16
    q, k, bias = (t.to(torch.bfloat16) for t in (q, k, bias))
    logits = q.double() @ k.double().transpose(-1, -2) + bias.double()
    assert torch.equal(logits.float().double(), logits)
    ref = torch.softmax(logits, -1) @ v.double()
    _check(_call(cuda_device, q, k, v, None, bias, softmax_scale=1.0), ref.float(), value)


def _quantised(q, k):
    (q, qs), (k, ks) = O.quantize_e4m3_per_head(q.float()), O.quantize_e4m3_per_head(k.float())
    return q, k, {"q_scale": qs, "k_scale": ks}


def _plan(B1, B2, S, D, fp8=False, Sk=None, max_ctas=0, rows_per_item=0):
    Sk = Sk or S
    d = _capi.AttentionDesc()
    d.B1, d.B2, d.Sq, d.Sk, d.D = B1, B2, S, Sk, D
    for n, keys in (("q_stride", S), ("k_stride", Sk), ("v_stride", Sk), ("out_stride", S)):
        getattr(d, n)[:] = [B2 * keys * D, keys * D, D]
    d.bias_stride[:], d.mask_row_stride, d.softmax_scale, d.max_ctas, d.rows_per_item = [S * Sk, Sk], Sk, D ** -0.5, max_ctas, rows_per_item
    d.qk_dtype, d.bias_dtype = _capi.AF3K_FP8_E4M3 if fp8 else _capi.AF3K_BF16, _capi.AF3K_BF16
    return _capi.describe_plan(d)


def _check_form(dev, B1, B2, S, D, qk, **other):
    """One row of items against the oracle, and the same bits as with another split of the work."""
    q, k, v, mask, bias = _inputs(B1, B2, S, D, S + D)
    scales, kw, on_dev = {}, {}, {}
    if qk != "bf16":
        q, k, scales = _quantised(q, k)
        kw = {"use_workspace": qk == "fp8"}
        on_dev = {n: t.to(dev) for n, t in scales.items()}
    out = _call(dev, q, k, v, mask, bias, **kw, **on_dev)
    assert torch.equal(_call(dev, q, k, v, mask, bias, **other, **kw, **on_dev), out)
    rows = [0, B1 // 2, B1 - 2, B1 - 1]
    st = O.error_stats(out[rows], O.oracle_fp32(q[rows], k[rows], v[rows], mask[rows], bias, **scales))
    limit = (2e-2, 2e-3) if qk == "bf16" else (6e-2, 6e-3)
    assert st["nan"] == 0 and st["max_abs"] <= limit[0] and st["mean_abs"] <= limit[1], st


@pytest.mark.parametrize("B1,B2,S,D,qk", [
    (99, 3, 130, 8, "bf16"), (99, 3, 130, 24, "bf16"), (46, 8, 136, 16, "bf16"), (78, 8, 256, 16, "bf16"), (77, 8, 250, 32, "bf16"), (41, 4, 640, 32, "bf16"),
    (46, 8, 136, 16, "fp8"), (99, 3, 136, 32, "fp8"), (41, 4, 640, 32, "fp8"), (46, 8, 136, 16, "fp8_no_workspace"), (99, 3, 136, 32, "fp8_no_workspace"),
    (41, 4, 640, 32, "fp8_no_workspace")])
def test_smaller_items_behind_the_last_full_round(cuda_device, B1, B2, S, D, qk):
    """Items of three or four rows, then items of two."""
    plan = _plan(B1, B2, S, D, qk != "bf16")
    tiles = B2 * ((S + 127) // 128)
    assert plan["rows_per_item"] > 2 and plan["items"] > -(-B1 // plan["rows_per_item"]) * tiles, plan
    _check_form(cuda_device, B1, B2, S, D, qk, rows_per_item=1)


@pytest.mark.parametrize("B1,B2,S,D,qk", [(5, 16, 700, 48, "bf16"), (7, 16, 900, 64, "bf16"), (150, 1, 130, 8, "bf16"), (7, 16, 904, 64, "fp8"),
                                          (7, 16, 904, 64, "fp8_no_workspace"), (149, 2, 264, 16, "fp8"), (149, 2, 264, 16, "fp8_no_workspace")])
def test_rows_that_do_not_fill_the_last_item(cuda_device, B1, B2, S, D, qk):
    """Items of one width, the last of them of fewer rows; a cap on the CTAs gives each CTA several of both."""
    _check_form(cuda_device, B1, B2, S, D, qk, max_ctas=B2 * 3)


@pytest.mark.parametrize("fp8", [False, True])
def test_items_of_one_and_two_query_tiles_on_one_cta(cuda_device, fp8):
    """Nine query tiles in pairs leave items of one; with five items to a CTA a slot of the Q buffers is skipped and used
    again."""
    q, k, v, mask, bias = _inputs(1, 10, 1100, 32, 3)
    scales = {}
    if fp8:
        q, k, scales = _quantised(q, k)
    ref = O.oracle_fp32(q, k, v, mask, bias, **scales)
    for ctas in (9, 11, 13):
        out = _call(cuda_device, q, k, v, mask, bias, max_ctas=ctas, **{n: t.to(cuda_device) for n, t in scales.items()})
        if fp8:
            assert O.error_stats(out, ref)["max_abs"] <= 6e-2, ctas
        else:
            _check(out, ref, ctas)


@pytest.mark.parametrize("D", [32, 40, 48, 56])
@pytest.mark.parametrize("B1,B2,S", [(1, 2, 77), (5, 3, 300), (2, 16, 1100)])
def test_heads_of_33_to_48_channels(cuda_device, B1, B2, S, D):
    """Q and K tiles in two parts (40 and 48 channels) beside the widths around them, channels strided as in [B1, S, B2, D]."""
    q, k, v, mask, bias = _inputs(B1, B2, S, D, S + D)
    q, k = (t.transpose(1, 2).contiguous().transpose(1, 2) for t in (q, k))
    _check(_call(cuda_device, q, k, v, mask, bias), O.oracle_fp32(q, k, v, mask, bias), (B1, B2, S, D))


@pytest.mark.parametrize("B1,B2,S,D", [(12, 2, 100, 32), (12, 2, 100, 64), (14, 2, 128, 16), (6, 2, 200, 48), (9, 2, 300, 32), (8, 2, 260, 64), (1, 4, 100, 32),
                                       (1, 6, 129, 64)])
@pytest.mark.parametrize("scale", [None, 1.0])
def test_several_items_on_one_cta(cuda_device, B1, B2, S, D, scale):
    """One, two or four streams and one to three key tiles per item, many items per CTA: a stream's result is stored under the tile
    that comes next, and the next item's Q tiles are scaled meanwhile (not at all with a scale of 1).  Logits that grow by more than the
    lazy bound between key tiles have the accumulator next to it rescaled at the same time."""
    q, k, v, mask, bias = _inputs(B1, B2, S, D, S + D + B1)
    if scale:
        q = (q * D ** -0.5).to(torch.bfloat16)
    bias[..., 128:] += 12
    bias[..., 256:] += 12
    kw = {"softmax_scale": scale} if scale else {}
    ref = O.oracle_fp32(q, k, v, mask, bias)
    if scale:
        logits = q.float() @ k.float().transpose(-1, -2) + bias.float()
        ref = torch.softmax(logits.masked_fill(~mask[:, None, None, :], -1e9), -1) @ v.float()
    out = _call(cuda_device, q, k, v, mask, bias, **kw)
    _check(out, ref, (B1, B2, S, D))
    for other in ({"max_ctas": 2}, {"max_ctas": 3}, {"max_ctas": 2, "rows_per_item": 2}, {"rows_per_item": 1}):
        assert torch.equal(_call(cuda_device, q, k, v, mask, bias, **kw, **other), out), other


@pytest.mark.parametrize("S", [300, 640, 1100, 1152])
@pytest.mark.parametrize("D", [8, 24, 32, 48, 64])
def test_bias_stages_of_query_tile_streams(cuda_device, S, D):
    """Two query tiles per item bring three bias stages (two from 33 channels on), one per item and shared ones two: more key tiles than
    stages, an odd number of query tiles, one item and several per CTA."""
    q, k, v, mask, bias = _inputs(1, 2, S, D, S + D)
    out = _call(cuda_device, q, k, v, mask, bias)
    _check(out, O.oracle_fp32(q, k, v, mask, bias), (S, D))
    assert _plan(1, 2, S, D)["streams"] == 1
    tiles = (S + 127) // 128
    for ctas in (1, 3, tiles + tiles % 2):
        plan = _plan(1, 2, S, D, max_ctas=ctas)
        pairs = ctas != 3 or tiles > 3
        assert plan["query_tile_streams"] == pairs and plan["bias_stages"] == (3 if pairs and D <= 32 else 2), plan
        assert torch.equal(_call(cuda_device, q, k, v, mask, bias, max_ctas=ctas), out), ctas


@pytest.mark.parametrize("B1,B2,S,Sk,D,max_ctas,q_buffers", [
    (1, 3, 300, 300, 64, 3, 1), (1, 3, 300, 200, 64, 3, 1), (1, 3, 300, 100, 32, 3, 2), (1, 7, 300, 300, 48, 5, 2), (1, 16, 2400, 2400, 64, 0, 1),
    (3, 16, 1400, 1400, 48, 0, 1), (5, 16, 1660, 1660, 48, 0, 1)])
def test_pair_of_query_tiles_behind_a_lone_one(cuda_device, B1, B2, S, Sk, D, max_ctas, q_buffers):
    """CTAs that begin with a lone query tile, on which one softmax warpgroup has no stream, and go on with a pair of them: that
    warpgroup scales the pair's second Q tile, from a slot that the lone tile's item went through without using it."""
    plan = _plan(B1, B2, S, D, Sk=Sk, max_ctas=max_ctas)
    tiles = (S + 127) // 128
    lone = lambda item: item % (tiles // 2 + 1) == tiles // 2
    assert tiles % 2 and plan["query_tile_streams"] and plan["q_buffers"] == q_buffers, plan
    assert any(lone(c) and not lone(c + plan["grid"]) for c in range(plan["items"] - plan["grid"])), plan
    q, k, v, mask, bias = _inputs(B1, B2, S, D, S + D, Sk)
    out = _call(cuda_device, q, k, v, mask, bias, max_ctas=max_ctas)
    _check(out, O.oracle_fp32(q, k, v, mask, bias), plan)
    on_dev = [t.to(cuda_device) for t in (q, k, v, mask, bias)]
    out = out.to(cuda_device)
    for _ in range(50):
        assert torch.equal(dot_product_attention(*on_dev, max_ctas=max_ctas, check_status=True), out)


@pytest.mark.parametrize("B1,B2,S,rows_per_item,max_ctas,streams", [(1, 3, 128, 0, 1, 1), (3, 2, 200, 2, 0, 2), (2, 1, 300, 2, 1, 2), (1, 1, 256, 0, 1, 2), (1, 2, 300, 0, 1, 2),
                                                                    (4, 1, 130, 3, 1, 3), (8, 1, 100, 4, 1, 4)])
def test_debug_dump_has_the_first_result(cuda_device, B1, B2, S, rows_per_item, max_ctas, streams):
    """Pair rows or query tiles, one item on a CTA and several: accumulator and sum of block 0's first stream are in the dump, and their
    quotient is the result but for its rounding to bf16."""
    D = 32
    other = {"rows_per_item": rows_per_item, "max_ctas": max_ctas}
    plan = _plan(B1, B2, S, D, **other)
    assert plan["streams"] == streams, plan
    lib = _capi.load()
    q, k, v, mask, bias = _inputs(B1, B2, S, D, S)
    dump = torch.full((4 * 128 * 128 + 2 * (2 * 256 * 8 + 4 * 256),), float("nan"), device=cuda_device)
    lib.af3k_debug_set_dump(dump.data_ptr())
    try:
        out = _call(cuda_device, q, k, v, mask, bias, **other)
    finally:
        lib.af3k_debug_set_dump(None)
    _check(out, O.oracle_fp32(q, k, v, mask, bias), plan)
    n = min(S, 128)
    _, _, acc, sums = dump[:4 * 128 * 128].view(4, 128, 128)[:, :n].cpu()
    want = acc[:, :D] / sums[:, 1:2]
    assert ((out[0, 0, :n].float() - want).abs() <= 2 ** -8 * want.abs()).all()


@pytest.mark.parametrize("Sk", [1, 16, 31, 32, 33, 64, 65, 80, 81, 96, 97, 112, 113, 128, 129, 160, 161, 192, 193, 224, 225, 256, 257, 288, 289, 336, 337, 385, 448,
                                449, 560, 561])
@pytest.mark.parametrize("qk,D", [("bf16", 24), ("bf16", 48), ("bf16", 64), ("fp8", 32)])
def test_key_tiles_of_every_width(cuda_device, Sk, qk, D):
    """The last key tile is as wide as the keys of a call need: first and last length of each width, with one to five tiles.  Several
    pair rows per item with a remainder, two query tiles, and (fp32 bias, a single pair row) the bias converted on the way in."""
    for B1, Sq in ((5, 140), (1, 70)):
        q, k, v, mask, bias = _inputs(B1, 3, Sq, D, Sk + D, Sk)
        mask[:, -1] = True
        bias[..., -1] += 3            # the last key counts
        scales = {}
        if qk == "fp8":
            q, k, scales = _quantised(q, k)
        bias = bias.float() if B1 == 1 else bias.to(torch.bfloat16)
        out = A.dot_product_attention_cpp(*(t.to(cuda_device) for t in (q, k, v, mask, bias)), **{n: t.to(cuda_device) for n, t in scales.items()}).cpu()
        ref = O.oracle_fp32(q, k, v, mask, bias, **scales)
        if qk == "fp8":
            assert O.error_stats(out, ref)["max_abs"] <= 6e-2, (B1, Sk)
        else:
            _check(out, ref, (B1, Sk, D))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B1,B2,Sq,Sk,D,pitch,offset,launches", [
    (1, 16, 129, 129, 32, 129, 0, (1, 1)), (1, 16, 140, 161, 24, 161, 1, (1, 1)), (1, 16, 250, 225, 48, 231, 2, (1, 1)), (2, 16, 200, 257, 32, 257, 3, (1, 1)),
    (1, 6, 400, 389, 64, 389, 5, (2, 2)), (1, 16, 400, 389, 64, 389, 5, (1, 1)), (1, 5, 385, 385, 32, 385, 0, (2, 2)), (1, 16, 385, 385, 32, 385, 0, (1, 1)),
    (1, 16, 1300, 1300, 24, 1300, 0, (1, 1)), (1, 16, 1290, 1301, 16, 1301, 1, (1, 2)), (1, 16, 2000, 2001, 16, 2001, 1, (1, 1)), (1, 20, 1100, 1030, 40, 1032, 4, (1, 2))])
def test_ragged_rows_of_several_key_tiles_converted_by_the_attention_kernel(cuda_device, dtype, B1, B2, Sq, Sk, D, pitch, offset, launches):
    """Rows that start anywhere, key tiles of 80 to 128 keys, more query tiles than SMs among them: the bits of the pass, whatever stands
    in front of, between and behind the rows.  launches: with an fp32 and with a bf16 bias (two: the pass, by its estimate, so that
    nothing is compared there but two ways into it)."""
    g = torch.Generator().manual_seed(Sk)
    q, k, v = (torch.randn(B1, B2, s, D, generator=g).to(cuda_device, torch.bfloat16) for s in (Sq, Sk, Sk))
    mask = (torch.rand(B1, Sk, generator=g) >= 0.1).to(cuda_device)
    mask[:, -1] = True
    flat = torch.full((B2 * Sq * pitch + 16,), float("nan"), device=cuda_device, dtype=dtype)
    bias = flat[offset:offset + B2 * Sq * pitch].view(B2, Sq, pitch)[:, :, :Sk]
    bias.copy_(torch.randn(B2, Sq, Sk, generator=g))
    bias[torch.rand(bias.shape, generator=g).to(cuda_device) < 0.02] = -float("inf")
    bias[..., -1] = 1
    lib = _capi.load()
    out = A.dot_product_attention_cpp(q, k, v, mask, bias)
    assert lib.af3k_last_launch_count() == launches[dtype is torch.bfloat16]
    staged = dot_product_attention(q, k, v, mask, bias, cache_bias=False, check_status=True)
    assert lib.af3k_last_launch_count() == 2 and not out.isnan().any()
    assert torch.equal(out, staged)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 2047, 2048, 300001])
def test_conversions_in_one_launch(cuda_device, n):
    """Three arrays of different lengths to bf16, one back: torch's roundings, infinities and NaN, nothing written behind the ends."""
    import ctypes
    lib = _capi.load()
    g = torch.Generator().manual_seed(n)
    lengths = [n, max(n // 3, 1), 5]
    src = [(torch.randn(m, generator=g) * 10.0 ** torch.randint(-45, 39, (m,), generator=g)).to(cuda_device) for m in lengths]
    src[0][0] = float("nan")
    src[2][:2] = torch.tensor([float("inf"), -3.4e38])
    dst = [torch.full((m + 8,), 7.0, device=cuda_device, dtype=torch.bfloat16) for m in lengths]
    stream = torch.cuda.current_stream().cuda_stream
    pointers = lambda ts: (ctypes.c_void_p * len(ts))(*(t.data_ptr() for t in ts))
    assert lib.af3k_cast(pointers(src), pointers(dst), (ctypes.c_int64 * 3)(*lengths), 3, _capi.AF3K_BF16, stream) == 0
    assert lib.af3k_last_launch_count() == 1
    for a, b, m in zip(src, dst, lengths):
        assert torch.equal(b[:m].nan_to_num(5.0), a.to(torch.bfloat16).nan_to_num(5.0)) and torch.equal(b[:m].isnan(), a.isnan()) and (b[m:] == 7).all()
    back = torch.full((n + 8,), 7.0, device=cuda_device)
    assert lib.af3k_cast(pointers(dst[:1]), pointers([back]), (ctypes.c_int64 * 1)(n), 1, _capi.AF3K_F32, stream) == 0
    assert torch.equal(back[:n].nan_to_num(5.0), dst[0][:n].float().nan_to_num(5.0)) and (back[n:] == 7).all()
    assert lib.af3k_cast(pointers([src[0][1:]]) if n > 1 else pointers(src[:1]), pointers(dst[:1]), (ctypes.c_int64 * 1)(n - 1), 1, _capi.AF3K_BF16, stream) == (4 if n > 1 else 0)


@pytest.mark.parametrize("form", ["contiguous", "permuted", "offset", "mixed"])
def test_fp32_operands_give_the_bits_of_their_bf16_forms(cuda_device, form):
    g = torch.Generator().manual_seed(4)
    B1, B2, S, D = 2, 4, 150, 24
    make = lambda: torch.randn(B1, S, B2, D, generator=g).to(cuda_device).permute(0, 2, 1, 3) if form == "permuted" else torch.randn(B1, B2, S, D, generator=g).to(cuda_device)
    q, k, v = make(), make(), make()
    if form == "offset":
        q = torch.cat([q.flatten(), q.flatten()[:1]])[1:].view(B1, B2, S, D)
    if form == "mixed":
        k, v = k.to(torch.bfloat16), v.double()
    bias = torch.randn(B2, S, S, generator=g).to(cuda_device)
    out = A.dot_product_attention_cpp(q, k, v, None, bias)
    assert out.dtype == torch.float32
    assert torch.equal(out, A.dot_product_attention_cpp(*(t.to(torch.bfloat16) for t in (q, k, v)), None, bias).float())


@pytest.mark.parametrize("Sk,pitch,offset", [(255, 255, 1), (256, 257, 0), (257, 257, 0), (263, 263, 2), (264, 268, 1), (513, 515, 0), (640, 641, 3)])
def test_conversion_of_fp32_rows_that_start_anywhere(cuda_device, Sk, pitch, offset):
    """A warp converts 256 columns of a row: lengths around whole pieces, rows of every remainder."""
    test_conversion_of_the_bias(cuda_device, Sk, pitch, offset, torch.float32)


@pytest.mark.parametrize("form", ["bias_in_place", "converted", "converted_anywhere", "two_launches", "rows", "fp8", "single_block", "module"])
def test_waits_are_counted_from_the_end_of_the_kernel_before(cuda_device, form):
    """A call under a block limit lets the next kernel's blocks in on the SMs that it leaves free, and goes on for several times what a
    single wait may take: the blocks that came in early must not have begun to count."""
    g = torch.Generator().manual_seed(7)
    lib = _capi.load()
    S = 100 if form == "converted_anywhere" else 200
    q, k, v, mask, bias = _inputs(64 if form == "rows" else 1, 4, S, 32, 7)
    scales = {}
    if form == "fp8":
        q, k, scales = _quantised(q, k)
        scales = {n: t.to(cuda_device) for n, t in scales.items()}
    q, k, v, mask, bias = (t.to(cuda_device) for t in (q, k, v, mask, bias))
    if form in ("converted", "two_launches"):
        bias = bias.float()
    if form == "converted_anywhere":
        bias = torch.cat([bias, bias[..., :1]], -1)[..., 1:]
    if form == "single_block":
        x, qb = torch.randn(S, 128, generator=g).to(cuda_device, torch.bfloat16), torch.randn(128, generator=g).to(cuda_device)
        w = [(torch.randn(128, 128, generator=g) * 0.1).to(cuda_device, torch.bfloat16) for _ in range(4)]
        call = lambda: A.self_attention_cpp(x, mask[0], bias, w[0], qb, *w[1:], 4)
    elif form == "module":
        m = A.GridSelfAttentionCpp(64, 4).to(cuda_device, torch.bfloat16)
        pair = torch.randn(40, 40, 64, generator=g).to(cuda_device, torch.bfloat16)
        call = lambda: m(pair, mask[0, :40])
    elif form in ("fp8", "two_launches"):
        if form == "fp8":
            bias = stage_bias(bias, 4, S, S, head_dim=32, **scales)
        call = lambda: dot_product_attention(q, k, v, mask, bias, cache_bias=False, **scales)
    else:
        call = lambda: A.dot_product_attention_cpp(q, k, v, mask, bias)
    with torch.no_grad():
        want = call()
        big = [t.to(cuda_device) for t in _inputs(192, 4, 512, 32, 8)]
        begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        assert read_status(cuda_device)[0] == 0
        lib.af3k_set_wait_limit_cycles(2_000_000)          # about a millisecond
        try:
            begin.record()
            before = dot_product_attention(*big, max_ctas=1)
            out = call()
            end.record()
            torch.cuda.synchronize()
        finally:
            lib.af3k_set_wait_limit_cycles(0)
    assert begin.elapsed_time(end) > 4
    assert read_status(cuda_device)[0] == 0
    assert torch.equal(out, want) and torch.equal(before, dot_product_attention(*big))


def test_fp32_operands_under_a_block_limit(cuda_device):
    """The library's conversions overlap the kernel before, and would wait on the SMs that the limit leaves free: such a call launches
    the pass over the bias and the attention kernel, and nothing of the library's behind them."""
    q, k, v, mask, bias = (t.to(cuda_device) for t in _inputs(2, 4, 150, 32, 11))
    bias = bias.float()
    lib = _capi.load()
    want = dot_product_attention(q, k, v, mask, bias, cache_bias=False, max_ctas=9)
    out = dot_product_attention(q.float(), k.float(), v.float(), mask, bias, cache_bias=False, max_ctas=9, check_status=True)
    assert lib.af3k_last_launch_count() == 2
    assert out.dtype == torch.float32 and torch.equal(out, want.float())
    assert torch.equal(out, A.dot_product_attention_cpp(q.float(), k.float(), v.float(), mask, bias))


def test_fp32_operands_that_are_lazily_negated(cuda_device):
    """A tensor whose negative bit is set holds the values before the change of sign."""
    g = torch.Generator().manual_seed(12)
    q, k, v = (torch.randn(2, 4, 50, 24, generator=g).to(cuda_device) for _ in range(3))
    bias = torch.randn(4, 50, 50, generator=g).to(cuda_device)
    want = A.dot_product_attention_cpp(-q, k, -v, None, bias)
    assert torch.equal(A.dot_product_attention_cpp(torch._neg_view(q), k, torch._neg_view(v), None, bias), want)
    x, w = q[0].reshape(50, 96).contiguous(), [torch.randn(96, 96, generator=g).to(cuda_device) * 0.1 for _ in range(4)]
    for ws in (w, [t.to(torch.bfloat16) for t in w]):       # packed in a launch that rounds the tokens too, and read in place
        call = lambda t: A.self_attention_cpp(t, None, bias, ws[0], torch.zeros(96, device=cuda_device), *ws[1:], 4)
        assert torch.equal(call(torch._neg_view(x)), call(-x))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B1,B2,S,pitch,offset,launches,captured", [
    (45, 4, 45, 45, 0, 1, 2), (62, 4, 62, 62, 1, 1, 2), (64, 4, 64, 68, 4, 1, 2), (38, 8, 33, 33, 0, 2, 2), (75, 4, 75, 75, 0, 2, 2), (100, 4, 62, 62, 1, 2, 2), (140, 4, 24, 28, 4, 2, 2),
    (140, 4, 31, 31, 0, 2, 2), (20, 16, 40, 44, 4, 2, 2), (1, 4, 129, 129, 0, 1, 1), (1, 4, 255, 255, 0, 1, 1), (1, 4, 1001, 1001, 0, 2, 2), (1, 3, 131, 131, 0, 2, 2)])
def test_short_calls_convert_their_bias_where_the_device_loses_little(cuda_device, dtype, B1, B2, S, pitch, offset, launches, captured):
    """Several pair rows per item, in place of which lone rows convert: only while that costs the device little, and not in a graph.
    Lone items of four heads.  The same bits on every way."""
    q, k, v, mask, _ = _inputs(B1, B2, S, 32, S)
    mask[:, -1] = True
    flat = torch.full((B2 * S * pitch + 16,), float("nan"), device=cuda_device, dtype=dtype)
    bias = flat[offset:offset + B2 * S * pitch].view(B2, S, pitch)[:, :, :S]
    bias.copy_(torch.randn(B2, S, S, generator=torch.Generator().manual_seed(S)))
    q, k, v, mask = (t.to(cuda_device) for t in (q, k, v, mask))
    lib = _capi.load()
    out = A.dot_product_attention_cpp(q, k, v, mask, bias)
    assert lib.af3k_last_launch_count() == launches
    assert torch.equal(out, dot_product_attention(q, k, v, mask, bias, cache_bias=False, check_status=True))
    assert lib.af3k_last_launch_count() == 2
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        replayed = A.dot_product_attention_cpp(q, k, v, mask, bias)
        count = lib.af3k_last_launch_count()
    graph.replay()
    assert count == captured and torch.equal(replayed, out)


@pytest.mark.parametrize("qk,D", [("bf16", 24), ("bf16", 48), ("fp8", 32)])
@pytest.mark.parametrize("Sk", [1, 31, 77, 97, 128, 129, 160, 161, 192, 193, 224, 225, 256, 257, 300, 389, 512, 513])
def test_results_do_not_depend_on_the_tiles_width(cuda_device, Sk, qk, D):
    """Narrow tiles leave out keys that do not exist and nothing else: the same bits as all tiles of 128 keys give (the kernels that
    write the debug dump have those only).  Several pair rows with a remainder, pairs of query tiles, a query tile of its own."""
    lib = _capi.load()
    dump = torch.empty(4 * 128 * 128 + 2 * (2 * 256 * 8 + 4 * 256), device=cuda_device)
    for B1, Sq, kw in ((7, 140, {}), (1, 400, {"max_ctas": 2}), (1, 70, {}), (5, 90, {"rows_per_item": 4})):
        q, k, v, mask, bias = _inputs(B1, 2, Sq, D, Sk + D, Sk)
        mask[:, -1] = True
        scales = {}
        if qk == "fp8":
            q, k, scales = _quantised(q, k)
        scales = {n: t.to(cuda_device) for n, t in scales.items()}
        out = _call(cuda_device, q, k, v, mask, bias, **kw, **scales)
        lib.af3k_debug_set_dump(dump.data_ptr())
        try:
            wide = _call(cuda_device, q, k, v, mask, bias, **kw, **scales)
        finally:
            lib.af3k_debug_set_dump(None)
        assert torch.equal(out, wide), (B1, Sq)
