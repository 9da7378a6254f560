"""Parity of the CUDA path (called through the C ABI of libaf3k.so) against the CPU oracles.

Tolerances are those of the path's specification, measured against the fp32 oracle on the same
stored inputs: bf16 max-abs <= 2e-2 and mean-abs <= 2e-3; fp8 (e4m3 q/k, de-quantised oracle)
max-abs <= 6e-2.
"""
import ctypes
import math

import pytest
import torch

import af3_kernels_b200 as A
from af3_kernels_b200 import _capi
from af3_kernels_b200.dpa import dot_product_attention, read_status
from oracle import attention_oracle as O

pytestmark = pytest.mark.gpu

BF16_MAX_ABS, BF16_MEAN_ABS = 2e-2, 2e-3
FP8_MAX_ABS = 6e-2


def _to(dev, *ts):
    return [t.to(dev) if t is not None else None for t in ts]


def _run(dev, q, k, v, mask, bias, **kw):
    qd, kd, vd, md, bd = _to(dev, q, k, v, mask, bias)
    for name in ("q_scale", "k_scale"):
        if kw.get(name) is not None:
            kw[name] = kw[name].to(dev)
    out = dot_product_attention(qd, kd, vd, md, bd, check_status=True, **kw)
    return out.cpu()


def _check_bf16(out, ref, what):
    st = O.error_stats(out, ref)
    assert st["nan"] == 0, (what, st)
    assert st["max_abs"] <= BF16_MAX_ABS and st["mean_abs"] <= BF16_MEAN_ABS, (what, st)
    return st


def test_loaded_library_is_the_cuda_one(cuda_device):
    lib = _capi.load()
    assert lib.af3k_version() >= 1000
    assert torch.cuda.get_device_capability(cuda_device)[0] == 10


def test_golden_vectors(cuda_device, golden):
    for name, c in golden.items():
        out = _run(cuda_device, c["q"], c["k"], c["v"], c["mask"], c["bias"])
        _check_bf16(out, c["ref_fp32"], name)
        if not name.startswith("fully_masked"):
            # against the restatement of the reference's own bf16 rounding scheme: both sit
            # within their own distance of the fp32 result
            o2 = O.ref_semantics(c["q"], c["k"], c["v"], c["mask"], c["bias"])
            st = O.error_stats(out, o2)
            assert st["max_abs"] <= 6e-2 + BF16_MAX_ABS and st["mean_abs"] <= 3e-3 + BF16_MEAN_ABS, (name, st)


@pytest.mark.parametrize("name", ["cfg1", "cfg3", "cfg4"])
def test_benchmark_configs_full_size(cuda_device, name):
    inp = O.make_inputs(name)
    out = _run(cuda_device, inp["q"], inp["k"], inp["v"], inp["mask"], inp["bias"])
    ref = O.oracle_fp32(inp["q"], inp["k"], inp["v"], inp["mask"], inp["bias"])
    _check_bf16(out, ref, name)


def test_cfg2_reduced_rows_against_oracle(cuda_device):
    inp = O.make_inputs("cfg2", rows=24)
    out = _run(cuda_device, inp["q"], inp["k"], inp["v"], inp["mask"], inp["bias"])
    ref = O.oracle_fp32(inp["q"], inp["k"], inp["v"], inp["mask"], inp["bias"])
    _check_bf16(out, ref, "cfg2 rows=24")


def test_cfg2_full_size_properties(cuda_device):
    dev = cuda_device
    g = torch.Generator(device=dev).manual_seed(0)
    B1, B2, S, D = 768, 4, 768, 32
    q = torch.randn(B1, B2, S, D, generator=g, device=dev).to(torch.bfloat16)
    k = torch.randn(B1, B2, S, D, generator=g, device=dev).to(torch.bfloat16)
    v = torch.randn(B1, B2, S, D, generator=g, device=dev).to(torch.bfloat16)
    bias = torch.randn(B2, S, S, generator=g, device=dev)
    mask = torch.rand(B1, S, generator=g, device=dev) >= 0.05
    q0 = q.clone()
    out = dot_product_attention(q, k, v, mask, bias, check_status=True)
    assert torch.equal(q, q0), "inputs must not be written"
    # (1) bit-reproducible
    again = dot_product_attention(q, k, v, mask, bias, check_status=True)
    assert torch.equal(out, again)
    # (2) rows are independent problems: a slice of the rows gives the same bits
    rows = torch.tensor([0, 5, 383, 767], device=dev)
    sub = dot_product_attention(q[rows], k[rows], v[rows], mask[rows], bias, check_status=True)
    assert torch.equal(sub, out[rows])
    # (3) the slice against the CPU oracle
    ref = O.oracle_fp32(q[rows].cpu(), k[rows].cpu(), v[rows].cpu(), mask[rows].cpu(), bias.cpu())
    _check_bf16(sub.cpu(), ref, "cfg2 full, row subset")
    # (4) softmax weights sum to one: V = 1 gives 1 everywhere
    ones = dot_product_attention(q, k, torch.ones_like(v), mask, bias, check_status=True)
    assert (ones.float() - 1.0).abs().max().item() <= 1e-2


def test_cfg5_fp8_reduced_rows(cuda_device):
    inp = O.make_inputs("cfg5", rows=6)
    out = _run(cuda_device, inp["q"], inp["k"], inp["v"], inp["mask"], inp["bias"],
               q_scale=inp["q_scale"], k_scale=inp["k_scale"])
    ref = O.oracle_fp32(inp["q"], inp["k"], inp["v"], inp["mask"], inp["bias"],
                        q_scale=inp["q_scale"], k_scale=inp["k_scale"])
    st = O.error_stats(out, ref)
    assert st["nan"] == 0 and st["max_abs"] <= FP8_MAX_ABS, st


def test_fp8_both_kernel_variants(cuda_device):
    """fp8 q/k run on two kernels: with a workspace the bias (divided by the head's logit scale in
    the staging pass) is added by the tensor core, without one the softmax threads add it in
    fp32.  Both against the de-quantised fp32 oracle, with small and with tiny quantisation
    scales (the value a masked key gets is scaled with them), and a fully masked row."""
    g = torch.Generator().manual_seed(77)
    B1, B2, S, D = 3, 2, 296, 32          # bias rows of 592 bytes: usable in place, no staging needed
    for amp in (1.0, 1e-3):
        qf = torch.randn(B1, B2, S, D, generator=g) * amp
        kf = torch.randn(B1, B2, S, D, generator=g) * amp
        v = torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16)
        bias = torch.randn(B2, S, S, generator=g).to(torch.bfloat16)
        mask = torch.rand(B1, S, generator=g) >= 0.1
        mask[1, :] = False
        q, qs = O.quantize_e4m3_per_head(qf)
        k, ks = O.quantize_e4m3_per_head(kf)
        ref = O.oracle_fp32(q, k, v, mask, bias, q_scale=qs, k_scale=ks)
        for use_ws in (True, False):
            out = _run(cuda_device, q, k, v, mask, bias, q_scale=qs, k_scale=ks, use_workspace=use_ws,
                       cache_bias=False)
            st = O.error_stats(out, ref)
            assert st["nan"] == 0 and st["max_abs"] <= FP8_MAX_ABS, (amp, use_ws, st)
            uniform = v[1].float().mean(dim=1, keepdim=True).expand(B2, S, D)
            assert (out[1].float() - uniform).abs().max().item() <= 1e-2, (amp, use_ws)
            lib = _capi.load()
            assert lib.af3k_last_launch_count() == (2 if use_ws else 1)


def test_cfg5_fp8_quarter_size_properties(cuda_device):
    dev = cuda_device
    g = torch.Generator(device=dev).manual_seed(0)
    B1, B2, S, D = 512, 4, 2048, 32
    qf = torch.randn(B1, B2, S, D, generator=g, device=dev)
    kf = torch.randn(B1, B2, S, D, generator=g, device=dev)
    v = torch.randn(B1, B2, S, D, generator=g, device=dev).to(torch.bfloat16)
    bias = torch.randn(B2, S, S, generator=g, device=dev).to(torch.bfloat16)
    mask = torch.rand(B1, S, generator=g, device=dev) >= 0.05
    q, qs = O.quantize_e4m3_per_head(qf)
    k, ks = O.quantize_e4m3_per_head(kf)
    del qf, kf
    out = dot_product_attention(q, k, v, mask, bias, q_scale=qs, k_scale=ks, check_status=True)
    again = dot_product_attention(q, k, v, mask, bias, q_scale=qs, k_scale=ks, check_status=True)
    assert torch.equal(out, again)
    rows = torch.tensor([0, 255, 511], device=dev)
    ref = O.oracle_fp32(q[rows].cpu(), k[rows].cpu(), v[rows].cpu(), mask[rows].cpu(), bias.cpu(),
                        q_scale=qs.cpu(), k_scale=ks.cpu())
    st = O.error_stats(out[rows].cpu(), ref)
    assert st["nan"] == 0 and st["max_abs"] <= FP8_MAX_ABS, st


@pytest.mark.parametrize("S", [1, 17, 127, 128, 129, 257])
@pytest.mark.parametrize("D", [24, 32, 48])
def test_odd_sequence_lengths(cuda_device, S, D):
    g = torch.Generator().manual_seed(S * 100 + D)
    B1, B2 = 3, 2
    q = torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16)
    k = torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16)
    v = torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16)
    bias = torch.randn(B2, S, S, generator=g)
    mask = torch.rand(B1, S, generator=g) >= 0.2
    mask[:, 0] = True
    out = _run(cuda_device, q, k, v, mask, bias)
    _check_bf16(out, O.oracle_fp32(q, k, v, mask, bias), (S, D))


@pytest.mark.parametrize("D", [8, 16, 40, 56, 64])
def test_other_head_dims(cuda_device, D):
    g = torch.Generator().manual_seed(D)
    q = torch.randn(2, 3, 200, D, generator=g).to(torch.bfloat16)
    k = torch.randn(2, 3, 200, D, generator=g).to(torch.bfloat16)
    v = torch.randn(2, 3, 200, D, generator=g).to(torch.bfloat16)
    bias = torch.randn(3, 200, 200, generator=g).to(torch.bfloat16)
    out = _run(cuda_device, q, k, v, None, bias)
    _check_bf16(out, O.oracle_fp32(q, k, v, None, bias), D)


def test_mask_and_bias_forms(cuda_device):
    g = torch.Generator().manual_seed(3)
    B1, B2, S, D = 4, 2, 150, 32
    q = torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16)
    k = torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16)
    v = torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16)
    bias = torch.randn(B2, S, S, generator=g)
    m1 = torch.rand(S, generator=g) >= 0.3
    m2 = m1[None, :].expand(B1, S).contiguous()
    ref = O.oracle_fp32(q, k, v, m2, bias)
    o1 = _run(cuda_device, q, k, v, m1, bias)                       # 1-D broadcasts over the batch
    o2 = _run(cuda_device, q, k, v, m2, bias)                       # 2-D
    o4 = _run(cuda_device, q, k, v, m2[:, None, None, :], bias)     # what the reference builds
    ob = _run(cuda_device, q, k, v, m2, bias[None])                 # 4-D bias [1, H, S, S]
    _check_bf16(o1, ref, "1-D mask")
    assert torch.equal(o1, o2) and torch.equal(o2, o4) and torch.equal(o2, ob)
    onone = _run(cuda_device, q, k, v, None, bias)
    _check_bf16(onone, O.oracle_fp32(q, k, v, None, bias), "no mask")


def test_fully_masked_row_is_uniform_over_real_keys(cuda_device):
    g = torch.Generator().manual_seed(4)
    B1, B2, S, D = 2, 2, 200, 32
    q = torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16)
    k = torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16)
    v = torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16)
    bias = torch.randn(B2, S, S, generator=g)
    mask = torch.rand(B1, S, generator=g) >= 0.1
    mask[0, :] = False
    out = _run(cuda_device, q, k, v, mask, bias)
    _check_bf16(out, O.oracle_fp32(q, k, v, mask, bias), "fully masked row")
    uniform = v[0].float().mean(dim=1, keepdim=True).expand(B2, S, D)
    assert (out[0].float() - uniform).abs().max().item() <= 1e-2


def test_rows_per_item_choices_give_identical_bits(cuda_device):
    g = torch.Generator().manual_seed(5)
    B1, B2, S, D = 11, 2, 300, 32
    q = torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16)
    k = torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16)
    v = torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16)
    bias = torch.randn(B2, S, S, generator=g).to(torch.bfloat16)
    mask = torch.rand(B1, S, generator=g) >= 0.05
    base = _run(cuda_device, q, k, v, mask, bias, rows_per_item=1)
    _check_bf16(base, O.oracle_fp32(q, k, v, mask, bias), "G=1")
    for G in range(2, 9):
        assert torch.equal(_run(cuda_device, q, k, v, mask, bias, rows_per_item=G), base), G


def test_capped_grid_gives_identical_bits(cuda_device):
    """max_ctas (SMs left to a collective running beside the kernel) changes which CTA takes which
    work item, nothing else."""
    g = torch.Generator().manual_seed(15)
    B1, B2, S, D = 40, 4, 300, 32
    q = torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16)
    k = torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16)
    v = torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16)
    bias = torch.randn(B2, S, S, generator=g).to(torch.bfloat16)
    mask = torch.rand(B1, S, generator=g) >= 0.05
    base = _run(cuda_device, q, k, v, mask, bias)
    for cap in (1, 7, 100, 140, 1000):
        assert torch.equal(_run(cuda_device, q, k, v, mask, bias, max_ctas=cap), base), cap


def test_strided_inputs_and_output(cuda_device):
    dev = cuda_device
    g = torch.Generator().manual_seed(6)
    B1, B2, S, D = 2, 4, 130, 32
    # [B, S, H, D] projections viewed as [B, H, S, D]: the usual layout after a fused QKV linear
    qkv = torch.randn(3, B1, S, B2, D, generator=g).to(torch.bfloat16).to(dev)
    q, k, v = (t.permute(0, 2, 1, 3) for t in qkv)
    assert not q.is_contiguous()
    bias = torch.randn(B2, S, S, generator=g).to(dev)
    mask = (torch.rand(B1, S, generator=g) >= 0.1).to(dev)
    out = dot_product_attention(q, k, v, mask, bias, check_status=True)
    ref = O.oracle_fp32(q.cpu(), k.cpu(), v.cpu(), mask.cpu(), bias.cpu())
    _check_bf16(out.cpu(), ref, "strided")
    dst = torch.zeros(B1, S, B2, D, dtype=torch.bfloat16, device=dev).permute(0, 2, 1, 3)
    dot_product_attention(q, k, v, mask, bias, out=dst, check_status=True)
    assert torch.equal(dst, out)


def test_output_padding_is_not_overwritten(cuda_device):
    dev = cuda_device
    g = torch.Generator().manual_seed(8)
    B1, B2, S, D = 2, 2, 77, 24
    q = torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16).to(dev)
    bias = torch.randn(B2, S, S, generator=g).to(dev)
    big = torch.full((B1, B2, S + 2, D + 8), 7.0, dtype=torch.bfloat16, device=dev)
    view = big[:, :, 1:S + 1, :D]
    dot_product_attention(q, q, q, None, bias, out=view, check_status=True)
    assert (big[:, :, 0] == 7).all() and (big[:, :, S + 1] == 7).all() and (big[..., D:] == 7).all()
    assert not (view == 7).all()


def test_reference_named_wrapper_and_dtype_checks(cuda_device):
    dev = cuda_device
    q = torch.randn(1, 2, 64, 32, device=dev).to(torch.bfloat16)
    bias = torch.zeros(2, 64, 64, device=dev)
    mask = torch.ones(64, dtype=torch.bool, device=dev)
    out = A.dot_product_attention_cpp(q, q, q, mask, bias, True, 64, 256)   # knobs accepted, ignored
    assert out.shape == q.shape and out.dtype == torch.bfloat16
    with pytest.raises(TypeError):
        A.dot_product_attention_cpp(q.half(), q.half(), q.half(), mask, bias)
    with pytest.raises(ValueError):
        A.dot_product_attention_cpp(q, q, q, mask, bias[:, :32])
    empty = A.dot_product_attention_cpp(q[:0], q[:0], q[:0], mask, bias)
    assert empty.shape == (0, 2, 64, 32)


def test_bounded_wait_reports_instead_of_hanging(cuda_device):
    lib = _capi.load()
    st = torch.zeros(4, dtype=torch.int32, device=cuda_device)
    assert lib.af3k_selftest_wait_timeout(5_000_000, st.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert st[0].item() == _capi.AF3K_STATUS_WAIT_TIMEOUT
    # the context is still usable afterwards
    q = torch.randn(1, 1, 32, 32, device=cuda_device).to(torch.bfloat16)
    out = dot_product_attention(q, q, q, None, torch.zeros(1, 32, 32, device=cuda_device), check_status=True)
    assert torch.isfinite(out.float()).all()


def test_launch_count(cuda_device):
    lib = _capi.load()
    q = torch.randn(1, 1, 64, 32, device=cuda_device).to(torch.bfloat16)
    dot_product_attention(q, q, q, None, torch.zeros(1, 64, 64, device=cuda_device), cache_bias=False)
    assert lib.af3k_last_launch_count() == 2          # fp32 bias: staging pre-pass + attention
    dot_product_attention(q, q, q, None, torch.zeros(1, 64, 64, device=cuda_device, dtype=torch.bfloat16))
    assert lib.af3k_last_launch_count() == 1
    assert read_status(cuda_device)[0] == 0


def test_staged_bias_is_reused_and_follows_in_place_updates(cuda_device):
    """A bias that needs the staging pass is staged once per tensor object and version: the second
    call with the same tensor launches one kernel, gives the same bits as a call that stages
    inside, and an in-place update of the bias is seen by the next call.  Same for fp8 q/k, whose
    copy also depends on the scales."""
    dev = cuda_device
    lib = _capi.load()
    g = torch.Generator().manual_seed(5)
    B1, B2, S, D = 3, 2, 200, 32
    q, k, v = (torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16).to(dev) for _ in range(3))
    bias = torch.randn(B2, S, S, generator=g).to(dev)
    mask = (torch.rand(B1, S, generator=g) >= 0.1).to(dev)
    inside = dot_product_attention(q, k, v, mask, bias, cache_bias=False, check_status=True)
    first = dot_product_attention(q, k, v, mask, bias, check_status=True)
    second = dot_product_attention(q, k, v, mask, bias, check_status=True)
    assert lib.af3k_last_launch_count() == 1
    assert torch.equal(first, inside) and torch.equal(second, inside)
    bias.mul_(-1.0)                                   # same object, new version
    flipped = dot_product_attention(q, k, v, mask, bias, check_status=True)
    assert torch.equal(flipped, dot_product_attention(q, k, v, mask, bias, cache_bias=False))
    assert not torch.equal(flipped, inside)
    # explicit handle
    from af3_kernels_b200.dpa import stage_bias
    handle = stage_bias(bias, B2, S, S)
    assert torch.equal(dot_product_attention(q, k, v, mask, handle, check_status=True), flipped)
    # fp8 q/k
    q8, qs = O.quantize_e4m3_per_head(q.float().cpu())
    k8, ks = O.quantize_e4m3_per_head(k.float().cpu())
    q8, k8, qs, ks = q8.to(dev), k8.to(dev), qs.to(dev), ks.to(dev)
    b16 = bias.to(torch.bfloat16)
    ref8 = dot_product_attention(q8, k8, v, mask, b16, q_scale=qs, k_scale=ks, cache_bias=False, check_status=True)
    for _ in range(2):
        got = dot_product_attention(q8, k8, v, mask, b16, q_scale=qs, k_scale=ks, check_status=True)
        assert torch.equal(got, ref8)
    assert lib.af3k_last_launch_count() == 1


def test_ordinary_calls_see_every_write_to_the_bias(cuda_device):
    """The reference's signatures keep no copy of a bias or of fp8 scales: a write that bumps no version counter
    (``.data``, as a collective or a kernel on the raw pointer) shows in the next call of the operator and of the blocks."""
    g = torch.Generator().manual_seed(9)
    dev = cuda_device
    B1, B2, S, D = 3, 4, 200, 32
    C = B2 * D
    q, k, v = (torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16).to(dev) for _ in range(3))
    mask = (torch.rand(B1, S, generator=g) >= 0.1).to(dev)
    w = [(torch.randn(C, C, generator=g) * C ** -0.5).to(torch.bfloat16).to(dev) for _ in range(5)]
    wide = [(torch.randn(96, 96, generator=g) * 0.1).to(torch.bfloat16).to(dev) for _ in range(5)]     # not a fused size
    x, pair, other = (torch.randn(*s, generator=g).to(torch.bfloat16).to(dev) for s in ((S, C), (B1, S, C), (B1, S, 96)))
    q8, qs = O.quantize_e4m3_per_head(q.float().cpu())
    k8, ks = O.quantize_e4m3_per_head(k.float().cpu())
    q8, k8, qs, ks = q8.to(dev), k8.to(dev), qs.to(dev), ks.to(dev)
    calls = {
        "operator": lambda b: A.dot_product_attention_cpp(q, k, v, mask, b),
        "operator, byte mask": lambda b: A.dot_product_attention_cpp(q, k, v, mask.to(torch.uint8), b),
        "operator, fp8": lambda b: A.dot_product_attention_cpp(q8, k8, v, mask, b, q_scale=qs, k_scale=ks),
        "grid block": lambda b: A._attention_cpp(pair, mask, b, *w, B2),
        "grid block, torch projections": lambda b: A._attention_cpp(other, mask, b, *wide, B2),
        "single block": lambda b: A.self_attention_cpp(x, mask[0], b, w[0], torch.zeros(C, device=dev), *w[1:4], B2),
        "single block, torch projections": lambda b: A.self_attention_cpp(x[:, :96], mask[0], b, wide[0], torch.zeros(96, device=dev), *wide[1:4], B2),
    }
    for name, call in calls.items():
        bias, new = (torch.randn(B2, S, S, generator=g).to(dev) for _ in range(2))
        first = call(bias)
        assert torch.equal(call(bias), first), name
        bias.data.copy_(new)
        assert torch.equal(call(bias), call(new.clone())), name
        assert not torch.equal(call(bias), first), name
    bias = torch.randn(B2, S, S, generator=g).to(dev)
    first = calls["operator, fp8"](bias)
    qs.data.mul_(0.5)
    assert torch.equal(calls["operator, fp8"](bias), calls["operator, fp8"](bias.clone()))
    assert not torch.equal(calls["operator, fp8"](bias), first)


def test_debug_dump_shows_the_tensor_core_stages(cuda_device):
    """The diagnostic build dumps the first logits tile: the logits as the tensor core delivers them
    (scaled Q K^T + bias + mask column), P as written to TMEM, the un-normalised accumulator and
    the row statistics.  Checking each against plain fp32
    math pins the operand layouts (swizzled K-major Q/K, MN-major V, P in TMEM, mask column)."""
    dev = cuda_device
    lib = _capi.load()
    g = torch.Generator().manual_seed(21)
    S, D = 128, 32
    q = torch.randn(1, 1, S, D, generator=g).to(torch.bfloat16).to(dev)
    k = torch.randn(1, 1, S, D, generator=g).to(torch.bfloat16).to(dev)
    v = torch.randn(1, 1, S, D, generator=g).to(torch.bfloat16).to(dev)
    bias = torch.randn(1, S, S, generator=g).to(torch.bfloat16).to(dev)
    mask = torch.rand(S, generator=g) >= 0.2
    mask[0] = True
    timeline_floats = 2 * (2 * 256 * 8 + 4 * 256)
    dump = torch.zeros(4 * 128 * 128 + timeline_floats, dtype=torch.float32, device=dev)
    lib.af3k_debug_set_dump(dump.data_ptr())
    try:
        out = dot_product_attention(q, k, v, mask.to(dev), bias, check_status=True)
    finally:
        lib.af3k_debug_set_dump(None)
    d = dump[: 4 * 128 * 128].view(4, 128, 128).cpu()
    # with bf16 q/k the tensor core delivers the finished logit: q is scaled and rounded to bf16 in
    # shared memory first (the reference's own first step), the bias is added by identity MMAs
    q_scaled = (q[0, 0].float().cpu() * D ** -0.5).to(torch.bfloat16).float()
    x_ref = q_scaled @ k[0, 0].float().cpu().T + bias[0].float().cpu()
    keep = mask[None, :].expand(S, S)
    assert (d[0][keep] - x_ref[keep]).abs().max().item() <= 1e-4          # attended keys
    assert (d[0][~keep] == -(2.0 ** 47)).all()                             # masked keys: exactly -2^47
    s_ref = q[0, 0].float().cpu() @ k[0, 0].float().cpu().T
    p_words = d[1][:, :64].contiguous().view(torch.int32)
    p_lo = (p_words << 16).view(torch.float32)
    p_hi = (p_words & -65536).view(torch.float32)
    p = torch.stack([p_lo, p_hi], dim=-1).reshape(S, S)                    # key 2c in the low half
    x = s_ref * D ** -0.5 + bias[0].float().cpu()
    x = x.masked_fill(~keep, float("-inf"))
    p_ref = torch.exp(x - x.max(dim=1, keepdim=True).values)
    assert (p - p_ref).abs().max().item() <= 8e-3                          # bf16 rounding of P
    o_ref = p @ v[0, 0].float().cpu()
    assert (d[2][:, :D] - o_ref).abs().max().item() <= 1e-3
    assert (d[3][:, 1] - p_ref.sum(dim=1)).abs().max().item() <= 2e-2 * p_ref.sum(dim=1).max().item()
    ref = O.oracle_fp32(q.cpu(), k.cpu(), v.cpu(), mask, bias.cpu())
    _check_bf16(out.cpu(), ref, "debug build")



@pytest.mark.parametrize("B1,B2,S,D", [(1, 16, 129, 24), (1, 16, 257, 48), (1, 16, 1152, 32), (1, 3, 640, 64), (2, 16, 512, 48), (3, 16, 200, 32),
                                       (1, 16, 1153, 16)])
def test_query_tiles_on_ctas_of_their_own(cuda_device, B1, B2, S, D):
    """Up to one CTA per SM every (row, head, query tile) gets a CTA of its own; a cap on the CTAs makes two query tiles
    (or rows) share one.  Same bits, and the oracle's result."""
    g = torch.Generator().manual_seed(B1 * S + D)
    q, k, v = (torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16) for _ in range(3))
    bias = torch.randn(B2, S, S, generator=g).to(torch.bfloat16)
    mask = torch.rand(B1, S, generator=g) >= 0.1
    own = _run(cuda_device, q, k, v, mask, bias)
    tiles = B1 * B2 * ((S + 127) // 128)
    assert torch.equal(_run(cuda_device, q, k, v, mask, bias, max_ctas=max(1, tiles // 2)), own)
    _check_bf16(own, O.oracle_fp32(q, k, v, mask, bias), (B1, B2, S, D))


@pytest.mark.parametrize("fp8,S", [(False, 200), (False, 77), (True, 128)])
def test_a_graph_converts_the_bias_it_is_given(cuda_device, fp8, S):
    """A bias that is staged first (fp32, ragged rows, fp8 scales), captured on the stream that was warmed up: a replay
    sees the values the bias holds then, whatever other biases were staged since."""
    g = torch.Generator().manual_seed(S)
    B1, B2, D = 3, 4, 32
    q, k, v = (torch.randn(B1, B2, S, D, generator=g).to(cuda_device, torch.bfloat16) for _ in range(3))
    scales = {}
    if fp8:
        q, k = q.to(torch.float8_e4m3fn), k.to(torch.float8_e4m3fn)
        scales = {n: torch.rand(B2, generator=g).to(cuda_device) + 0.5 for n in ("q_scale", "k_scale")}
    biases = [torch.randn(B2, S, S, generator=g).to(cuda_device) for _ in range(8)]
    bias = biases[0].clone()
    call = lambda b: A.dot_product_attention_cpp(q, k, v, None, b, **scales)
    want = [call(b) for b in biases]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        call(bias)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            out = call(bias)
    torch.cuda.current_stream().wait_stream(side)
    again = [call(b) for b in biases]
    assert all(torch.equal(a, b) for a, b in zip(again, want))
    for i in (0, 3, 5):
        bias.copy_(biases[i])
        graph.replay()
        assert torch.equal(out, want[i]), i
    torch.cuda.synchronize()


def test_out_counts_as_written(cuda_device):
    """A result written into a caller's tensor bumps its version, as any in-place operator does: a staged copy made of
    that tensor as a bias is not used again."""
    q = torch.ones(1, 2, 40, 32, dtype=torch.bfloat16, device=cuda_device)
    out = torch.empty_like(q)
    before = out._version
    A.dot_product_attention(q, q, q, None, torch.zeros(2, 40, 40, device=cuda_device), out=out)
    assert out._version > before


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_bias_of_another_shape_is_reshaped(cuda_device, dtype):
    """As many elements in another three (or four) dimensions: read as the [B2, Sq, Sk] tensor it reshapes to, on every
    route a bias takes (in place, staged, staged by the caller, single block, host tensors)."""
    from af3_kernels_b200.dpa import stage_bias
    g = torch.Generator().manual_seed(2)
    B2, S, D = 4, 64, 16
    q, k, v = (torch.randn(2, B2, S, D, generator=g).to(cuda_device, torch.bfloat16) for _ in range(3))
    bias = torch.randn(B2, S, S, generator=g).to(cuda_device, dtype)
    want = A.dot_product_attention(q, k, v, None, bias)
    w = [torch.randn(S, S, generator=g).to(cuda_device, torch.bfloat16) * 0.1 for _ in range(4)]
    x, qb = q[0, 0].repeat(1, B2), torch.zeros(S, device=cuda_device)
    block = lambda b: A.self_attention_cpp(x, None, b, w[0], qb, *w[1:], B2)
    want_block = block(bias)
    for shape in ((1, B2 * S, S), (B2 * S, 1, S), (S, B2, S), (1, B2, S, S), (B2 * S * S,)):
        b = bias.reshape(shape)
        assert torch.equal(A.dot_product_attention(q, k, v, None, b), want), shape
        assert torch.equal(A.dot_product_attention(q, k, v, None, b, cache_bias=False), want), shape
        assert torch.equal(A.dot_product_attention(q, k, v, None, stage_bias(b, B2, S, S)), want), shape
        assert torch.equal(block(b), want_block), shape
        assert torch.equal(A.dot_product_attention_host(q.cpu(), k.cpu(), v.cpu(), None, b.cpu()), want.cpu()), shape


@pytest.mark.parametrize("fp8,workspace", [(False, False), (True, True), (True, False)])
@pytest.mark.parametrize("B1,B2,S,D", [(1, 3, 77, 24), (2, 4, 200, 32), (3, 2, 129, 64)])
def test_gated_result_of_every_kernel_variant(cuda_device, fp8, workspace, B1, B2, S, D):
    """The descriptor's gate through the C ABI, rows with a pitch of their own: bf16 q and k, and fp8 on both of its
    kernels (with a workspace the tensor core adds the bias, without one the softmax threads do)."""
    g = torch.Generator().manual_seed(S)
    dev = cuda_device
    q, k, v = (torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16) for _ in range(3))
    scales = {}
    if fp8:
        if D % 16:
            pytest.skip("fp8 rows are 16-byte multiples")
        q, k = q.to(torch.float8_e4m3fn), k.to(torch.float8_e4m3fn)
        scales = {n: torch.rand(B2, generator=g) * 0.5 + 0.5 for n in ("q_scale", "k_scale")}
    pitch = (S + 7) // 8 * 8
    bias = torch.randn(B2, S, pitch, generator=g).to(torch.bfloat16)
    gate = (torch.randn(B1, S, B2 + 1, D, generator=g) * 3).to(torch.bfloat16)      # [B1, S, H, D]: one head more than used
    mask = torch.rand(B1, S, generator=g) >= 0.1
    gated = gate[:, :, :B2].permute(0, 2, 1, 3)
    ref = O.oracle_fp32(q, k, v, mask, bias[:, :, :S], **scales) * torch.sigmoid(gated.float())
    qd, kd, vd, bd, gd, md = (t.to(dev) for t in (q, k, v, bias, gate, mask))
    sd = {n: t.to(dev) for n, t in scales.items()}
    out = torch.empty(B1, B2, S, D, dtype=torch.bfloat16, device=dev)
    d = _capi.AttentionDesc()
    d.B1, d.B2, d.Sq, d.Sk, d.D = B1, B2, S, S, D
    for name, t in (("q_stride", qd), ("k_stride", kd), ("v_stride", vd), ("out_stride", out), ("gate_stride", gd[:, :, :B2].permute(0, 2, 1, 3))):
        getattr(d, name)[:] = list(t.stride()[:3])
    d.bias_stride[:] = [S * pitch, pitch]
    d.mask_row_stride, d.softmax_scale = S, D ** -0.5
    d.qk_dtype, d.bias_dtype, d.gate = (_capi.AF3K_FP8_E4M3 if fp8 else _capi.AF3K_BF16), _capi.AF3K_BF16, gd.data_ptr()
    lib, p = _capi.load(), lambda t: None if t is None else t.data_ptr()
    n = lib.af3k_dot_product_attention_workspace(ctypes.byref(d), p(bd)) if workspace else 0
    ws = torch.empty(n, dtype=torch.uint8, device=dev) if n else None
    _capi.check(lib.af3k_dot_product_attention(
        ctypes.byref(d), p(qd), p(kd), p(vd), p(bd), p(md.view(torch.uint8)), p(out), p(sd.get("q_scale")), p(sd.get("k_scale")), p(ws), n,
        None, torch.cuda.current_stream().cuda_stream))
    if fp8:
        assert O.error_stats(out.cpu(), ref)["max_abs"] <= FP8_MAX_ABS
    else:
        _check_bf16(out.cpu(), ref, (B1, B2, S, D))
