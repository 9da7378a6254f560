"""GPU parity of the two attention blocks and the grid modules (fused passes, and projections through
torch for the sizes those do not take) against golden outputs of the reference's PyTorch models and the fp32 block
oracles.  The blocks compute in bf16, so errors are judged against the size of the outputs:
max-abs <= 4 % of the largest reference magnitude, mean-abs <= 2 % of the mean magnitude (four
bf16 roundings in a row: projections, P, gated product, output projection)."""
import os
import socket

import pytest
import torch

import af3_kernels_b200 as A
from af3_kernels_b200.dpa import read_status
from oracle import attention_oracle as O
from test_blocks_oracle import blocks, grid_args, self_args  # noqa: F401  (fixture + helpers)

pytestmark = pytest.mark.gpu


def _close(out, ref, what):
    o, r = out.float().cpu(), ref.float()
    err = (o - r).abs()
    assert torch.isfinite(o).all(), what
    assert err.max().item() <= 0.04 * r.abs().max().item(), (what, err.max().item(), r.abs().max().item())
    assert err.mean().item() <= 0.02 * r.abs().mean().item(), (what, err.mean().item(), r.abs().mean().item())


def _grid_module(c, dev, cls=None):
    N, C, H, T = (int(v) for v in c["meta"])
    m = (cls or A.GridSelfAttentionCpp)(C, H, bool(T))
    m.load_state_dict({k[2:]: v for k, v in c.items() if k.startswith("w/")})
    return m.to(dev).eval()


def test_grid_module_matches_reference_model(cuda_device, blocks):
    for tag, c in blocks.items():
        if not tag.startswith("grid"):
            continue
        m = _grid_module(c, cuda_device)
        with torch.no_grad():
            out = m(c["pair"].to(cuda_device), c["mask"].to(cuda_device))
        assert out.shape == c["out"].shape and out.dtype == torch.float32
        _close(out, c["out"], tag)
    assert read_status(cuda_device)[0] == 0


def test_attention_cpp_operator_signature_path(cuda_device, blocks):
    c = blocks["grid_n24_c64_h2"]
    dev = cuda_device
    pair, mask, ln_w, ln_b, w_bias, w_q, w_k, w_v, w_g, w_o = (t.to(dev) for t in grid_args(c))
    x = torch.nn.functional.layer_norm(pair, (pair.shape[-1],), ln_w, ln_b)
    bias = torch.nn.functional.linear(x, w_bias).permute(2, 0, 1)
    rep = lambda w: A.vnni_repack_tensor(w.T.contiguous(), 2, 32)     # what the reference module does
    out = A._attention_cpp(x.to(torch.bfloat16), mask, bias, rep(w_q), rep(w_k), rep(w_v), rep(w_g),
                           w_o.T.contiguous(), 2, False, 64, 0)
    assert out.dtype == torch.bfloat16
    _close(out, c["out"], "_attention_cpp")


def test_self_attention_cpp_matches_reference_model(cuda_device, blocks):
    dev = cuda_device
    for tag, c in blocks.items():
        if not tag.startswith("self"):
            continue
        N, C, H = (int(v) for v in c["meta"])
        x, mask, logits, w_q, b_q, w_k, w_v, w_g = (t.to(dev) for t in self_args(c))
        out = A.self_attention_cpp(x, mask, logits, w_q.T.contiguous(), b_q, w_k.T.contiguous(),
                                   w_v.T.contiguous(), w_g.T.contiguous(), H)
        assert out.shape == (N, C) and out.dtype == torch.float32
        _close(out, c["out"], tag)


def test_grid_module_larger_shape_against_oracle(cuda_device):
    torch.manual_seed(3)
    N, C, H = 200, 128, 4
    m = A.GridSelfAttentionCpp(C, H, False)
    with torch.no_grad():
        for lin in (m.q_projection, m.k_projection):
            lin.weight.mul_(4.0)
        m.pair_bias_projection.weight.mul_(8.0)
    pair = torch.randn(N, N, C)
    mask = torch.rand(N, N) >= 0.05
    sd = m.state_dict()
    ref = O.grid_block_fp32(pair, mask, sd["act_norm.weight"], sd["act_norm.bias"],
                            sd["pair_bias_projection.weight"], sd["q_projection.weight"],
                            sd["k_projection.weight"], sd["v_projection.weight"],
                            sd["gating_query.weight"], sd["output_projection.weight"], H)
    m = m.to(cuda_device).eval()
    with torch.no_grad():
        out = m(pair.to(cuda_device), mask.to(cuda_device))
        again = m(pair.to(cuda_device), mask.to(cuda_device))
    _close(out, ref, "grid N=200")
    assert torch.equal(out, again)


def test_distributed_module_single_rank_equals_plain_module(cuda_device, blocks):
    import torch.distributed as dist
    c = blocks["grid_n36_c48_h2_t"]
    with socket.socket() as s:
        s.bind(("127.0.0.1", 0))
        port = s.getsockname()[1]
    os.environ.setdefault("NCCL_NVLS_ENABLE", "0")
    dist.init_process_group("nccl", init_method=f"tcp://127.0.0.1:{port}", rank=0, world_size=1,
                            device_id=cuda_device)
    try:
        plain = _grid_module(c, cuda_device)
        sharded = _grid_module(c, cuda_device, A.DistributedGridSelfAttentionCpp)
        pair, mask = c["pair"].to(cuda_device), c["mask"].to(cuda_device)
        with torch.no_grad():
            a = plain(pair, mask)
            b = sharded(pair, mask, COMM_SPLIT=3)
        assert a.shape == b.shape
        # same math on row pieces; the projection GEMMs may pick another tiling for another M
        assert (a - b).abs().max().item() <= 2e-2 * a.abs().max().item()
    finally:
        dist.destroy_process_group()


def test_fused_projection_kernel_matches_plain_gemms(cuda_device):
    """af3k_qkvg_projection: q, k, v head-major with q pre-scaled, gate row-major, against fp32
    matmuls of the same bf16 operands (bf16 rounding of the result only), on a ragged row count and
    for every head count the kernel takes."""
    from af3_kernels_b200.fused_ops import _stacked_projection_weights, qkvg_projection
    from af3_kernels_b200.dpa import read_status
    dev = cuda_device
    g = torch.Generator().manual_seed(3)
    for R, N, H in ((3, 200, 4), (1, 37, 2), (2, 129, 16), (5, 256, 8)):
        C, D = 128, 128 // H
        x = torch.randn(R, N, C, generator=g).to(torch.bfloat16).to(dev)
        ws = [(torch.randn(C, C, generator=g) * 0.1).to(torch.bfloat16).to(dev) for _ in range(4)]   # [in, out]
        w4 = _stacked_projection_weights(*ws)
        assert w4.shape == (4 * C, C)
        scale = D ** -0.5
        q, k, v, gate = qkvg_projection(x, w4, H, scale)
        torch.cuda.synchronize()
        assert read_status(dev)[0] == 0
        ref = [x.float() @ w.float() for w in ws]
        ref[0] = ref[0] * scale
        for got, want in zip((q, k, v), ref[:3]):
            want = want.view(R, N, H, D).permute(0, 2, 1, 3)
            assert got.shape == want.shape
            assert (got.float() - want).abs().max().item() <= 2e-2 * max(1.0, want.abs().max().item()), (R, N, H)
        assert (gate.float() - ref[3]).abs().max().item() <= 2e-2 * max(1.0, ref[3].abs().max().item())


def test_self_block_replays_from_a_cuda_graph(cuda_device):
    """The block is two short launches (the projections, the attention kernel with the gate); its
    calls into the library allocate nothing the graph allocator cannot serve and never synchronise,
    so the whole block can be captured once and replayed - with results identical to the eager call."""
    dev = cuda_device
    g = torch.Generator().manual_seed(31)
    N, C, H = 200, 64, 4
    x = torch.randn(N, C, generator=g).to(torch.bfloat16).to(dev)
    ws = [(torch.randn(C, C, generator=g) * C ** -0.5).to(torch.bfloat16).to(dev) for _ in range(4)]
    qb = (torch.randn(C, generator=g) * 0.1).to(torch.bfloat16).to(dev)
    bias = torch.randn(H, N, N, generator=g).to(torch.bfloat16).to(dev)
    mask = (torch.arange(N) < N - 17).to(dev)
    call = lambda: A.self_attention_cpp(x, mask, bias, ws[0], qb, ws[1], ws[2], ws[3], H)
    with torch.no_grad():
        ref = call()
        side = torch.cuda.Stream(device=dev)
        side.wait_stream(torch.cuda.current_stream(dev))
        with torch.cuda.stream(side):
            call()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=side):
                out = call()
        torch.cuda.current_stream(dev).wait_stream(side)
        out.zero_()
        graph.replay()
        torch.cuda.synchronize(dev)
    assert torch.equal(out, ref)
    assert read_status(dev)[0] == 0


def test_fused_front_matches_the_two_kernels_it_replaces(cuda_device):
    """af3k_pair_front (LayerNorm + pair bias + q/k/v/gate projections from the raw pair) against
    af3k_pair_bias followed by af3k_qkvg_projection: both round the normalised pair to bf16 before
    the projections; odd sizes cover tiles that straddle pair rows and the ragged last tile."""
    from af3_kernels_b200.fused_ops import _stacked_projection_weights, pair_front, qkvg_projection
    from af3_kernels_b200.pair_bias import layernorm_pair_bias
    dev = cuda_device
    for R, N, H, Hb in ((5, 200, 4, 4), (3, 128, 4, 2), (2, 37, 8, 1), (130, 130, 4, 4)):
        g = torch.Generator().manual_seed(100 + N)
        pair = (torch.randn(R, N, 128, generator=g) * 2.0 + 0.3).to(torch.bfloat16).to(dev)
        ln_w = (1.0 + 0.2 * torch.randn(128, generator=g)).to(dev)
        ln_b = (0.1 * torch.randn(128, generator=g)).to(dev)
        bw = (torch.randn(Hb, 128, generator=g) * 0.3).to(dev)
        ws = [(torch.randn(128, 128, generator=g) * 128 ** -0.5).to(torch.bfloat16).to(dev) for _ in range(4)]
        w4 = _stacked_projection_weights(*ws)
        D = 128 // H
        normed, bias_ref = layernorm_pair_bias(pair, ln_w, ln_b, bw)
        q_ref, k_ref, v_ref, g_ref = qkvg_projection(normed, w4, H, D ** -0.5)
        bias, q, k, v, gate = pair_front(pair, ln_w, ln_b, 1e-5, bw, w4, H, D ** -0.5)
        torch.cuda.synchronize(dev)
        assert read_status(dev)[0] == 0
        # the two LayerNorms order their arithmetic differently, so a normalised value may land on the
        # neighbouring bf16 now and then: the projections agree to a few bf16 ulps of their scale
        for a, b in ((q, q_ref), (k, k_ref), (v, v_ref), (gate, g_ref)):
            s_ = b.float().abs().max().item()
            assert (a.float() - b.float()).abs().max().item() <= 2.0 ** -6 * s_
            assert (a.float() - b.float()).abs().mean().item() <= 2.0 ** -10 * s_
        scale = bias_ref.float().abs().max().item()
        assert (bias.float() - bias_ref.float()).abs().max().item() <= 2.0 ** -7 * scale + 1e-3


@pytest.mark.parametrize("N,C,H,dtype,transpose", [
    (1, 128, 4, torch.bfloat16, False), (5, 64, 4, torch.float32, True), (64, 128, 4, torch.bfloat16, True),
    (100, 64, 2, torch.bfloat16, False), (129, 128, 2, torch.float32, False), (131, 128, 4, torch.float32, True),
    (192, 64, 4, torch.bfloat16, True), (261, 64, 1, torch.bfloat16, False), (261, 64, 4, torch.float32, True)])
def test_fused_grid_module_against_oracle(cuda_device, N, C, H, dtype, transpose):
    """The three-launch module over what its kernels branch on: one row tile and less, tiles that straddle
    pair rows, tiles shared by four / two CTAs and several tiles per CTA, both widths, both pair types, both
    orientations, one to four heads of bias."""
    torch.manual_seed(N + C)
    m = A.GridSelfAttentionCpp(C, H, transpose)
    with torch.no_grad():
        m.act_norm.weight.add_(0.2 * torch.randn(C))
        m.act_norm.bias.add_(0.1 * torch.randn(C))
        for lin in (m.q_projection, m.k_projection):
            lin.weight.mul_(3.0)
        m.pair_bias_projection.weight.mul_(4.0)
    m = m.to(dtype).eval()
    pair = (torch.randn(N, N, C) * 2.0 + 0.5).to(dtype)
    mask = torch.rand(N, N) >= 0.1
    mask[:, 0] = True
    sd = m.state_dict()
    ref = O.grid_block_fp32(pair, mask, *(sd[k].float() for k in (
        "act_norm.weight", "act_norm.bias", "pair_bias_projection.weight", "q_projection.weight", "k_projection.weight",
        "v_projection.weight", "gating_query.weight", "output_projection.weight")), H, transpose)
    m = m.to(cuda_device)
    with torch.no_grad():
        out = m(pair.to(cuda_device), mask.to(cuda_device))
        # new values in the same parameters are seen
        m.output_projection.weight.neg_()
        flipped = m(pair.to(cuda_device), mask.to(cuda_device))
    assert out.dtype == dtype and out.shape == (N, N, C)
    _close(out, ref, (N, C, H, dtype, transpose))
    assert torch.equal(flipped, -out)
    assert read_status(cuda_device)[0] == 0


@pytest.mark.parametrize("N,C,H,dtype", [(1, 64, 4, torch.bfloat16), (77, 384, 16, torch.bfloat16), (128, 200, 5, torch.float32),
                                         (129, 768, 16, torch.bfloat16), (700, 384, 16, torch.float32), (1100, 512, 8, torch.bfloat16)])
def test_self_block_against_oracle(cuda_device, N, C, H, dtype):
    """Single block over what its projection kernel branches on: rows short of a tile and one past it, K blocks
    short of 64 channels, fewer and more K blocks than stages, both tile widths; odd N stages the bias."""
    g = torch.Generator().manual_seed(N)
    x = torch.randn(N, C, generator=g).to(dtype)
    ws = [(torch.randn(C, C, generator=g) * C ** -0.5).to(dtype) for _ in range(4)]        # [in, out]
    qb = (torch.randn(C, generator=g) * 0.3).to(dtype)
    bias = torch.randn(H, N, N, generator=g).to(dtype)
    mask = torch.arange(N) < N - N // 9
    ref = O.self_block_fp32(x, mask, bias, ws[0].T, qb, ws[1].T, ws[2].T, ws[3].T, H)
    dev = cuda_device
    out = A.self_attention_cpp(x.to(dev), mask.to(dev), bias.to(dev), ws[0].to(dev), qb.to(dev), *(w.to(dev) for w in ws[1:]), H)
    assert out.dtype == dtype and out.shape == (N, C)
    _close(out, ref, (N, C, H, dtype))
    assert read_status(dev)[0] == 0


@pytest.mark.parametrize("N,C,dtype", [(24, 128, torch.bfloat16), (129, 64, torch.float32), (200, 128, torch.float32)])
def test_kernels_that_start_under_the_previous_ones_wait_for_them(cuda_device, N, C, dtype):
    """Every kernel of a chain reads what the one before wrote (and overwrites buffers that it read): modules in both
    orientations, a plain call and the single block, back to back, on two streams and from a graph, give the bits of
    the same chain with a synchronisation behind every call."""
    g = torch.Generator().manual_seed(21)
    H, D = 4, C // 4
    mods = []
    for t in (False, True):
        m = A.GridSelfAttentionCpp(C, H, t)
        with torch.no_grad():
            for p in m.parameters():
                p.copy_(torch.randn(p.shape, generator=g) * (C ** -0.5 if p.dim() == 2 else 0.1))
            m.act_norm.weight.add_(1.0)
        mods.append(m.to(cuda_device, dtype).eval())
    pair0 = torch.randn(N, N, C, generator=g).to(cuda_device, dtype)
    mask = (torch.rand(N, N, generator=g) >= 0.1).to(cuda_device)
    w = [(torch.randn(C, C, generator=g) * C ** -0.5).to(cuda_device, dtype) for _ in range(4)]
    qb = torch.zeros(C, device=cuda_device, dtype=dtype)

    def chain(pair, between):
        for i in range(6):
            pair = mods[i % 2](pair, mask)
            between()
            x = pair.reshape(N, N, H, D).permute(0, 2, 1, 3).to(torch.bfloat16)
            pair = A.dot_product_attention_cpp(x, x, x, mask, x[:H, 0, :, :1].expand(H, N, N)).permute(0, 2, 1, 3).reshape(N, N, C).to(dtype)
            between()
            row = A.self_attention_cpp(pair[0], mask[0], pair.permute(2, 0, 1)[:H].contiguous(), *w[:1], qb, *w[1:], H)
            between()
            pair = pair + row
        return pair

    with torch.no_grad():
        want = chain(pair0, torch.cuda.synchronize)
        got = [chain(pair0, lambda: None) for _ in range(5)]
        streams = [torch.cuda.Stream(), torch.cuda.Stream()]
        for s in streams * 2:
            s.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(s):
                got.append(chain(pair0, lambda: None))
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = chain(pair0, lambda: None)
        for _ in range(3):
            graph.replay()
        torch.cuda.synchronize()
        got.append(out)
    for i, r in enumerate(got):
        assert torch.equal(r, want), i
    assert read_status(cuda_device)[0] == 0


def _block_calls(kind, C, dtype, device, seed):
    """-> (parameters, call): one block of the given kind and a call of it on fixed inputs."""
    g = torch.Generator().manual_seed(seed)
    H, N = 4, 72
    normal = lambda *s, std=1.0: (torch.randn(*s, generator=g) * std).to(device, dtype)
    mask = (torch.rand(N, N, generator=g) >= 0.1).to(device)
    if kind == "module":
        m = A.GridSelfAttentionCpp(C, H, bool(seed % 2)).to(device, dtype).eval()
        pair = normal(N, N, C)
        params = list(m.parameters())
        with torch.no_grad():
            for p in params:
                p.copy_(normal(*p.shape, std=C ** -0.5 if p.dim() == 2 else 0.3))
        return params, lambda: m(pair, mask)
    ws = [normal(C, C, std=C ** -0.5) for _ in range(5)]
    bias = normal(H, N, N).to(torch.bfloat16)        # read in place: the staged copy of another bias is not the subject
    if kind == "grid":
        pair = normal(3, N, C)
        return ws, lambda: A._attention_cpp(pair, mask[:3], bias, *ws, H)
    x, qb = normal(N, C), normal(C, std=0.1)
    return ws[:4] + [qb], lambda: A.self_attention_cpp(x, mask[0], bias, ws[0], qb, *ws[1:4], H)


@pytest.mark.parametrize("kind,C,dtype", [("module", 128, torch.bfloat16), ("module", 64, torch.float32), ("grid", 128, torch.float32),
                                          ("grid", 64, torch.bfloat16), ("self", 64, torch.bfloat16), ("self", 224, torch.float32)])
def test_blocks_compute_with_the_parameters_as_they_are(cuda_device, kind, C, dtype):
    """New values are seen by the next call and by the next replay of a graph captured on the stream that was warmed
    up, however they were written (``.data`` bumps no version counter), and however many other blocks ran since."""
    with torch.no_grad():
        params, call = _block_calls(kind, C, dtype, cuda_device, 1)
        values, want = [], []
        for seed in (1, 2, 3):
            p, c = _block_calls(kind, C, dtype, cuda_device, 1)
            for i, t in enumerate(p):
                t.copy_(torch.randn(t.shape, generator=torch.Generator().manual_seed(10 * seed + i)) * C ** -0.5)
            values.append([t.clone() for t in p])
            want.append(c())

        def load(i):
            for t, v in zip(params, values[i]):
                t.data.copy_(v)

        load(0)
        assert torch.equal(call(), want[0])
        load(1)
        assert torch.equal(call(), want[1])
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            call()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=side):
                out = call()
        torch.cuda.current_stream().wait_stream(side)
        keep = []
        for seed in range(20):
            keep.append(_block_calls(kind, C, dtype, cuda_device, 100 + seed))
            keep[-1][1]()
        for i in (1, 2, 0):
            for t, v in zip(params, values[i]):
                t.copy_(v)
            graph.replay()
            assert torch.equal(out, want[i]), i
        torch.cuda.synchronize()
    assert read_status(cuda_device)[0] == 0


def test_a_part_of_the_weights_is_not_taken_for_the_whole(cuda_device):
    """Views that differ in their extent only: a block on the corner of a larger block's weights."""
    g = torch.Generator().manual_seed(8)
    H, N = 4, 40
    ws = [(torch.randn(256, 256, generator=g) * 0.1).to(cuda_device, torch.bfloat16) for _ in range(4)]
    for C in (256, 128):
        x = torch.randn(N, C, generator=g).to(torch.bfloat16)
        bias = torch.randn(H, N, N, generator=g).to(torch.bfloat16)
        part = [w[:C, :C] for w in ws]
        qb = torch.zeros(C, dtype=torch.bfloat16)
        out = A.self_attention_cpp(x.to(cuda_device), None, bias.to(cuda_device), part[0], qb.to(cuda_device), *part[1:], H)
        cpu = [w.cpu() for w in part]
        _close(out, O.self_block_fp32(x, torch.ones(N, dtype=torch.bool), bias, cpu[0].T, qb, *(w.T for w in cpu[1:]), H), C)


@pytest.mark.parametrize("N,C,H", [(1, 64, 4), (77, 72, 3), (130, 200, 5), (300, 384, 16), (1100, 512, 8), (129, 1024, 16), (3600, 72, 3)])
def test_self_block_reads_weights_of_any_layout(cuda_device, N, C, H):
    """Weights kept `[in, out]`, `[out, in]`, as parts of larger matrices, mixed, and in forms that are packed first
    (odd pitch, odd offset, fp32 with the same values) give the same bits, on channel counts short of and past whole
    64-column blocks."""
    g = torch.Generator().manual_seed(C)
    dev = cuda_device
    x = torch.randn(N, C, generator=g).to(torch.bfloat16)
    ws = [(torch.randn(C, C, generator=g) * C ** -0.5).to(torch.bfloat16) for _ in range(4)]        # [in, out]
    qb = (torch.randn(C, generator=g) * 0.3).to(torch.bfloat16)
    bias = torch.randn(H, N, N, generator=g).to(torch.bfloat16)

    def part(w, rows, cols, r0, c0):
        big = torch.full((rows, cols), float("nan"), dtype=w.dtype, device=dev)
        big[r0:r0 + C, c0:c0 + C] = w.to(dev)
        return big[r0:r0 + C, c0:c0 + C]

    forms = {
        "in_out": lambda w: w.to(dev).contiguous(),
        "out_in": lambda w: w.T.contiguous().to(dev).T,
        "part": lambda w: part(w, C + 3, C + 16, 2, 8),
        "part_t": lambda w: part(w.T, C + 3, C + 16, 2, 8).T,
        "odd_pitch": lambda w: part(w, C, C + 1, 0, 0),
        "odd_offset": lambda w: part(w, C, C + 8, 0, 1),
        "f32": lambda w: w.float().to(dev),
        "f32_t": lambda w: w.float().T.contiguous().to(dev).T,
    }
    ref = O.self_block_fp32(x, torch.ones(N, dtype=torch.bool), bias, ws[0].T, qb, *(w.T for w in ws[1:]), H)
    call = lambda w: A.self_attention_cpp(x.to(dev), None, bias.to(dev), w[0], qb.to(dev), *w[1:], H)
    want = call([forms["out_in"](w) for w in ws])
    _close(want, ref, (N, C, H))
    for name, form in forms.items():
        assert torch.equal(call([form(w) for w in ws]), want), name
    mixed = [forms[n](w) for n, w in zip(("in_out", "out_in", "part", "part_t"), ws)]
    assert torch.equal(call(mixed), want)
    assert read_status(dev)[0] == 0


@pytest.mark.parametrize("C", [64, 128])
def test_parameters_on_another_device_are_refused(cuda_device, C):
    """A module or weights left on the host: an exception before anything is launched."""
    H, N = 4, 24
    dev, bf16 = cuda_device, torch.bfloat16
    pair, mask = torch.zeros(N, N, C, device=dev, dtype=bf16), torch.ones(N, N, dtype=torch.bool, device=dev)
    bias = torch.zeros(H, N, N, device=dev, dtype=bf16)
    w = [torch.zeros(C, C, dtype=bf16) for _ in range(5)]
    on = [t.to(dev) for t in w]
    m = A.GridSelfAttentionCpp(C, H).to(bf16)
    with torch.no_grad():
        with pytest.raises(ValueError, match="device"):
            m(pair, mask)
        m.to(dev).output_projection.cpu()
        with pytest.raises(ValueError, match="device"):
            m(pair, mask)
        for i in range(5):
            mixed = [w[j] if j == i else on[j] for j in range(5)]
            with pytest.raises(ValueError, match="device"):
                A._attention_cpp(pair, mask, bias, *mixed, H)
            if i < 4:
                with pytest.raises(ValueError, match="device"):
                    A.self_attention_cpp(pair[0], mask[0], bias, mixed[0], torch.zeros(C, device=dev), *mixed[1:4], H)
        with pytest.raises(ValueError, match="device"):
            A.self_attention_cpp(pair[0], mask[0], bias, on[0], torch.zeros(C), *on[1:4], H)
        q = torch.zeros(1, 2, 16, 32, device=dev, dtype=bf16)
        with pytest.raises(ValueError, match="device"):
            A.dot_product_attention(q, q, q, None, torch.zeros(2, 16, 16, device=dev), out=q.cpu())
    torch.cuda.synchronize()
    assert read_status(dev)[0] == 0


@pytest.mark.parametrize("C,dtype,transpose", [(64, torch.bfloat16, False), (128, torch.float32, True), (128, torch.bfloat16, False)])
def test_output_projection_has_a_gradient(cuda_device, C, dtype, transpose):
    """Outside no_grad the result carries the gradient of the output projection (out = gated Wo^T is linear in it), and is
    the result under no_grad up to bf16 rounding; module and functional block."""
    g = torch.Generator().manual_seed(C)
    H, N = 4, 40
    m = A.GridSelfAttentionCpp(C, H, transpose).to(cuda_device, dtype)
    pair = torch.randn(N, N, C, generator=g).to(cuda_device, dtype)
    mask = torch.ones(N, N, dtype=torch.bool, device=cuda_device)
    bias = torch.randn(H, N, N, generator=g).to(cuda_device, torch.bfloat16)
    wo = m.output_projection.weight
    for call in (lambda: m(pair, mask), lambda: A._attention_cpp(pair, mask, bias, *m._weights(), H)):
        with torch.no_grad():
            want = call()
        out = call()
        assert out.dtype == dtype and out.requires_grad and not want.requires_grad
        scale = want.float().abs().max().item()
        assert (out.detach().float() - want.float()).abs().max().item() <= 2.0 ** -7 * scale
        wo.grad = None
        (out.float() * want.float()).sum().backward()
        # sum(out * c) is linear in Wo: its derivative along Wo itself is its value
        along, value = (wo.grad.float() * wo.detach().float()).sum().item(), (out.detach().float() * want.float()).sum().item()
        assert abs(along - value) <= 2e-2 * abs(value)


def test_norm_and_bias_modules_that_were_hooked_or_replaced_run(cuda_device):
    """At 64 channels LayerNorm and bias projection are the module's own: hooks on them fire, and one put in their place
    is used."""
    C, H, N = 64, 4, 24
    m = A.GridSelfAttentionCpp(C, H).to(cuda_device).eval()
    pair = torch.randn(N, N, C, generator=torch.Generator().manual_seed(1)).to(cuda_device)
    mask = torch.ones(N, N, dtype=torch.bool, device=cuda_device)
    with torch.no_grad():
        plain = m(pair, mask)
        seen = []
        hooks = [x.register_forward_hook(lambda mod, a, out: seen.append(type(mod))) for x in (m.act_norm, m.pair_bias_projection)]
        hooked = m(pair, mask)
        assert seen == [torch.nn.LayerNorm, torch.nn.Linear]
        _close(hooked, plain.cpu(), "hooked")
        for h in hooks:
            h.remove()
        assert torch.equal(m(pair, mask), plain)
        m.act_norm = torch.nn.LayerNorm(C, elementwise_affine=False, device=cuda_device)
        _close(m(pair, mask), plain.cpu(), "without affine parameters (they were one and zero)")


def _gate_values(device):
    """Every bf16 gate from -88.5 to 88.5, on 128 channels (below -128 ln 2 = -88.7 the exponential is past fp32 and the
    sigmoid, under 2^-128, is zero)."""
    bits = torch.arange(2 ** 16, dtype=torch.int32).to(torch.uint16).view(torch.bfloat16)
    g = bits[bits.float().abs() <= 88.5]
    return torch.nn.functional.pad(g, (0, -g.numel() % 128)).view(-1, 128).to(device)


def _gated(weighted, gate):
    """weighted * sigmoid(gate) in 64 bits, and the tolerance of its bf16 rounding: half an ulp (relative 2^-8), the
    rounding of the exponent (up to 128, so 2^-18 ln 2) with a few fp32 ulps, and the smallest bf16 step below the normal
    range."""
    want = weighted.double() * torch.sigmoid(gate.double())
    return want, want.abs() * (2.0 ** -8 + 2.0 ** -17) + 2.0 ** -133


@pytest.mark.parametrize("factor", [1.0, 2.0 ** 100])
def test_sigmoid_gate_over_every_gate(cuda_device, factor):
    """The gate kernel and the gated output pass (identity weights), down to where the sigmoid is denormal."""
    from af3_kernels_b200 import _capi
    from af3_kernels_b200.fused_ops import sigmoid_gate
    gate = _gate_values(cuda_device)
    w = torch.full_like(gate, factor)
    want, tol = _gated(w, gate)
    got = sigmoid_gate(w, gate)
    assert ((got.double() - want).abs() <= tol).all()
    import ctypes
    out = torch.empty(gate.shape, device=cuda_device)
    eye = torch.eye(128, device=cuda_device, dtype=torch.bfloat16)
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    i64 = ctypes.c_longlong
    _capi.check(_capi.load().af3k_grid_out(p(w), p(gate), p(eye), p(out), _capi.AF3K_F32, i64(gate.shape[0]), i64(128), None,
                                           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert ((out.double() - want).abs() <= tol).all()


@pytest.mark.parametrize("R,N", [(3, 50), (40, 129), (160, 160)])
def test_bias_of_a_narrow_fp32_pair_is_that_of_the_fp32_normalised_pair(cuda_device, R, N):
    """64 channels, fp32: LayerNorm and bias projection against 64 bits.  x and the weights enter as two bf16 parts
    (2^-16 relative each) and the sums are fp32, so the bound is half a bf16 ulp of the result (2^-8 relative) plus 2^-14
    of the sum of absolute products; a bias of the rounded x is off by up to 2^-8 of it.  Tiles split over CTAs and not."""
    import ctypes
    from af3_kernels_b200 import _capi
    g = torch.Generator().manual_seed(R)
    C, H, Hb, dev = 64, 4, 3, cuda_device
    pair = (torch.randn(R, N, C, generator=g) * 2 + 0.3).to(dev)
    gamma, beta = (1 + 0.2 * torch.randn(C, generator=g)).to(dev), (0.1 * torch.randn(C, generator=g)).to(dev)
    bw = (torch.randn(Hb, C, generator=g) * 0.3).to(dev)
    w4 = torch.zeros(4 * C, C, dtype=torch.bfloat16, device=dev)
    pitch = (N + 7) // 8 * 8
    bias = torch.empty(Hb, R, pitch, dtype=torch.bfloat16, device=dev)
    q, k, v, gate = (torch.empty(R * N * C, dtype=torch.bfloat16, device=dev) for _ in range(4))
    p, i64, f = (lambda t: ctypes.c_void_p(t.data_ptr())), ctypes.c_longlong, ctypes.c_float
    _capi.check(_capi.load().af3k_grid_front(
        p(pair), ctypes.c_int32(_capi.AF3K_F32), p(gamma), p(beta), f(1e-5), p(bw), i64(Hb), p(w4), i64(R), i64(N), i64(C), i64(H), f(1.0),
        ctypes.c_int32(0), p(bias), i64(pitch), p(q), p(k), p(v), p(gate), None, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    x = torch.nn.functional.layer_norm(pair.double(), (C,), gamma.double(), beta.double(), 1e-5)
    want = torch.einsum("rnc,hc->hrn", x, bw.double())
    size = torch.einsum("rnc,hc->hrn", x.abs(), bw.double().abs())
    err = (bias[:, :, :N].double() - want).abs()
    assert (err <= want.abs() * 2.0 ** -8 + size * 2.0 ** -14).all(), (err / size).max()


@pytest.mark.parametrize("C", [64, 128])
@pytest.mark.parametrize("R,N", [(2, 30), (70, 90), (200, 200)])
def test_grid_block_reads_weights_of_any_layout(cuda_device, R, N, C):
    """`[out, in]` weights are read where they are (bf16 by TMA, fp32 converted on the way in), others are packed first:
    the same bits for the same values, with a tile's outputs on four, two and one CTAs."""
    g = torch.Generator().manual_seed(C + N)
    H, dev = 4, cuda_device
    pair = torch.randn(R, N, C, generator=g).to(dev, torch.bfloat16)
    mask = (torch.rand(R, N, generator=g) >= 0.1).to(dev)
    bias = torch.randn(H, N, N, generator=g).to(dev, torch.bfloat16)
    ws = [(torch.randn(C, C, generator=g) * C ** -0.5).to(dev, torch.bfloat16) for _ in range(5)]      # [in, out]
    out_in = lambda w: w.T.contiguous().T
    forms = {"out_in": out_in, "in_out": lambda w: w, "f32": lambda w: out_in(w.float()), "f32_in_out": lambda w: w.float(),
             "odd_offset": lambda w: torch.nn.functional.pad(w.T.reshape(-1), (1, 0))[1:].view(C, C).T}
    with torch.no_grad():
        res = {n: A._attention_cpp(pair, mask, bias, *map(f, ws), H) for n, f in forms.items()}
        mixed = A._attention_cpp(pair, mask, bias, *[f(w) for f, w in zip(forms.values(), ws)], H)
    for n, r in res.items():
        assert torch.equal(r, res["out_in"]), n
    assert torch.equal(mixed, res["out_in"])
    assert read_status(dev)[0] == 0


class _Subclass(A.GridSelfAttentionCpp):      # takes the module's general way
    pass


class _Scaled(torch.nn.Linear):
    """A Linear whose weight is not what its parameters hold."""

    def __getattr__(self, name):
        value = super().__getattr__(name)
        return value * 2 if name == "weight" else value


@pytest.mark.parametrize("C", [64, 128])
@pytest.mark.parametrize("form", ["plain", "mask_1d", "mask_uint8", "mask_3d", "float32", "hook", "replaced", "weight_in_dict", "layer_in_dict", "functional", "half_norm", "trains_output"])
def test_module_call_straight_from_python(cuda_device, C, form):
    """Whatever parameters, layers, masks and modes a module is called with: the bits of the general way, and hooks run."""
    g = torch.Generator().manual_seed(C)
    N = 40
    plain, general = A.GridSelfAttentionCpp(C, 4, True).to(cuda_device, torch.bfloat16), _Subclass(C, 4, True).to(cuda_device, torch.bfloat16)
    calls = []
    for m in (plain, general):
        if form == "float32":
            m.float()
        if form == "half_norm":
            m.act_norm.half()
        if form == "replaced":
            m.k_projection = _Scaled(C, C, bias=False).to(cuda_device, torch.bfloat16)
        if form == "hook":
            m.act_norm.register_forward_hook(lambda *a: calls.append(1))
    params = [(torch.randn(p.shape, generator=g) * (C ** -0.5 if p.dim() == 2 else 0.2)).to(cuda_device) for p in plain.parameters()]
    with torch.no_grad():
        for m in (plain, general):
            for p, value in zip(m.parameters(), params):
                p.copy_(value)
    if form == "weight_in_dict":
        for m in (plain, general):
            m.v_projection.__dict__["weight"] = m.v_projection.weight.detach() * 3
    if form == "layer_in_dict":
        for m in (plain, general):
            other = torch.nn.Linear(C, C, bias=False).to(cuda_device, torch.bfloat16)
            other.weight.data.copy_(m.v_projection.weight.detach() * 3)
            m.__dict__["v_projection"] = other
    pair = torch.randn(N, N, C, generator=g).to(cuda_device, torch.float32 if form == "float32" else torch.bfloat16)
    mask = (torch.rand(N, N, generator=g) >= 0.2).to(cuda_device)
    mask = {"mask_1d": mask[0], "mask_uint8": mask.to(torch.uint8), "mask_3d": mask[:, None, None, :]}.get(form, mask)
    call = lambda m: m(pair, mask)
    if form == "functional":
        new = {n: (p.detach() * 1.5) for n, p in plain.named_parameters()}
        call = lambda m: torch.func.functional_call(m, new, (pair, mask))
    with torch.enable_grad() if form == "trains_output" else torch.no_grad():
        out, want = call(plain), call(general)
    assert torch.equal(out, want) and out.dtype == pair.dtype
    assert out.requires_grad == (form == "trains_output")
    assert len(calls) == (2 if form == "hook" and C == 64 else 0)
    assert read_status(cuda_device)[0] == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_single_block_and_operator_straight_from_python(cuda_device, dtype):
    """Masks in other forms take the general way: the same bits; what is refused is refused on both."""
    g = torch.Generator().manual_seed(5)
    N, C, H = 70, 96, 4
    x = torch.randn(N, C, generator=g).to(cuda_device, dtype)
    ws = [(torch.randn(C, C, generator=g) * 0.1).to(cuda_device, dtype) for _ in range(4)]
    qb, bias = torch.randn(C, generator=g).to(cuda_device), torch.randn(H, N, N, generator=g).to(cuda_device, dtype)
    mask = (torch.rand(N, generator=g) >= 0.2).to(cuda_device)
    for forms in ((None, torch.ones_like(mask)), (mask, mask.to(torch.uint8), mask[None], mask.float().reshape(1, 1, N))):
        outs = [A.self_attention_cpp(x, m, bias, ws[0], qb, *ws[1:], H) for m in forms]
        assert all(torch.equal(o, outs[0]) for o in outs) and outs[0].dtype == dtype
    # [in, out] weights as views of [out, in] ones, and other strides
    views = [w.t().contiguous().t() for w in ws]
    assert torch.equal(A.self_attention_cpp(x, mask, bias, views[0], qb, *views[1:], H), outs[0])
    strided = [torch.cat([w, w])[:, :].as_strided((C, C), (C, 1)) for w in ws]
    assert torch.equal(A.self_attention_cpp(x, mask, bias, strided[0], qb, *strided[1:], H), outs[0])
    q = x.reshape(1, N, H, C // H).permute(0, 2, 1, 3)
    outs = [A.dot_product_attention_cpp(q, q, q, m, bias) for m in (mask, mask.to(torch.uint8), mask[None, None, None])]
    assert all(torch.equal(o, outs[0]) for o in outs)
    for bad in (mask[:-1], torch.ones(3, N, dtype=torch.bool, device=cuda_device)):
        with pytest.raises(ValueError):
            A.dot_product_attention_cpp(q, q, q, bad, bias)
        with pytest.raises(ValueError):
            A.self_attention_cpp(x, bad, bias, ws[0], qb, *ws[1:], H)
    with pytest.raises(ValueError):
        A.dot_product_attention_cpp(q, q, q, mask, bias, False, 0)


@pytest.mark.parametrize("N,C,H", [(900, 704, 11), (1030, 520, 13)])
def test_projection_tiles_of_256_columns(cuda_device, N, C, H):
    """Where tiles of 128 columns would take two rounds of CTAs; matrices that end inside such a tile."""
    test_self_block_reads_weights_of_any_layout(cuda_device, N, C, H)
