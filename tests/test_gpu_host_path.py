"""The operator's host-tensor path (row blocks pipelined over PCIe): same result as the device
path, through the reference's own call signature."""
import pytest
import torch

import af3_kernels_b200 as A
from oracle import attention_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [True, False])
def test_host_tensors_give_the_device_result(cuda_device, pinned):
    g = torch.Generator().manual_seed(31)
    B1, B2, S, D = 13, 2, 200, 32
    q = torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16)
    k = torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16)
    v = torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16)
    bias = torch.randn(B2, S, S, generator=g)                      # fp32, as the reference's callers pass it
    mask = torch.rand(B1, S, generator=g) >= 0.1
    if pinned:
        q, k, v, bias, mask = (t.pin_memory() for t in (q, k, v, bias, mask))
    out = A.dot_product_attention_cpp(q, k, v, mask, bias)          # host in, host out
    assert not out.is_cuda and out.shape == (B1, B2, S, D) and out.dtype == torch.bfloat16
    dev = cuda_device
    ref_dev = A.dot_product_attention_cpp(q.to(dev), k.to(dev), v.to(dev), mask.to(dev), bias.to(dev))
    assert torch.equal(out, ref_dev.cpu())
    st = O.error_stats(out, O.oracle_fp32(q, k, v, mask, bias))
    assert st["nan"] == 0 and st["max_abs"] <= 2e-2, st
    # uneven row blocks, 1-D mask, preallocated output
    out2 = torch.empty_like(out)
    A.dot_product_attention_host(q, k, v, mask[0], bias, out=out2, chunks=5)
    ref2 = A.dot_product_attention_cpp(q.to(dev), k.to(dev), v.to(dev), mask[0].to(dev), bias.to(dev))
    assert torch.equal(out2, ref2.cpu())


def test_host_path_rejects_cuda_tensors(cuda_device):
    q = torch.zeros(1, 1, 8, 32, dtype=torch.bfloat16, device=cuda_device)
    with pytest.raises(ValueError):
        A.dot_product_attention_host(q, q, q, None, torch.zeros(1, 8, 8))


@pytest.mark.parametrize("B1,chunks", [(40, 8), (41, 3), (40, 1)])
def test_host_row_blocks_give_the_device_result(cuda_device, B1, chunks):
    """Enough rows that the call is cut into halving row blocks on three streams (10 MB of q, k, v; blocks
    of at least 2 MB), with a bias the kernel cannot read in place and one mask row per batch row."""
    g = torch.Generator().manual_seed(7)
    B2, S, D = 4, 331, 32
    q, k, v = (torch.randn(B1, B2, S, D, generator=g).to(torch.bfloat16).pin_memory() for _ in range(3))
    bias = torch.randn(B2, S, S, generator=g).to(torch.bfloat16)
    mask = torch.rand(B1, S, generator=g) >= 0.1
    out = A.dot_product_attention_host(q, k, v, mask, bias, chunks=chunks)
    ref = A.dot_product_attention_cpp(*(t.to(cuda_device) for t in (q, k, v, mask, bias)))
    assert torch.equal(out, ref.cpu())


def test_host_call_refuses_a_mask_of_one_block(cuda_device):
    """A mask with as many rows as a row block has, not as the call has, is refused as it is for CUDA tensors."""
    q = torch.zeros(40, 4, 331, 32, dtype=torch.bfloat16)
    bias = torch.zeros(4, 331, 331, dtype=torch.bfloat16)
    with pytest.raises(ValueError):
        A.dot_product_attention_host(q, q, q, torch.ones(20, 331, dtype=torch.bool), bias, chunks=2)


def test_host_calls_hold_no_more_memory_the_more_there_are(cuda_device):
    """Forty pipelined calls reserve what two do."""
    g = torch.Generator().manual_seed(3)
    q = torch.randn(40, 4, 331, 32, generator=g).to(torch.bfloat16).pin_memory()
    bias = torch.randn(4, 331, 331, generator=g).pin_memory()
    mask = (torch.rand(40, 331, generator=g) >= 0.1).pin_memory()
    first = A.dot_product_attention_host(q, q, q, mask, bias).clone()
    A.dot_product_attention_host(q, q, q, mask, bias)
    held = torch.cuda.memory_reserved()
    for _ in range(40):
        assert torch.equal(A.dot_product_attention_host(q, q, q, mask, bias), first)
    assert torch.cuda.memory_reserved() == held
