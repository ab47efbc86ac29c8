"""Packed rows whose document boundaries fall on and around the kernels' blocks, tensor-core kernels against the
CUDA-core ones.  Both round O and the gradients to bf16 once; the tensor-core kernels also round P and dS to bf16
(2^-9 of each term, independent): 2^-8 of the largest value covers the two, 2e-2 is the class the parity tests use.
A one-token document's dS = P (dP - D) is zero; formed from two fp32 sums of 64 products of up to 4 x 4 it is off by
64 x 16 x 2^-24 = 6e-5 at most, times |k| <= 4 and the scale 1/8: 3e-5 absolute."""
import pytest
import torch

from mlx_train_perf_b200.attention.api import flash_attention
from mlx_train_perf_b200.attention.segments import PackedMask

pytestmark = pytest.mark.gpu

LENGTHS = [[300], [1] * 40, [127, 1, 128, 129], [64, 64, 31, 33, 32, 300], [1, 639], [513, 2, 1, 1, 61, 130],
           [2050, 1, 200]]


def _run(q, k, v, d_o, seg, impl):
    q, k, v = (t.clone().requires_grad_(True) for t in (q, k, v))
    o = flash_attention(q, k, v, scale=q.shape[-1] ** -0.5, segments=seg, impl=impl)
    return (o.detach(), *torch.autograd.grad(o, (q, k, v), d_o))


@pytest.mark.parametrize("impl", ["tc1", "tc2", "tcg"])
@pytest.mark.parametrize("lengths", LENGTHS)
def test_boundaries(cuda_device, lengths, impl):
    s, g = sum(lengths), torch.Generator().manual_seed(len(lengths))
    ids = torch.repeat_interleave(torch.arange(len(lengths)), torch.tensor(lengths)).int()[None]
    first = torch.tensor([0] + lengths[:-1]).cumsum(0)
    starts = torch.repeat_interleave(first, torch.tensor(lengths)).int()[None]
    q, d_o = (torch.randn(1, 4, s, 64, generator=g).bfloat16().to(cuda_device) for _ in range(2))
    k, v = (torch.randn(1, 2, s, 64, generator=g).bfloat16().to(cuda_device) for _ in range(2))
    seg = PackedMask(seg_id=ids.to(cuda_device), seg_start=starts.to(cuda_device))
    want = _run(q, k, v, d_o, seg, "simt")
    got = _run(q, k, v, d_o, seg, impl)
    for a, b in zip(got, want):
        assert (a - b).abs().max() <= 2e-2 * b.abs().max() + 3e-5
    # starts that are only a lower bound (nothing skipped): the ids alone decide
    loose = PackedMask(seg_id=seg.seg_id, seg_start=torch.zeros_like(seg.seg_start))
    for a, b in zip(_run(q, k, v, d_o, loose, impl), got):
        assert (a - b).abs().max() <= 2e-2 * b.abs().max() + 3e-5


@pytest.mark.parametrize("d", [64, 96, 128])
def test_gradient_in_another_layout(cuda_device, d):
    """d_o as it comes back through `o.transpose(1, 2)` is read where it lies: the same bits as its copy in o's
    layout; layouts the kernels cannot read are copied."""
    g, s = torch.Generator().manual_seed(d), 333
    q, k, v = (torch.randn(2, h, s, d, generator=g).bfloat16().to(cuda_device) for h in (4, 2, 2))
    base = torch.randn(2, s, 4, d + 8, generator=g).bfloat16().to(cuda_device)
    views = [base[..., :d].transpose(1, 2), base[..., 8:].contiguous().transpose(1, 2),
             base[..., 4:d + 4].transpose(1, 2),                      # not 16-byte aligned
             base[:1, :, :, :d].transpose(1, 2).expand(2, 4, s, d)]   # batches share memory
    for d_o in views:
        want = _run(q, k, v, d_o.contiguous(), None, "auto")
        for a, b in zip(_run(q, k, v, d_o, None, "auto"), want):
            assert torch.equal(a, b)
