"""Merging of per-split (max, sum-exp, target) triples: parts around the number the block spreads them over, rows
around a block's 32, against the fp64 logsumexp.  Bound: each part's weight exp(m_p - m) and the sum of `parts`
positive terms are off by (parts + 8) 2^-24 relatively at most, lse by that plus the roundings of m + log s."""
import ctypes as C

import pytest
import torch

from mlx_train_perf_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("parts", [1, 2, 15, 16, 17, 203])
@pytest.mark.parametrize("n", [1, 31, 33, 700])
def test_combine(cuda_device, parts, n):
    g = torch.Generator().manual_seed(parts * 1000 + n)
    m = torch.randn(parts, n, generator=g) * 20
    s = torch.rand(parts, n, generator=g) * 100 + 1e-3
    t = torch.zeros(parts, n)
    t[torch.randint(0, parts, (n,), generator=g), torch.arange(n)] = torch.randn(n, generator=g)
    if parts > 1:                       # a part that holds nothing
        m[0, ::3], s[0, ::3] = float("-inf"), 0.0
    targets = torch.arange(n)
    targets[1::4] = -100
    buf = torch.stack([m, s, t], dim=1).contiguous().to(cuda_device)     # part p: rows m, s, t
    tg, out = targets.to(cuda_device), torch.empty(3, n, device=cuda_device)
    _lib.check(_lib.load().b200tp_linear_ce_combine(
        C.c_void_p(buf.data_ptr()), parts, n, C.c_void_p(tg.data_ptr()), -100, C.c_void_p(out[0].data_ptr()),
        C.c_void_p(out[1].data_ptr()), C.c_void_p(out[2].data_ptr()),
        C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    lse, nll, tgt = out.double().cpu()
    want = torch.logsumexp(m.double() + s.double().log(), dim=0)
    bound = 2.0 ** -24 * (parts + 8 + 2 * want.abs())
    valid = targets != -100
    assert ((lse - want).abs() <= bound).all()
    assert (tgt[valid] == t.sum(0).double()[valid]).all() and (tgt[~valid] == 0).all()
    assert ((nll - (want - tgt)).abs()[valid] <= bound[valid] + 2.0 ** -23 * want.abs()[valid]).all()
    assert (nll[~valid] == 0).all()
