"""Dense bf16 losses at sizes that run on CTA pairs (an even number of 128-row blocks with D >= 2048, or 16 blocks and
more), against the fp64 evaluation of the oracle: last blocks of one row, a last pair of one block, partial vocab and
column tiles, several chunks, both forms of the gradient and a trained head's.

Bounds: forward, D / 16 accumulation steps at 2^-23 of the running sum, |h| |w| at most; gradients, g and the result are
rounded to bf16 (2^-9 of each term and of each element, so 4e-3 of a row's or column's norm; 1e-2 leaves room for
cancellation) beside what the forward's error moves g by."""
import pytest
import torch

from mlx_train_perf_b200 import configs
from mlx_train_perf_b200.core import loss as L
from mlx_train_perf_b200.core.loss import DenseHead, fused_linear_ce
from oracle import linear_ce as oc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize(("n", "d", "v"), [(129, 2048, 300), (256, 2056, 257), (500, 2176, 16640), (2049, 72, 700),
                                           (2177, 264, 1000), (3000, 128, 255)])
def test_against_fp64(cuda_device, n, d, v):
    inp = configs.ce_dense(n, d, v, dtype=torch.bfloat16, ignore_frac=0.05, seed=n + v)
    ct = torch.linspace(0.5, 1.5, n) * torch.where(torch.arange(n) % 2 == 0, 1.0, -1.0)
    r_nll, r_lse, r_tgt = oc.naive_linear_ce(inp.hidden, inp.weight, inp.targets, dtype=torch.float64)
    r_dh, r_dw = oc.chunked_backward(inp.hidden, inp.weight, inp.targets, r_lse, ct.double(), chunk_size=4096,
                                     dtype=torch.float64, want_dw=True)
    z = (d / 16 + 4) * 2.0 ** -23 * inp.hidden.float().norm(dim=1).max() * inp.weight.float().norm(dim=1).max()
    fwd = float(z) + 2.0 ** -22 * r_lse.abs().max().item()
    dev, ign = cuda_device, inp.targets == configs.IGNORE_INDEX
    for trained in (False, True):
        w = inp.weight.to(dev).requires_grad_(trained)
        h = inp.hidden.to(dev).requires_grad_(True)
        nll, lse, tgt = fused_linear_ce(h, DenseHead(w, trainable=trained), inp.targets.to(dev))
        grads = torch.autograd.grad(nll, [h, w] if trained else [h], ct.to(dev))
        L.check_device_status()
        for x, y in ((nll, r_nll), (lse, r_lse), (tgt, r_tgt)):
            assert (x.detach().double().cpu() - y).abs().max().item() <= fwd
        dh = grads[0].double().cpu()
        assert (dh[ign] == 0).all()
        assert ((dh - r_dh).norm(dim=1) <= (1e-2 + 2 * fwd) * r_dh.norm(dim=1)).all()
        if trained:
            dw = grads[1].double().cpu()
            assert ((dw - r_dw).norm(dim=1) <= (1e-2 + 2 * fwd) * r_dw.norm(dim=1) + 1e-3 * r_dw.norm(dim=1).mean()).all()
