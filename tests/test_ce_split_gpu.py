"""fp32 losses on the tensor cores (three bf16 planes an operand) against fp64 and against the CUDA-core kernels.

Bounds: a logit is a sum of D exact products, dropped terms below 2^-25 of each; its segments of 128 round towards
zero at most nine times at 2^-23 of the running sum, and there are D / 128 additions of them: (9 + D / 128) 2^-23 of the
largest partial sum, |h| |w| at most.  Probabilities move by that, d_hidden rows by it times sum_v |g_v| |W_v|, plus
the same for the second contraction over V."""
import math

import pytest
import torch

from mlx_train_perf_b200 import parallel
from mlx_train_perf_b200.core import loss as L
from mlx_train_perf_b200.core.loss import DenseHead, fused_linear_ce, reduced_linear_cross_entropy
from oracle import linear_ce as oc

pytestmark = pytest.mark.gpu


def _inputs(n, d, v):
    g = torch.Generator().manual_seed(n + d + v)
    w = torch.randn(v, d, generator=g) * d ** -0.5
    h = torch.randn(n, d, generator=g)
    t = torch.randint(0, v, (n,), generator=g)
    h += torch.linspace(0, 20, n)[:, None] * w[t]
    t[2::7] = -100
    return h, w, t


def _run(dev, h, w, t, ct, impl="split"):
    h, t, head = h.to(dev), t.to(dev), DenseHead(w.to(dev), trainable=False)
    _, _, tgt, lse, nll = L.ce_forward_raw(h, head, t, impl=impl)
    dh = L.ce_backward_raw(h, head, t, lse, ct.to(dev), impl=impl)
    L.check_device_status()
    return nll.cpu(), lse.cpu(), tgt.cpu(), dh.cpu()


# rows, hidden sizes and vocabularies around tiles, k blocks and accumulator segments; several chunks; shares
@pytest.mark.parametrize(("n", "d", "v"), [(1, 8, 1), (1, 64, 257), (127, 72, 255), (128, 128, 512), (129, 136, 4099),
                                           (60, 1024, 17000), (300, 264, 2500), (33, 2056, 600)])
def test_against_fp64(cuda_device, n, d, v):
    h, w, t = _inputs(n, d, v)
    ct = torch.linspace(-1, 1.5, n)
    nll, lse, tgt, dh = _run(cuda_device, h, w, t, ct)
    r_nll, r_lse, r_tgt = oc.naive_linear_ce(h, w, t, dtype=torch.float64)
    r_dh, _ = oc.chunked_backward(h, w, t, r_lse, ct.double(), chunk_size=4096, dtype=torch.float64)
    rows = h.double().norm(dim=1) * w.double().norm(dim=1).max()
    z = (9 + d / 128) * 2.0 ** -23 * rows + 2.0 ** -22 * (1 + r_lse.abs())
    ok = t != -100
    assert ((lse.double() - r_lse).abs() <= z).all()
    assert ((tgt.double() - r_tgt).abs() <= z)[ok].all() and ((nll.double() - r_nll).abs() <= 2 * z)[ok].all()
    assert (nll[~ok] == 0).all() and (dh[~ok] == 0).all()
    wn = w.double().norm(dim=1).max()
    bound = ct.double().abs() * wn * 2 * (z + (9 + v / 128) * 2.0 ** -23)
    assert ((dh.double() - r_dh).norm(dim=1) <= bound + 1e-12).all()
    # no less precise than the CUDA cores, up to the last rounding of the results
    s_nll, s_lse, _, s_dh = _run(cuda_device, h, w, t, ct, impl="simt")
    assert (lse.double() - r_lse).norm() <= (s_lse.double() - r_lse).norm() + 2.0 ** -24 * r_lse.norm()
    assert (dh.double() - r_dh).norm() <= (s_dh.double() - r_dh).norm() + 2.0 ** -24 * r_dh.norm()


def test_accumulates_into_fp32(cuda_device):
    h, w, t = _inputs(70, 264, 5000)
    dev, ct = cuda_device, torch.ones(70)
    head = DenseHead(w.to(dev), trainable=False)
    out = L.ce_forward_buffer(h.to(dev), head, t.to(dev), impl="split")
    base = torch.randn(70 * 264 + 1, device=dev)[1:].reshape(70, 264)      # not 16-byte aligned
    buf = torch.empty(70 * 264 + 1, device=dev)[1:].reshape(70, 264).copy_(base)
    one = L.ce_backward_raw(h.to(dev), head, t.to(dev), out[3], ct.to(dev), impl="split")
    L.ce_backward_raw(h.to(dev), head, t.to(dev), out[3], ct.to(dev), out=buf, accumulate=True,
                      out_dtype=torch.float32, impl="split")
    assert torch.equal(buf, base + one)        # added once, after the shares' own sum


@pytest.mark.parametrize("what", ["inf", "nan", "largest", "cotangent"])
def test_values_without_planes(cuda_device, what):
    """bf16 cannot hold them: the CUDA-core kernels give the result, bit for bit theirs."""
    h, w, t = _inputs(40, 64, 700)
    ct = torch.ones(40)
    if what == "inf":
        w[5] = 0
        w[5, 3] = -math.inf
        h[:, 3] = h[:, 3].abs() + 0.1
    elif what == "nan":
        h[7, 2] = math.nan
    elif what == "largest":
        w[9] = 0
        w[9, 1] = -3.4e38
        h[:, 1] = h[:, 1].abs().clamp(max=0.9)
    else:
        ct[3] = math.inf
    for a, b in zip(_run(cuda_device, h, w, t, ct), _run(cuda_device, h, w, t, ct, impl="simt")):
        if what == "cotangent" and a.ndim == 1:
            continue                      # the forward saw no such value
        if what == "cotangent":           # nor did the saved lse come from the same kernels
            assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isinf(), b.isinf())
            continue
        assert torch.equal(a.nan_to_num(7e7), b.nan_to_num(7e7))


@pytest.mark.parametrize(("n", "d", "v", "push"), [(1, 64, 257, 3.0), (129, 136, 4099, 20.0), (60, 1024, 17000, 20.0),
                                                   (40, 264, 2500, -90.0)])
def test_forward_that_forms_the_gradient(cuda_device, n, d, v, push):
    """Same bounds as above; at push -90 logits lie 69 and more above the target's and the CUDA cores take over."""
    dev, (h, w, t) = cuda_device, _inputs(n, d, v)
    h = h + torch.linspace(0, push - 20, n)[:, None] * w[t]
    ct = torch.linspace(-1, 1.5, n)
    r_nll, r_lse, _ = oc.naive_linear_ce(h, w, t, dtype=torch.float64)
    r_dh, _ = oc.chunked_backward(h, w, t, r_lse, ct.double(), chunk_size=4096, dtype=torch.float64)
    assert push > 0 or r_nll.max() > 75
    hd, td, head = h.to(dev), t.to(dev), DenseHead(w.to(dev), trainable=False)
    rows, state = L.ce_forward_grad(hd, head, td, impl="split")
    got = [L.ce_backward_grad(hd, head, td, rows, state, ct.to(dev), impl="split") for _ in range(2)]
    L.check_device_status()
    assert torch.equal(got[0], got[1])
    s_nll, s_lse, _, s_dh = _run(dev, h, w, t, ct, impl="simt")
    if push < 0:
        for a, b in ((rows[1], s_lse), (rows[2], s_nll), (got[0], s_dh)):
            assert torch.equal(a.cpu(), b)
        return
    _, lse, nll = rows.double().cpu()
    dh, ok = got[0].double().cpu(), t != -100
    z = (9 + d / 128) * 2.0 ** -23 * h.double().norm(dim=1) * w.double().norm(dim=1).max() + 2.0 ** -22 * (1 + r_lse.abs())
    assert ((lse - r_lse).abs() <= z).all() and ((nll - r_nll).abs() <= 2 * z)[ok].all()
    wn = w.double().norm(dim=1).max()
    assert ((dh - r_dh).norm(dim=1) <= ct.double().abs() * wn * 2 * (2 * z + (9 + v / 128) * 2.0 ** -23) + 1e-12).all()
    # no less precise than the recomputing form, up to the last rounding of the results
    assert (dh - r_dh).norm() <= (s_dh.double() - r_dh).norm() + 2.0 ** -24 * r_dh.norm()


def test_forward_that_forms_the_gradient_without_planes(cuda_device):
    h, w, t = _inputs(40, 64, 700)
    w[5] = 0
    w[5, 3] = -math.inf
    h[:, 3] = h[:, 3].abs() + 0.1
    dev, ct = cuda_device, torch.ones(40)
    hd, td, head = h.to(dev), t.to(dev), DenseHead(w.to(dev), trainable=False)
    rows, state = L.ce_forward_grad(hd, head, td, impl="split")
    dh = L.ce_backward_grad(hd, head, td, rows, state, ct.to(dev), impl="split")
    nll, lse, tgt, s_dh = _run(dev, h, w, t, ct, impl="simt")
    for a, b in ((rows[0], tgt), (rows[1], lse), (rows[2], nll), (dh, s_dh)):
        assert torch.equal(a.cpu().nan_to_num(7e7), b.nan_to_num(7e7))


def test_trained_head_keeps_one_kind_of_logits(cuda_device):
    """A size that would be split: with the head trained, forward and backward are the CUDA-core ones."""
    n, d, v = 300, 1024, 1000
    h, w, t = (x.to(cuda_device) for x in _inputs(n, d, v))
    out = []
    for impl in ("auto", "simt"):
        hh, ww = h.clone().requires_grad_(True), w.clone().requires_grad_(True)
        nll, lse, _ = fused_linear_ce(hh, DenseHead(ww), t, impl=impl)
        loss, _ = reduced_linear_cross_entropy(hh, DenseHead(ww), t, impl=impl)
        out.append((nll.detach(), lse, loss.detach(), *torch.autograd.grad(nll.sum(), (hh, ww)),
                    *torch.autograd.grad(loss, (hh, ww))))
    for a, b in zip(*out):
        assert torch.equal(a, b)
    assert n * d * v >= 2 ** 28 and not torch.equal(fused_linear_ce(h, DenseHead(w, trainable=False), t)[1], out[0][1])


def test_trained_shards_keep_one_kind_of_logits(cuda_device, monkeypatch):
    """The vocabulary-sharded operator with d_weight, two shards that would each be split: lse and the gradients come from
    the same logits, so the distance to fp64 is no larger than the CUDA cores', up to the last rounding of the results."""
    n, d, v = 128, 1024, 4099
    (h, w, t), ct = _inputs(n, d, v), torch.linspace(-1, 1.5, n)
    _, r_lse, _ = oc.naive_linear_ce(h, w, t, dtype=torch.float64)
    r_dh, r_dw = oc.chunked_backward(h, w, t, r_lse, ct.double(), chunk_size=4096, dtype=torch.float64, want_dw=True)
    hd, td, ctd = h.to(cuda_device), t.to(cuda_device), ct.to(cuda_device)
    shards = [parallel.shard_dense_head(w.to(cuda_device), 2, rank) for rank in range(2)]
    assert min(head.weight.shape[0] for head, _ in shards) * n * d >= 2 ** 28
    err = {}
    for impl in ("auto", "simt"):
        ops = [parallel.VocabShardedLinearCE(head, lo, impl=impl) for head, lo in shards]
        parts = torch.stack([L.ce_forward_buffer(hd, head, td, v_offset=lo, impl=impl, want_lse=False)[:3]
                             for head, lo in shards])
        monkeypatch.setattr(parallel, "gather_partials", lambda local, group=None: parts)
        dh, dw = torch.zeros(n, d, dtype=torch.float64), []
        for op in ops:
            monkeypatch.setattr(op, "_reduce", lambda partial, dtype: partial)
            _, lse, _ = op.forward(hd, td)
            dw.append(torch.full_like(op.head.weight, float("nan")))
            dh += op.backward(hd, td, lse, ctd, d_weight=dw[-1]).double().cpu()
        L.check_device_status()
        err[impl] = [(dh - r_dh).norm(), (torch.cat(dw).double().cpu() - r_dw).norm()]
    for got, cores, ref in zip(err["auto"], err["simt"], (r_dh, r_dw)):
        assert got <= cores + 2.0 ** -24 * ref.norm(), (float(got / ref.norm()), float(cores / ref.norm()))


@pytest.mark.parametrize(("n", "d", "v", "what"), [(1, 8, 1, "planes"), (129, 136, 4099, "planes"),
                                                   (300, 264, 25000, "planes"), (129, 136, 4095, "inf")])
def test_gradient_of_the_weight(cuda_device, n, d, v, what):
    """Against the CUDA cores' d_weight; with a value that has no planes it is theirs, bit for bit (one chunk).  Bound: g moves by
    the errors of z and lse (as above, for both kinds), the sum over n rows by n 2^-24 of its terms, for both."""
    h, w, t = _inputs(n, d, v)
    if what == "inf":
        w[0] = 0
        w[0, 3] = -math.inf
        h[:, 3] = h[:, 3].abs() + 0.1
    ct, out = torch.linspace(-1, 1.5, n).to(cuda_device), []
    hd, td, head = h.to(cuda_device), t.to(cuda_device), DenseHead(w.to(cuda_device))
    for impl in ("split", "simt"):
        lse = L.ce_forward_raw(hd, head, td, impl=impl)[3]
        dw = torch.full_like(head.weight, 7.0)
        dh = L.ce_backward_raw(hd, head, td, lse, ct, impl=impl, d_weight=dw)
        out.append((dh.cpu(), dw.cpu()))
    L.check_device_status()
    if what == "inf":
        for a, b in zip(*out):
            assert torch.equal(a.nan_to_num(7e7), b.nan_to_num(7e7))
        return
    z = (9 + d) * 2.0 ** -23 * (h.norm(dim=1) * w.norm(dim=1).max()).max() + 2.0 ** -20
    terms = ct.abs().cpu() @ h.abs()                  # a row of d_weight, were every |g| as large as |ct|
    assert ((out[0][1] - out[1][1]).abs() <= (4 * z + n * 2.0 ** -23) * terms + 1e-12).all()


@pytest.mark.parametrize("what", ["one row", "all rows", "no planes"])
def test_void_sums_of_a_large_call(cuda_device, what):
    """Logits 69 and more above a target's, at a size where the planes are the faster form: the backward computes them
    again from planes, bit for bit as the recomputing backward does from the same lse, and the CUDA cores give the result
    only where a value has none."""
    n, d, v = 200, 1024, 2600
    dev, (h, w, t) = cuda_device, _inputs(n, d, v)
    assert n * d * v >= 2 ** 28
    if what == "no planes":
        w[5] = 0
        w[5, 3] = -math.inf
        h[:, 3] = h[:, 3].abs() + 0.1
    else:
        rows = slice(17, 18) if what == "one row" else slice(None)
        h[rows] += -110.0 * w[t[rows].clamp(min=0)]
    ct = torch.linspace(-1, 1.5, n)
    hd, td, head = h.to(dev), t.to(dev), DenseHead(w.to(dev), trainable=False)
    rows, state = L.ce_forward_grad(hd, head, td, impl="auto")
    got = [L.ce_backward_grad(hd, head, td, rows, state, ct.to(dev), impl="auto") for _ in range(2)]
    L.check_device_status()
    assert torch.equal(got[0].nan_to_num(7e7), got[1].nan_to_num(7e7))
    flags = state[:12].view(torch.int32).tolist()
    s_nll, s_lse, _, s_dh = _run(dev, h, w, t, ct, impl="simt")
    if what == "no planes":
        assert flags == [1, 1, 1]
        for a, b in ((rows[1], s_lse), (rows[2], s_nll), (got[0], s_dh)):
            assert torch.equal(a.cpu().nan_to_num(7e7), b.nan_to_num(7e7))
        return
    assert flags == [1, 0, 0]
    assert torch.equal(got[0], L.ce_backward_raw(hd, head, td, rows[1], ct.to(dev), impl="auto"))
    r_nll, r_lse, _ = oc.naive_linear_ce(h, w, t, dtype=torch.float64)
    r_dh, _ = oc.chunked_backward(h, w, t, r_lse, ct.double(), chunk_size=4096, dtype=torch.float64)
    assert r_nll.max() > 75
    lse, dh = rows[1].double().cpu(), got[0].double().cpu()
    assert (lse - r_lse).norm() <= (s_lse.double() - r_lse).norm() + 2.0 ** -24 * r_lse.norm()
    assert (dh - r_dh).norm() <= (s_dh.double() - r_dh).norm() + 2.0 ** -24 * r_dh.norm()


@pytest.mark.parametrize("n", [16, 130])
def test_target_logit_that_overflows(cuda_device, n):
    """Finite operands whose product is below fp32's range: the target's logit is -inf, its row's loss +inf, everything
    else finite, as on the CUDA cores (the larger call would compute void sums again from planes)."""
    d, v, dev = 1024, 2100, cuda_device
    h, w, t = _inputs(n, d, v)
    w[5], h[:, 3], t[4] = 0, 3.0, 5
    w[5, 3] = -3e38
    ct = torch.linspace(-1, 1.5, n)
    hd, td, head = h.to(dev), t.to(dev), DenseHead(w.to(dev), trainable=False)
    rows, state = L.ce_forward_grad(hd, head, td, impl="split")
    dh = L.ce_backward_grad(hd, head, td, rows, state, ct.to(dev), impl="split").cpu()
    nll, lse, tgt, s_dh = _run(dev, h, w, t, ct, impl="simt")
    assert nll[4].item() == math.inf and lse.isfinite().all()
    for a, b in ((rows[0], tgt), (rows[1], lse), (rows[2], nll), (dh, s_dh)):
        a, ok = a.cpu(), b.isfinite()
        assert torch.equal(a.isfinite(), ok) and torch.equal(a[~ok], b[~ok])
        a, b, ok = (x[torch.arange(n) != 4] for x in (a, b, ok))        # (that row of d_hidden holds 1e38)
        # logits of up to 40 at (9 + D) 2^-23 of themselves for both kinds: 1e-2 of a probability at most
        assert (a[ok] - b[ok]).norm() <= 1e-2 * b[ok].norm()
