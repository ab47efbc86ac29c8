"""The forward that also forms the gradient of a frozen head, against the fp64 evaluation of the oracle.

Bound, per row of d_hidden in the 2-norm: the exponentials are rounded to bf16 before the second contraction
(2^-9 of each term at most, errors independent) and the result is rounded once (2^-9 of each element), so a row is
off by at most 2 x 2^-9 = 4e-3 of its norm unless its terms cancel; 1e-2 leaves room for that.  On top, the target's
term (p - 1) W_t with p = exp(tgt - lse) <= 1 moves by the absolute error of tgt - lse: an error of the target's
logit is in both and cancels, their roundings to fp32 (2^-24 each) and those of the logarithm and the scale (as much
again) do not.  It is what limits rows whose target is certain.
Forward: D / 16 accumulation steps per logit, each off by at most 2^-23 of the running sum, beside the 1e-5 that small
logits are held to.
"""
import pytest
import torch

from mlx_train_perf_b200 import configs
from mlx_train_perf_b200.core import loss as L
from mlx_train_perf_b200.core.loss import DenseHead, QuantizedHead, fused_linear_ce
from oracle import linear_ce as oc

pytestmark = pytest.mark.gpu


def _run(dev, hidden, head, targets, ct):
    h = hidden.to(dev).requires_grad_(True)
    nll, lse, tgt = fused_linear_ce(h, head, targets.to(dev))
    (nll * ct.to(dev)).sum().backward(retain_graph=True)
    first = h.grad.clone()
    h.grad = None
    (nll * ct.to(dev)).sum().backward()
    torch.cuda.synchronize()
    L.check_device_status()
    assert torch.equal(first, h.grad)            # the forward's sums serve a second backward unchanged
    return nll.detach().cpu(), lse.detach().cpu(), tgt.detach().cpu(), h.grad.double().cpu()


def _check(got, hidden, w, targets, ct):
    nll, lse, tgt, dh = got
    r_nll, r_lse, r_tgt = oc.naive_linear_ce(hidden, w, targets, dtype=torch.float64)
    r_dh, _ = oc.chunked_backward(hidden, w, targets, r_lse, ct.double(), chunk_size=4096, dtype=torch.float64)
    top = max(r_lse.abs().max().item(), r_tgt.abs().max().item())
    fwd = 1e-5 + hidden.shape[1] / 16 * 2.0 ** -23 * top
    for x, y in ((nll, r_nll), (lse, r_lse), (tgt, r_tgt)):
        assert (x.double() - y).abs().max().item() < fwd
    ign = targets == configs.IGNORE_INDEX
    assert (dh[ign] == 0).all() and (nll[ign] == 0).all()
    err, norm = (dh - r_dh)[~ign].norm(dim=1), r_dh[~ign].norm(dim=1)
    floor = 2.0 ** -22 * top * ct.double().abs()[~ign] * w[targets[~ign]].double().norm(dim=1)
    assert (err <= 1e-2 * norm + floor).all(), (err / (1e-2 * norm + floor)).max().item()


# rows around a tile, hidden sizes around a k block and a column tile, vocabularies around a tile, dense ones in one
# chunk, the 4-bit ones below over several; few rows share each tile's contraction over many CTAs, many rows do not
SHAPES = [(1, 8, 1), (1, 64, 257), (127, 72, 255), (128, 256, 512), (129, 264, 4099), (60, 1024, 33000),
          (300, 320, 16385), (1500, 136, 2049)]


@pytest.mark.parametrize("certain", [False, True])
@pytest.mark.parametrize(("n", "d", "v"), SHAPES)
def test_dense(cuda_device, n, d, v, certain):
    inp = configs.ce_dense(n, d, v, dtype=torch.bfloat16, ignore_frac=0.05 if n > 1 else 0.0, seed=n + v)
    if certain:      # targets from unlikely to certain: pushed towards their weight rows by up to 30
        t = inp.targets.clamp(min=0)
        push = torch.linspace(0, 30, n)[:, None]
        inp.hidden = (inp.hidden.float() + push * inp.weight[t].float()).to(torch.bfloat16)
    ct = torch.linspace(0.5, 1.5, n) * torch.where(torch.arange(n) % 2 == 0, 1.0, -1.0)
    got = _run(cuda_device, inp.hidden, DenseHead(inp.weight.to(cuda_device), trainable=False), inp.targets, ct)
    if v == 1:       # the loss of the only class is zero and so is its gradient
        assert got[3].abs().max() < 1e-5 and got[0].abs().max() < 1e-5
        return
    _check(got, inp.hidden, inp.weight, inp.targets, ct)


@pytest.mark.parametrize("params", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize(("n", "d", "v"), [(1, 64, 300), (130, 320, 4099), (70, 128, 40000)])
def test_int4(cuda_device, n, d, v, params):
    inp = configs.ce_quant(n, d, v, ignore_frac=0.05 if n > 1 else 0.0, seed=v)
    sc, bi = inp.scales.to(params), inp.biases.to(params)
    w = oc.dequantize_int4(inp.w_q, sc, bi, out_dtype=torch.bfloat16)
    head = QuantizedHead(*(x.to(cuda_device) for x in (inp.w_q, sc, bi)))
    ct = torch.full((n,), 1.0 / n)
    _check(_run(cuda_device, inp.hidden, head, inp.targets, ct), inp.hidden, w, inp.targets, ct)


@pytest.mark.parametrize("quant", [False, True])
@pytest.mark.parametrize("scale", [20.0, 200.0])
def test_logits_far_above_the_target(cuda_device, quant, scale):
    """Logits 70 and more above the target's leave the range of the fixed reference: the backward then computes
    them again.  At 20 some rows do, at 200 all; ignored rows' logits (reference: vocab row 0) do as well, to no effect."""
    n, d, v = 200, 128, 20000
    if quant:
        inp = configs.ce_quant(n, d, v, ignore_frac=0.1, seed=3)
        w = oc.dequantize_int4(inp.w_q, inp.scales, inp.biases, out_dtype=torch.bfloat16)
        head = QuantizedHead(*(x.to(cuda_device) for x in (inp.w_q, inp.scales, inp.biases)))
    else:
        inp = configs.ce_dense(n, d, v, dtype=torch.bfloat16, ignore_frac=0.1, seed=3)
        w, head = inp.weight, DenseHead(inp.weight.to(cuda_device), trainable=False)
    hidden = (inp.hidden.float() * scale).to(torch.bfloat16)
    ct = torch.full((n,), 1.0 / n)
    got = _run(cuda_device, hidden, head, inp.targets, ct)
    nll, lse, _, dh = got
    r_nll, r_lse, _ = oc.naive_linear_ce(hidden, w, inp.targets, dtype=torch.float64)
    assert r_nll.max() > 80
    r_dh, _ = oc.chunked_backward(hidden, w, inp.targets, r_lse, ct.double(), chunk_size=4096, dtype=torch.float64)
    # fp32 sums of 128 products of size up to 4 scale: 2^-24 of the largest partial sum per addition
    assert ((lse.double() - r_lse).abs() <= 2e-6 * scale * 4).all()
    assert torch.isfinite(nll).all()
    # a probability moves by the absolute error of its logit, and g is rounded to bf16
    assert ((dh - r_dh).norm() / r_dh.norm()).item() < 1e-2


def test_no_gradient_wanted_runs_the_plain_forward(cuda_device):
    inp = configs.ce_dense(100, 128, 3000, dtype=torch.bfloat16, seed=1)
    head = DenseHead(inp.weight.to(cuda_device), trainable=False)
    h, t = inp.hidden.to(cuda_device), inp.targets.to(cuda_device)
    a = fused_linear_ce(h, head, t)
    b = fused_linear_ce(h.clone().requires_grad_(True), head, t)
    assert a[0].grad_fn is None and b[0].grad_fn is not None
    for x, y in zip(a, b):
        assert (x - y.detach()).abs().max().item() < 1e-5


@pytest.mark.parametrize("operand", ["hidden", "weight"])
def test_misaligned_operands_are_refused(cuda_device, operand):
    """Before any kernel reads them: the row kernels load whole 16-byte words."""
    from mlx_train_perf_b200.errors import LossInputError
    n, d, v = 40, 64, 300
    h = torch.zeros(n * d + 1, dtype=torch.bfloat16, device=cuda_device)[1:].reshape(n, d)
    w = torch.zeros(v * d + 1, dtype=torch.bfloat16, device=cuda_device)[1:].reshape(v, d)
    h, w = (h, w.clone()) if operand == "hidden" else (h.clone(), w)
    assert (h.data_ptr() | w.data_ptr()) % 16 != 0
    t = torch.zeros(n, dtype=torch.int64, device=cuda_device)
    with pytest.raises(LossInputError, match="16-byte aligned"):
        fused_linear_ce(h.requires_grad_(True), DenseHead(w, trainable=False), t)
    with pytest.raises(LossInputError, match="16-byte aligned"):
        fused_linear_ce(h.detach(), DenseHead(w, trainable=False), t)


@pytest.mark.parametrize("kind", ["dense", "quant", "fp32"])
def test_ignored_rows_do_not_void_the_sums(cuda_device, kind):
    """Their gradient is zero whatever their logits are; the reference of such a row is the logit of vocab row 0."""
    n, d, v = 200, 128, 20000
    if kind == "quant":
        inp = configs.ce_quant(n, d, v, seed=3)
        w = oc.dequantize_int4(inp.w_q, inp.scales, inp.biases, out_dtype=torch.bfloat16)
        head = QuantizedHead(*(x.to(cuda_device) for x in (inp.w_q, inp.scales, inp.biases)))
    else:
        inp = configs.ce_dense(n, d, v, dtype=torch.float32 if kind == "fp32" else torch.bfloat16, seed=3)
        w, head = inp.weight, DenseHead(inp.weight.to(cuda_device), trainable=False)
    t = inp.targets.clone()
    t[::3] = configs.IGNORE_INDEX
    ign = t == configs.IGNORE_INDEX
    hidden = torch.where(ign[:, None], inp.hidden.float() * 200, inp.hidden.float()).to(inp.hidden.dtype)
    ct = torch.full((n,), 1.0 / n)
    impl = "split" if kind == "fp32" else "tc"
    hd, td = hidden.to(cuda_device), t.to(cuda_device)
    rows, state = L.ce_forward_grad(hd, head, td, impl=impl)
    dh = L.ce_backward_grad(hd, head, td, rows, state, ct.to(cuda_device), impl=impl)
    L.check_device_status()
    r_nll, r_lse, _ = oc.naive_linear_ce(hidden, w, t, dtype=torch.float64)
    zmax = (hidden.double() @ w.double().T).max(dim=1).values - hidden.double() @ w.double()[0]
    assert zmax[ign].max() > 80 and r_nll.max() < 60
    assert state[:4].view(torch.int32).item() == 0
    # D / 16 accumulation steps at 2^-23 of the running sum, |h| |w| at most, and the roundings of lse
    z = (d / 16 + 4) * 2.0 ** -23 * hidden.double().norm(dim=1) * w.double().norm(dim=1).max()
    assert ((rows[1].double().cpu() - r_lse).abs() <= z + 2.0 ** -22 * r_lse.abs()).all()
    r_dh, _ = oc.chunked_backward(hidden, w, t, r_lse, ct.double(), chunk_size=4096, dtype=torch.float64)
    assert (dh[ign.to(cuda_device)] == 0).all()
    assert ((dh.double().cpu() - r_dh).norm() / r_dh.norm()).item() < 1e-2


@pytest.mark.parametrize(("kind", "n", "d"), [("bf16", 4, 64), ("fp32", 4, 64), ("fp32", 128, 1024)])
@pytest.mark.parametrize(("weight", "ct"), [(3e9, 1.0), (1.0, 1e-20)])
def test_products_at_the_ends_of_fp32(cuda_device, kind, n, d, weight, ct):
    """Logits 66 above the target's are inside the reference's range; 3000 exponentials of e^66 times weights of 3e9 are
    not inside fp32's, and exp(ref - lse) times a cotangent of 1e-20 is not either.  p = 1 / 2999 everywhere but at the
    target, so d_hidden = ct (mean of the other rows - W_t), to the rounding of p and of the result (2^-9 each; fp32:
    (9 + 3000 / 128) 2^-23 for the sum) and what 2^-22 of lse = 74 moves p by."""
    v = 3000
    dtype = torch.bfloat16 if kind == "bf16" else torch.float32
    w, h = torch.zeros(v, d), torch.zeros(n, d)
    w[:, 0], w[:, 1] = 1.0, weight
    w[7] = 0.0
    h[:, 0] = 66.0
    t = torch.full((n,), 7)
    impl = "tc" if kind == "bf16" else "split"
    hd, td, head = (h.to(dtype).to(cuda_device), t.to(cuda_device),
                    DenseHead(w.to(dtype).to(cuda_device), trainable=False))
    rows, state = L.ce_forward_grad(hd, head, td, impl=impl)
    for _ in range(2):
        dh = L.ce_backward_grad(hd, head, td, rows, state, torch.full((n,), ct, device=cuda_device), impl=impl)
        L.check_device_status()
        want = torch.zeros(n, d, dtype=torch.float64)
        want[:, 0], want[:, 1] = ct, ct * float(torch.tensor(weight).to(dtype))
        tol = 1e-2 if kind == "bf16" else 1e-4
        assert ((dh.double().cpu() - want).abs() <= tol * want.abs()).all(), dh[:, :2]


def test_accumulations_are_short(cuda_device):
    """Hidden states of zero make every exponential 1, so a row's sum in `state` is that of the weights but the target's.
    One large row and many small ones: where the large one is in the accumulator, a step of 16 rows loses up to an ulp
    (2^-23) of it towards zero, 1024 x 2^-23 in an accumulation of 16384 rows (over all 131072, which are one chunk and
    one share here, eight times as much); the parts' sums and the small rows add 2 % at most."""
    n, d, v, dev = 1000, 4096, 131072, cuda_device
    w = torch.randn(v, d, generator=torch.Generator(device=dev).manual_seed(v), device=dev) * 2.0 ** -8
    w[17] = 300 * torch.randn(d, generator=torch.Generator(device=dev).manual_seed(17), device=dev)
    w = w.to(torch.bfloat16)
    h, t = torch.zeros(n, d, dtype=torch.bfloat16, device=dev), torch.full((n,), 5, device=dev)
    _, state = L.ce_forward_grad(h, DenseHead(w, trainable=False), t)
    L.check_device_status()
    at = 256 + (4 * n + 255) // 256 * 256
    sums = state[at:at + (state.numel() - at) // (4 * n * d) * (4 * n * d)].view(torch.float32).reshape(-1, n, d)
    assert sums.shape[0] == 1
    want = w.sum(dim=0, dtype=torch.float64) - w[5].double()
    rel = (sums[0].double() - want).norm(dim=1) / want.norm()
    assert rel.max().item() <= 1.02 * 1024 * 2.0 ** -23, rel.max().item() * 2.0 ** 23


@pytest.mark.parametrize("what", ["targets out of range", "inf weight", "nan hidden"])
def test_values_outside_the_ordinary(cuda_device, what):
    """What the recomputing pair gives: a target outside the vocabulary has no logit (loss = lse, d_hidden = ct sum of
    p W); a value that is not finite reaches the same rows, as one that is not finite."""
    n, d, v = 130, 64, 700
    inp = configs.ce_dense(n, d, v, dtype=torch.bfloat16, ignore_frac=0.05, seed=5)
    h, w, t = inp.hidden.clone(), inp.weight.clone(), inp.targets.clone()
    if what == "targets out of range":
        t[3], t[9] = v, -7
    elif what == "inf weight":
        t[3] = 5                                  # (also the logit of a target)
        w[5], w[5, 3] = 0, float("-inf")
        h[:, 3] = h[:, 3].abs() + 0.1
    else:
        h[7, 2] = float("nan")
    hd, td, head = h.to(cuda_device), t.to(cuda_device), DenseHead(w.to(cuda_device), trainable=False)
    ct = torch.full((n,), 0.5, device=cuda_device)
    rows, state = L.ce_forward_grad(hd, head, td)
    dh = L.ce_backward_grad(hd, head, td, rows, state, ct)
    _, _, tgt, lse, nll = L.ce_forward_raw(hd, head, td, impl="tc")
    want = L.ce_backward_raw(hd, head, td, lse, ct, impl="tc")
    L.check_device_status()
    # sums of the same logits in another order; g rounded to bf16 in one and its exponentials in the other (see above)
    for a, b in ((rows[0], tgt), (rows[1], lse), (rows[2], nll)):
        assert torch.equal(a.isfinite(), b.isfinite())
        ok = b.isfinite()
        assert (a[ok] - b[ok]).abs().max() <= 1e-5 * (1 + b[ok].abs().max())
    ok = want.isfinite()      # (not where a g of zero meets an infinite weight: ignored rows too)
    assert torch.equal(dh.isfinite(), ok)
    a, b = dh.double()[ok], want.double()[ok]
    assert (a - b).norm() <= 1e-2 * b.norm()


# single CTAs and pairs, with shares (some of which the narrower last chunk leaves empty) and without
@pytest.mark.parametrize(("n", "d", "v", "units"), [(60, 1024, 5000, 4), (129, 264, 4099, 1), (300, 320, 2561, 2),
                                                    (256, 2056, 3000, 3), (2177, 264, 2600, 4), (1500, 2112, 1100, 2)])
def test_dense_over_several_chunks(cuda_device, monkeypatch, n, d, v, units):
    """A chunk bound of `units` x 256 vocabulary rows: sums added up over the chunks, shares among them."""
    monkeypatch.setitem(L._RESERVED, "tc", units)
    inp = configs.ce_dense(n, d, v, dtype=torch.bfloat16, ignore_frac=0.05, seed=n + v)
    ct = torch.linspace(0.5, 1.5, n) * torch.where(torch.arange(n) % 2 == 0, 1.0, -1.0)
    _check(_run(cuda_device, inp.hidden, DenseHead(inp.weight.to(cuda_device), trainable=False), inp.targets, ct),
           inp.hidden, inp.weight, inp.targets, ct)
