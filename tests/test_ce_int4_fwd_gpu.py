"""The forward that expands a 4-bit head into tensor memory against the chunk-wise form: the same bf16 weights, fp32
accumulation, row sums in another order.  A logit's accumulation rounds towards zero at each of its D / 16 steps, at
2^-23 of the running sum; both forms do, so their logits differ by less than 2 D / 16 such steps of |h| |w|."""
import pytest
import torch

from mlx_train_perf_b200 import configs
from mlx_train_perf_b200.core import loss as L
from mlx_train_perf_b200.core.loss import QuantizedHead

pytestmark = pytest.mark.gpu


# rows around an MMA's 16-row granularity, its 256 columns, a CTA's 320 tokens and several groups of them; vocabularies
# around a 128-row tile; hidden sizes with odd numbers of k blocks, one, and those whose parameters load eight at a time
@pytest.mark.parametrize("params", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize(("n", "d", "v"), [(1, 64, 1), (15, 64, 127), (17, 192, 129), (128, 512, 4000), (255, 320, 3000),
                                           (257, 1024, 20011), (320, 64, 700), (321, 128, 700), (700, 448, 2500)])
def test_against_chunked(cuda_device, n, d, v, params):
    inp = configs.ce_quant(n, d, v, ignore_frac=0.05 if n > 1 else 0.0, seed=n + v)
    head = QuantizedHead(inp.w_q.to(cuda_device), inp.scales.to(params).to(cuda_device),
                         inp.biases.to(params).to(cuda_device))
    h, t = inp.hidden.to(cuda_device), inp.targets.to(cuda_device)
    got = L.ce_forward_raw(h, head, t, v_offset=0, impl="tc")
    want = L.ce_forward_raw(h, head, t, v_offset=0, impl="tc_chunked")
    L.check_device_status()
    z = 2 * (d / 16 + 4) * 2.0 ** -23 * h.float().norm(dim=1).max() * 0.16 * d ** 0.5     # |w| <= 8 scales of 0.02
    for a, b in zip(got[2:], want[2:]):
        assert (a - b).abs().max() <= z + 2.0 ** -22 * b.abs().max()
    # a shard of the vocabulary: targets outside it have no logit here
    off = L.ce_forward_raw(h, head, t, v_offset=v // 2, impl="tc")
    ref = L.ce_forward_raw(h, head, t, v_offset=v // 2, impl="tc_chunked")
    assert ((off[2] == 0) == (ref[2] == 0)).all() and (off[3] - ref[3]).abs().max() <= z + 2.0 ** -22 * ref[3].abs().max()
