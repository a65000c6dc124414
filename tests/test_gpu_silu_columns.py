"""The gated product's quantizer on both sides of the line from four to eight elements a thread (2048 threads an SM), through routed layers."""
import numpy as np
import pytest

import oracle_lib as O
from gpu_util import assert_bits, need_gpu
from test_gpu_moe import _layer, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ff,beyond", [(2048, -1), (2048, 0), (2080, 0)])  # just below, at the line, a last CTA that is not full
def test_gated_product_of_many_columns(ff, beyond):
    torch = need_gpu()
    import cera_b200 as cb
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    _run(cb.Q8_0, n_expert=4, n_used=2, hidden=64, ff=ff, n=-(-sms * 16384 // (2 * ff)) + beyond, seed=71)


# The quants, scales and sums of the halves (Q4_1, Q4_K: the minimum's term) all enter the down rows, which a call of fewer than sixteen tokens forms
# token by token: the parts, below the line, give the same bits.  Tokens' sizes bring gates through +-88 and +-134, and to zero, infinity and NaN
@pytest.mark.parametrize("t", [O.Q4_1, O.Q4_K, O.Q8_0])
def test_eight_elements_equal_four(t):
    torch = need_gpu()
    import cera_b200 as cb
    n, experts, hidden = 15, 16, 256
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    ff = -(-sms * 16384 // (n * experts * 256)) * 256
    assert n * experts * ff >= sms * 16384 > 8 * experts * ff
    moe = cb.MoeFfn(experts, experts, hidden, ff, t, *_layer(t, experts, hidden, ff, 5), max_tokens=n)
    x = O.synth_normal(n * hidden, 6, 1.0).reshape(n, hidden)
    x *= np.float32([0, 1e-6, 1e-3, 0.03, 0.3, 1, 3, 10, 40, 90, 130, 200, 300, 1, 1])[:, None]
    x[13, 7], x[14, 9] = np.inf, np.nan
    x[14, 40] = -np.inf
    x = torch.from_numpy(x).cuda()
    whole = moe(x).cpu().numpy()
    parts = np.concatenate([moe(x[:7]).cpu().numpy(), moe(x[7:]).cpu().numpy()])
    nan = np.isnan(parts)
    assert np.array_equal(np.isnan(whole), nan) and not nan[:13].any()
    assert np.isfinite(whole[:13]).all() and np.abs(whole[12]).max() > 1e3 * np.abs(whole[5]).max()
    assert_bits(np.where(nan, 0, whole), np.where(nan, 0, parts), O.NAMES[t])
    moe.close()
