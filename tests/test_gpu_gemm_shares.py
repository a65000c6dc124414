"""Products whose last round of tiles is shared out along k, and that pairs of CTAs do, against the same rows in a small product."""
import numpy as np
import pytest

import oracle_lib as O
from gpu_util import need_gpu

pytestmark = pytest.mark.gpu


# tiles beyond a multiple of the SMs: the fewest (most shares of a tile) and as many as two shares each leave room for; ragged rows and tokens
@pytest.mark.parametrize("t", [O.Q4_K, O.Q5_K, O.Q6_K])
@pytest.mark.parametrize("rows,x_tiles,beyond,k", [(256, 4, 1, 2048), (256, 4, 71, 2304), (128, 3, 2, 4352), (128, 8, 5, 2048), (128, 8, 66, 2048)])
def test_shared_tiles_equal_whole_ones(t, rows, x_tiles, beyond, k):
    torch = need_gpu()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    check(t, (sms + beyond + x_tiles - 1) // x_tiles * rows - 5, x_tiles * 128 - 3, k)


# Q6_K on both sides of its line between pairs and single CTAs (short k); odd token tiles (a pair's last half is empty; one and three tiles go without pairs), odd row tiles, a row and a token beyond a tile
@pytest.mark.parametrize("t", [O.Q4_K, O.Q5_K, O.Q6_K])
@pytest.mark.parametrize("m,n,k", [(6145, 602, 1024), (6528, 513, 2048), (30800, 100, 512), (30721, 129, 256), (10300, 257, 768), (700, 1000, 2304),
                                   (4093, 500, 512), (1000, 140, 256), (8190, 200, 1024), (4096, 640, 512)])
def test_pairs_equal_small_products(t, m, n, k):
    check(t, m, n, k)


def check(t, m, n, k):
    torch = need_gpu()
    import cera_b200 as cb
    part = 600
    raw = cb.quantize_weights(t, cb.synth_normal(m * k, seed=m, sigma=0.02)).cpu().numpy().reshape(-1)
    w = cb.QuantWeight(t, m, k, raw)
    assert w.prepare_gemm()
    acts = cb.quantize_q8_0(cb.synth_normal(n * k, seed=k, sigma=1.0), k=k, n=n)
    x = acts.quants.view(n, k // 32, 32).double() * acts.scales.view(n, k // 32, 1).double()
    got = cb.gemm_preq(w, acts, torch.full((m, n), float("nan"), device="cuda"))
    per_row = raw.size // m
    for a in (0, min(m // 2, m - part), m - part):
        few = cb.QuantWeight(t, part, k, np.ascontiguousarray(raw[a * per_row:(a + part) * per_row]))
        assert few.prepare_gemm()
        want = cb.gemm_preq(few, acts)
        # k / 256 partial sums, none above |w| |x|, added in two orders; the minimum's product drops parts below 2^-22
        size = cb.dequantize_rows(few).double().norm(dim=1)[:, None] * x.reshape(n, k).norm(dim=1)[None]
        bound = (2 * (k // 256 + 1) * 2.0 ** -24 + 2.0 ** -22) * size
        assert bool(((got[a:a + part].double() - want.double()).abs() <= bound).all()), f"{O.NAMES[t]} rows from {a}"
