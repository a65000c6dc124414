"""One-token paths that form their operands themselves, against the same operation in separate calls: equal to the last bit."""
import numpy as np
import pytest

import oracle_lib as O
from gpu_util import need_gpu

pytestmark = pytest.mark.gpu


def _column(k, seed):
    """A column with the blocks a quantizer can go wrong at: zeros, one value, NaN, infinity, subnormal maxima, ties."""
    x = O.synth_normal(k, seed, 1.5)
    for i, v in enumerate((0.0, 1e-40, np.nan, np.inf, 63.5)):
        if k >= 32 * (i + 2):
            x[32 * i] = v
            if i in (0, 1):
                x[32 * i:32 * i + 32] = v
            if i == 4:  # scale 0.5: values half way between two quants
                x[32 * i:32 * i + 32] = np.tile(np.float32([63.5, 0.25, -0.25, 0.75, -0.75, 1.25, 31.75, -63.5]), 4)
    return x


@pytest.mark.parametrize("k,n", [(32, 1), (96, 3), (256, 2), (4096, 5)])
def test_contiguous_quantizer_equals_the_strided_one(k, n):
    torch = need_gpu()
    import cera_b200 as cb
    x = torch.from_numpy(np.stack([_column(k, 3 + j) for j in range(n)])).cuda()
    a, b = cb.quantize_q8_0(x.reshape(-1), k=k, n=n), cb.quantize_columns(x.T.contiguous(), k, n)
    odd = torch.cat([torch.zeros(1, device="cuda"), x.reshape(-1)])[1:]  # not on a 16-byte boundary
    for c in (b, cb.quantize_q8_0(odd, k=k, n=n)):
        for f in ("quants", "scales", "sums"):
            assert torch.equal(getattr(a, f).view(torch.uint8), getattr(c, f).view(torch.uint8)), f
