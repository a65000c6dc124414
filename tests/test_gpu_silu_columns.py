"""The gated product's quantizer on both sides of the line from four to eight elements a thread (148 SMs x 2048 threads), through a routed layer."""
import pytest

from gpu_util import need_gpu
from test_gpu_moe import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ff,n", [(2048, 591), (2048, 592), (2080, 600)])  # just below, at the line, a last CTA that is not full
def test_gated_product_of_many_columns(ff, n):
    need_gpu()
    import cera_b200 as cb
    _run(cb.Q8_0, n_expert=4, n_used=2, hidden=64, ff=ff, n=n, seed=71)
