"""The router of a one-token step - a cluster of CTAs forms the logits, the first one picks - at the edges of its rounds of 32 experts."""
import pytest

import goletar_ref as G
from goletar_util import TOL, config, error, mingru, moe, tokens
from gpu_util import need_gpu
from test_gpu_goletar import feed, load

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [8, 72, 520])  # vectors of four a lane holds: some lanes none, one, several
@pytest.mark.parametrize("experts,top", [(1, 1), (4, 4), (5, 3), (31, 8), (32, 1), (33, 4), (64, 2), (65, 8)])
def test_router_of_one_token(tmp_path, experts, top, width):
    need_gpu()
    cfg = config([mingru(width=8, mlp=moe(experts=experts, top=top, ff=24))], width=width)
    w = G.random_weights(cfg, 131 + experts)
    m = load(tmp_path / "m", cfg, w, "float32", 16)
    toks = tokens(6, cfg["vocab"], 132)
    assert error(feed(m, toks, [1]), G.logits(toks, cfg, w)) < TOL["float32"]
    m.close()
