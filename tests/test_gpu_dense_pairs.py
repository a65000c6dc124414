"""Dense products whose tiles two CTAs share, inside layered models, at the edges of their tiles of 256 weight rows."""
import pytest

import goletar_ref as G
from goletar_util import TOL, config, error, mingru, moe, tokens
from gpu_util import need_gpu
from test_gpu_goletar import feed, load

pytestmark = pytest.mark.gpu


# experts' products: one whole pair of row tiles, one beyond a row short, and an odd count of them with the last pair half empty; columns: a tile
# and a bit, and last tiles of one column and of all but one.  The recurrence's product: its own row tiles
@pytest.mark.parametrize("ff,width,n", [(256, 100, 129), (250, 72, 255), (1100, 136, 300), (512, 72, 385), (640, 72, 200)])
def test_experts(tmp_path, ff, width, n):
    need_gpu()
    cfg = config([mingru(width=8, mlp=moe(experts=2, top=2, ff=ff))], width=width)
    w = G.random_weights(cfg, 141)
    m = load(tmp_path / "m", cfg, w, "bfloat16", n)
    toks = tokens(n, cfg["vocab"], 142)
    assert error(feed(m, toks, [n]), G.logits(toks, cfg, w)) < TOL["bfloat16"]
    m.close()


@pytest.mark.parametrize("width,n", [(683, 1793), (640, 2047), (1000, 1300)])  # 17, 15 and 24 row tiles; columns cut at 256
def test_one_matrix(tmp_path, width, n):
    need_gpu()
    cfg = config([mingru(width=width)])
    w = G.random_weights(cfg, 143)
    m = load(tmp_path / "m", cfg, w, "bfloat16", n)
    toks = tokens(n, cfg["vocab"], 144)
    assert error(feed(m, toks, [n]), G.logits(toks, cfg, w)) < TOL["bfloat16"]
    m.close()
