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


# three token tiles: 128 x 256 tiles of single CTAs, the last round shared
@pytest.mark.parametrize("t", [O.Q4_K, O.Q5_K])
def test_shared_tiles_of_single_wide_ctas(t):
    check(t, 28670, 383, 2048)


# one token tile of q, k and v together, every row tile shared along k: a weight's first tiles follow another's last, token-major
@pytest.mark.parametrize("n", [100, 128])
def test_shared_tiles_of_several_weights(n):
    torch = need_gpu()
    import cera_b200 as cb
    from cera_b200.model import Role
    width, kv, vocab = 4096, 1024, 256
    model = cb.CudaModel(n_layers=1, hidden_size=width, intermediate_size=512, n_heads=32, n_kv_heads=8, head_dim=128, vocab_size=vocab, rope_theta=10000.0,
                         rms_norm_eps=1e-5, rope_type=0, kv_f16=0, max_seq_len=n)
    raw = {}
    for role, rows, cols in ((Role.TOKEN_EMBD, vocab, width), (Role.OUTPUT, vocab, width), (Role.ATTN_Q, width, width), (Role.ATTN_K, kv, width), (Role.ATTN_V, kv, width),
                             (Role.ATTN_OUTPUT, width, width), (Role.FFN_GATE, 512, width), (Role.FFN_UP, 512, width), (Role.FFN_DOWN, width, 512)):
        raw[role] = cb.quantize_weights(O.Q4_K, cb.synth_normal(rows * cols, seed=int(role) + 1, sigma=0.02))
        model.add_tensor(role, 0, O.Q4_K, rows, cols, raw[role])
    ones = np.ones(width, dtype=np.float32)
    for role in (Role.OUTPUT_NORM, Role.ATTN_NORM, Role.FFN_NORM):
        model.add_tensor(role, 0, cb.types.F32, 1, width, ones)
    torch.cuda.synchronize()
    model.finalize()
    tokens = (np.arange(n) * 7 % vocab).astype(np.uint32)
    model.forward_prefill(tokens, 0)
    k_got, v_got = (np.asarray(c).reshape(-1).view(np.float32).reshape(n, kv) for c in model.state_snapshot()["layers"][0])
    model.close()
    rows = cb.dequantize_rows(cb.QuantWeight(O.Q4_K, vocab, width, raw[Role.TOKEN_EMBD]))
    weight = torch.ones(width, device="cuda")
    pairs = lambda a: np.hypot(a[:, ::2].astype(np.float64), a[:, 1::2].astype(np.float64))  # noqa: E731  what the rotation leaves of keys
    for role, got in ((Role.ATTN_K, pairs(k_got)), (Role.ATTN_V, v_got.astype(np.float64))):
        w = cb.QuantWeight(O.Q4_K, kv, width, raw[role])
        size = cb.dequantize_rows(w).double().norm(dim=1).cpu().numpy()
        for j in (0, 1, 63, n - 1):
            acts = cb.rmsnorm_q8_0(rows[int(tokens[j])].contiguous(), weight, 1e-5)[1]
            want = cb.gemm_preq(w, acts)[:, 0].cpu().numpy()[None]
            norm = float((acts.quants.view(-1, 32).double() * acts.scales.view(-1, 1).double()).norm())
            bound = (2 * (width // 256 + 1) * 2.0 ** -24 + 2.0 ** -22) * size * norm  # as below
            if role == Role.ATTN_K:  # two values, turned by a cosine and a sine of 24 bits
                want, bound = pairs(want), (bound[::2] + bound[1::2]) + 2.0 ** -22 * (size[::2] + size[1::2]) * norm
            assert (np.abs(got[j] - want[0]) <= bound).all(), (role, j)


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
