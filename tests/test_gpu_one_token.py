"""One-token paths that form their operands themselves, against the same operation in separate calls: equal to the last bit."""
import numpy as np
import pytest

import oracle_lib as O
from gpu_util import assert_bits, need_gpu
from test_gpu_moe import _layer

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


@pytest.mark.parametrize("t", O.QUANT_TYPES)
@pytest.mark.parametrize("m,k", [(1, 256), (9, 512), (70, 768), (33, 4096), (300, 1024), (20, 14336)])
def test_gemv_equals_quantizer_and_product(t, m, k):
    torch = need_gpu()
    import cera_b200 as cb
    w = cb.QuantWeight(t, m, k, cb.quantize_weights(t, cb.synth_normal(m * k, seed=m + k, sigma=0.05)))
    x = torch.from_numpy(O.synth_normal(k, k, 1.0)).cuda()
    odd = torch.cat([torch.zeros(1, device="cuda"), x])[1:]
    want = cb.gemm_preq(w, cb.quantize_q8_0(x))[:, 0]
    for v in (x, odd):
        assert_bits(cb.gemv(w, v).cpu().numpy(), want.cpu().numpy(), f"{O.NAMES[t]} {m} x {k}")


@pytest.mark.parametrize("t", O.QUANT_TYPES)
def test_gemv_over_its_own_operand(t):
    torch = need_gpu()
    import cera_b200 as cb
    n = 4096
    w = cb.QuantWeight(t, n, n, cb.quantize_weights(t, cb.synth_normal(n * n, seed=3, sigma=0.05)))
    x = torch.from_numpy(O.synth_normal(n, 4, 1.0)).cuda()
    want = cb.gemv(w, x)
    assert_bits(cb.gemv(w, x, x).cpu().numpy(), want.cpu().numpy(), O.NAMES[t])


# both sides of the lines between one launch and two: rows of one, two and four warps, few and many of them; a column of 10240 and beyond
@pytest.mark.parametrize("t", O.QUANT_TYPES)
@pytest.mark.parametrize("m,k", [(1184, 2048), (1200, 2048), (2400, 256), (4730, 5376), (4760, 5376), (4760, 8448), (70, 9216), (70, 9728), (2047, 14336), (2048, 14336),
                                 (2048, 14848)])
def test_gemv_in_one_launch_or_two(t, m, k):
    test_gemv_equals_quantizer_and_product(t, m, k)


@pytest.mark.parametrize("t", [O.Q4_0, O.Q4_1, O.Q8_0])
@pytest.mark.parametrize("m,k", [(5, 128), (17, 384), (3, 32768), (11, 160)])
def test_gemv_of_32_element_formats_equals_quantizer_and_product(t, m, k):
    test_gemv_equals_quantizer_and_product(t, m, k)


# experts: fewer, as many and more than the cluster has warps; widths whose items do not fill a warp, and that take several rounds
@pytest.mark.parametrize("t,experts,used,hidden,ff,softmax", [
    (O.Q4_0, 1, 1, 32, 32, False), (O.Q4_0, 8, 2, 96, 160, True), (O.Q8_0, 33, 4, 2080, 64, False), (O.Q4_1, 64, 16, 256, 96, True),
    (O.Q4_0, 65, 5, 512, 2112, False), (O.Q8_0, 256, 16, 64, 32, True), (O.Q4_K, 8, 3, 512, 256, False), (O.Q5_K, 16, 4, 256, 768, True),
    (O.Q6_K, 12, 2, 1280, 512, False), (O.Q4_0, 4, 2, 8224, 64, False)])
@pytest.mark.parametrize("biased", [False, True])
def test_one_token_equals_the_first_of_two(t, experts, used, hidden, ff, softmax, biased):
    torch = need_gpu()
    import cera_b200 as cb
    gate, up, down, router = _layer(t, experts, hidden, ff, 100 + experts)
    bias = O.synth_normal(experts, 5, 0.3) if biased else None
    moe = cb.MoeFfn(experts, used, hidden, ff, t, gate, up, down, router, exp_probs_b=bias, max_tokens=4)
    x = torch.from_numpy(O.synth_normal(2 * hidden, 7, 1.0).reshape(2, hidden)).cuda()
    two = moe(x, softmax_gate=softmax, want_routing=True)
    one = moe(x[:1], softmax_gate=softmax, want_routing=True)
    plain = moe(x[:1], softmax_gate=softmax)
    for a, b, what in zip(one, two, ("out", "ids", "weights")):
        assert_bits(a[0].cpu().numpy(), b[0].cpu().numpy(), what)
    assert_bits(plain.cpu().numpy(), one[0].cpu().numpy(), "without routing")
    moe.close()


# rows an SM in eights, and the lone warps of a CTA that shared memory leaves: the line between the two register budgets lies at 21
@pytest.mark.parametrize("t,k,share,warps", [(O.Q4_K, 512, 18, 18), (O.Q4_K, 512, 25, 25), (O.Q4_K, 1536, 32, 28), (O.Q5_K, 512, 21, 21), (O.Q5_K, 512, 22, 22),
                                             (O.Q5_K, 1536, 32, 25), (O.Q6_K, 512, 18, 18), (O.Q6_K, 512, 22, 22), (O.Q6_K, 1536, 32, 21)])
def test_gemv_of_many_rows_equals_its_parts(t, k, share, warps):
    torch = need_gpu()
    import cera_b200 as cb
    assert _lone_warps(t, k, share) == warps
    m, part = torch.cuda.get_device_properties(0).multi_processor_count * 8 * share - 3, 1000
    raw = cb.quantize_weights(t, cb.synth_normal(m * k, seed=share, sigma=0.02)).cpu().numpy()
    x = torch.from_numpy(O.synth_normal(k, 5, 1.0)).cuda()
    w = cb.QuantWeight(t, m, k, raw)
    got = cb.gemv(w, x).cpu().numpy()
    assert_bits(cb.gemm_preq(w, cb.quantize_q8_0(x))[:, 0].cpu().numpy(), got, f"{O.NAMES[t]} quantized ahead")
    per_row = raw.size // m
    for a in (0, m // 2, m - part):
        rows = np.ascontiguousarray(raw.reshape(-1)[a * per_row:(a + part) * per_row])
        assert_bits(got[a:a + part], cb.gemv(cb.QuantWeight(t, part, k, rows), x).cpu().numpy(), f"{O.NAMES[t]} rows from {a}")


def _lone_warps(t, k, share):
    """The warps that the product in reference order gives a CTA: its share of the row groups, or what 224 KB hold beside the column."""
    segment = {O.Q4_K: 2304, O.Q5_K: 2816, O.Q6_K: 3456}[t]
    room = 224 * 1024 - (2112 + k + k // 32 * 8 + k // 16 * 4)
    most = {s: min(32, room // (s * segment + 2 * 1024 + 2 * 640)) for s in (8, 4, 2)}
    if share <= most[8] or share <= most[4]:
        return share
    return most[4] if 4 * most[4] >= 3 * min(share, 32) else min(share, most[2])
