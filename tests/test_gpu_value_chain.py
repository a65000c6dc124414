"""Value chains of decode attention around the edges of what one load and one block of loads bring."""
import pytest

pytestmark = pytest.mark.gpu


# blocks of 32 positions: none, one, a remainder, the last of several, past the one-launch form
@pytest.mark.parametrize("kv_f16", [0, 1])
@pytest.mark.parametrize("nh,nkv,hd,seq", [(4, 1, 128, 31), (4, 1, 128, 32), (8, 2, 64, 33), (8, 2, 64, 63), (4, 1, 256, 64), (8, 4, 128, 65), (4, 2, 128, 95),
                                           (8, 2, 64, 97), (4, 1, 128, 1056), (16, 4, 128, 1537), (8, 2, 64, 1600), (6, 2, 96, 2081)])
def test_value_chain_block_edges(nh, nkv, hd, seq, kv_f16):
    from test_gpu_reference_order import test_decode_attention_bits
    test_decode_attention_bits(nh, nkv, hd, seq, kv_f16)
