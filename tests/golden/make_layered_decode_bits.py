"""Writes tests/golden/layered_decode_bits.json: CRC-32 of the logits' bits of two small layered models (Goletar, Piditar; f32 and bf16),
decoded token by token on a B200.  Their matrices are of the sizes at which the one-column products share a row among one, two, four
or eight warps.  The order of those sums is part of what a program sees: one last bit grows to a bf16 step, and at a router whose experts
are almost level to another pick.

    python tests/golden/make_layered_decode_bits.py
"""
import json
import os
import pathlib
import sys
import tempfile
import zlib

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.dirname(HERE))
sys.path.insert(0, os.path.dirname(os.path.dirname(HERE)))
import goletar_ref as G  # noqa: E402
import goletar_util as GU  # noqa: E402
import piditar_ref as P  # noqa: E402
import piditar_util as PU  # noqa: E402

GOLETAR = GU.config([GU.mingru(width=1024, mlp=GU.moe(ff=512, experts=8, top=2, limit=4.0)),
                     GU.attention(heads=16, dim=128, rot_dim=64, vdim=128, kv_rank=512, scale=0.07, mlp=GU.moe(ff=200, experts=8, top=2, limit=4.0))],
                    width=1024, vocab=9001)
PIDITAR = PU.config([PU.rglru(width=1024, blocks=4, mlp=PU.unit(ff=2101)),
                     PU.attention(heads=32, kv_heads=8, dim=128, vdim=64, rot=128, mlp=PU.unit(ff=512)),
                     PU.mamba2(heads=32, vdim=64, state=64, mlp=PU.unit(ff=4200))], width=1024, vocab=4200)
N_TOKENS = 4


def build(name, dtype):
    """CRC-32 of the logits after each token."""
    from cera_b200 import load_model
    ref, cfg = {"goletar": (G, GOLETAR), "piditar": (P, PIDITAR)}[name]
    with tempfile.TemporaryDirectory() as d:
        d = pathlib.Path(d)
        ref.save(d, cfg, ref.random_weights(cfg, 51))
        model = load_model(d, dtype=dtype, max_seq_len=16)
    out = [zlib.crc32(np.ascontiguousarray(model.forward(t, i), dtype=np.float32).tobytes()) for i, t in enumerate(GU.tokens(N_TOKENS, cfg["vocab"], 52))]
    model.close()
    return out


def main():
    out = {f"{n}_{t}": build(n, t) for n in ("goletar", "piditar") for t in ("float32", "bfloat16")}
    with open(sys.argv[1] if len(sys.argv) > 1 else os.path.join(HERE, "layered_decode_bits.json"), "w") as f:
        json.dump(out, f)


if __name__ == "__main__":
    main()
