"""Edges of the decode attention: every head grouping, contexts around its 16-token rounds and its splits, ragged positions."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from oracle import mfq_oracle as O  # noqa: E402
from tyloquant_b200 import decoder as D  # noqa: E402
from test_decoder_gpu import _block_oracle  # noqa: E402
from test_nint_gpu import rel_l2  # noqa: E402


@pytest.mark.parametrize("heads,kv", [(4, 4), (4, 2), (8, 2), (8, 1)])
@pytest.mark.parametrize("max_ctx", [80, 1400])
def test_contexts_and_groups(heads, kv, max_ctx):
    cfg = dict(hidden=heads * 128, n_q_heads=heads, n_kv_heads=kv, ffn=64, vocab=64, layers=1, max_ctx=max_ctx, max_batch=2)
    dec, blobs = D.random_decoder(**cfg, seed=heads + kv, keep_blobs=True, distinct_layers=1)
    w = {k: O.dequant_nint(O.unpack_nint(b)) for k, b in blobs[0].items()}
    h_in = np.random.default_rng(heads).standard_normal((2, cfg["hidden"])).astype(np.float32)
    h_in[1] *= 30.0   # sharp scores
    for ctx in [c for c in (0, 1, 15, 16, 17, 63, 64, 79, 500, 1399) if c < max_ctx]:
        dec.fill_cache(ctx, seed=ctx)
        kc = [dec.read_cache(0, r, 0, ctx + 1).float().cpu().numpy()[:, :ctx] for r in range(2)]
        vc = [dec.read_cache(0, r, 1, ctx + 1).float().cpu().numpy()[:, :ctx] for r in range(2)]
        for rows in (1, 2):
            got = dec.layer(0, torch.from_numpy(h_in[:rows]).cuda()).cpu().numpy()
            for r in range(rows):
                want, _, _ = _block_oracle(h_in[r], w, kc[r], vc[r], ctx, heads, kv)
                assert rel_l2(got[r] - h_in[r], want - h_in[r]) <= 3e-3, (ctx, rows, r)
    dec.free()
