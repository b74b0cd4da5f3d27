"""Batches whose CTAs have an SM each, with 16 warps: chunks of 4 tiles and of 8, an SM for every CTA exactly and one too few, sequences without a
sealed tile, and the few that run 8 warps a CTA; every sequence against the oracle over the bytes the GPU wrote."""
import numpy as np
import pytest

from helpers import ATTN_MAX_ABS, ATTN_REL_L2, attn_close, cpu_twin_of, orc, pkg

pytestmark = pytest.mark.gpu


# at 148 SMs and 4 heads 37 chunks fit: one of 4 tiles each, one more; chunks of 8; 8 heads: 18 of 8 tiles; 3 short sequences
@pytest.mark.parametrize("H,QH,tiles", [(4, 24, [1, 0, 3, 4, 2, 4]), (4, 24, [4 * 31, 4, 3, 1, 0, 2, 4]), (4, 24, [4 * 31, 5, 3, 1, 0, 2, 4]), (4, 24, [8 * 34, 1, 8, 0]),
                                        (8, 64, [17, 40, 8, 63, 1]), (4, 24, [2, 3, 1]), (2, 16, [64, 3, 4, 20, 9, 1])])
def test_small_batches(H, QH, tiles):
    import torch

    scale, rng = 128 ** -0.5, np.random.default_rng(len(tiles))
    lengths = [128 * t + int(rng.integers(1 if t == 0 else 0, 128)) for t in tiles]
    layers, pages = [], 2 * max(tiles) + 4
    for i, n in enumerate(lengths):
        L = pkg().KvarnLayer(128, H, QH, pages, torch.from_numpy(orc.shuffled_table(i, pages, pages)))
        L.append(*(torch.from_numpy(orc.synth_kv(n + i, n, H, 128, j)).cuda() for j in (1, 2)), torch.arange(n, dtype=torch.int32, device="cuda"))
        layers.append(L)
    q = orc.synth_q(QH, len(lengths), QH, 128)
    pos = torch.tensor([n - 1 for n in lengths], dtype=torch.int32, device="cuda")
    batch = pkg().DecodeBatch(layers, lengths)
    out = batch.attn_decode(torch.from_numpy(q).cuda(), pos, scale)
    assert all(torch.equal(out, batch.attn_decode(torch.from_numpy(q).cuda(), pos, scale)) for _ in range(5))
    for i, (L, n) in enumerate(zip(layers, lengths)):
        want = cpu_twin_of(L).attention(q[i:i + 1], [n - 1], scale, QH, threads=4, kv_total=n)
        ok, msg = attn_close(out[i:i + 1].float().cpu().numpy(), want, ATTN_MAX_ABS, ATTN_REL_L2)
        assert ok, (i, n, msg)
        assert L.errors() == 0
