"""How a head's pages are dealt to splits and warps: with and without an open tile of one key to 127, less than a page a split, a round, a round
and a bit, several, and just below and above the eight from which the pages alone are shared; against the oracle over the bytes the GPU
wrote.  (Every page once, over all sizes: tests/cpp/shares_check.cpp.)

Balanced caches: the deal does not depend on it, and ATTN_MAX_ABS is not a bound there.  16 bits against the largest of a row leave an error of
0.5 / 32639 of it in every q' scale_K, with codes up to 15 over 128 dims up to 28 / 32639 = 8.6e-4 of it (rms) in a logit, which other_K, 1
otherwise, multiplies: at 18,977 tokens and two iterations the output was 1.1e-3 .. 1.3e-3 of the largest off, whatever the deal.  Three times
that is allowed."""
import numpy as np
import pytest

from helpers import ATTN_MAX_ABS, ATTN_REL_L2, Twin, attn_close, cpu_twin_of, orc

pytestmark = pytest.mark.gpu


# splits: 37 (4 heads, a row block), 6 (8 heads, three), 18 (8 heads, a row block)
@pytest.mark.parametrize("H,QH,rows", [(4, 24, 1), (8, 64, 3), (8, 8, 2)])
@pytest.mark.parametrize("T", [3 * 128, 26 * 128 + 1, 27 * 128 + 127, 72 * 128 + 16, 73 * 128 + 64, 147 * 128, 148 * 128 + 33])
def test_shares(H, QH, rows, T):
    import torch

    D, scale = 128, 128 ** -0.5
    tw = Twin(D=D, H=H, QH=QH, capacity_tokens=T, seed=T)
    k, v = (torch.from_numpy(orc.synth_kv(T, T, H, D, i)).to(tw.dev) for i in (1, 2))
    at = torch.arange(T, dtype=torch.int32, device=tw.dev)
    tw.gpu.append(k[:T - rows], v[:T - rows], at[:T - rows])
    q = orc.synth_q(T, rows, QH, D)
    out = tw.gpu.attn_verify(torch.from_numpy(q).to(tw.dev), k[T - rows:], v[T - rows:], at[T - rows:], scale, T)
    want = cpu_twin_of(tw.gpu).attention(q, list(range(T - rows, T)), scale, QH, threads=8, kv_total=T)
    ok, msg = attn_close(out.float().cpu().numpy(), want, ATTN_MAX_ABS, ATTN_REL_L2)
    assert ok, msg
    # a key range that begins inside a page: what it holds, and the rest, merge to the same
    if rows == 1:
        from helpers import pkg

        cut = T // 3 + 5
        parts = [[x.clone() for x in tw.gpu.attn_decode_partial(torch.from_numpy(q[0]).to(tw.dev), at[T - 1:], scale, T, a, b)] for a, b in ((0, cut), (cut, T))]
        both = pkg().merge_partials(*(torch.stack(x) for x in zip(*parts)))
        ok, msg = attn_close(both.float().cpu().numpy(), want[0], ATTN_MAX_ABS, ATTN_REL_L2)
        assert ok, msg
    assert tw.gpu.errors() == 0


# 24 rows a head of eight: two blocks of 16 rows, 9 splits of 8 warps (56 pages a split are seven rounds, 57 eight), or three blocks of 8
# rows, 6 splits of up to 16 warps
@pytest.mark.parametrize("T,iters,rounds", [(252 * 128 + 5, 0, 6), (253 * 128 + 127, 0, 6), (400 * 128 + 97, 0, 8), (401 * 128, 0, 8), (252 * 128 + 127, 2, 7), (253 * 128 + 1, 2, 8),
                                            (300 * 128 + 64, 2, 8)])
def test_many_rounds(T, iters, rounds):
    import torch

    from helpers import pkg

    D, H, QH, rows, scale = 128, 8, 64, 3, 128 ** -0.5
    splits = 9 if iters else pkg().capi.load().kvb_split_capacity(T, H, QH, rows, 1)  # (balanced: blocks of 16 rows)
    most_warps = 8 if splits == 9 else 16
    assert splits in (6, 9) and -(-2 * (T // 128) // splits) > (rounds - 1) * most_warps  # of the CTA with the most pages
    tw = Twin(D=D, H=H, QH=QH, capacity_tokens=T, seed=T, iters=iters)
    k, v = (torch.from_numpy(orc.synth_kv(T, T, H, D, i)).to(tw.dev) for i in (1, 2))
    at = torch.arange(T, dtype=torch.int32, device=tw.dev)
    tw.gpu.append(k[:T - rows], v[:T - rows], at[:T - rows])
    q = orc.synth_q(T, rows, QH, D)
    out = tw.gpu.attn_verify(torch.from_numpy(q).to(tw.dev), k[T - rows:], v[T - rows:], at[T - rows:], scale, T)
    want = cpu_twin_of(tw.gpu).attention(q, list(range(T - rows, T)), scale, QH, threads=8, kv_total=T)
    ok, msg = attn_close(out.float().cpu().numpy(), want, *((3 * 1.3e-3, 3 * 1.3e-3) if iters else (ATTN_MAX_ABS, ATTN_REL_L2)))
    assert ok, msg
    assert tw.gpu.errors() == 0
