"""head_dim 256 on the warp-level int8 kernel (two 128-dim slices per key): decode and verify steps against the oracle.

Tolerance: the kernel's integers keep 22 bits of q' * scale_K and 23 of p * scale_V, its sums are fp32 -- what is left is the
rounding of the fp16 output: at most 2^-11 of a value (max-abs <= 2^-11 of the largest), 2^-11 / sqrt(3) of the norm where
mantissas are spread evenly.  Both with 10 % on top."""
import numpy as np
import pytest

from helpers import Twin, attn_close, cpu_twin_of, orc

pytestmark = pytest.mark.gpu

MAX_ABS, REL_L2 = 1.1 * 2.0 ** -11, 1.1 * 2.0 ** -11 / 3 ** 0.5


@pytest.mark.parametrize("H,QH,T,iters", [(4, 24, 1, 0), (4, 24, 63, 16), (4, 24, 128, 0), (4, 24, 129, 16), (2, 16, 191, 0), (1, 7, 256, 0), (8, 8, 2049, 16),
                                          (4, 24, 9000, 0), (4, 24, 9001, 16)])
def test_decode_and_verify(H, QH, T, iters):
    import torch

    D, scale = 256, 1.0 / 16.0
    tw = Twin(D=D, H=H, QH=QH, capacity_tokens=T + 8, seed=T, iters=iters)
    k, v = orc.synth_kv(T, T + 8, H, D, 1), orc.synth_kv(T, T + 8, H, D, 2)
    dev = tw.dev

    def on_gpu(x):
        return torch.from_numpy(x).to(dev)

    tw.gpu.append(on_gpu(k[:T]), on_gpu(v[:T]), torch.arange(T, dtype=torch.int32, device=dev))
    q = orc.synth_q(T, 1, QH, D)
    pos = torch.tensor([T - 1], dtype=torch.int32, device=dev)
    out = tw.gpu.attn_decode(on_gpu(q[0]), pos, scale, T)
    want = cpu_twin_of(tw.gpu).attention(q, [T - 1], scale, QH, threads=4, kv_total=T)
    ok, msg = attn_close(out.float().cpu().numpy(), want[0], MAX_ABS, REL_L2)
    assert ok, "decode: " + msg
    # two key ranges of the same decode, merged
    from helpers import pkg

    cut = T // 2
    parts = [[x.clone() for x in tw.gpu.attn_decode_partial(on_gpu(q[0]), pos, scale, T, a, b)] for a, b in ((0, cut), (cut, T))]
    both = pkg().merge_partials(*(torch.stack(x) for x in zip(*parts)))
    ok, msg = attn_close(both.float().cpu().numpy(), want[0], MAX_ABS, REL_L2)
    assert ok, "merged ranges: " + msg
    for width in (2, 5, 8):  # every width appends at T again: rows of several 8-row blocks, some of them across a seal
        qv = orc.synth_q(T + width, width, QH, D)
        at = np.arange(T, T + width, dtype=np.int32)
        out = tw.gpu.attn_verify(on_gpu(qv), on_gpu(k[T:T + width]), on_gpu(v[T:T + width]), on_gpu(at), scale, T + 8)
        want = cpu_twin_of(tw.gpu).attention(qv, at, scale, QH, threads=4, kv_total=T + width)
        ok, msg = attn_close(out.float().cpu().numpy(), want, MAX_ABS, REL_L2)
        assert ok, "verify of %d rows: %s" % (width, msg)
    assert tw.gpu.errors() == 0


# tokens in the cache before the chunk, tokens of the chunk: one row tile and several (128 rows of G heads), ragged ends of
# pages and tiles, an open tile, an empty prefix, several key ranges
@pytest.mark.parametrize("H,QH,ctx,T,iters", [(4, 24, 0, 9, 0), (4, 24, 0, 64, 16), (2, 16, 0, 65, 0), (4, 24, 127, 21, 16), (4, 24, 128, 22, 0), (1, 7, 191, 300, 16),
                                              (8, 8, 1000, 129, 0), (4, 24, 3000, 40, 16), (4, 4, 4096, 128, 0)])
def test_chunk(H, QH, ctx, T, iters):
    """The tcgen05 chunk kernel: operands of 22 significant bits and fp32 sums leave the rounding of the output."""
    import torch

    D, scale = 256, 1.0 / 16.0
    tw = Twin(D=D, H=H, QH=QH, capacity_tokens=ctx + T, seed=ctx + T, iters=iters)
    k, v = orc.synth_kv(T, ctx + T, H, D, 1), orc.synth_kv(T, ctx + T, H, D, 2)
    q = orc.synth_q(T, T, QH, D)
    gk, gv, gq = (torch.from_numpy(x).to(tw.dev) for x in (k, v, q))
    at = torch.arange(ctx + T, dtype=torch.int32, device=tw.dev)
    if ctx:
        tw.gpu.append(gk[:ctx], gv[:ctx], at[:ctx])
    out = tw.gpu.attn_prefill(gq, gk[ctx:], gv[ctx:], at[ctx:], scale, ctx + T)
    want = cpu_twin_of(tw.gpu).attention(q, np.arange(ctx, ctx + T, dtype=np.int32), scale, QH, threads=4, kv_total=ctx + T)
    assert tw.gpu.errors() == 0
    ok, msg = attn_close(out.float().cpu().numpy(), want, MAX_ABS, REL_L2)
    assert ok, msg


def test_chunk_far_from_one():
    """Scales of 2^-10 in K, 2^11 in V and one row of the open tile 2^4 above the rest: the split operands follow them."""
    import torch

    D, H, QH, T, scale = 256, 2, 8, 300, 16.0
    tw = Twin(D=D, H=H, QH=QH, capacity_tokens=T, seed=3)
    k = (orc.synth_kv(1, T, H, D, 1).astype(np.float32) * 2.0 ** -10).astype(np.float16)
    v = (np.clip(orc.synth_kv(1, T, H, D, 2).astype(np.float32), -2, 2) * 2.0 ** 9).astype(np.float16)
    v[T - 7] *= 4
    q = orc.synth_q(1, T, QH, D)
    at = torch.arange(T, dtype=torch.int32, device=tw.dev)
    out = tw.gpu.attn_prefill(*(torch.from_numpy(x).to(tw.dev) for x in (q, k, v)), at, scale, T)
    want = cpu_twin_of(tw.gpu).attention(q, np.arange(T, dtype=np.int32), scale, QH, threads=4, kv_total=T)
    assert tw.gpu.errors() == 0
    ok, msg = attn_close(out.float().cpu().numpy(), want, MAX_ABS, REL_L2)
    assert ok, msg
