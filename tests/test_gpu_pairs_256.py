"""Steps at head_dim 256, two warps a page: fewer pages than pairs of a CTA, a page each, one more, several; page ids read in batches of 32;
open tiles from one key to 127 (a 16-key group a pair); against the oracle over the bytes the GPU wrote.

Tolerance: the kernel's integers keep 22 bits of q' * scale_K and 23 of p * scale_V, its sums are fp32: what is left is the rounding of
the fp16 output, at most 2^-11 of a value, 2^-11 / sqrt(3) of the norm, with 10 % on top."""
import numpy as np
import pytest

from helpers import Twin, attn_close, cpu_twin_of, orc

pytestmark = pytest.mark.gpu

MAX_ABS, REL_L2 = 1.1 * 2.0 ** -11, 1.1 * 2.0 ** -11 / 3 ** 0.5


# two splits of eight pairs (64 CTAs a split), pages = 2 (T / 128); then more splits, up to 1,536 keys as a cluster
@pytest.mark.parametrize("H,QH,T,rows,iters", [(8, 64, 127, 8, 0), (8, 64, 128, 8, 2), (8, 64, 385, 8, 0), (8, 64, 1024, 8, 2), (8, 64, 1169, 8, 0),
                                               (8, 64, 2063, 8, 2), (8, 64, 4096 + 16, 8, 0), (8, 64, 2 * 8 * 33 * 64 + 145, 8, 0),
                                               (4, 24, 1536, 2, 0), (4, 24, 1537, 2, 0), (4, 24, 3200, 1, 2), (1, 3, 9000, 1, 0), (4, 24, 5000, 5, 2)])
def test_pairs(H, QH, T, rows, iters):
    import torch

    D, scale = 256, 1.0 / 16.0
    tw = Twin(D=D, H=H, QH=QH, capacity_tokens=T, seed=T, iters=iters)
    k, v = (torch.from_numpy(orc.synth_kv(T, T, H, D, i)).to(tw.dev) for i in (1, 2))
    at = torch.arange(T, dtype=torch.int32, device=tw.dev)
    tw.gpu.append(k[:T - rows], v[:T - rows], at[:T - rows])
    q = orc.synth_q(T, rows, QH, D)
    out = tw.gpu.attn_verify(torch.from_numpy(q).to(tw.dev), k[T - rows:], v[T - rows:], at[T - rows:], scale, T)
    want = cpu_twin_of(tw.gpu).attention(q, list(range(T - rows, T)), scale, QH, threads=8, kv_total=T)
    ok, msg = attn_close(out.float().cpu().numpy(), want, MAX_ABS, REL_L2)
    assert ok, msg
    assert tw.gpu.errors() == 0


@pytest.mark.parametrize("slice_", [0, 1])
@pytest.mark.parametrize("what", ["scale", "zero point", "dim"])
def test_factor_not_finite(slice_, what):
    """A factor of V that is not finite reaches the rows that see its key or tile, in its slice, and nothing else."""
    import torch

    D, H, QH, T, key = 256, 4, 24, 512, 300
    tw = Twin(D=D, H=H, QH=QH, capacity_tokens=T, seed=T)
    k, v = (torch.from_numpy(orc.synth_kv(T, T, H, D, i)).to(tw.dev) for i in (1, 2))
    q = torch.from_numpy(orc.synth_q(T, 1, QH, D)[0]).to(tw.dev)
    tw.gpu.append(k, v, torch.arange(T, dtype=torch.int32, device=tw.dev))
    for page in ((4, 5) if what == "dim" else (4,)):  # a scale row: 4 other_V | 2 scales | 2 zero points
        row = tw.gpu.v_scale[int(tw.table[page]), 1, 32 * slice_ + 5 if what == "dim" else key % 64]
        row[{"dim": 1, "scale": 4 + slice_, "zero point": 6 + slice_}[what]] = float("inf")
    pos = torch.tensor([T - 1], dtype=torch.int32, device=tw.dev)
    for end, bad in ((256, False), (T, True)):
        o = tw.gpu.attn_decode_partial(q, pos, 1.0 / 16.0, T, 0, end)[2]
        nan = torch.isnan(o.view(H, QH // H, 2, 128))
        want = torch.zeros_like(nan)
        want[1, :, slice_] = bad
        assert torch.equal(nan, want)
