"""Steps over short contexts, whose splits merge as a thread-block cluster: around the longest such context, one split to eight, both head
dims, balanced and not, one row block and two, against the oracle over the bytes the GPU wrote."""
import numpy as np
import pytest

from helpers import ATTN_MAX_ABS, ATTN_REL_L2, Twin, attn_close, cpu_twin_of, orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,H,QH", [(128, 4, 24), (128, 2, 16), (128, 8, 8), (256, 4, 24)])
@pytest.mark.parametrize("T,rows", [(1, 1), (127, 1), (130, 2), (383, 1), (1025, 2), (3071, 1), (3072, 3), (3073, 1)])
@pytest.mark.parametrize("iters", [0, 2])
def test_short_steps(D, H, QH, T, rows, iters):
    import torch

    rows = min(rows, T)
    tw = Twin(D=D, H=H, QH=QH, capacity_tokens=T, seed=T + D, iters=iters)
    dev = tw.dev
    k, v = (torch.from_numpy(orc.synth_kv(T, T, H, D, i)).to(dev) for i in (1, 2))
    at = torch.arange(T, dtype=torch.int32, device=dev)
    if T > rows:
        tw.gpu.append(k[:T - rows], v[:T - rows], at[:T - rows])
    q = orc.synth_q(T, rows, QH, D)
    scale = 1.0 / np.sqrt(D)
    pos = at[T - rows:]
    if rows == 1:
        out = tw.gpu.append_decode(torch.from_numpy(q[0]).to(dev), k[T - 1:], v[T - 1:], pos, scale, T)[None]
    else:
        out = tw.gpu.attn_verify(torch.from_numpy(q).to(dev), k[T - rows:], v[T - rows:], pos, scale, T)
    want = cpu_twin_of(tw.gpu).attention(q, list(range(T - rows, T)), scale, QH, threads=4, kv_total=T)
    ok, msg = attn_close(out.float().cpu().numpy(), want, ATTN_MAX_ABS, ATTN_REL_L2)
    assert ok, msg
    assert tw.gpu.errors() == 0
