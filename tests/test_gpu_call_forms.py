"""Forms of the attention calls that a caller may choose freely: buffers that are only as aligned as their elements, rows without
a key, a descriptor that says less than the planes hold, values that are not finite.  Everything is compared with another form
of the same call or with the oracle over the bytes of the cache."""
import ctypes as C

import numpy as np
import pytest

from helpers import ATTN_MAX_ABS, ATTN_REL_L2, PREFILL_MAX_ABS, PREFILL_REL_L2, Twin, attn_close, cpu_twin_of, orc, pkg

pytestmark = pytest.mark.gpu


def _filled(D, H, QH, T, iters=0, seed=1, room=16):
    import torch

    tw = Twin(D=D, H=H, QH=QH, capacity_tokens=T + room, seed=seed, iters=iters)
    if T:
        k, v = orc.synth_kv(seed, T, H, D, 1), orc.synth_kv(seed, T, H, D, 2)
        tw.gpu.append(torch.from_numpy(k).to(tw.dev), torch.from_numpy(v).to(tw.dev), torch.arange(T, dtype=torch.int32, device=tw.dev))
    return tw


def _partial(tw, q, pos, kv_len, packed):
    """m, l, o of chunk rows q at positions pos, exported into `packed` (m | l | o)."""
    rows = q.shape[0] * tw.QH
    tw.gpu.attn_chunk_partial_packed(q, pos, 1.0 / np.sqrt(tw.D), kv_len, packed)
    return packed[:rows], packed[rows:2 * rows], packed[2 * rows:2 * rows + rows * tw.D].view(rows, tw.D)


@pytest.mark.parametrize("D", [128, 256])
@pytest.mark.parametrize("H,QH,tokens", [(1, 7, 1), (3, 9, 1), (1, 7, 3), (1, 5, 7), (1, 7, 11)])
def test_packed_partials_of_an_odd_number_of_rows(D, H, QH, tokens):
    """o starts 2 * rows floats behind the base of a packed buffer: 8 bytes off a 16-byte boundary for an odd number of rows.
    The same bits as from a buffer that starts 8 bytes later, where o is 16-byte aligned."""
    import torch

    T = 500
    tw = _filled(D, H, QH, T)
    rows = tokens * QH
    assert rows % 2 == 1
    q = torch.from_numpy(orc.synth_q(2, tokens, QH, D)).to(tw.dev)
    pos = torch.arange(T - tokens, T, dtype=torch.int32, device=tw.dev)
    n = rows * (D + 2)
    a, b = torch.full((n + 4,), 7.0, device=tw.dev), torch.full((n + 4,), 7.0, device=tw.dev)
    got = _partial(tw, q, pos, T, a[:n])
    want = _partial(tw, q, pos, T, b[2:n + 2])
    assert all(torch.equal(x, y) for x, y in zip(got, want))
    assert torch.all(a[n:] == 7.0) and torch.all(b[n + 2:] == 7.0)
    out = pkg().cache.merge_partials_packed(a[:n].contiguous(), 1, rows, D, torch.empty((rows, D), dtype=torch.float16, device=tw.dev))
    ref = cpu_twin_of(tw.gpu).attention(q.cpu().numpy(), np.arange(T - tokens, T, dtype=np.int32), 1.0 / np.sqrt(D), QH, threads=4, kv_total=T)
    ok, msg = attn_close(out.float().cpu().numpy().reshape(ref.shape), ref, *((PREFILL_MAX_ABS, PREFILL_REL_L2) if D == 128 and tokens * QH // H >= 32 else (ATTN_MAX_ABS, ATTN_REL_L2)))
    assert ok, msg
