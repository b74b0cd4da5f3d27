"""The same call over and over: one answer, bit for bit and finite, whatever the CTAs of a call leave in shared memory for the next ones.
Ragged batches and single sequences on every instance of the decode kernel (8, 12 and 16 warps, 8 and 16 rows a block, both head dims)."""
import numpy as np
import pytest

from helpers import ATTN_MAX_ABS, ATTN_REL_L2, attn_close, cpu_twin_of, orc, pkg

pytestmark = pytest.mark.gpu

CALLS = 60


def _sequence(gen, H, QH, T, D=128, iters=0, room=8):
    import torch

    lp = 2 * ((T + room + 127) // 128 + 1)
    L = pkg().KvarnLayer(D, H, QH, lp, torch.randperm(lp, generator=gen, device="cuda").to(torch.int32), sinkhorn_iters=iters)
    for at in range(0, T, 8192):
        n = min(8192, T - at)
        k, v = (torch.randn((n, H, D), generator=gen, device="cuda").half() for _ in range(2))
        L.append(k, v, torch.arange(at, at + n, dtype=torch.int32, device="cuda"))
    return L


def _oracle(L, q, T, rows=1):
    got = cpu_twin_of(L).attention(q.cpu().numpy().reshape(rows, L.q_heads, L.head_dim), np.arange(T - rows, T, dtype=np.int32), 1.0 / np.sqrt(L.head_dim), L.q_heads,
                                   threads=8, kv_total=T)
    return got if rows > 1 else got[0]


@pytest.mark.parametrize("H,QH", [(4, 24), (8, 32), (2, 16)])
@pytest.mark.parametrize("lengths", [[35646, 9000, 16383, 128, 127, 1, 60001, 4097, 20000, 31, 8192, 52345], [30000 - 37 * i for i in range(20)]])
def test_ragged_batches(H, QH, lengths):
    import torch

    gen = torch.Generator(device="cuda")
    gen.manual_seed(QH)
    layers = [_sequence(gen, H, QH, n) for n in lengths]
    batch = pkg().DecodeBatch(layers, lengths)
    pos = torch.tensor([n - 1 for n in lengths], dtype=torch.int32, device="cuda")
    scale = 1.0 / np.sqrt(128)
    for _ in range(3):
        q = torch.randn((len(lengths), QH, 128), generator=gen, device="cuda").half()
        first = batch.attn_decode(q, pos, scale)
        for i in (0, len(lengths) // 2):
            ok, msg = attn_close(first[i].float().cpu().numpy(), _oracle(layers[i], q[i], lengths[i]), ATTN_MAX_ABS, ATTN_REL_L2)
            assert ok, msg
        outs = [batch.attn_decode(q, pos, scale) for _ in range(CALLS // 3)]
        assert torch.isfinite(first).all() and all(torch.equal(first, x) for x in outs)
    assert all(L.errors() == 0 for L in layers)


# pages per CTA from less than one a warp to several rounds: 8, 12 and 16 warps; 16-row blocks; balanced caches; 256 dims
@pytest.mark.parametrize("D,H,QH,T,rows,iters", [(128, 4, 24, 1500, 1, 0), (128, 4, 24, 35646, 1, 0), (128, 4, 24, 60001, 1, 0), (128, 4, 24, 100003, 1, 0), (128, 4, 24, 33000, 4, 0),
                                                 (128, 4, 24, 20011, 1, 16), (128, 4, 24, 20011, 3, 16), (256, 4, 24, 30011, 1, 16), (256, 4, 24, 20000, 5, 0)])
def test_one_sequence(D, H, QH, T, rows, iters):
    import torch

    gen = torch.Generator(device="cuda")
    gen.manual_seed(T)
    L = _sequence(gen, H, QH, T, D, iters)
    q = torch.randn((rows, QH, D), generator=gen, device="cuda").half()
    n = rows * QH * (D + 2)
    pos = torch.arange(T - rows, T, dtype=torch.int32, device="cuda")
    outs = [L.attn_chunk_partial_packed(q, pos, 1.0 / np.sqrt(D), T, torch.full((n,), float("nan"), device="cuda")) for _ in range(CALLS)]
    assert torch.isfinite(outs[0]).all() and all(torch.equal(outs[0], x) for x in outs[1:])
    out = pkg().cache.merge_partials_packed(outs[0], 1, rows * QH, D, torch.empty((rows * QH, D), dtype=torch.float16, device="cuda"))
    want = _oracle(L, q, T, rows)
    ok, msg = attn_close(out.float().cpu().numpy().reshape(want.shape), want, ATTN_MAX_ABS, ATTN_REL_L2)
    assert ok, msg
    assert L.errors() == 0
