"""Steps whose attention starts beside their append, against the append and the attention called one after the other: the same bits.
Bounds from the length itself to many times as many splits as pages, so that the tile a step completes, or opens again after a
roll-back, is read by other CTAs than those of the last split."""
import numpy as np
import pytest

from helpers import Twin, orc, pkg

pytestmark = pytest.mark.gpu


def _pair(D, H, QH, T, iters):
    import torch

    k, v = (torch.from_numpy(orc.synth_kv(T, T + 16, H, D, i)).cuda() for i in (1, 2))
    at = torch.arange(T + 16, dtype=torch.int32, device="cuda")
    layers = [Twin(D=D, H=H, QH=QH, capacity_tokens=T + 16, seed=T, iters=iters).gpu for _ in range(2)]
    for L in layers:
        if T:
            L.append(k[:T], v[:T], at[:T])
    return layers, at


def _same(a, b):
    import torch

    torch.cuda.synchronize()
    assert all(torch.equal(x, y) for x, y in zip((a.stage, a.k_code, a.v_code, a.k_scale, a.v_scale), (b.stage, b.k_code, b.v_code, b.k_scale, b.v_scale)))
    assert a.errors() == 0 and b.errors() == 0


def _rows(L, q, pos, bound):
    import ctypes as C

    import torch

    out, n = torch.empty_like(q), q.shape[0]
    ptr = [C.c_void_p(x.data_ptr()) for x in (q, pos, pos[n - 1:], L.workspace(bound, n), out)]
    pkg().capi.check(pkg().capi.load().kvb_attn_rows(C.byref(L.c), ptr[0], ptr[1], n, ptr[2], 1.0 / np.sqrt(L.head_dim), bound, ptr[3], ptr[4], torch.cuda.current_stream().cuda_stream))
    return out


@pytest.mark.parametrize("D,iters", [(128, 0), (128, 16), (256, 16)])
@pytest.mark.parametrize("T", [125, 253, 1021, 4093])
@pytest.mark.parametrize("bound", [0, 3000, 9000, 70000])
def test_decode_steps_across_a_seal(D, iters, T, bound):
    import torch

    H, QH, bound = 4, 24, max(bound, T + 6)
    (a, b), at = _pair(D, H, QH, T, iters)
    scale = 1.0 / np.sqrt(D)
    for s in range(6):
        q, k, v = (torch.from_numpy(x).cuda() for x in (orc.synth_q(T + s, 1, QH, D)[0], orc.synth_kv(T + s, 1, H, D, 3), orc.synth_kv(T + s, 1, H, D, 4)))
        pos = at[T + s:T + s + 1]
        got = a.append_decode(q, k, v, pos, scale, bound)
        b.append(k, v, pos)
        assert torch.equal(got, b.attn_decode(q, pos, scale, bound)), s
    _same(a, b)


# rows from a sealed tile on that was rolled back into, over one that the step completes, inside the open tile
@pytest.mark.parametrize("D,iters", [(128, 0), (128, 16), (256, 0)])
@pytest.mark.parametrize("T,back", [(256, 3), (259, 7), (384, 100), (1030, 8), (300, 0)])
@pytest.mark.parametrize("width", [1, 3, 5, 8])
@pytest.mark.parametrize("bound", [0, 9000])
def test_verify_steps_after_a_roll_back(D, iters, T, back, width, bound):
    import torch

    H, QH, p, bound = 4, 24, T - back, max(bound, T + 16)
    (a, b), at = _pair(D, H, QH, T, iters)
    for s in range(2):  # the second step re-opens what the first one has just sealed, or follows it
        q, k, v = (torch.from_numpy(x).cuda() for x in (orc.synth_q(T + s, width, QH, D), orc.synth_kv(T + s, width, H, D, 3), orc.synth_kv(T + s, width, H, D, 4)))
        pos = at[p + s:p + s + width]
        got = a.attn_verify(q, k, v, pos, 1.0 / np.sqrt(D), bound)
        b.append(k, v, pos)
        assert torch.equal(got, _rows(b, q, pos, bound)), s
    _same(a, b)


@pytest.mark.parametrize("D,iters", [(128, 0), (256, 16)])
@pytest.mark.parametrize("T,tokens", [(0, 1), (0, 3), (120, 8), (250, 9), (300, 40), (384, 300)])
@pytest.mark.parametrize("bound", [0, 20000])
def test_chunks(D, iters, T, tokens, bound):
    import torch

    H, QH, bound = 4, 24, max(bound, T + tokens)
    layers = [Twin(D=D, H=H, QH=QH, capacity_tokens=T + tokens, seed=T, iters=iters).gpu for _ in range(2)]
    k, v = (torch.from_numpy(orc.synth_kv(T, T + tokens, H, D, i)).cuda() for i in (1, 2))
    q, at = torch.from_numpy(orc.synth_q(T, tokens, QH, D)).cuda(), torch.arange(T + tokens, dtype=torch.int32, device="cuda")
    a, b = layers
    for L in layers:
        if T:
            L.append(k[:T], v[:T], at[:T])
    got = [a.attn_prefill(q, k[T:], v[T:], at[T:], 1.0 / np.sqrt(D), bound) for _ in range(2)]  # the second call writes the same rows again
    b.append(k[T:], v[T:], at[T:])
    torch.cuda.synchronize()
    want = b.attn_prefill(q, k[T:], v[T:], at[T:], 1.0 / np.sqrt(D), bound)
    assert torch.equal(got[0], want) and torch.equal(got[1], want)
    _same(a, b)
