"""Chunks whose rows see one key range are finished in chunk_kernel itself (head_dim 128): no partials, no merge kernel.  Compared
with the merge kernel's route -- taken by an output that starts at no 16-byte boundary -- and with the oracle."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from helpers import PREFILL_MAX_ABS, PREFILL_REL_L2, ROOT, Twin, attn_close, cpu_twin_of, orc, pkg

pytestmark = pytest.mark.gpu


# split walks of one and several key tiles, the second stream without a tile, ragged row tiles; two row tiles a CTA, the last one
# alone or with few rows; rows of a group that end inside a row tile (7 and 3 query heads a KV head).  Which walk a shape takes at 148
# SMs: tests/cpp/chunk_shape_check.cpp
@pytest.mark.parametrize("H,QH,ctx,tokens,dtype,iters", [(4, 24, 0, 780, 0, 0), (8, 64, 0, 128, 0, 16), (8, 64, 0, 290, 1, 0), (4, 28, 5, 680, 0, 16), (4, 24, 0, 1024, 0, 0),
                                                         (8, 24, 130, 1000, 1, 16), (8, 64, 0, 1023, 0, 0), (1, 3, 0, 20, 0, 0), (2, 16, 0, 8, 1, 0)])
def test_finished_rows(H, QH, ctx, tokens, dtype, iters):
    import torch

    D, T = 128, ctx + tokens
    scale = 1.0 / np.sqrt(D)
    k, v, qn = orc.synth_kv(T, T, H, D, 1), orc.synth_kv(T, T, H, D, 2), orc.synth_q(T, tokens, QH, D)
    got = []
    for shift in (0, 1):  # elements
        tw = Twin(D=D, H=H, QH=QH, capacity_tokens=T, seed=T, dtype=dtype, iters=iters)
        kd, vd, q = (torch.from_numpy(x).to(tw.dev).to(tw.gpu.dtype) for x in (k, v, qn))
        at = torch.arange(T, dtype=torch.int32, device=tw.dev)
        if ctx:
            tw.gpu.append(kd[:ctx], vd[:ctx], at[:ctx])
        ws = tw.gpu.prefill_workspace(T, tokens).fill_(float("nan"))
        buf = torch.full((q.numel() + 16,), 7.0, dtype=q.dtype, device=tw.dev)
        out = buf[8 + shift:8 + shift + q.numel()]
        args = [C.c_void_p(x.data_ptr()) for x in (q, kd[ctx:], vd[ctx:], at[ctx:])]
        pkg().capi.check(pkg().capi.load().kvb_attn_prefill(C.byref(tw.gpu.c), *args, tokens, scale, T, C.c_void_p(ws.data_ptr()), C.c_void_p(out.data_ptr()), None))
        torch.cuda.synchronize()
        assert torch.all(buf[:8 + shift] == 7.0) and torch.all(buf[8 + shift + q.numel():] == 7.0)
        assert tw.gpu.errors() == 0
        assert torch.isnan(ws).all() if shift == 0 else not torch.isnan(ws).all()  # partials are written for the merge kernel alone
        got.append(out.view(tokens, QH, D).float().cpu().numpy())
    # both routes round the same sums (fp32 sums in another order) to the output type
    assert np.abs(got[0] - got[1]).max() <= np.abs(got[1]).max() * (2.0 ** -8 if dtype else 2.0 ** -11)
    rows = np.unique(np.concatenate([np.arange(0, tokens, max(1, tokens // 6)), [tokens - 1]]))
    bits = q.view(torch.int16).cpu().numpy().view(np.uint16)[rows] if dtype else qn[rows]
    want = cpu_twin_of(tw.gpu).attention(bits, np.arange(ctx, T, dtype=np.int32)[rows], scale, QH, dtype=dtype, threads=8, kv_total=T)
    tol = (PREFILL_MAX_ABS, PREFILL_REL_L2) if dtype == 0 else (2.0 ** -7, 2.0 ** -7)  # bf16: half a unit of the output, 2^-9 of a value, and of P's, K's and V's rounding
    ok, msg = attn_close(got[0][rows], want, *tol)
    assert ok, msg


def _both_routes(call, numel, dtype):
    """What `call(out)` writes to an output at a 16-byte boundary (finished in the chunk kernel) and to one element further (merged)."""
    import torch

    outs = []
    for shift in (0, 1):
        buf = torch.full((numel + 16,), 7.0, dtype=dtype, device="cuda")
        out = buf[8 + shift:8 + shift + numel]
        call(C.c_void_p(out.data_ptr()))
        torch.cuda.synchronize()
        assert torch.all(buf[:8 + shift] == 7.0) and torch.all(buf[8 + shift + numel:] == 7.0)
        outs.append(out.float())
    return outs


@pytest.mark.parametrize("H,QH,ctx,tokens,iters", [(8, 64, 140, 290, 0), (8, 64, 250, 8, 16), (8, 24, 130, 1000, 16), (4, 24, 300, 40, 0)])
@pytest.mark.parametrize("bad", [-7, 1 << 20])
def test_finished_rows_over_a_bad_page(H, QH, ctx, tokens, iters, bad):
    """A table entry of the prefix outside the pool: reported, its tile left out, by either route."""
    import torch

    D, T = 128, ctx + tokens
    k, v, q = (torch.from_numpy(x).cuda() for x in (orc.synth_kv(T, T, H, D, 1), orc.synth_kv(T, T, H, D, 2), orc.synth_q(T, tokens, QH, D)))
    at = torch.arange(T, dtype=torch.int32, device="cuda")

    def rows(entry):
        def call(out):  # each on a cache of its own: a long chunk cannot be rolled back
            tw = Twin(D=D, H=H, QH=QH, capacity_tokens=T, seed=T, iters=iters)
            tw.gpu.append(k[:ctx], v[:ctx], at[:ctx])
            if entry is not None:
                tw.gpu.table[1] = entry
            args = [C.c_void_p(x.data_ptr()) for x in (q, k[ctx:], v[ctx:], at[ctx:])]
            ws = tw.gpu.prefill_workspace(T, tokens)
            pkg().capi.check(pkg().capi.load().kvb_attn_prefill(C.byref(tw.gpu.c), *args, tokens, 1.0 / np.sqrt(D), T, C.c_void_p(ws.data_ptr()), out, None))
            assert tw.gpu.errors() == (0 if entry is None else pkg().capi.ERR_PAGE_RANGE)

        return _both_routes(call, q.numel(), q.dtype)

    whole, got = rows(None), rows(bad)
    assert torch.isfinite(got[0]).all() and not torch.equal(got[0], whole[0])
    for a, b in (whole, got):
        assert (a - b).abs().max() <= b.abs().max() * 2.0 ** -11


@pytest.mark.parametrize("H,QH,T,rows", [(8, 64, 250, 8), (4, 24, 200, 8), (4, 32, 130, 5), (8, 64, 60, 4)])
def test_finished_rows_of_attn_rows(H, QH, T, rows):
    """Rows that are in the cache already, in any order, some of them without a key: zeros there, the others by either route alike."""
    import torch

    D = 128
    tw = Twin(D=D, H=H, QH=QH, capacity_tokens=T, seed=T)
    at = torch.arange(T, dtype=torch.int32, device=tw.dev)
    tw.gpu.append(*(torch.from_numpy(orc.synth_kv(T, T, H, D, i)).to(tw.dev) for i in (1, 2)), at)
    qn = orc.synth_q(T, rows, QH, D)
    q = torch.from_numpy(qn).to(tw.dev)
    seen = np.array([T - 1, -1, 0, T // 2, 127, -1, T - 2, 64][:rows]).clip(max=T - 1).astype(np.int32)
    pos, lib, ws = torch.from_numpy(seen).to(tw.dev), pkg().capi.load(), tw.gpu.workspace(T, rows).fill_(float("nan"))

    def call(out):
        pkg().capi.check(lib.kvb_attn_rows(C.byref(tw.gpu.c), C.c_void_p(q.data_ptr()), C.c_void_p(pos.data_ptr()), rows, C.c_void_p(at[T - 1:].data_ptr()), 1.0 / np.sqrt(D), T,
                                           C.c_void_p(ws.data_ptr()), out, None))

    a, b = (x.view(rows, QH, D) for x in _both_routes(call, q.numel(), q.dtype))
    assert tw.gpu.errors() == 0
    none = torch.from_numpy(seen < 0).to(tw.dev)
    assert torch.all(a[none] == 0.0) and torch.all(b[none] == 0.0)
    assert (a - b).abs().max() <= b.abs().max() * 2.0 ** -11
    want = cpu_twin_of(tw.gpu).attention(qn[seen >= 0], seen[seen >= 0], 1.0 / np.sqrt(D), QH, threads=8, kv_total=T)
    ok, msg = attn_close(a[~none].cpu().numpy(), want, PREFILL_MAX_ABS, PREFILL_REL_L2)
    assert ok, msg


@pytest.fixture(scope="module")
def gives_up(tmp_path_factory):
    """The chunk kernel built with waits that never look at their barrier: every one of them gives up at once, no MMA is issued."""
    if shutil.which("nvcc") is None:
        pytest.skip("needs nvcc on the GPU machine")
    home = os.path.join(ROOT, "ninfer-3080-iq3_s_b200")
    pkg().capi.load()
    lib = str(tmp_path_factory.mktemp("gives_up") / "libchunk.so")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-DKVB_CHUNK_PROBES=0u",
                    os.path.join(home, "csrc", "kvb_prefill.cu"), "-o", lib, "-L", home, "-lkvarn_b200", "-Xlinker", "-rpath", "-Xlinker", home], check=True)
    return C.CDLL(lib).kvb_attn_prefill


# finished in the kernel (two row tiles a CTA, split keys with tiles for both streams and for one), and merged
@pytest.mark.parametrize("H,QH,ctx,tokens,shift", [(4, 24, 0, 780, 0), (8, 64, 0, 290, 0), (1, 3, 0, 20, 0), (4, 24, 0, 780, 1), (4, 24, 900, 40, 0)])
def test_a_chunk_that_gives_up(gives_up, H, QH, ctx, tokens, shift):
    """A wait that runs out is reported, the rows are zeros and nothing beside them is touched; the next call is as if nothing had been."""
    import torch

    D, T = 128, ctx + tokens
    k, v, q = orc.synth_kv(T, T, H, D, 1), orc.synth_kv(T, T, H, D, 2), orc.synth_q(T, tokens, QH, D)
    for call in (gives_up, pkg().capi.load().kvb_attn_prefill):
        tw = Twin(D=D, H=H, QH=QH, capacity_tokens=T, seed=T)
        kd, vd, qd = (torch.from_numpy(x).to(tw.dev) for x in (k, v, q))
        at = torch.arange(T, dtype=torch.int32, device=tw.dev)
        if ctx:
            tw.gpu.append(kd[:ctx], vd[:ctx], at[:ctx])
        ws = tw.gpu.prefill_workspace(T, tokens).fill_(float("nan"))
        buf = torch.full((qd.numel() + 16,), 7.0, dtype=qd.dtype, device=tw.dev)
        out = buf[8 + shift:8 + shift + qd.numel()]
        args = [C.c_void_p(x.data_ptr()) for x in (qd, kd[ctx:], vd[ctx:], at[ctx:])]
        assert call(C.byref(tw.gpu.c), *args, tokens, C.c_float(1.0 / np.sqrt(D)), T, C.c_void_p(ws.data_ptr()), C.c_void_p(out.data_ptr()), None) == 0
        torch.cuda.synchronize()
        assert torch.all(buf[:8 + shift] == 7.0) and torch.all(buf[8 + shift + qd.numel():] == 7.0)
        if call is gives_up:
            assert tw.gpu.errors() == pkg().capi.ERR_WAIT_TIMEOUT
            assert torch.all(out == 0.0)
        else:
            assert tw.gpu.errors() == 0
            got = out.view(tokens, QH, D).float().cpu().numpy()
            rows = np.array([0, tokens // 2, tokens - 1])
            want = cpu_twin_of(tw.gpu).attention(q[rows], np.arange(ctx, T, dtype=np.int32)[rows], 1.0 / np.sqrt(D), QH, threads=8, kv_total=T)
            ok, msg = attn_close(got[rows], want, PREFILL_MAX_ABS, PREFILL_REL_L2)
            assert ok, msg
