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


@pytest.mark.parametrize("D", [128, 256])
@pytest.mark.parametrize("op,tokens", [("decode", 1), ("verify", 3), ("verify", 8), ("prefill", 40)])
def test_workspace_at_any_float(D, op, tokens):
    """A workspace of the queried size that starts 4, 8 or 12 bytes behind a 16-byte boundary: the same bits, and nothing
    written outside it."""
    import torch

    H, QH, T, scale = 4, 24, 700, 1.0 / np.sqrt(D)
    tw = _filled(D, H, QH, T, room=64)
    lib, capi = pkg().capi.load(), pkg().capi
    q = torch.from_numpy(orc.synth_q(3, tokens, QH, D)).to(tw.dev)
    k, v = (torch.from_numpy(orc.synth_kv(4, tokens, H, D, i)).to(tw.dev) for i in (1, 2))
    pos = torch.arange(T, T + tokens, dtype=torch.int32, device=tw.dev)
    rows = min(tokens, 8)
    need = lib.kvb_prefill_workspace_bytes(T + tokens, H, QH, D, tokens) if op == "prefill" else lib.kvb_workspace_bytes(T + tokens, H, QH, D, rows, 1)
    outs = []
    for shift in (0, 1, 2, 3):
        buf = torch.full((need // 4 + 16,), 7.0, device=tw.dev)
        ws, out = buf[4 + shift:], torch.empty_like(q)
        ptr = [C.c_void_p(x.data_ptr()) for x in (q, k, v, pos, ws, out)]
        if op == "decode":
            tw.gpu.append(k, v, pos)
            capi.check(lib.kvb_attn_decode(C.byref(tw.gpu.c), ptr[0], ptr[3], scale, T + tokens, ptr[4], ptr[5], None))
        elif op == "verify":
            capi.check(lib.kvb_attn_verify(C.byref(tw.gpu.c), *ptr[:4], tokens, scale, T + tokens, ptr[4], ptr[5], None))
        else:
            capi.check(lib.kvb_attn_prefill(C.byref(tw.gpu.c), *ptr[:4], tokens, scale, T + tokens, ptr[4], ptr[5], None))
        torch.cuda.synchronize()
        assert torch.all(buf[:4 + shift] == 7.0) and torch.all(buf[4 + shift + need // 4:] == 7.0)
        outs.append(out)
    assert all(torch.equal(outs[0], x) for x in outs[1:])
    assert tw.gpu.errors() == 0


@pytest.mark.parametrize("D", [128, 256])
@pytest.mark.parametrize("tokens", [1, 4, 8, 9, 40])
def test_rows_without_a_key(D, tokens):
    """A position of -1 (a rank whose range of a sharded sequence is empty passes it for every row): the row's partial is that of
    no key at all, whatever the workspace held before, and the rows beside it are as without it."""
    import torch

    H, QH = 4, 24
    q = torch.from_numpy(orc.synth_q(5, tokens, QH, D)).to("cuda")
    none = torch.full((tokens,), -1, dtype=torch.int32, device="cuda")
    n = tokens * QH * (D + 2)

    def run(tw, pos, kv_len):
        for ws in (tw.gpu.workspace(kv_len, min(tokens, 8)), tw.gpu.prefill_workspace(kv_len, tokens)):
            ws.fill_(3.0)
        return [x.clone() for x in _partial(tw, q, pos, kv_len, torch.full((n,), 7.0, device="cuda"))]

    tw = _filled(D, H, QH, 0)
    m, l, o = run(tw, none, 128)
    assert torch.all(m == float("-inf")) and torch.all(l == 0) and torch.all(o == 0)
    T = 700
    tw = _filled(D, H, QH, T)
    pos = torch.arange(T - tokens, T, dtype=torch.int32, device="cuda")
    want = run(tw, pos, T)
    pos[:tokens // 2] = -1
    got = run(tw, pos, T)
    cut = tokens // 2 * QH
    assert torch.all(got[0][:cut] == float("-inf")) and torch.all(got[1][:cut] == 0) and torch.all(got[2][:cut] == 0)
    assert all(torch.equal(a[cut:], b[cut:]) for a, b in zip(got, want))
    assert tw.gpu.errors() == 0


@pytest.mark.parametrize("T,tokens", [(300, 1), (900, 5), (130, 8), (500, 40)])
def test_a_balanced_cache_of_256_dims_read_without_the_count(T, tokens):
    """At head_dim 256 the balancing factors lie in the planes and are applied whatever sinkhorn_iters the reader gives."""
    import torch

    H, QH, D, scale = 4, 24, 256, 1.0 / 16.0
    tw = _filled(D, H, QH, T, iters=16)
    q = torch.from_numpy(orc.synth_q(6, tokens, QH, D)).to(tw.dev)
    pos = torch.arange(T - tokens, T, dtype=torch.int32, device=tw.dev)
    n = tokens * QH * (D + 2)
    want = _partial(tw, q, pos, T, torch.empty(n, device=tw.dev))
    tw.gpu.c.sinkhorn_iters = 0
    got = _partial(tw, q, pos, T, torch.empty(n, device=tw.dev))
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    out = pkg().merge_partials(*(x.unsqueeze(0) for x in got))
    ref = cpu_twin_of(tw.gpu).attention(q.cpu().numpy(), pos.cpu().numpy(), scale, QH, threads=4, kv_total=T)
    ok, msg = attn_close(out.float().cpu().numpy().reshape(ref.shape), ref, ATTN_MAX_ABS, ATTN_REL_L2)
    assert ok, msg


def _causal_run(tw, q, k, v, T, entry):
    import torch

    pos = torch.arange(T, T + q.shape[0], dtype=torch.int32, device=tw.dev)
    return getattr(tw.gpu, entry)(q, k, v, pos, 1.0 / np.sqrt(tw.D), T + q.shape[0])


@pytest.mark.parametrize("T,tokens,at,entry", [(300, 5, 2, "attn_verify"), (125, 5, 1, "attn_verify"), (255, 8, 7, "attn_verify"), (120, 8, 0, "attn_verify"),
                                               (300, 40, 17, "attn_prefill"), (100, 60, 30, "attn_prefill")])
def test_non_finite_v_reaches_the_rows_that_see_it(T, tokens, at, entry):
    """One row of a step at head_dim 256 overflows in V, in the open tile or in one that the step seals: the rows before it are as
    if that key's V were zero, the rows from it on are not a number."""
    import torch

    H, QH, D = 4, 24, 256
    q, k, v = (torch.from_numpy(x).cuda() for x in (orc.synth_q(7, tokens, QH, D), orc.synth_kv(8, tokens, H, D, 1), orc.synth_kv(8, tokens, H, D, 2)))
    out = {}
    for name, value in (("zero", 0.0), ("inf", float("inf")), ("nan", float("nan"))):
        tw = _filled(D, H, QH, T, room=64)
        v[at] = 0.0
        v[at, 1:3, 77] = value
        out[name] = _causal_run(tw, q, k, v, T, entry).float().view(tokens, H, QH // H, D)
        assert tw.gpu.errors() == 0
    assert torch.isfinite(out["zero"]).all()
    for name in ("inf", "nan"):
        hit, ref = out[name], out["zero"]
        assert torch.equal(hit[:at], ref[:at]) and torch.equal(hit[:, [0, 3]], ref[:, [0, 3]])
        assert torch.isnan(hit[at:, 1:3]).all()


@pytest.mark.parametrize("what", ["scale", "zero point", "dim"])
def test_non_finite_factors_of_a_page(what):
    """A V factor of tile 1 (of token 150, or of a dim) is infinite in the planes, slice 1 only: key ranges without that token (that
    tile) are unaffected, ranges with it are not a number in that slice."""
    import torch

    H, QH, D, T = 4, 24, 256, 400
    tw = _filled(D, H, QH, T)
    q = torch.from_numpy(orc.synth_q(9, 1, QH, D)[0]).to(tw.dev)
    pos = torch.tensor([T - 1], dtype=torch.int32, device=tw.dev)

    def ranges():
        return [[x.clone() for x in tw.gpu.attn_decode_partial(q, pos, 1.0 / 16.0, T, a, b)] for a, b in ((0, 128), (128, 150), (150, 151), (140, 170), (256, T), (0, T))]

    def row(token):
        return tw.gpu.v_scale[int(tw.table[token // 64]), :, token % 64]

    if what == "dim":  # dim 200: entry 0 of scale row 50 of either page
        for page in (2, 3):
            row(64 * page + 50)[:, 0] = 0.0
    else:
        row(150)[:, 5 if what == "scale" else 7] = 0.0
    want = ranges()
    if what == "dim":
        for page in (2, 3):
            row(64 * page + 50)[:, 0] = float("inf")
        hit = [False, True, True, True, False, True]
    else:
        row(150)[:, 5 if what == "scale" else 7] = float("-inf")
        if what == "zero point":  # the whole factor leaves with it
            row(150)[:, 5] = 0.0
        hit = [False, False, True, True, False, True]
    got = ranges()
    for g, w, h in zip(got, want, hit):
        assert torch.equal(g[0], w[0]) and torch.equal(g[1], w[1])
        if h:
            assert torch.isnan(g[2][:, 128:]).all() and torch.isfinite(g[2][:, :128]).all()
        elif what == "dim":
            assert torch.equal(g[2], w[2])
        else:
            assert torch.allclose(g[2], w[2], rtol=0, atol=float(w[2].abs().max()) * 2.0 ** -21)  # another largest scale of the page


def _chunk_reference(tw, q_bits, at, T, dtype=0, without=None):
    """The oracle's attention over the bytes of the GPU's cache, the keys [a, b) of `without` left out."""
    cpu, scale = cpu_twin_of(tw.gpu), 1.0 / np.sqrt(tw.D)
    if without is None:
        return cpu.attention(q_bits, at, scale, tw.QH, dtype=dtype, threads=8, kv_total=T)
    parts = [cpu.attention(q_bits, at, scale, tw.QH, dtype=dtype, threads=8, kv_total=T, key_begin=a, key_end=b, want_partials=True)[1:]
             for a, b in ((0, without[0]), (without[1], T))]
    return np.stack([orc.merge_partials(*(np.stack([p[i][t] for p in parts]) for i in range(3))) for t in range(len(at))])


@pytest.mark.parametrize("entry,T,tokens", [("attn_decode", 700, 1), ("attn_verify", 300, 5), ("attn_verify", 125, 8), ("attn_prefill", 0, 64), ("attn_prefill", 700, 40)])
@pytest.mark.parametrize("iters", [0, 16])
def test_bf16_rows_of_256_dims(entry, T, tokens, iters):
    """The engine's own type and geometry.  What is left is the rounding of the output: 2^-9 of a value at most, 10 % on top."""
    import torch

    from helpers import from_bits, to_bits

    H, QH, D, end = 4, 24, 256, T + tokens
    tw = Twin(D=D, H=H, QH=QH, capacity_tokens=end, seed=T, dtype=1, iters=iters)
    kb, vb = (to_bits(orc.synth_kv(13, end, H, D, i), 1) for i in (1, 2))
    qb = to_bits(orc.synth_q(13, tokens, QH, D), 1)
    k, v, q = (from_bits(x, 1).to(tw.dev) for x in (kb, vb, qb))
    pos = torch.arange(end, dtype=torch.int32, device=tw.dev)
    if T:
        tw.gpu.append(k[:T], v[:T], pos[:T])
    if entry == "attn_decode":
        tw.gpu.append(k[T:], v[T:], pos[T:])
        out = tw.gpu.attn_decode(q[0], pos[T:], 1.0 / 16.0, end).unsqueeze(0)
    else:
        out = getattr(tw.gpu, entry)(q, k[T:], v[T:], pos[T:], 1.0 / 16.0, end)
    assert out.dtype == torch.bfloat16 and tw.gpu.errors() == 0
    want = _chunk_reference(tw, qb, np.arange(T, end, dtype=np.int32), end, dtype=1)
    ok, msg = attn_close(out.float().cpu().numpy(), want, 1.1 * 2.0 ** -8, 1.1 * 2.0 ** -8 / 3 ** 0.5)
    assert ok, msg


# key ranges per row 17 .. 32, 33 .. 64, 65 .. 128: a CTA per row merges them
@pytest.mark.parametrize("H,QH,ctx,tokens", [(8, 8, 12000, 9), (4, 4, 16300, 9), (2, 4, 33000, 9), (4, 24, 16384, 32)])
@pytest.mark.parametrize("D", [128, 256])
def test_chunks_over_many_key_ranges(D, H, QH, ctx, tokens):
    """... as output and as the merged partial of a chunk."""
    import torch

    T, scale = ctx + tokens, 1.0 / np.sqrt(D)
    tw = _filled(D, H, QH, T, room=0, seed=14)
    qn = orc.synth_q(15, tokens, QH, D)
    q, at = torch.from_numpy(qn).to(tw.dev), np.arange(ctx, T, dtype=np.int32)
    pos = torch.from_numpy(at).to(tw.dev)
    m, l, o = _partial(tw, q, pos, T, torch.empty(tokens * QH * (D + 2), device=tw.dev))
    merged = pkg().merge_partials(m[None], l[None], o[None]).view(tokens, QH, D)
    k, v = (torch.from_numpy(orc.synth_kv(14, T, H, D, i)[ctx:]).to(tw.dev) for i in (1, 2))
    out = tw.gpu.attn_prefill(q, k, v, pos, scale, T)
    assert tw.gpu.errors() == 0
    want = _chunk_reference(tw, qn, at, T)
    tol = (PREFILL_MAX_ABS, PREFILL_REL_L2) if D == 128 else (ATTN_MAX_ABS, ATTN_REL_L2)
    for what, x in (("output", out), ("partial", merged)):
        ok, msg = attn_close(x.float().cpu().numpy(), want, *tol)
        assert ok, what + ": " + msg


@pytest.mark.parametrize("D,H,QH,ctx,tokens,cuts", [(256, 4, 24, 900, 3, (128, 512)), (256, 4, 24, 900, 8, (200, 450)), (256, 4, 24, 900, 50, (128, 512)), (256, 2, 16, 500, 200, (100, 300)),
                                                    (128, 4, 24, 900, 50, (128, 512))])
def test_chunk_partials_of_tile_ranges(D, H, QH, ctx, tokens, cuts):
    """The rows of a chunk over three caches that hold consecutive tile ranges (the last one also the rows themselves): the merged
    partials are the attention over the whole sequence."""
    import torch

    T = ctx + tokens
    k, v, qn = orc.synth_kv(16, T, H, D, 1), orc.synth_kv(16, T, H, D, 2), orc.synth_q(16, tokens, QH, D)
    cuts = [0] + [c // 128 * 128 for c in cuts] + [T]
    whole = _filled(D, H, QH, 0, room=T)
    whole.gpu.append(*(torch.from_numpy(x).to(whole.dev) for x in (k, v)), torch.arange(T, dtype=torch.int32, device=whole.dev))
    parts = []
    for i, (a, b) in enumerate(zip(cuts, cuts[1:])):
        tw = _filled(D, H, QH, 0, room=b - a + 128, seed=i)
        if b > a:
            tw.gpu.append(*(torch.from_numpy(x[a:b].copy()).to(tw.dev) for x in (k, v)), torch.arange(b - a, dtype=torch.int32, device=tw.dev))
        last = i == len(cuts) - 2
        at = torch.arange(ctx - a, T - a, dtype=torch.int32, device=tw.dev) if last else torch.full((tokens,), b - a - 1, dtype=torch.int32, device=tw.dev)
        parts.append([x.clone() for x in _partial(tw, torch.from_numpy(qn).to(tw.dev), at, max(b - a, 1), torch.empty(tokens * QH * (D + 2), device=tw.dev))])
    out = pkg().merge_partials(*(torch.stack(x) for x in zip(*parts))).view(tokens, QH, D)
    want = _chunk_reference(whole, qn, np.arange(ctx, T, dtype=np.int32), T)
    ok, msg = attn_close(out.float().cpu().numpy(), want, *((PREFILL_MAX_ABS, PREFILL_REL_L2) if D == 128 else (ATTN_MAX_ABS, ATTN_REL_L2)))
    assert ok, msg


@pytest.mark.parametrize("D,H,QH,ctx,tokens", [(128, 4, 24, 900, 8), (128, 4, 24, 900, 40), (128, 8, 64, 600, 300), (256, 4, 24, 900, 5), (256, 4, 24, 900, 40), (256, 2, 16, 500, 90)])
@pytest.mark.parametrize("bad", [-7, 1 << 20])
def test_bad_page_in_the_prefix_of_a_chunk(D, H, QH, ctx, tokens, bad):
    """A table entry outside the pool: reported in the error word, and the keys of its page (at 128 dims from 32 rows on: of its
    tile) are left out."""
    import torch

    T, page = ctx + tokens, 5
    tw = _filled(D, H, QH, T, room=0, seed=17)
    tw.gpu.table[page] = bad
    qn, at = orc.synth_q(18, tokens, QH, D), np.arange(ctx, T, dtype=np.int32)
    m, l, o = _partial(tw, torch.from_numpy(qn).to(tw.dev), torch.from_numpy(at).to(tw.dev), T, torch.empty(tokens * QH * (D + 2), device=tw.dev))
    out = pkg().merge_partials(m[None], l[None], o[None]).view(tokens, QH, D)
    assert tw.gpu.errors() == pkg().capi.ERR_PAGE_RANGE
    tw.gpu.table[page] = 0  # for the oracle: a page it may read (its keys are left out)
    tile = D == 128 and tokens * QH // H >= 32
    want = _chunk_reference(tw, qn, at, T, without=(page // 2 * 128, (page // 2 + 1) * 128) if tile else (64 * page, 64 * (page + 1)))
    ok, msg = attn_close(out.float().cpu().numpy(), want, *((PREFILL_MAX_ABS, PREFILL_REL_L2) if tile else (ATTN_MAX_ABS, ATTN_REL_L2)))
    assert ok, msg


@pytest.mark.parametrize("D", [128, 256])
@pytest.mark.parametrize("bound", [400, 20000])
@pytest.mark.parametrize("newest", [-48, -50, -129, -100000])
def test_a_newest_position_below_zero(D, bound, newest):
    """No key is there: zeros by every entry point, on any number of splits, and what an append says of the positions."""
    import torch

    H, QH, scale = 4, 24, 1.0 / np.sqrt(D)
    tw = _filled(D, H, QH, 300, room=20000)
    L, bad = tw.gpu, pkg().capi.ERR_POSITIONS

    def rows(n, heads):
        return torch.ones((n, heads, D), dtype=torch.float16, device=tw.dev)

    def zeros(out, errors):
        torch.cuda.synchronize()
        assert torch.all(out == 0.0) and L.errors() == errors
        L.error_word.zero_()

    at = torch.arange(newest - 39, newest + 1, dtype=torch.int32, device=tw.dev)
    zeros(L.attn_decode(rows(1, QH)[0], at[39:], scale, bound), 0)
    zeros(L.append_decode(rows(1, QH)[0], rows(1, H), rows(1, H), at[39:], scale, bound), bad)
    for n in (2, 5, 8):
        zeros(L.attn_verify(rows(n, QH), rows(n, H), rows(n, H), at[40 - n:], scale, bound), bad)
    zeros(L.attn_prefill(rows(40, QH), rows(40, H), rows(40, H), at, scale, bound), bad)
    if D == 128:
        zeros(pkg().DecodeBatch([L, L], [bound, bound]).attn_decode(rows(2, QH), at[39:].repeat(2), scale), 0)
