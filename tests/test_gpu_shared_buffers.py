"""Steps whose buffers share memory: a workspace that begins with k, v and the positions, an output in the place of q, a token further,
over k or over the positions.  The rows of the step are read before anything is written over them: the same bits as with
buffers of their own."""
import ctypes as C

import numpy as np
import pytest

from helpers import Twin, orc, pkg

pytestmark = pytest.mark.gpu


def _run(D, H, QH, T, op, tokens, bound, place):
    """One step on a fresh cache; `place` maps the sizes (in 16-bit elements) of q, k, v, pos, ws and out to their offsets in one buffer."""
    import torch

    lib, capi = pkg().capi.load(), pkg().capi
    tw = Twin(D=D, H=H, QH=QH, capacity_tokens=max(T + tokens, bound), seed=T, iters=0)
    kv = [torch.from_numpy(orc.synth_kv(T + 1, T + tokens, H, D, i)).to(tw.dev) for i in (1, 2)]
    at = torch.arange(T + tokens, dtype=torch.int32, device=tw.dev)
    if T:
        tw.gpu.append(kv[0][:T], kv[1][:T], at[:T])
    q = torch.from_numpy(orc.synth_q(T, tokens, QH, D)).to(tw.dev)
    need = lib.kvb_prefill_workspace_bytes(bound, H, QH, D, tokens) if op == "prefill" else lib.kvb_workspace_bytes(bound, H, QH, D, tokens, 1)
    size = {"q": q.numel(), "k": tokens * H * D, "v": tokens * H * D, "pos": 2 * tokens, "ws": (need + 31) // 32 * 16, "out": q.numel()}
    offset = place(size)
    buf = torch.zeros(max(offset[x] + size[x] for x in size) + 64, dtype=torch.int16, device=tw.dev)
    for name, x in (("q", q), ("k", kv[0][T:]), ("v", kv[1][T:]), ("pos", at[T:])):
        buf[offset[name]:offset[name] + size[name]] = x.contiguous().view(torch.int16).flatten()
    ptr = {x: C.c_void_p(buf.data_ptr() + 2 * offset[x]) for x in size}
    scale = 1.0 / np.sqrt(D)
    torch.cuda.synchronize()
    if op == "decode":
        capi.check(lib.kvb_append_decode(C.byref(tw.gpu.c), ptr["q"], ptr["k"], ptr["v"], ptr["pos"], scale, bound, ptr["ws"], None, ptr["out"], None))
    else:
        call = lib.kvb_attn_verify if op == "verify" else lib.kvb_attn_prefill
        capi.check(call(C.byref(tw.gpu.c), ptr["q"], ptr["k"], ptr["v"], ptr["pos"], tokens, scale, bound, ptr["ws"], ptr["out"], None))
    torch.cuda.synchronize()
    assert tw.gpu.errors() == 0
    g = tw.gpu
    return [buf[offset["out"]:offset["out"] + size["out"]].clone(), g.stage, g.k_code, g.v_code, g.k_scale, g.v_scale]


def _apart(size):
    at, out = 0, {}
    for name, n in size.items():
        out[name] = at
        at += (n + 63) // 64 * 64
    return out


@pytest.mark.parametrize("D,T,op,tokens,bound", [(128, 700, "decode", 1, 701), (128, 4095, "decode", 1, 9000), (256, 700, "decode", 1, 2000), (128, 2000, "verify", 3, 2003), (128, 127, "verify", 8, 9000),
                                                 (256, 700, "verify", 5, 705), (128, 700, "prefill", 40, 9000), (256, 500, "prefill", 40, 6000), (128, 0, "prefill", 780, 780)])
def test_a_workspace_over_the_rows_of_the_step(D, T, op, tokens, bound):
    def over(size):
        at = _apart(size)
        at.update(k=at["ws"], v=at["ws"] + size["k"])
        assert size["k"] + size["v"] <= size["ws"]
        return at

    want = _run(D, 4, 24, T, op, tokens, bound, _apart)
    got = _run(D, 4, 24, T, op, tokens, bound, over)
    assert all((a == b).all() for a, b in zip(got, want))


# 780 tokens alone: finished in the chunk kernel where the output allows it
@pytest.mark.parametrize("D,T,op,tokens", [(128, 0, "prefill", 780), (128, 0, "verify", 8), (128, 300, "decode", 1), (256, 300, "prefill", 40)])
@pytest.mark.parametrize("where", ["q", "a token after q", "k", "positions"])
def test_an_output_over_what_the_step_reads(D, T, op, tokens, where):
    H, QH, bound = 4, 24, T + tokens

    def over(size):
        at = _apart(size)
        free = max(at[x] + size[x] for x in size)
        if where == "q":
            at["out"] = at["q"]
        elif where == "a token after q":
            at["out"] = at["q"] = (free + 63) // 64 * 64
            at["out"] += QH * D
        else:  # `where` lies inside the output
            at["out"] = (free + 63) // 64 * 64
            at["k" if where == "k" else "pos"] = at["out"] + (0 if where == "k" else 64)
        return at

    want = _run(D, H, QH, T, op, tokens, bound, _apart)
    got = _run(D, H, QH, T, op, tokens, bound, over)
    assert all((a == b).all() for a, b in zip(got[1:], want[1:]))
    if T == 0 and where in ("a token after q", "positions"):  # merged by the merge kernel: the same sums in another order, rounded to fp16
        import torch

        a, b = (x[0].view(torch.float16).float() for x in (got, want))
        assert (a - b).abs().max() <= b.abs().max() * 2.0 ** -11
    else:
        assert (got[0] == want[0]).all()
