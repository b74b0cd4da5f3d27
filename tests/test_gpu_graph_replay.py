"""Steps as an engine replays them: append and attention captured once, replayed with new rows, positions and queries, the appended rows in the
cache; against the same steps launched one by one on a twin, and the oracle over the bytes the GPU wrote."""
import numpy as np
import pytest

from helpers import ATTN_MAX_ABS, ATTN_REL_L2, PREFILL_MAX_ABS, PREFILL_REL_L2, Twin, attn_close, cpu_twin_of, orc, pkg

pytestmark = pytest.mark.gpu


def _captured(call):
    """`call` captured behind a call of its own (the first use of a kernel on a device sets it up)."""
    import torch

    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        call()
    torch.cuda.current_stream().wait_stream(stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call()
    return graph


# one split, clusters (128 dims) and their like with a merge kernel, several rounds; two rows a warp; the tensor cores' chunk kernel; balanced
@pytest.mark.parametrize("D,H,QH,T,rows,iters", [(128, 4, 24, 60, 1, 0), (128, 4, 24, 126, 4, 0), (128, 4, 24, 1500, 1, 0), (128, 4, 24, 2998, 3, 16), (128, 4, 24, 20000, 1, 0),
                                                 (128, 4, 24, 9000, 8, 0), (256, 4, 24, 60, 1, 0), (256, 4, 24, 1405, 1, 2), (256, 4, 24, 5000, 5, 2)])
def test_steps(D, H, QH, T, rows, iters):
    import torch

    steps, scale = 3, 1.0 / np.sqrt(D)
    tw = [Twin(D=D, H=H, QH=QH, capacity_tokens=T + (steps + 1) * rows, seed=T, iters=iters) for _ in range(2)]
    n = T + steps * rows
    k, v = (torch.from_numpy(orc.synth_kv(T, n, H, D, i)).cuda() for i in (1, 2))
    q = torch.from_numpy(orc.synth_q(T, steps * rows, QH, D)).cuda().view(steps, rows, QH, D)
    at = torch.arange(n, dtype=torch.int32, device="cuda")
    for t in tw:
        t.gpu.append(k[:T], v[:T], at[:T])

    def step(layer, qs, ks, vs, pos, out):
        if rows == 1:
            layer.append_decode(qs[0], ks, vs, pos, scale, n, out=out[0])
        else:
            layer.attn_verify(qs, ks, vs, pos, scale, n, out=out)

    bufs = [torch.empty_like(x) for x in (q[0], k[:rows], v[:rows], at[:rows], q[0])]
    for b, x in zip(bufs, (q[0], k[T:T + rows], v[T:T + rows], at[T:T + rows])):
        b.copy_(x)
    graph = _captured(lambda: step(tw[0].gpu, *bufs))  # (the rows of the first step, appended once ahead of its replay)
    for s in range(steps):
        a, b = T + s * rows, T + (s + 1) * rows
        for buf, x in zip(bufs, (q[s], k[a:b], v[a:b], at[a:b])):
            buf.copy_(x)
        graph.replay()
        out = torch.empty_like(q[s])
        step(tw[1].gpu, q[s], k[a:b], v[a:b], at[a:b], out)
        assert torch.equal(bufs[4], out)
        want = cpu_twin_of(tw[0].gpu).attention(q[s].cpu().numpy(), list(range(a, b)), scale, QH, threads=8, kv_total=b)
        wide = D == 128 and rows * QH // H >= 32
        ok, msg = attn_close(out.float().cpu().numpy(), want, *((PREFILL_MAX_ABS, PREFILL_REL_L2) if wide else (ATTN_MAX_ABS, ATTN_REL_L2)))
        assert ok, msg
    assert all(t.gpu.errors() == 0 for t in tw)


@pytest.mark.parametrize("lengths", [[1, 300, 1500, 700], [20000, 9000, 128, 35646, 8192, 100, 16383, 4097]])
def test_batches(lengths):
    import torch

    H, QH, scale = 4, 24, 128 ** -0.5
    layers, room = [], 40
    for i, n in enumerate(lengths):
        L = pkg().KvarnLayer(128, H, QH, 2 * (n // 128 + 3), torch.from_numpy(orc.shuffled_table(i, 2 * (n // 128 + 3), 2 * (n // 128 + 3))))
        L.append(*(torch.from_numpy(orc.synth_kv(n, n + room, H, 128, j)).cuda()[:n] for j in (1, 2)), torch.arange(n, dtype=torch.int32, device="cuda"))
        layers.append(L)
    batch = pkg().DecodeBatch(layers, [n + room for n in lengths])
    q = torch.zeros((len(lengths), QH, 128), dtype=torch.float16, device="cuda")
    pos, out = torch.tensor([n - 1 for n in lengths], dtype=torch.int32, device="cuda"), torch.empty_like(q)
    graph = _captured(lambda: batch.attn_decode(q, pos, scale, out=out))
    for s in (0, room):  # the same graph over longer caches
        if s:
            for L, n in zip(layers, lengths):
                L.append(*(torch.from_numpy(orc.synth_kv(n, n + room, H, 128, j)).cuda()[n:] for j in (1, 2)), torch.arange(n, n + room, dtype=torch.int32, device="cuda"))
            pos += room
        qn = orc.synth_q(s, len(lengths), QH, 128)
        q.copy_(torch.from_numpy(qn))
        graph.replay()
        for i, (L, n) in enumerate(zip(layers, lengths)):
            want = cpu_twin_of(L).attention(qn[i:i + 1], [n + s - 1], scale, QH, threads=8, kv_total=n + s)
            ok, msg = attn_close(out[i:i + 1].float().cpu().numpy(), want, ATTN_MAX_ABS, ATTN_REL_L2)
            assert ok, (i, n, msg)
        assert all(L.errors() == 0 for L in layers)
