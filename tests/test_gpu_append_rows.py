"""The rows an append reads and the codes it writes at their edges: rows that start at any 2-byte boundary, values that lie exactly in the
middle between two codes, rows without any spread.  The oracle's bytes, all of them."""
import numpy as np
import pytest

from helpers import Twin, orc

pytestmark = pytest.mark.gpu


def _planes(layer):
    return [x.cpu().numpy() for x in (layer.k_code, layer.v_code)] + [x.cpu().numpy().view(np.uint16) for x in (layer.k_scale, layer.v_scale, layer.stage)]


@pytest.mark.parametrize("D", [128, 256])
@pytest.mark.parametrize("T,iters", [(1, 0), (129, 0), (300, 0), (256, 3)])
@pytest.mark.parametrize("shift", [1, 4, 7])
def test_rows_at_any_boundary(D, T, iters, shift):
    import torch

    H, QH = 4, 24
    k, v = (torch.from_numpy(orc.synth_kv(0, T, H, D, i)).cuda() for i in (1, 2))
    at = torch.arange(T, dtype=torch.int32, device="cuda")
    got = []
    for s in (0, shift):
        layer = Twin(D=D, H=H, QH=QH, capacity_tokens=T, seed=3, iters=iters).gpu
        rows = []
        for x in (k, v):
            buf = torch.zeros(x.numel() + 8, dtype=x.dtype, device="cuda")
            rows.append(buf[s:s + x.numel()].view(x.shape))
            rows[-1].copy_(x)
        layer.append(*rows, at)
        got.append(_planes(layer))
    assert all((a == b).all() for a, b in zip(*got))


@pytest.mark.parametrize("kind", ["middles", "constant", "two values"])
def test_codes_at_the_middle(kind):
    """Rotated values of 256 dims that are small whole numbers, exact in fp16: a row of 0 .. 30 has scale 2, its odd values lie in the
    middle between two codes (rounded away from zero)."""
    import torch

    D, H, T = 256, 2, 128
    rng = np.random.default_rng(5)
    d = np.zeros((T, H, D))
    if kind == "middles":
        for t in range(T):
            for h in range(H):
                for s in range(2):
                    d[t, h, 128 * s + rng.permutation(128)[:4]] = (30, 1, 15, 7)
    elif kind == "two values":
        d[:, :, ::64] = 3
    h2 = np.ones((1, 1))
    while h2.shape[0] < D:
        h2 = np.block([[h2, h2], [h2, -h2]])
    x = d @ h2 / 16
    rows = x.astype(np.float16)
    assert (rows == x).all()
    tw = Twin(D=D, H=H, QH=H, capacity_tokens=T, seed=1)
    at = torch.arange(T, dtype=torch.int32, device="cuda")
    dev = torch.from_numpy(rows).cuda()
    tw.gpu.append(dev, dev, at)
    tw.cpu.append(rows, rows, 0)
    got = _planes(tw.gpu)
    want = [tw.cpu.k_code, tw.cpu.v_code, np.asarray(tw.cpu.k_scale).view(np.uint16), np.asarray(tw.cpu.v_scale).view(np.uint16)]
    assert all((np.asarray(a).reshape(-1) == np.asarray(b).reshape(-1)).all() for a, b in zip(got, want))
    if kind == "middles":
        assert got[1].max() > 0x0F


@pytest.mark.parametrize("D", [128, 256])
@pytest.mark.parametrize("shift", [0, 3])
@pytest.mark.parametrize("before,T", [(0, 16), (3, 17), (0, 32), (5, 33), (0, 48), (0, 49), (60, 64), (100, 30), (90, 300), (120, 140)])
def test_few_rows_and_many(D, shift, before, T):
    """Rows of a tile that a warp each rotates, and more: tiles left open, completed, and a long append that begins inside one.  The oracle's
    stage and planes."""
    import torch

    H, QH = 4, 24
    tw = Twin(D=D, H=H, QH=QH, capacity_tokens=before + T, seed=2)
    k, v = (orc.synth_kv(T, before + T, H, D, i) for i in (1, 2))
    if before:
        tw.append(k[:before], v[:before])
    rows = []
    for x in (k, v):
        x = torch.from_numpy(x[before:]).cuda()
        buf = torch.zeros(x.numel() + 8, dtype=x.dtype, device="cuda")
        rows.append(buf[shift:shift + x.numel()].view(x.shape))
        rows[-1].copy_(x)
    tw.gpu.append(*rows, torch.arange(before, before + T, dtype=torch.int32, device="cuda"))
    tw.cpu.append(k[before:].view(np.uint16), v[before:].view(np.uint16), before, 0)
    tw.len = before + T
    assert tw.live_stage_equal()
    assert all(tw.planes_equal().values()) and tw.gpu.errors() == 0
