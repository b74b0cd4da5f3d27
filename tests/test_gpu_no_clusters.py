"""A device, or a part of one, that holds no cluster of a short step's CTAs: the step takes the merge kernel's route, to the same bits."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from helpers import ATTN_MAX_ABS, ATTN_REL_L2, ROOT, Twin, attn_close, cpu_twin_of, orc, pkg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def without(tmp_path_factory):
    if shutil.which("nvcc") is None:
        pytest.skip("needs nvcc on the GPU machine")
    home = os.path.join(ROOT, "ninfer-3080-iq3_s_b200")
    pkg().capi.load()
    lib = str(tmp_path_factory.mktemp("no_clusters") / "libstep.so")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-DKVB_NO_CLUSTERS",
                    os.path.join(home, "csrc", "kvb_attn.cu"), "-o", lib, "-L", home, "-lkvarn_b200", "-Xlinker", "-Bsymbolic", "-Xlinker", "-rpath", "-Xlinker", home], check=True)
    return C.CDLL(lib)


@pytest.mark.parametrize("D,H,QH,T,rows,iters", [(128, 4, 24, 1500, 1, 0), (128, 4, 24, 3000, 2, 16), (128, 2, 16, 130, 3, 0), (128, 4, 24, 100, 4, 0), (256, 4, 24, 1400, 1, 2), (256, 4, 24, 1536, 3, 0)])
def test_short_steps_without_clusters(without, D, H, QH, T, rows, iters):
    import torch

    tw = Twin(D=D, H=H, QH=QH, capacity_tokens=T, seed=T, iters=iters)
    at = torch.arange(T, dtype=torch.int32, device=tw.dev)
    tw.gpu.append(*(torch.from_numpy(orc.synth_kv(T, T, H, D, i)).to(tw.dev) for i in (1, 2)), at)
    qn = orc.synth_q(T, rows, QH, D)
    q = torch.from_numpy(qn).to(tw.dev)
    ws = tw.gpu.workspace(T, rows)
    want = cpu_twin_of(tw.gpu).attention(qn, list(range(T - rows, T)), 1.0 / np.sqrt(D), QH, threads=4, kv_total=T)
    outs = []
    for lib, merged in ((pkg().capi.load(), False), (without, True)):
        ws.fill_(float("nan"))
        out = torch.empty_like(q)
        assert lib.kvb_attn_rows(C.byref(tw.gpu.c), C.c_void_p(q.data_ptr()), C.c_void_p(at[T - rows:].data_ptr()), rows, C.c_void_p(at[T - 1:].data_ptr()),
                                 C.c_float(1.0 / np.sqrt(D)), T, C.c_void_p(ws.data_ptr()), C.c_void_p(out.data_ptr()), None) == 0
        torch.cuda.synchronize()
        assert torch.isnan(ws).all() != merged  # partials for the merge kernel
        ok, msg = attn_close(out.float().cpu().numpy(), want, ATTN_MAX_ABS, ATTN_REL_L2)
        assert ok, msg
        outs.append(out)
    assert torch.equal(*outs)
    assert tw.gpu.errors() == 0
