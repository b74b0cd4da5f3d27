"""Decode and verify steps whose waits for a chunk of K, or of V, give up at once while the chunk is still on its way: reported, nothing
written beside the output, and the call behind it is as if nothing had been.  The kernels are built for it: no wait of the library is
made to run out."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from helpers import ROOT, Twin, orc, pkg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def builds(tmp_path_factory):
    if shutil.which("nvcc") is None:
        pytest.skip("needs nvcc on the GPU machine")
    home = os.path.join(ROOT, "ninfer-3080-iq3_s_b200")
    pkg().capi.load()
    made = {}
    for what in "KV":
        lib = str(tmp_path_factory.mktemp("gives_up") / ("libstep_%s.so" % what))
        made[what] = lib, subprocess.Popen(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                                            "-DKVB_STEP_PROBES_%s=0u" % what, os.path.join(home, "csrc", "kvb_attn.cu"), "-o", lib, "-L", home, "-lkvarn_b200",
                                            "-Xlinker", "-Bsymbolic", "-Xlinker", "-rpath", "-Xlinker", home])
    for lib, build in made.values():
        assert build.wait() == 0
    return {what: C.CDLL(lib) for what, (lib, _) in made.items()}


# clusters and splits with a merge kernel, one page a warp and several, one row block a warp and two, both head dims
@pytest.mark.parametrize("D,H,QH,T,rows,iters", [(128, 4, 24, 1500, 1, 0), (128, 4, 24, 3000, 4, 16), (128, 8, 64, 20000, 1, 0), (128, 8, 64, 9000, 2, 16), (128, 8, 40, 9001, 3, 0),
                                                 (256, 4, 24, 1400, 1, 0), (256, 8, 64, 5000, 2, 16)])
@pytest.mark.parametrize("what", ["K", "V"])
def test_a_step_that_gives_up(builds, what, D, H, QH, T, rows, iters):
    import torch

    tw = Twin(D=D, H=H, QH=QH, capacity_tokens=T, seed=T, iters=iters)
    at = torch.arange(T, dtype=torch.int32, device=tw.dev)
    tw.gpu.append(*(torch.from_numpy(orc.synth_kv(T, T, H, D, i)).to(tw.dev) for i in (1, 2)), at)
    q = torch.from_numpy(orc.synth_q(T, rows, QH, D)).to(tw.dev)
    ws = tw.gpu.workspace(T, rows)
    buf = torch.empty(q.numel() + 16, dtype=q.dtype, device=tw.dev)

    def rows_of(lib):
        buf.fill_(7.0)
        assert lib.kvb_attn_rows(C.byref(tw.gpu.c), C.c_void_p(q.data_ptr()), C.c_void_p(at[T - rows:].data_ptr()), rows, C.c_void_p(at[T - 1:].data_ptr()),
                                 C.c_float(1.0 / np.sqrt(D)), T, C.c_void_p(ws.data_ptr()), C.c_void_p(buf[8:].data_ptr()), None) == 0
        torch.cuda.synchronize()
        assert torch.all(buf[:8] == 7.0) and torch.all(buf[-8:] == 7.0)
        return buf[8:-8].clone(), tw.gpu.errors()

    library = pkg().capi.load()
    want, errors = rows_of(library)
    assert errors == 0 and torch.isfinite(want).all()
    assert rows_of(builds[what])[1] == pkg().capi.ERR_WAIT_TIMEOUT
    tw.gpu.error_word.zero_()
    got, errors = rows_of(library)
    assert errors == 0 and torch.equal(got, want)
