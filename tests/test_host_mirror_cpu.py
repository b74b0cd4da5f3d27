"""The C++ mirror of the reference's operator interface compiles against the C ABI and keeps the reference's error
behaviour on the host (no GPU needed: every checked path returns before a launch)."""
import os
import shutil
import subprocess

import pytest

from helpers import ROOT, pkg


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs the CUDA toolkit headers")
def test_host_mirror_compiles_and_rejects_bad_arguments(tmp_path):
    pkg().build()
    libdir = os.path.join(ROOT, "ninfer-3080-iq3_s_b200")
    exe = str(tmp_path / "host_mirror_check")
    subprocess.run(["nvcc", "-std=c++17", "-x", "cu", "-I", os.path.join(libdir, "host"), os.path.join(ROOT, "tests", "cpp", "host_mirror_check.cpp"),
                    "-o", exe, "-L", libdir, "-lkvarn_b200", "-Xlinker", "-rpath", "-Xlinker", libdir], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "host mirror: ok" in r.stdout


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs the CUDA toolkit headers")
def test_engine_shim_compiles_and_refuses_what_the_reference_refuses(tmp_path):
    pkg().build()
    libdir = os.path.join(ROOT, "ninfer-3080-iq3_s_b200")
    exe = str(tmp_path / "engine_shim_check")
    subprocess.run(["nvcc", "-std=c++17", "-x", "cu", "-I", os.path.join(libdir, "host"), os.path.join(ROOT, "tests", "cpp", "engine_shim_check.cpp"),
                    "-o", exe, "-L", libdir, "-lkvarn_b200", "-Xlinker", "-rpath", "-Xlinker", libdir], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "engine shim: ok" in r.stdout


@pytest.mark.gpu
@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc on the GPU machine")
def test_engine_shim_on_the_gpu_equals_the_c_abi(tmp_path):
    """The engine-shaped launchers (Tensor / PagedKV*LayerView values, op-owned stage) against the C ABI called
    directly on a second, identical cache: prompt chunk, verify step, append + cached decode, bit for bit."""
    libdir = os.path.join(ROOT, "ninfer-3080-iq3_s_b200")
    pkg().capi.load()  # fails loudly if the library is missing
    exe = str(tmp_path / "engine_shim_gpu")
    subprocess.run(["nvcc", "-std=c++17", "-x", "cu", "-I", os.path.join(libdir, "host"), os.path.join(ROOT, "tests", "cpp", "engine_shim_gpu.cpp"),
                    "-o", exe, "-L", libdir, "-lkvarn_b200", "-Xlinker", "-rpath", "-Xlinker", libdir], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "engine shim on the GPU: ok" in r.stdout


def _run_host_check(tmp_path, name):
    exe = str(tmp_path / name)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", os.path.join(ROOT, "ninfer-3080-iq3_s_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", name + ".cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_device_setup_is_done_before_any_thread_goes_on(tmp_path):
    assert "once per device: ok" in _run_host_check(tmp_path, "once_check")


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_chunk_workspaces_cover_every_smaller_call(tmp_path):
    assert "chunk shapes: ok" in _run_host_check(tmp_path, "chunk_shape_check")


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_what_of_a_step_runs_beside_what(tmp_path):
    assert "step: ok" in _run_host_check(tmp_path, "step_check")


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_warps_that_share_rows_leave_together(tmp_path):
    assert "walk: ok" in _run_host_check(tmp_path, "walk_check")


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_every_page_is_dealt_once(tmp_path):
    assert "shares: ok" in _run_host_check(tmp_path, "shares_check")


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_the_schedule_of_a_batch(tmp_path):
    assert "batch plan: ok" in _run_host_check(tmp_path, "batch_plan_check")


def test_chunk_workspaces_are_what_a_call_can_use():
    """24 / 4 heads, 148 SMs: an 8-row verify step takes 74 partials a row at 128 dims and the narrow kernel's at 256; a short prompt
    takes one key range, a chunk at 256 dims three."""
    lib = pkg().capi.load()
    part = {D: 128 * (D + 2) * 4 for D in (128, 256)}
    assert lib.kvb_workspace_bytes(131072, 4, 24, 128, 8, 1) <= 4 * 74 * part[128] + 64
    assert lib.kvb_workspace_bytes(131072, 4, 24, 256, 8, 1) <= 4 * 37 * 16 * 258 * 4 + 64
    assert lib.kvb_prefill_workspace_bytes(777, 4, 24, 128, 777) <= 4 * 37 * 2 * part[128] + 64
    assert lib.kvb_prefill_workspace_bytes(17408, 4, 24, 256, 1024) <= 1.1 * 4 * 48 * 3 * part[256]
