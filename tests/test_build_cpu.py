"""The build script: the C library needs no torch, and the Python calls follow torch and Python.  Compilers are replaced by a script
that writes down its call and its output file."""
import importlib.metadata
import importlib.util
import os
import re
import shutil
import stat
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture
def script(tmp_path, monkeypatch):
    spec = importlib.util.spec_from_file_location("bonsai_b200_build_test", os.path.join(ROOT, "p40-kernel_b200", "build.py"))
    b = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(b)
    for tool in ("nvcc", "cxx"):
        path = tmp_path / tool
        path.write_text('#!/bin/sh\necho %s >> %s/log\nwhile [ "$1" != -o ]; do shift; done\necho made > "$2"\n' % (tool, tmp_path))
        path.chmod(path.stat().st_mode | stat.S_IXUSR)
    monkeypatch.setattr(b, "LIB", str(tmp_path / "lib.so"))
    monkeypatch.setattr(b, "CALLS", str(tmp_path / "calls.so"))
    if hasattr(b, "CALLS_STAMP"):
        monkeypatch.setattr(b, "CALLS_STAMP", str(tmp_path / "stamps" / "calls.stamp"))
    monkeypatch.setattr(b, "NVCC", str(tmp_path / "nvcc"))
    monkeypatch.setenv("CXX", str(tmp_path / "cxx"))
    b.stale.__defaults__ = (b.LIB, None)
    b.log = lambda: (tmp_path / "log").read_text().split()
    return b


def test_library_without_torch(script, monkeypatch):
    monkeypatch.setitem(sys.modules, "torch", None)
    script.build()
    assert script.log() == ["nvcc"] and os.path.exists(script.LIB)


def test_calls_are_built_again_for_another_torch(script, monkeypatch):
    script.build()
    assert script.log() == ["nvcc", "cxx"]
    script.build()
    assert script.log() == ["nvcc", "cxx"]
    real = importlib.metadata.version
    monkeypatch.setattr(importlib.metadata, "version", lambda name: "99.0" if name == "torch" else real(name))
    script.build()
    assert script.log() == ["nvcc", "cxx", "cxx"]


def test_a_failed_compiler_leaves_the_old_file(script, tmp_path):
    script.build()
    (tmp_path / "nvcc").write_text('#!/bin/sh\nwhile [ "$1" != -o ]; do shift; done\necho half > "$2"\nexit 1\n')
    with pytest.raises(Exception):
        script.build(force=True)
    assert open(script.LIB).read() == "made\n"


def test_list_kernel_keeps_its_registers(tmp_path):
    """By the compiler's own count no form of the list kernel spills more than a few bytes: a spill in the multiply costs more than what is
    gained around it (116 bytes at 640 threads were a tenth of the time)."""
    spec = importlib.util.spec_from_file_location("bonsai_b200_build_spills", os.path.join(ROOT, "p40-kernel_b200", "build.py"))
    b = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(b)
    if not shutil.which(b.NVCC):
        pytest.skip("no nvcc")
    forms = {"512, 5, false": 0, "640, 4, false": 0, "768, 3, false": 24, "512, 5, true": 8}
    src = tmp_path / "forms.cu"
    src.write_text('#include "gemv_chain.cuh"\nusing namespace b200;\n' + "".join(
        f"template __global__ void b200::gemv_chain_kernel<{f}>(const ChainOp *__restrict__, const int, const ChainGeom, unsigned int *, "
        "uint8_t *, const ChainPeers);\n" for f in forms))
    run = subprocess.run([b.NVCC, *[f for f in b.FLAGS if f != "-shared"], "-Xptxas", "-v", f"-I{b.CSRC}", "-c", str(src), "-o", str(tmp_path / "forms.o")],
                         capture_output=True, text=True)
    assert run.returncode == 0, run.stderr[-2000:]
    spilt = {}
    for threads, steps, ranks, stores in re.findall(r"properties for \S*gemv_chain_kernelILi(\d+)ELi(\d)ELb(\d)E\S*\n.*?(\d+) bytes spill stores", run.stderr):
        spilt[f"{threads}, {steps}, {'true' if ranks == '1' else 'false'}"] = int(stores)
    assert set(spilt) == set(forms), run.stderr[-2000:]
    assert all(spilt[f] <= most for f, most in forms.items()), spilt


def test_mat_mul_kernel_keeps_its_registers(tmp_path):
    """The same of the many-token mat-mul, whose warps have 72 registers a thread: pairs of CTAs spill nothing, single CTAs three words."""
    spec = importlib.util.spec_from_file_location("bonsai_b200_build_spills16", os.path.join(ROOT, "p40-kernel_b200", "build.py"))
    b = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(b)
    if not shutil.which(b.NVCC):
        pytest.skip("no nvcc")
    forms = {"64, 1": 12, "128, 2": 0}
    src = tmp_path / "forms16.cu"
    src.write_text('#include "gemm_tc16.cuh"\nusing namespace b200;\n' + "".join(
        f"template __global__ void b200::gemm_tc16_kernel<{f}>(float *, const T16Params, const float *__restrict__, float *, unsigned int *, "
        "const __grid_constant__ Tc16Maps);\n" for f in forms))
    run = subprocess.run([b.NVCC, *[f for f in b.FLAGS if f != "-shared"], "-Xptxas", "-v", f"-I{b.CSRC}", "-c", str(src), "-o", str(tmp_path / "forms16.o")],
                         capture_output=True, text=True)
    assert run.returncode == 0, run.stderr[-2000:]
    spilt = {f"{n}, {ctas}": int(stores) for n, ctas, stores in
             re.findall(r"properties for \S*gemm_tc16_kernelILi(\d+)ELi(\d)E\S*\n.*?(\d+) bytes spill stores", run.stderr)}
    assert set(spilt) == set(forms) and all(spilt[f] <= most for f, most in forms.items()), spilt or run.stderr[-2000:]


def test_attention_kernel_spills_nothing(tmp_path):
    """The CUDA-core attention: shared memory lets three CTAs of either size on an SM, and with the registers that three leave nothing is spilled."""
    spec = importlib.util.spec_from_file_location("bonsai_b200_build_spills_attn", os.path.join(ROOT, "p40-kernel_b200", "build.py"))
    b = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(b)
    if not shutil.which(b.NVCC):
        pytest.skip("no nvcc")
    src = tmp_path / "forms_attn.cu"
    src.write_text('#include "ops.cuh"\nusing namespace b200;\n' + "".join(
        f"template __global__ void b200::attn_kernel<{w}>(const float *, const float *, const float *, float *, int, int, int, float);\n" for w in (2, 4)))
    run = subprocess.run([b.NVCC, *[f for f in b.FLAGS if f != "-shared"], "-Xptxas", "-v", f"-I{b.CSRC}", "-c", str(src), "-o", str(tmp_path / "forms_attn.o")],
                         capture_output=True, text=True)
    assert run.returncode == 0, run.stderr[-2000:]
    spilt = re.findall(r"properties for \S*11attn_kernelILi(\d)E\S*\n.*?(\d+) bytes spill stores", run.stderr)
    assert sorted(spilt) == [("2", "0"), ("4", "0")], spilt or run.stderr[-2000:]
