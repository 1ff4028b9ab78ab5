"""How kernels are launched: per-device launch attributes, and overlapped
launches that begin only when they may."""
import glob
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "sparseops_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_no_launch_attribute_behind_a_process_wide_static():
    """Function attributes and occupancies belong to a device: no kernel's
    launch may keep them in one static for the whole process."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = open(path).read()
        found = re.findall(r"static (?:int|bool|size_t) \w+(?: = [^;{]*)?;", text)
        assert not found, (os.path.basename(path), found)


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.exists(f"{CUDA}/include/cuda_runtime.h"),
                    reason="needs g++ and the CUDA headers")
def test_launch_helpers_against_a_fake_runtime(tmp_path):
    exe = str(tmp_path / "launch_test")
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-Wextra", "-I", CSRC, "-isystem", f"{CUDA}/include", "-o", exe,
                    os.path.join(ROOT, "tests", "cpp", "launch_test.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


def test_overlapped_launches_wait_or_belong_to_a_chain():
    """A kernel launched by launch_overlapped waits (overlap_begin, or
    overlap_wait after its plan's loads); one that does not wait until its end
    (overlap_end) is launched through an OverlapChain, whose first launch is a
    plain one."""
    def kernels(pattern):  # names of the kernels whose body calls it
        out = set()
        for path in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")):
            if path.endswith("pdl.cuh"):
                continue
            text = open(path).read()
            for m in re.finditer(pattern, text):
                head = text[:m.start()]
                out.add(re.findall(r"(\w+_kernel)\(", head[head.rindex("__global__"):])[0])
        return out

    late = kernels(r"overlap_end\(\)")
    assert late
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        text = open(path).read()
        for m in re.finditer(r"launch_overlapped\(\s*(\w+)", text):
            name = m.group(1)
            if name == "kern":  # a local: the last kernel named before it
                name = re.findall(r"auto\*? kern = (\w+_kernel)|OverlapChain|auto kern\b", text[:m.start()])[-1]
            assert name.endswith("_kernel") and name not in late, (os.path.basename(path), m.group(0), name)
    waits = kernels(r"overlap_begin\(\)|overlap_wait\(\)")
    assert not waits & late


@pytest.mark.gpu
@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("k", [3, 12, 16, 32])
def test_spmm_on_two_devices(cuda, k, f32):
    """The same SpMM form on two GPUs of one process (forms with more than
    48 KB of shared memory among them)."""
    import torch
    from sparseops_b200 import CSR_Matrix, SpMM_csr, synth
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    n = 5000
    rp, ci, v = synth.banded_random(n, 16.0, 64, seed=1)
    dt = torch.float32 if f32 else torch.float64
    X = torch.rand(n, k, dtype=dt, generator=torch.Generator().manual_seed(1))
    out = []
    for d in range(2):
        with torch.cuda.device(d):
            dev = f"cuda:{d}"
            A = CSR_Matrix(n, n, torch.from_numpy(rp.astype(np.int64)).to(dev), torch.from_numpy(ci.astype(np.int64)).to(dev),
                           torch.from_numpy(v).to(dev, dt))
            Y = torch.zeros(n, k, dtype=dt, device=dev)
            SpMM_csr(1.0, A, X.to(dev), 0.0, Y)
            out.append(Y.cpu())
    assert torch.equal(out[0], out[1])
