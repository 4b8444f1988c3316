"""The solve's FP64 reciprocal (reciprocal.h) over its range, on the host and, in
the kernels' form, against CUDA's division (gpu).

Bound: the last Newton step leaves an error of 2^-88 before its rounding, so the
result is 1 / d rounded, or its neighbour where 1 / d lies between two doubles
within that: one unit in the last place of the correctly rounded quotient.
"""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "bd-cudatag_gb300" / "csrc"


def arguments():
    rng = np.random.default_rng(9)
    d = np.concatenate([
        np.exp(rng.uniform(np.log(1e-12), np.log(3.4e38), 200_000)),
        np.arange(1.0, 65537.0),                                           # sample counts
        np.nextafter(2.0 ** np.arange(-39, 128), 0.0), 2.0 ** np.arange(-39, 128),
        [1e-12, 8.5e37, 1.7e38, 3.4e38],                                   # seeds below the normal floats
    ])
    return np.ascontiguousarray(d)


def within_one_ulp(got, d):
    want = 1.0 / d  # correctly rounded
    assert np.abs(got.view(np.int64) - want.view(np.int64)).max() <= 1


def test_host(tmp_path):
    src = tmp_path / "r.cpp"
    src.write_text('#include "reciprocal.h"\n'
                   'extern "C" void run(const double* d, double* r, long n) {\n'
                   '    for (long i = 0; i < n; ++i) r[i] = bdmath::reciprocal(d[i]);\n}\n')
    lib = tmp_path / "r.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", f"-I{CSRC}", str(src),
                    "-o", str(lib)], check=True)
    d = arguments()
    got = np.empty_like(d)
    run = ctypes.CDLL(str(lib)).run
    run.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_long]
    run(d.ctypes.data, got.ctypes.data, d.size)
    within_one_ulp(got, d)


@pytest.mark.gpu
def test_device(tmp_path):
    torch = pytest.importorskip("torch")
    import build  # the package's own flags
    src = tmp_path / "r.cu"
    src.write_text('#include "reciprocal.h"\n'
                   '__global__ void k(const double* d, double* r, double* q, int n) {\n'
                   '    const int i = blockIdx.x * blockDim.x + threadIdx.x;\n'
                   '    if (i < n) { r[i] = bdmath::reciprocal(d[i]); q[i] = 1.0 / d[i]; }\n}\n'
                   'extern "C" int run(const double* d, double* r, double* q, int n) {\n'
                   '    k<<<(n + 255) / 256, 256>>>(d, r, q, n);\n'
                   '    return static_cast<int>(cudaDeviceSynchronize());\n}\n')
    lib = tmp_path / "r.so"
    subprocess.run([build.nvcc(), build.ARCH, "-fmad=false", "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                    f"-I{CSRC}", str(src), "-o", str(lib), "-lcudart"], check=True)
    d = arguments()
    dev = torch.from_numpy(d).cuda()
    got, quotient = torch.empty_like(dev), torch.empty_like(dev)
    torch.cuda.synchronize()
    run = ctypes.CDLL(str(lib)).run
    run.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int]
    assert run(dev.data_ptr(), got.data_ptr(), quotient.data_ptr(), d.size) == 0
    assert np.array_equal(quotient.cpu().numpy(), 1.0 / d)
    within_one_ulp(got.cpu().numpy(), d)
