"""The exponential of the tensor-core four-phonon delta terms (exp_neg.cuh) over its range, against extended precision:
the bound its comment states, on the host and as the device computes it."""
import ctypes as ct
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "spring_b200", "csrc")
BOUND = 2.3e-16


def _points():
    rng = np.random.default_rng(0)
    edge = (2 * np.arange(58) + 1) * 0.5 * np.log(2.0)          # the reduction's rounding turns over here
    edge = np.concatenate([edge, np.nextafter(edge, 0.0), np.nextafter(edge, 41.0)])
    x = np.concatenate([[0.0, 40.0, 5e-324, 1e-300, 1e-17, np.log(2.0), np.nextafter(40.0, 0.0)], edge,
                        np.arange(58) * np.log(2.0), rng.uniform(0.0, 40.0, 400000), 10.0 ** rng.uniform(-18.0, 1.6, 100000)])
    return np.ascontiguousarray(x[(x >= 0.0) & (x <= 40.0)])


def _check(x, y):
    ref = np.exp(-x.astype(np.longdouble))                      # 64-bit mantissa
    assert np.finfo(np.longdouble).nmant >= 63
    assert np.max(np.abs(y.astype(np.longdouble) / ref - 1.0)) <= BOUND
    assert y[0] == 1.0


def test_exp_neg_on_the_host(tmp_path):
    src = tmp_path / "e.cpp"
    src.write_text('#include "exp_neg.cuh"\nextern "C" void run(long n, const double* x, double* y) '
                   '{ for (long i = 0; i < n; ++i) y[i] = spring::exp_neg(x[i]); }\n')
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(src),
                    "-o", str(tmp_path / "e.so")], check=True)
    x = _points()
    y = np.zeros_like(x)
    p = ct.c_void_p
    ct.CDLL(str(tmp_path / "e.so")).run(ct.c_long(len(x)), p(x.ctypes.data), p(y.ctypes.data))
    _check(x, y)


@pytest.mark.gpu
def test_exp_neg_on_the_device(tmp_path):
    from spring_b200.build import ARCH, nvcc
    src = tmp_path / "e.cu"
    src.write_text('#include "exp_neg.cuh"\n'
                   '__global__ void k(long n, const double* x, double* y) '
                   '{ long i = blockIdx.x * (long)blockDim.x + threadIdx.x; if (i < n) y[i] = spring::exp_neg(x[i]); }\n'
                   'extern "C" int run(long n, const double* x, double* y) { k<<<(n + 255) / 256, 256>>>(n, x, y); '
                   'return cudaDeviceSynchronize(); }\n')
    subprocess.run([nvcc(), *ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I", CSRC, str(src),
                    "-o", str(tmp_path / "e.so")], check=True)
    import torch
    x = _points()
    dx = torch.from_numpy(x).cuda()
    dy = torch.zeros_like(dx)
    torch.cuda.synchronize()
    p = ct.c_void_p
    assert ct.CDLL(str(tmp_path / "e.so")).run(ct.c_long(len(x)), p(dx.data_ptr()), p(dy.data_ptr())) == 0
    _check(x, dy.cpu().numpy())
