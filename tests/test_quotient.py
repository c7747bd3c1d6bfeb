"""The CPML quotient of csrc/quotient.h has the bits of the division for every
numerator: normal, near the smallest floats, subnormal, zero, infinite, NaN.
On the host, and on the device against CUDA's division."""
import ctypes
import subprocess

import numpy as np
import pytest

from conftest import ROOT

HOST = r"""
#include "quotient.h"
extern "C" void quotients(const float* a, const float* K, float* q, float* div, long n) {
  for (long i = 0; i < n; ++i) {
    q[i] = fwigb::over<CALL>(a[i], K[i] * fwigb::kQuotientScale, 1.0f / K[i] / fwigb::kQuotientScale);
    div[i] = a[i] / K[i];
  }
}
"""
DEVICE = r"""
#include "quotient.h"
__global__ void k(const float* a, const float* K, float* q, float* div, long n) {
  const long i = blockIdx.x * 256L + threadIdx.x;
  if (i < n) {
    q[i] = fwigb::over<CALL>(a[i], K[i] * fwigb::kQuotientScale, 1.0f / K[i] / fwigb::kQuotientScale);
    div[i] = a[i] / K[i];
  }
}
extern "C" int quotients(const float* a, const float* K, float* q, float* div, long n) {
  k<<<static_cast<unsigned>((n + 255) / 256), 256>>>(a, K, q, div, n);
  return cudaDeviceSynchronize();
}
"""


def _samples():
    """(a, K): every exponent, random significands; quotients next to the midpoint of two floats; special values."""
    rng = np.random.default_rng(3)
    per = 4000
    K = (1.0 + rng.integers(0, 1 << 23, (277, per)) * 2.0 ** -23).astype(np.float32)
    K[:, :3] = 1.0, 2.0, np.nextafter(np.float32(2.0), np.float32(0.0))
    m = 1.0 + rng.integers(0, 1 << 23, (277, per)) * 2.0 ** -23
    a = np.ldexp(m, np.arange(-149, 128)[:, None]).astype(np.float32)  # (subnormal ones rounded)
    # a = round(K (Q + 1/2) ulp): the quotient is within half an ulp of a / K of a midpoint, some of them by little
    Q = rng.integers(1 << 23, 1 << 24, (277, per)) + 0.5
    b = np.ldexp(K.astype(np.float64) * Q, np.arange(-173, 104)[:, None] - 1).astype(np.float32)
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, np.finfo(np.float32).max, 2.0 ** -149, -(2.0 ** -149),
                        2.0 ** -126, 2.0 ** -100, np.nextafter(np.float32(2.0 ** -100), np.float32(0.0))], np.float32)
    Ks = np.array([1.0, 1.25, 1.9999999, 2.0], np.float32)
    A = np.concatenate([a.ravel(), -a.ravel(), b.ravel(), np.repeat(special, len(Ks))])
    return A, np.concatenate([K.ravel(), K.ravel(), K.ravel(), np.tile(Ks, len(special))])


def _check(q, div):
    same = (q.view(np.uint32) == div.view(np.uint32)) | (np.isnan(q) & np.isnan(div))
    assert same.all(), int((~same).sum())
    assert np.isnan(div).sum() == 4 and np.isinf(div).sum() == 8 and (div == 0).sum() >= 8


@pytest.mark.parametrize("call", ["true", "false"])
def test_quotient_has_the_bits_of_the_division(call, tmp_path):
    src, lib = tmp_path / "q.cpp", tmp_path / "q.so"
    src.write_text(HOST.replace("CALL", call))
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", f"{ROOT}/fwiflow.jl_gb300/csrc",
                    "-o", str(lib), str(src)], check=True)
    a, K = _samples()
    q, div = np.empty_like(a), np.empty_like(a)
    p = [x.ctypes.data_as(ctypes.c_void_p) for x in (a, K, q, div)]
    ctypes.CDLL(str(lib)).quotients(*p, ctypes.c_long(a.size))
    _check(q, div)


@pytest.mark.gpu
@pytest.mark.parametrize("call", ["true", "false"])
def test_quotient_has_the_bits_of_cudas_division(call, gpu_lib, fw, tmp_path):
    import torch
    from fwiflow_gb300 import build

    src, lib = tmp_path / "q.cu", tmp_path / "q.so"
    src.write_text(DEVICE.replace("CALL", call))
    subprocess.run([build.nvcc_path(), *build.ARCH, "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-shared",
                    "-Xcompiler", "-fPIC", "-I", f"{ROOT}/fwiflow.jl_gb300/csrc", "-o", str(lib), str(src)], check=True)
    a, K = _samples()
    t = [torch.from_numpy(x).cuda() for x in (a, K)] + [torch.empty(a.size, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    p = [ctypes.c_void_p(x.data_ptr()) for x in t]
    assert ctypes.CDLL(str(lib)).quotients(*p, ctypes.c_long(a.size)) == 0
    _check(t[2].cpu().numpy(), t[3].cpu().numpy())
