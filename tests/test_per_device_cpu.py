"""Threads of one process may drive a device each. What a launch needs on its device (a kernel's opt-in to more shared memory than the default) has to
be set there, not only on the device that was first. Checked without a GPU: a stand-in for the CUDA runtime's functions keeps track per device."""
import os
import shutil
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
LIB = os.path.join(os.path.dirname(HERE), "flodl_b200", "_C.so")

FAKE = r"""
#include <cuda_runtime_api.h>
#include <string.h>
static int dev, n, launches, refused;
static struct { const void* f; int dev; size_t bytes; } allowed[512];
static int encode(void) { return 0; }
extern "C" {
void fake_set_device(int d) { dev = d; }
int fake_launches(void) { return launches; }
int fake_refused(void) { return refused; }
cudaError_t cudaGetDevice(int* d) { *d = dev; return cudaSuccess; }
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveClusters(int* v, const void*, const cudaLaunchConfig_t*) { *v = 36; return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** p, unsigned long long, cudaDriverEntryPointQueryResult* r) {
  *p = (void*)encode;
  if (r) *r = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize && n < 512) { allowed[n].f = f; allowed[n].dev = dev; allowed[n++].bytes = (size_t)v; }
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  ++launches;
  if (c->dynamicSmemBytes <= 48 * 1024) return cudaSuccess;
  for (int i = 0; i < n; ++i)
    if (allowed[i].f == f && allowed[i].dev == dev && allowed[i].bytes >= c->dynamicSmemBytes) return cudaSuccess;
  ++refused;
  return cudaErrorInvalidValue;
}
}
"""

WORKER = r"""
import ctypes, sys
import torch  # noqa: F401  (the library's dependencies)
fake, lib = ctypes.CDLL(sys.argv[1]), ctypes.CDLL(sys.argv[2])
P, L = ctypes.c_void_p, ctypes.c_longlong
f32 = ctypes.c_float
A = P(1 << 20)      # an address that nothing reads


def gemm(M, N, K, config=-1, a_mn=0, fp32=0):
    m, k = (M, K) if not a_mn else (K, M)
    return lib.fb_gemm_bf16(A, A, A, M, N, K, L(k), L(K), L(N), a_mn, 0, fp32, None, 0, 0, None, L(0), None, 0, 1, config, A, None)


def attention(S, p_drop, mask, backward):
    s = (L * 3)(S * 64, 64, S * 64)
    seed = ctypes.c_ulonglong(1)
    if not backward:
        return lib.fb_attn_fwd(A, A, A, A, A, mask, 1, 1, S, s, s, f32(0.125), 0, f32(p_drop), seed, None, A, None)
    return lib.fb_attn_bwd(A, A, A, A, A, A, mask, A, A, A, A, 1, 1, S, s, s, s, f32(0.125), 0, f32(p_drop), seed, None, A, None)


def everything():
    rc = {("gemm", c): gemm(512, 768, 256, c) for c in range(6)}
    rc["gemm few tiles"] = gemm(77, 768, 768)
    rc["gemm two pairs"] = gemm(4096, 512, 2048)
    for S in (128, 300):
        for back in (False, True):
            for p_drop in (0.0, 0.1):
                for mask in (None, A):
                    rc["attention", S, back, p_drop, mask is None] = attention(S, p_drop, mask, back)
    for stride in (1, 2):
        rc["conv", stride] = lib.fb_conv_fprop(A, A, A, None, 4, 32, 32, 16, 16 * stride, 3, stride, 1, A, None)
        rc["conv filter gradient", stride] = lib.fb_conv_wgrad(A, A, A, 4, 32, 32, 16, 16 * stride, 3, 3, stride, 1, A, None)
    return {k: v for k, v in rc.items() if v}


for device in (0, 1, 5, 0):
    fake.fake_set_device(device)
    before = fake.fake_launches()
    failed = everything()
    assert not failed, (device, failed)
    assert fake.fake_launches() - before >= 28
assert fake.fake_refused() == 0
print("PER_DEVICE_OK")
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_every_launch_is_prepared_on_its_own_device(tmp_path):
    src, so, worker = tmp_path / "fake.cpp", tmp_path / "libfake.so", tmp_path / "worker.py"
    src.write_text(FAKE)
    worker.write_text(WORKER)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", f"-I{cuda}/include", str(src), "-o", str(so)], check=True)
    r = subprocess.run([sys.executable, str(worker), str(so), LIB], env=dict(os.environ, LD_PRELOAD=str(so), CUDA_VISIBLE_DEVICES=""), capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "PER_DEVICE_OK" in r.stdout, r.stdout[-2000:] + r.stderr[-3000:]
