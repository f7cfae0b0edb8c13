"""Fusion on several devices of one process, on the CPU: the library's host code linked to a stand-in for
the CUDA runtime, in which the shared memory that a kernel may take is granted per device.  A program of
its own, which neither links nor loads the CUDA runtime or driver: no GPU can be reached from it."""
import os
import shutil
import subprocess

import pytest

RUNTIME = r'''
#include <stdio.h>
#include <map>
#include <utility>
#include <cuda_runtime_api.h>
#include "vissat_gb300.h"
static int device = 0, launches = 0;
static std::map<std::pair<int, const void *>, size_t> granted;
static bool fits(const void *f, size_t smem) {
    auto it = granted.find({device, f});
    return smem <= (it == granted.end() ? 48u * 1024u : it->second);
}
extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaGetSymbolAddress(void **, const void *) { return cudaErrorInvalidValue; }
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int bytes) {
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) granted[{device, f}] = bytes;
    return bytes <= 227 * 1024 ? cudaSuccess : cudaErrorInvalidValue;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int, size_t smem, unsigned) {
    *n = fits(f, smem) ? 1 : 0;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **) {
    if (!fits(f, c->dynamicSmemBytes)) return cudaErrorInvalidValue;
    ++launches;
    return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) { static void *handle; return &handle; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, void *, void *, void *, void *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPopCallConfiguration(void *, void *, size_t *, void *) { return 1; }
cudaError_t __cudaGetKernel(void *, const void *) { return cudaErrorInvalidValue; }
cudaError_t __cudaLaunchKernel(void *, dim3, dim3, void **, size_t, cudaStream_t) { return cudaErrorInvalidValue; }
}
namespace vs {
int launch_blur_f32(const float *, float *, long long, long long, cudaStream_t) { return 0; }
}
int main() {
    const float *stack = reinterpret_cast<const float *>(1 << 20);       // never followed: nothing runs
    float *out = reinterpret_cast<float *>(1 << 30);
    const int views[] = {3, 50, 64, 65, 100, 128, 129, 256, 257, 512}, devices[] = {0, 1, 0, 2};
    int bad = 0;
    for (int layout = 0; layout < 2; ++layout)
        for (int v : views)
            for (int d : devices) {
                device = d;
                const int before = launches;
                const int status = vs_fuse_dsms(stack, layout, v, 9, 16, out, 0, nullptr, 0, nullptr);
                if (status == 0 && launches == before + 1) continue;
                printf("%d views, layout %d, device %d: status %d\n", v, layout, d, status);
                ++bad;
            }
    return bad != 0;
}
'''



def test_every_device_fuses(tmp_path):
    from vissatsatellitestereo_gb300 import build
    if shutil.which('g++') is None:
        pytest.skip('needs g++')
    build.build()
    src, exe = tmp_path / 'devices.cpp', tmp_path / 'devices'
    src.write_text(RUNTIME)
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), 'include')
    objs = [os.path.join(build.BUILD, o) for o in ('core.o', 'fuse.o')]
    subprocess.run(['g++', '-std=c++17', '-I', cuda, '-I', build.INCLUDE, '-o', str(exe), str(src), *objs], check=True)
    p = subprocess.run([str(exe)], capture_output=True, text=True)
    assert p.returncode == 0, p.stdout
