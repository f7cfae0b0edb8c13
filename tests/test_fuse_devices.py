"""Fusion on several devices of one process, on the CPU: the library's host code linked to a stand-in for
the CUDA runtime, in which the shared memory that a kernel may take is granted per device."""
import ctypes
import os
import shutil
import subprocess

import pytest

RUNTIME = r'''
#include <map>
#include <utility>
#include <cuda_runtime_api.h>
static int device = 0, launches = 0;
static std::map<std::pair<int, const void *>, size_t> granted;
static bool fits(const void *f, size_t smem) {
    auto it = granted.find({device, f});
    return smem <= (it == granted.end() ? 48u * 1024u : it->second);
}
extern "C" {
void fake_set_device(int d) { device = d; }
int fake_launches() { return launches; }
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
'''


@pytest.fixture(scope='module')
def fuse(tmp_path_factory):
    from vissatsatellitestereo_gb300 import build
    if shutil.which('g++') is None:
        pytest.skip('needs g++')
    build.build()
    d = tmp_path_factory.mktemp('fake')
    src, so = d / 'runtime.cpp', d / 'libfuse.so'
    src.write_text(RUNTIME)
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), 'include')
    objs = [os.path.join(build.BUILD, o) for o in ('core.o', 'fuse.o')]
    subprocess.run(['g++', '-std=c++17', '-shared', '-fPIC', '-I', include, '-o', str(so), str(src), *objs], check=True)
    return ctypes.CDLL(str(so))


@pytest.mark.parametrize('layout', [0, 1])
@pytest.mark.parametrize('views', [3, 50, 64, 65, 100, 128, 129, 256, 257, 512])
def test_every_device_fuses(fuse, views, layout):
    stack, out = (ctypes.c_void_p(1 << 20), ctypes.c_void_p(1 << 30))       # never followed: nothing runs
    for device in (0, 1, 0, 2):
        fuse.fake_set_device(device)
        before = fuse.fake_launches()
        i64 = ctypes.c_int64
        status = fuse.vs_fuse_dsms(stack, layout, i64(views), i64(9), i64(16), out, 0, None, ctypes.c_size_t(0), None)
        assert status == 0 and fuse.fake_launches() == before + 1, device
