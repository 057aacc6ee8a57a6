"""Host side of ``inq_prefill_attention`` against a CUDA runtime of our own (no GPU, no launch): what a query
that the runtime refuses does to that call and to the next one."""
import ctypes
import os
import subprocess

import pytest

from inquant import _native as N

PACKAGE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "inquant-open-source_b200")
RUNTIME = r"""
#include <cuda_runtime.h>
#include <string.h>
extern "C" {
int fake_registers = 168, fake_failures = 0, fake_launches = 0;
int fake_refusals = 0;   // of launches
static int encode(...) { return 0; }
void** __cudaRegisterFatBinary(void*) { static void* handle; return &handle; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
static struct { dim3 grid, block; size_t shared; cudaStream_t stream; } call;
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t shared, cudaStream_t stream) {
  call.grid = grid; call.block = block; call.shared = shared; call.stream = stream;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* shared, void* stream) {
  *grid = call.grid; *block = call.block; *shared = call.shared; *(cudaStream_t*)stream = call.stream;
  return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "refused by the test"; }
cudaError_t cudaGetDevice(int* device) { *device = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* value, cudaDeviceAttr, int) { *value = 148; return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
  if (fake_failures > 0) { --fake_failures; return cudaErrorUnknown; }
  memset(a, 0, sizeof *a);
  a->numRegs = fake_registers;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** p, unsigned long long, cudaDriverEntryPointQueryResult* r) {
  *p = (void*)encode;
  *r = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { ++fake_launches; return cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) {
  if (fake_refusals > 0) { --fake_refusals; return cudaErrorUnknown; }
  ++fake_launches;
  return cudaSuccess;
}
}
"""


@pytest.fixture
def library(tmp_path):
    """The object files of the real host code, linked against the runtime above."""
    import build
    build.build_library()
    source, target = tmp_path / "runtime.cpp", tmp_path / "prefill_host.so"
    source.write_text(RUNTIME)
    objects = [os.path.join(PACKAGE, "build", name) for name in ("prefill.o", "lib.o")]
    subprocess.run(["g++", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I/usr/local/cuda/include", "-o", str(target), str(source), *objects], check=True)
    lib = ctypes.CDLL(str(target))
    lib.inq_last_error.restype = ctypes.c_char_p
    return lib


def _call(lib, dtype):
    args = N.PrefillArgs()
    args.q, args.k, args.v, args.out, args.status = 4096, 8192, 12288, 16384, 20480   # never read on the host
    for name in "qkvo":
        setattr(args, f"{name}_stride_h", 128 * 128)
        setattr(args, f"{name}_stride_t", 128)
    args.q_heads, args.kv_heads, args.q_tokens, args.kv_tokens = 4, 2, 64, 128
    args.dtype, args.scale = dtype, 0.1
    return lib.inq_prefill_attention(ctypes.byref(args), None)


@pytest.mark.parametrize("dtype", [N.F16, N.BF16])
def test_a_query_that_fails_once_is_reported_and_does_not_outlive_the_call(library, dtype):
    failures, launches = ctypes.c_int.in_dll(library, "fake_failures"), ctypes.c_int.in_dll(library, "fake_launches")
    failures.value = 1
    assert _call(library, dtype) == N.ERR_CUDA
    assert b"refused by the test" in library.inq_last_error() and launches.value == 0
    assert _call(library, dtype) == N.OK and launches.value == 1
    failures.value = 1                       # a yes is kept
    assert _call(library, dtype) == N.OK and launches.value == 2 and failures.value == 1


def test_a_kernel_with_too_few_registers_is_not_launched(library):
    ctypes.c_int.in_dll(library, "fake_registers").value = 160
    assert _call(library, N.BF16) == N.ERR_UNSUPPORTED
    assert ctypes.c_int.in_dll(library, "fake_launches").value == 0


def test_a_refused_launch_is_reported_and_not_repeated(library):
    ctypes.c_int.in_dll(library, "fake_refusals").value = 1
    assert _call(library, N.BF16) == N.ERR_CUDA
    assert b"refused by the test" in library.inq_last_error() and ctypes.c_int.in_dll(library, "fake_launches").value == 0
    assert _call(library, N.BF16) == N.OK and ctypes.c_int.in_dll(library, "fake_launches").value == 1
