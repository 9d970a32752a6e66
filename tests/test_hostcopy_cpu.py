"""The threaded device-to-host copy (vh_hostcopy.cuh) over a stand-in for the
CUDA runtime with two devices, whose copies are memcpy and whose events, as the
runtime's, are recorded in streams of their own device only."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RUNTIME = r"""
#pragma once
#include <cstddef>
#include <cstdlib>
#include <cstring>
typedef int cudaError_t;
enum { cudaSuccess = 0, cudaErrorInvalidResourceHandle = 400 };
struct FakeStream { int dev; };
struct FakeEvent { int dev; };
typedef FakeStream* cudaStream_t;
typedef FakeEvent* cudaEvent_t;
enum cudaMemoryType { cudaMemoryTypeUnregistered, cudaMemoryTypeHost, cudaMemoryTypeDevice, cudaMemoryTypeManaged };
struct cudaPointerAttributes { cudaMemoryType type; int device; void *devicePointer, *hostPointer; };
enum cudaMemcpyKind { cudaMemcpyDeviceToHost, cudaMemcpyDefault };
enum cudaStreamCaptureStatus { cudaStreamCaptureStatusNone };
enum { cudaEventDisableTiming = 2, cudaStreamNonBlocking = 1 };
extern thread_local int g_dev;       // the thread's current device
extern const char *g_src, *g_src_end;  // the one device array and its device
extern int g_src_dev;
inline cudaError_t cudaGetDevice(int* d) { *d = g_dev; return 0; }
inline cudaError_t cudaSetDevice(int d) { g_dev = d; return 0; }
inline cudaError_t cudaGetLastError() { return 0; }
template <class T> cudaError_t cudaMallocHost(T** p, size_t n) { *p = (T*)std::malloc(n); return 0; }
inline cudaError_t cudaFreeHost(void* p) { std::free(p); return 0; }
inline cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (FakeStream*)std::malloc(4); (*s)->dev = g_dev; return 0; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (FakeEvent*)std::malloc(4); (*e)->dev = g_dev; return 0; }
inline cudaError_t cudaStreamDestroy(cudaStream_t s) { std::free(s); return 0; }
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return 0; }
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return e->dev == s->dev ? 0 : cudaErrorInvalidResourceHandle; }
inline cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return 0; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t) { return 0; }
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { return 0; }
inline cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) { *c = cudaStreamCaptureStatusNone; return 0; }
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  const bool dev = p >= g_src && p < g_src_end;
  *a = {dev ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered, dev ? g_src_dev : -2, nullptr, nullptr};
  return 0;
}
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return 0; }
"""

MAIN = r"""
#include "vh_hostcopy.cuh"
#include <cstdio>
#include <vector>
thread_local int g_dev = 0;
const char *g_src, *g_src_end;
int g_src_dev;
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
int main(int, char** av) {
  const size_t n = (33u << 20) + 4097;
  std::vector<char> src(n), dst(n);
  for (size_t i = 0; i < n; i++) src[i] = (char)(i * 7 + i / 4093);
  g_src = src.data();
  g_src_end = g_src + n;
  const int what = std::atoi(av[1]);
  if (what == 0) {
    // the array and its stream on device 1, the caller on device 0, then on 1
    g_src_dev = 1;
    FakeStream s{1};
    HostCopy h;
    for (int cur : {0, 1, 0}) {
      g_dev = cur;
      std::memset(dst.data(), 0, n);
      CHECK(h.copy(dst.data(), src.data(), n, &s) == cudaSuccess);
      CHECK(g_dev == cur);
      CHECK(dst == src);
    }
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("hostcopy")
    (d / "cuda_runtime.h").write_text(RUNTIME)
    (d / "main.cpp").write_text(MAIN)
    exe = d / "run"
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", str(d), "-I",
                    os.path.join(ROOT, "viral_b200", "csrc"), str(d / "main.cpp"), "-o", str(exe)], check=True)
    return str(exe)


def test_the_array_on_another_device_than_the_callers(program):
    r = subprocess.run([program, "0"], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
