"""Launches of the decode attention: its host code, linked against a runtime that is kept to the rule that more than 48 KiB of
dynamic shared memory have to be asked for kernel by kernel and device by device, and that says how many CTAs fit an SM."""
import shutil
import subprocess

import pytest

from create_llm_by_cupy_b200.ops import build as B

PROGRAM = r"""
#include <cuda_runtime_api.h>
#include <cassert>
#include <cstdio>
#include <map>
#include <thread>
#include <utility>
#include <vector>
#include <mutex>

static thread_local int device = 0;
static std::mutex mu;
static std::map<std::pair<int, const void*>, int> allowed;
static int refuse = 0, launches = 0, asked = 0, warps = 0, per_sm = 0;
static int cluster = 0, clusters = 0;
static long ctas = 0;

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return ""; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int v) {
  std::lock_guard<std::mutex> lock(mu);
  ++asked;
  if (refuse > 0) { --refuse; return cudaErrorMemoryAllocation; }
  allowed[{device, f}] = v;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int threads, size_t smem, unsigned) {
  const int by_regs = 65536 / (128 * threads), by_smem = int(227 * 1024 / (smem + 12 * 1024));
  *n = by_regs < by_smem ? by_regs : by_smem;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* f, int threads, size_t smem) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(n, f, threads, smem, 0);
}
// GPCs of 18 SMs (and a rest of 4); a cluster lies within one of them
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void* f, const cudaLaunchConfig_t* c) {
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, c->blockDim.x, c->dynamicSmemBytes);
  const int cs = c->attrs[0].val.clusterDim.x;
  *n = 8 * (18 * per_sm / cs) + 4 * per_sm / cs;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  std::lock_guard<std::mutex> lock(mu);
  const auto at = allowed.find({device, f});
  if (int(c->dynamicSmemBytes) > (at == allowed.end() ? 48 * 1024 : at->second)) return cudaErrorInvalidValue;
  ++launches;
  ctas = long(c->gridDim.x) * c->gridDim.y * c->gridDim.z;
  cluster = c->gridDim.x;
  {
    cudaLaunchAttribute at[1];
    at[0].val.clusterDim.x = cluster;
    cudaLaunchConfig_t one = *c;
    one.attrs = at;
    cudaOccupancyMaxActiveClusters(&clusters, f, &one);
  }
  warps = c->blockDim.x / 32;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, c->blockDim.x, c->dynamicSmemBytes);
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaErrorInvalidValue; }
unsigned __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return 0; }
void** __cudaRegisterFatBinary(void*) { static void* p; return &p; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
int b200_gemm_skinny() { return 0; }                         // linked, not called
int b200_gemm_skinny_swiglu() { return 0; }
int b200_decode_attn(const void*, const void*, const void*, void*, const void*, int, int, int, int, int, float, cudaStream_t);
int b200_decode_attn_append(const void*, void*, void*, void*, const void*, const void*, const void*, int, int, int, int, int, int,
                            int, float, cudaStream_t);
}
namespace b200 {
int num_sms() { return 148; }
int* status_ptr() { return nullptr; }
}

// Addresses that the host code only looks at; B sequences, 4 query heads to each of 2 KV heads, a cache of T keys.
static int call(bool append, int D, int B, int T) {
  char* m = reinterpret_cast<char*>(4096);
  return append ? b200_decode_attn_append(m, m, m, m, m, m, m, B, 8, 2, T, D, 12 * D, T - 1, 0.1f, nullptr)
                : b200_decode_attn(m, m, m, m, m, B, 8, 2, T, D, 0.1f, nullptr);
}

int main() {
  for (int d : {3, 0, 3, 63, 64, 200})                       // also more devices than are remembered
    for (int D : {32, 64, 128})
      for (int T : {1, 40, 4096})
        for (int B : {1, 8, 100})
          for (bool append : {false, true}) {
            device = d;
            if (call(append, D, B, T) != 0) { std::printf("refused: device %d D %d B %d T %d\n", d, D, B, T); return 1; }
          }
  device = 7;                                                // a request that fails is made again by the next call
  refuse = 1;
  assert(call(true, 128, 1, 100) != 0 && call(true, 128, 1, 100) == 0);
  const int before = asked;
  for (int i = 0; i < 5; ++i) assert(call(true, 128, 8, 4000) == 0);
  assert(asked == before);                                   // and one that was granted is not
  std::vector<std::thread> ts;
  for (int d = 20; d < 28; ++d)
    ts.emplace_back([d] {
      device = d;
      for (int i = 0; i < 200; ++i) assert(call(i & 1, 128, 4, 2000) == 0);
    });
  for (auto& t : ts) t.join();
  assert(launches > 8 * 200);

  // A grid that could run at the same time does, whatever its head dimension, keys and sequences; otherwise four warps
  device = 0;
  for (int D : {32, 64, 128})
    for (int T : {1, 31, 33, 97, 101, 300, 700, 3000, 20000})
      for (int B = 1; B <= 1100; B += B < 80 ? 1 : 37)
        for (bool append : {false, true}) {
          assert(call(append, D, B, T) == 0);
          assert(warps <= 4 || ctas / cluster <= clusters);
          int one = 0;
          cudaOccupancyMaxActiveBlocksPerMultiprocessor(&one, nullptr, 32, 2 * 32 * D * 2);
          if (20 * 2 * B <= 19L * one * 148) {
            if (ctas > long(per_sm) * 148) {
              std::printf("D %d B %d T %d: %ld CTAs of %d warps, %d to an SM\n", D, B, T, ctas, warps, per_sm);
              return 1;
            }
          } else {
            assert(ctas == 2 * B && warps == 4);
          }
        }
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_every_device_is_asked_and_grids_run_at_once(tmp_path):
    B.build()
    src, exe = tmp_path / "devices.cpp", tmp_path / "devices"
    src.write_text(PROGRAM)
    obj = B.OUT_DIR / B.OBJ_DIR_NAME / "decode.o"
    subprocess.run(["g++", "-std=c++17", "-O1", "-UNDEBUG", "-pthread", "-I", str(B.Path(B._nvcc()).resolve().parent.parent / "include"),
                    str(src), str(obj), "-o", str(exe)], check=True)
    run = subprocess.run([str(exe)], timeout=60, capture_output=True, text=True)
    assert run.returncode == 0, run.stdout + run.stderr
