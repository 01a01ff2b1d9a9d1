"""The library's device allocations and the scratch it keeps between calls, against a CUDA runtime
that is played by the test: no device, and none driven out of memory."""
import subprocess

from conftest import ROOT

FAKE_MAIN = r"""
#include "device_memory.cuh"
#include <cstdint>
#include <cstdio>
#include <map>
#include <set>

// ---- the runtime: two devices of `room` bytes, pools, a last error
static int device = 0;
static size_t room[2], kept[2];  // free bytes; bytes that the device's pool keeps
static cudaError_t last = cudaSuccess;
static bool no_pools = false, no_threshold = false;
static std::map<cudaMemPool_t, int> live;
static cudaError_t set(cudaError_t e) { if (e != cudaSuccess) last = e; return e; }
static char arena;
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaMalloc(void** p, size_t n) {
  if (n > room[device]) return set(cudaErrorMemoryAllocation);
  room[device] -= n; *p = &arena; return cudaSuccess;
}
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t) {
  if (!live.count(pool)) return set(cudaErrorInvalidValue);
  const int d = live[pool];
  if (n <= kept[d]) { *p = &arena; return cudaSuccess; }
  if (n - kept[d] > room[d]) return set(cudaErrorMemoryAllocation);
  room[d] -= n - kept[d]; kept[d] = n; *p = &arena; return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* pool, const cudaMemPoolProps* props) {
  if (no_pools) return set(cudaErrorNotSupported);
  static intptr_t next = 16;
  *pool = (cudaMemPool_t)(next += 16); live[*pool] = props->location.id; return cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t pool) { live.erase(pool); return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) {
  return no_threshold ? set(cudaErrorInvalidValue) : cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t pool, size_t) {
  if (!live.count(pool)) return set(cudaErrorInvalidValue);
  const int d = live[pool]; room[d] += kept[d]; kept[d] = 0; return cudaSuccess;
}
}

#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
int main() {
  using namespace gwmb;
  void* p = nullptr;
  float* f = nullptr;
  room[0] = room[1] = 1000;
  // a runtime without pools: the default pool, and no error left for a launch to report
  no_pools = true;
  CHECK(scratch_alloc(&p, 100, nullptr) == cudaSuccess && room[0] == 900 && last == cudaSuccess);
  no_pools = false;
  // a pool whose threshold cannot be set is given up whole
  no_threshold = true;
  CHECK(scratch_alloc(&p, 100, nullptr) == cudaSuccess && live.empty() && last == cudaSuccess);
  no_threshold = false;
  room[0] = 1000;
  // both devices keep scratch
  CHECK(scratch_alloc(&p, 600, nullptr) == cudaSuccess && kept[0] == 600);
  device = 1;
  CHECK(scratch_alloc(&p, 600, nullptr) == cudaSuccess && kept[1] == 600 && live.size() == 2);
  // an allocation that finds no room takes the kept scratch back
  CHECK(device_alloc(&f, 900) == cudaSuccess && last == cudaSuccess && kept[1] == 0 && room[1] == 100);
  // one that does not fit at all fails cleanly
  CHECK(device_alloc(&f, 5000) == cudaErrorMemoryAllocation && last == cudaSuccess);
  CHECK(device_alloc_async(&f, 5000, nullptr) == cudaErrorMemoryAllocation && last == cudaSuccess);
  CHECK(scratch_alloc(&p, 5000, nullptr) == cudaErrorMemoryAllocation && last == cudaSuccess && live.size() == 2);
  // trimming reaches the other device's pool too
  device = 0;
  CHECK(scratch_alloc(&p, 600, nullptr) == cudaSuccess && kept[0] == 600);
  device = 1;
  trim_scratch();
  CHECK(kept[0] == 0 && room[0] == 1000);
  // pools that died with their context are replaced
  live.clear();
  room[1] = 1000;
  CHECK(scratch_alloc(&p, 100, nullptr) == cudaSuccess && last == cudaSuccess);  // the default pool this once
  CHECK(scratch_alloc(&p, 100, nullptr) == cudaSuccess && live.size() == 1 && last == cudaSuccess);
  std::puts("ok");
  return 0;
}
"""


def test_allocations_against_a_played_runtime(tmp_path):
    src = tmp_path / "memory.cpp"
    src.write_text(FAKE_MAIN)
    exe = tmp_path / "memory"
    csrc = f"{ROOT}/gpu-wm-next_b200/csrc"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", csrc, "-I", "/usr/local/cuda/include", "-o", str(exe), str(src),
                    f"{csrc}/device_memory.cpp"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout


def test_every_device_allocation_goes_through_it():
    import glob
    import re
    for path in glob.glob(f"{ROOT}/gpu-wm-next_b200/csrc/*"):
        if not path.endswith("device_memory.cpp") and not path.endswith("device_memory.cuh"):
            assert not re.search(r"cudaMalloc(Async|FromPoolAsync)?\(", open(path).read()), path
