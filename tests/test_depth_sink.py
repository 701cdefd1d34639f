"""The depth sink's staging ring: made only by runs that it pays for (a fresh
graph with a small result copies it with one driver copy), and the rows arrive
whole with and without it.  The first test runs sink.cpp on the CPU against a
stand-in for the CUDA runtime that counts what is pinned."""
import subprocess

import numpy as np
import pytest

import ibfs_b200 as ib
import oracle
from ibfs_b200 import build

PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include <cuda_runtime.h>
#include "internal.h"

static size_t pinned = 0;
static int allocs = 0, events = 0, streams = 0;
static bool refuse = false;
extern "C" {
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
  a->type = cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  streams++;
  *s = reinterpret_cast<cudaStream_t>(&streams);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { streams--; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  events++;
  *e = reinterpret_cast<cudaEvent_t>(&events);
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { events--; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaErrorNotReady; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaHostRegister(void*, size_t n, unsigned) {
  if (refuse) return cudaErrorMemoryAllocation;
  allocs++;
  pinned += n;
  return cudaSuccess;
}
cudaError_t cudaHostUnregister(void*) { allocs--; pinned = 0; return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) {
  allocs++;
  pinned += n;
  *p = std::malloc(n);
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { allocs--; std::free(p); return cudaSuccess; }
}

static int bad = 0;
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); bad = 1; } } while (0)

int main() {
  using namespace ibfs;
  const size_t MB = 1u << 20;
  {
    DepthSink s;  // small results: no ring until they add up
    for (int i = 0; i < 31; i++) CHECK(!s.ring_pays(MB));
    CHECK(pinned == 0 && allocs == 0);
    CHECK(s.ring_pays(MB));
    DepthSink big;
    CHECK(!big.ring_pays(32 * MB - 1));
    DepthSink whole;
    CHECK(whole.ring_pays(32 * MB));
  }
  {
    DepthSink s;
    const size_t V = 100003, n = 701;  // rows straddle slots: 70 MB
    std::vector<uint8_t> src(V * n), dst(V * n);
    for (size_t i = 0; i < src.size(); i++) src[i] = (uint8_t)(i * 2654435761u >> 24);
    for (int turn = 0; turn < 2; turn++) {
      std::fill(dst.begin(), dst.end(), 0);
      CHECK(s.begin(0, dst.data(), src.data()) == cudaSuccess);
      CHECK(allocs == 1 && pinned == 32 * MB);
      for (size_t r = 0; r < n; r++)  // rows out of order
        CHECK(s.push((r * 37 % n) * V, V) == cudaSuccess);
      CHECK(s.finish() == cudaSuccess);
      CHECK(std::memcmp(dst.data(), src.data(), src.size()) == 0);
      CHECK(s.ring_pays(1));
    }
    s.release();
    CHECK(allocs == 0 && pinned == 0 && events == 0 && streams == 0);
    refuse = true;  // no pinned memory: an error, and nothing kept
    CHECK(s.begin(0, dst.data(), src.data()) == cudaErrorMemoryAllocation);
    CHECK(allocs == 0 && events == 0 && streams == 0);
    refuse = false;
    CHECK(s.begin(0, dst.data(), src.data()) == cudaSuccess);
    CHECK(s.push(0, src.size()) == cudaSuccess && s.finish() == cudaSuccess);
    CHECK(std::memcmp(dst.data(), src.data(), src.size()) == 0);
  }
  CHECK(allocs == 0 && events == 0 && streams == 0);
  return bad;
}
"""


def test_ring_is_made_when_it_pays(tmp_path):
    src, exe = tmp_path / "sink_test.cpp", tmp_path / "sink_test"
    src.write_text(PROGRAM)
    subprocess.run(["g++", *build.CXX_FLAGS, f"-I{build.CSRC}", str(src),
                    f"{build.CSRC}/sink.cpp", "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("n,turns", [(1, 2), (1000, 5), (3400, 2)])  # 10 kB, 10 MB, 34 MB
def test_host_rows_before_and_after_the_ring(n, turns):
    beg, col = ib.gen_chung_lu(10007, 120000, 2.1, 900.0, seed=15)
    with ib.Graph.from_csr(beg, col) as g:
        for turn in range(turns):
            src = ib.sample_sources(beg, col, n, seed=turn)
            ref, _ = oracle.bfs_auto(beg, col, src)
            assert np.array_equal(g.run(src, mode=ib.MODE_PERSISTENT).depth, ref)
