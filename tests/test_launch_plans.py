"""What launch plans keep per device and kernel (csrc/gsq_host.h), asked for by many threads at once: the header compiled by the host
compiler against stand-ins for the CUDA calls it makes. No GPU."""

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "vllm-gsqrco-exl3_b200", "csrc")

HARNESS = r"""
#include "gsq_host.h"
#include <condition_variable>
#include <cstdio>
#include <mutex>
#include <thread>
#include <vector>

static std::mutex mu;
static std::condition_variable cv;
static int calls, inside, together;

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
// clusters of cs CTAs: 100 / cs; the first `together` callers leave at the same time
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t* c) {
  std::unique_lock<std::mutex> l(mu);
  ++calls;
  if (++inside >= together) cv.notify_all();
  cv.wait(l, [] { return inside >= together; });
  *n = 100 / (int)c->attrs[0].val.clusterDim.x;
  return cudaSuccess;
}
}
int gsq::record_cuda_error(cudaError_t e) { return (int)e; }

static gsq::ClusterCount kept;
static int ask(int cs) {
  int n = -1;
  const int rc = gsq::max_clusters(kept, (const void*)&kept, cs, 512, 227 * 1024, 148, &n);
  return rc == 0 ? n : -2;
}

int main() {
  constexpr int THREADS = 96;
  int bad = 0;
  for (int cs : {8, 4}) {
    std::vector<int> got(THREADS);
    std::vector<std::thread> t;
    inside = 0;
    together = THREADS;
    for (int i = 0; i < THREADS; ++i) t.emplace_back([&, i] { got[i] = ask(cs); });
    for (auto& x : t) x.join();
    for (int n : got) bad += n != 100 / cs;
  }
  together = 0;
  const int before = calls;
  for (int i = 0; i < 3; ++i)
    for (int cs : {1, 2, 4, 8}) bad += ask(cs) != (cs == 1 ? 148 : 100 / cs);
  std::printf("%d %d\n", bad, calls - before);
  return 0;
}
"""


def test_cluster_counts_asked_for_by_many_threads(tmp_path):
    src, exe = tmp_path / "h.cpp", tmp_path / "h"
    src.write_text(HARNESS)
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.check_call([os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-isystem", cuda, str(src), "-o", str(exe)])
    bad, asked_again = map(int, subprocess.check_output([str(exe)], timeout=60).split())
    assert bad == 0
    assert asked_again == 1   # the driver is asked for cluster size 2 alone, and once: what 96 threads found for 4 and 8 is kept
