"""The count of resident clusters, against a CUDA runtime of the test's own (no GPU): what it returns, what it remembers, and
that it leaves an error alone that the caller has pending."""
import os
import subprocess

from basedxl_b200 import build

PROGRAM = r"""
#include <stdio.h>
#include <thread>
#include <vector>
#include "bxl_host.h"

static cudaError_t pending = cudaSuccess;   // the runtime's last error
static int answer = 33, queries = 0;
static bool failing = false;
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) {
  ++queries;
  if (failing) return pending = cudaErrorInvalidValue;
  *n = answer;
  return cudaSuccess;
}
cudaError_t cudaPeekAtLastError() { return pending; }
cudaError_t cudaGetLastError() { cudaError_t e = pending; pending = cudaSuccess; return e; }
}
namespace bxl { int sm_count() { return 148; } }
static const void* const kernel = "a kernel";
#define CHECK(c) if (!(c)) { printf("line %d: %s\n", __LINE__, #c); return 1; }

template <typename Cache>
static int ask(Cache& cache, int width) { return bxl::resident_clusters(kernel, 512, 1024, width, cache); }
static std::atomic<int> a[64][5], b[64][5];
int main() {
  CHECK(ask(a, 4) == 33 && ask(a, 4) == 33 && queries == 1);        // asked once
  answer = 80;
  CHECK(ask(a, 2) == 74);                                           // never more than SMs / width
  pending = cudaErrorLaunchTimeout;                                 // somebody else's
  failing = true;
  CHECK(ask(b, 4) == 37 && pending == cudaErrorLaunchTimeout);
  pending = cudaSuccess;
  CHECK(ask(b, 2) == 74 && pending == cudaSuccess);                 // its own failure leaves nothing behind
  failing = false, answer = 33;
  CHECK(ask(b, 4) == 33);                                           // and what was not asked then is asked now
  std::vector<std::thread> threads;
  bool ok[8];
  for (int i = 0; i < 8; ++i) threads.emplace_back([&, i] { ok[i] = true; for (int k = 0; k < 1000; ++k) ok[i] &= ask(a, 4) == 33; });
  for (auto& t : threads) t.join();
  for (bool o : ok) CHECK(o);
  return 0;
}
"""


def test_resident_clusters_leaves_the_callers_error_alone(tmp_path):
    src = tmp_path / "clusters.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "clusters"
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build._nvcc()))), "include")
    subprocess.check_call(["g++", "-std=c++17", "-I", build.CSRC, "-I", cuda, str(src), "-o", str(exe), "-lpthread"])
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0, run.stdout
