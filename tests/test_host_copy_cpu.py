"""The copier of large host arrays (csrc/hostcopy.cpp) against a stand-in for the CUDA runtime whose copies are plain
ones: bytes of every length come through, and where an allocation fails (each of the first ones in turn) the copy takes
the ordinary way instead of throwing into its C caller. Contexts that copy at once share a bounded number of copiers,
which the last one gives back."""
import os
import pathlib
import subprocess

import pytest

ROOT = pathlib.Path(__file__).parent.parent
CUDA = pathlib.Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"

MAIN = r"""
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <thread>
#include <vector>
#include "internal.h"

static std::atomic<int> pinned{0}, made{0};  // slot memories that are there; that were made
static thread_local int fail_at = -1;  // the allocation of this thread that fails, counted down
void* operator new(size_t n) {
  if (fail_at == 0) throw std::bad_alloc();
  if (fail_at > 0) --fail_at;
  void* p = std::malloc(n);
  if (!p) throw std::bad_alloc();
  return p;
}
void* operator new(size_t n, const std::nothrow_t&) noexcept {
  try { return operator new(n); } catch (...) { return nullptr; }
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

extern "C" {
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)std::malloc(1); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { ++pinned; ++made; *p = std::malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { --pinned; std::free(p); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { a->type = cudaMemoryTypeUnregistered; return cudaSuccess; }
}

int main() {
  for (int k = -1; k < 24; ++k) {
    mycel_ctx c;
    mycel::host_copy_attach(&c);
    for (size_t n : {(size_t)1000, (size_t)1 << 20, ((size_t)1 << 20) + 1, (size_t)9 * 1000 * 1000 + 7}) {
      std::vector<char> h(n), d(n), back(n);
      for (size_t i = 0; i < n; ++i) h[i] = (char)(i * 2654435761u >> 13);
      try {
        fail_at = k;
        const bool bad = mycel::copy_in(&c, d.data(), h.data(), n) != cudaSuccess ||
                         mycel::copy_out(&c, back.data(), d.data(), n) != cudaSuccess;
        fail_at = -1;
        if (bad || d != h || back != h) return std::printf("bytes differ: failing allocation %d, length %zu\n", k, n), 1;
      } catch (...) {
        fail_at = -1;
        return std::printf("threw: failing allocation %d, length %zu\n", k, n), 1;
      }
    }
    mycel::host_copy_release(&c);
  }
  if (pinned != 0) return std::puts("slots left behind by the last context"), 1;
  // six contexts that copy at once and end one after another: a bounded number of copiers, none for each context
  made = 0;
  mycel_ctx cs[6];
  std::atomic<int> wrong{0}, most{0};
  for (auto& c : cs) mycel::host_copy_attach(&c);
  std::vector<std::thread> ts;
  for (int t = 0; t < 6; ++t)
    ts.emplace_back([&, t] {
      for (int k = 0; k < 12; ++k) {
        const size_t n = ((size_t)1 << 20) + 1000 * t + k;
        std::vector<char> h(n, (char)(t + k)), d(n), back(n);
        mycel::copy_in(&cs[t], d.data(), h.data(), n);
        mycel::copy_out(&cs[t], back.data(), d.data(), n);
        if (back != h) ++wrong;
        const int now = pinned;
        if (now > most) most = now;
      }
      mycel::host_copy_release(&cs[t]);
    });
  for (auto& t : ts) t.join();
  if (wrong || most > 2 || made > 2 || pinned != 0)
    return std::printf("%d wrong, %d copiers at once, %d made, %d left\n", wrong.load(), most.load(), made.load(), pinned.load()), 1;
  return std::puts("ok"), 0;
}
"""


@pytest.mark.skipif(not (CUDA / "cuda_runtime.h").exists(), reason="no CUDA headers")
def test_copies_and_failing_allocations(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    csrc = ROOT / "mycel_b200/csrc"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{CUDA}", f"-I{csrc}", str(tmp_path / "main.cpp"),
                    str(csrc / "hostcopy.cpp"), "-o", str(tmp_path / "t")], check=True)
    r = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, timeout=120)
    assert r.stdout.strip() == "ok", r.stdout + r.stderr[-500:]
