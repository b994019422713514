"""The self-collision stage's device buffers when an allocation fails while they
grow (a fake of the CUDA allocator, no device): nothing is freed twice or kept,
the capacity is 0, no last run is left to read back, and the next growth
succeeds. Every allocation of every kind of growth fails once."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "garmentcraft_b200", "csrc")

PROBE = r"""
#include <cstdio>
#include <cstdlib>
#include <functional>
#include <set>
#include "k3d_selbst_host.h"
using namespace k3d;

static std::set<void*> lebt;
static int bis = -1, zahl = 0, letzter = 0, fehler = 0;  // the call number `bis` fails
extern "C" {
cudaError_t cudaMalloc(void** p, size_t) {
  if (zahl++ == bis) return cudaError_t(letzter = cudaErrorMemoryAllocation);
  *p = std::malloc(1);
  lebt.insert(*p);
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  if (!lebt.erase(p)) ++fehler;  // twice, or never allocated
  else std::free(p);
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { const int e = letzter; letzter = 0; return cudaError_t(e); }
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
}
namespace k3d {
size_t selbst_scan_tmp_words(int64_t n) { return size_t(n); }
cudaError_t selbst_hash_zaehlen(const SelbstArgs&, cudaStream_t) { return cudaSuccess; }
cudaError_t selbst_hash_fuellen_und_paare_zaehlen(const SelbstArgs&, cudaStream_t) { return cudaSuccess; }
cudaError_t selbst_paare_und_federn(const SelbstArgs&, uint32_t, uint32_t, uint32_t, cudaStream_t) { return cudaSuccess; }
cudaError_t selbst_zeilen_zaehlen(const SelbstArgs&, cudaStream_t) { return cudaSuccess; }
cudaError_t selbst_zeilen(const SelbstArgs&, cudaStream_t) { return cudaSuccess; }
int selbst_launches_per_run(bool) { return 0; }
cudaError_t selbst_stoss_zaehlen(const SelbstArgs&, cudaStream_t) { return cudaSuccess; }
cudaError_t selbst_stoss_antwort(const SelbstArgs&, int, unsigned long long*, cudaStream_t) { return cudaSuccess; }
int selbst_stoss_launches(int) { return 0; }
}

int main() {
  SelbstHost H;
  H.s.n = 100;
  H.s.rsize = 8;
  struct Art {
    const char* name;
    std::function<cudaError_t(uint32_t)> f;
    std::function<uint32_t()> cap;
    std::vector<void*>* v;
  } arten[] = {
      {"schnitte", [&](uint32_t c) { return selbst_grow_schnitte(H, c); }, [&] { return H.s.cap_s; }, &H.schn},
      {"wege", [&](uint32_t c) { return selbst_grow_wege(H, c, c); }, [&] { return H.s.hp2.cap | H.s.hk2.cap; }, &H.wege},
      {"kanten", [&](uint32_t c) { return selbst_grow_edge_hash(H, c); }, [&] { return H.s.cap_ek; }, &H.hashk},
      {"paare", [&](uint32_t c) { return selbst_grow_pairs(H, c); }, [&] { return H.s.cap_pairs | H.s.cap_inc; }, &H.pairs},
      {"zeilen", [&](uint32_t c) { return selbst_grow_zeilen(H, c); }, [&] { return H.s.cap_sf; }, &H.sf}};
  for (Art& a : arten) {
    for (int k = 0;; ++k) {
      bis = -1;
      if (a.f(64) != cudaSuccess || a.cap() == 0) std::printf("%s: grows\n", a.name), ++fehler;
      H.ran = true;
      zahl = 0;
      bis = k;
      const cudaError_t e = a.f(1000);
      if (e == cudaSuccess) {
        if (zahl > k) std::printf("%s: call %d failed, the growth did not\n", a.name, k), ++fehler;
        if (k < 3) ++fehler;
        break;
      }
      if (a.cap() != 0 || !a.v->empty() || H.ran || letzter != 0)
        std::printf("%s: call %d leaves capacity %u, %zu buffers, ran %d, error %d\n", a.name, k, a.cap(), a.v->size(),
                    int(H.ran), letzter), ++fehler;
    }
  }
  selbst_free(H);
  if (!lebt.empty()) std::printf("%zu buffers leak\n", lebt.size()), ++fehler;
  return fehler ? 1 : 0;
}
"""


def test_wachsen_scheitert(tmp_path):
    src, exe = tmp_path / "probe.cpp", tmp_path / "probe"
    src.write_text(PROBE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=address,undefined", "-include", "math.h", "-I", CSRC,
                    "-I/usr/local/cuda/include", str(src), os.path.join(CSRC, "k3d_selbst_host.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
