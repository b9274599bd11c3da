"""The pixel list of the row-maxima peak scans, run lane by lane on the CPU.

The lanes of a warp share a short list in shared memory. Only __syncwarp orders
their accesses; ballots and reductions order none. Here each lane is a host
thread: __syncwarp is a barrier with memory order, every other collective
exchanges values with relaxed atomics, and ThreadSanitizer reports two accesses
of a list word that nothing orders. The scans are the functions of the kernels'
headers, compiled as they stand."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "hammerhead.jl_b200", "csrc")

SHIM = r"""
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <sched.h>
#include <set>
#include <thread>
#include <vector>
using std::isnan; using std::max; using std::min;
#define __device__
#define __forceinline__ inline
static thread_local int my_lane;
struct Tid { struct { operator int() const { return my_lane; } } x; };
static Tid threadIdx;
static std::atomic<unsigned> slot[2][32], arrived{0}, phase{0};
// a meeting of the 32 lanes that orders no other memory
static void meet(std::memory_order o) {
  const unsigned p = phase.load(o == std::memory_order_relaxed ? o : std::memory_order_acquire);
  if (arrived.fetch_add(1, o == std::memory_order_relaxed ? o : std::memory_order_acq_rel) == 31) {
    arrived.store(0, std::memory_order_relaxed);
    phase.fetch_add(1, o == std::memory_order_relaxed ? o : std::memory_order_acq_rel);
  } else {
    while (phase.load(o == std::memory_order_relaxed ? o : std::memory_order_acquire) == p) sched_yield();
  }
}
static thread_local int turn_ = 0;
template <class F> static unsigned gather(unsigned v, unsigned r, const F& f) {
  auto& s = slot[turn_ ^= 1];
  s[my_lane].store(v, std::memory_order_relaxed);
  meet(std::memory_order_relaxed);
  for (int k = 0; k < 32; ++k) r = f(r, k, s[k].load(std::memory_order_relaxed));
  return r;
}
static unsigned __ballot_sync(unsigned, bool p) {
  return gather(p, 0u, [](unsigned r, int k, unsigned v) { return r | v << k; });
}
static bool __any_sync(unsigned m, bool p) { return __ballot_sync(m, p) != 0; }
static unsigned __reduce_max_sync(unsigned, unsigned v) {
  return gather(v, 0u, [](unsigned r, int, unsigned x) { return std::max(r, x); });
}
static unsigned __shfl_xor_sync(unsigned, unsigned v, int o) {
  return gather(v, 0u, [o](unsigned r, int k, unsigned x) { return k == (my_lane ^ o) ? x : r; });
}
static void __syncwarp(unsigned = 0xffffffffu) { meet(std::memory_order_acq_rel); }
static int __popc(unsigned x) { return __builtin_popcount(x); }
static int __ffs(unsigned x) { return __builtin_ffs((int)x); }
static float __int_as_float(int x) { float f; memcpy(&f, &x, 4); return f; }
static unsigned __float_as_uint(float f) { unsigned u; memcpy(&u, &f, 4); return u; }
static unsigned fkey(float v) { return __float_as_uint(v) | 0x80000000u; }
static unsigned grp_mask(int) { return 0xffffffffu; }
struct Found {  // every pixel a lane reports
  std::vector<unsigned> e;
  void insert(uint32_t, uint32_t l, int) { e.push_back(~l); }
};
"""

MAIN = r"""
static unsigned rnd = 12345;
static float noise(int levels) { rnd = rnd * 1664525u + 1013904223u; return (float)((rnd >> 16) % levels) / levels; }
template <int N, int LANES, class F> static int run(int levels, int K, const F& scan) {
  constexpr int WIN = 32 / LANES, LD = N + 1;
  std::vector<std::vector<float>> R(WIN, std::vector<float>(N * LD));
  std::vector<std::vector<uint32_t>> rmax(WIN, std::vector<uint32_t>(N));
  std::vector<std::vector<uint16_t>> list(WIN, std::vector<uint16_t>(2 * LANES));
  for (int w = 0; w < WIN; ++w)
    for (int c = 0; c < N; ++c)
      for (int r = 0; r < N; ++r) {
        R[w][c * LD + r] = noise(levels);
        rmax[w][r] = std::max(rmax[w][r], __float_as_uint(R[w][c * LD + r]));
      }
  std::vector<Found> found(32);
  std::vector<std::thread> lanes;
  for (int k = 0; k < 32; ++k)
    lanes.emplace_back([&, k] {
      my_lane = k;
      const int w = k / LANES;
      scan(found[k], R[w].data(), rmax[w].data(), list[w].data(), k % LANES);
    });
  for (auto& t : lanes) t.join();
  // every regional maximum down to a bound is found once, K of them or all there are
  int bad = 0;
  for (int w = 0; w < WIN; ++w) {
    std::multiset<unsigned> want, got;
    for (int c = 0; c < N; ++c)
      for (int r = 0; r < N; ++r) {
        bool m = true;
        for (int dc = -1; dc <= 1; ++dc)
          for (int dr = -1; dr <= 1; ++dr) {
            const int i = r + dr, j = c + dc;
            if ((!dr && !dc) || i < 0 || i >= N || j < 0 || j >= N) continue;
            const bool earlier = dc < 0 || (dc == 0 && dr < 0);
            const float x = R[w][j * LD + i], v = R[w][c * LD + r];
            m = m && (earlier ? !(x > v) : !(x >= v));
          }
        if (m) want.insert(r + c * N);
      }
    for (int k = 0; k < LANES; ++k) got.insert(found[w * LANES + k].e.begin(), found[w * LANES + k].e.end());
    bad += got.size() < std::min<size_t>(K, want.size());
    auto value = [&](unsigned e) { return R[w][e / N * LD + e % N]; };
    float bound = 2.f;
    for (unsigned e : got) bound = std::min(bound, value(e));
    std::multiset<unsigned> above;
    for (unsigned e : want)
      if (value(e) >= bound) above.insert(e);
    bad += above != got;
  }
  return bad;
}
int main() {
  int bad = 0;
  static int K;  // 40 is more than the row maxima that stand out: the bound falls to 0
  for (int levels : {1, 3, 50})
    for (int k : {2, 5, 40}) {
      K = k;
      CASES
    }
  printf("%d\n", bad);
}
"""

ROWS = """
    bad += run<N, 32>(levels, K, [](Found& f, const float* R, const uint32_t* m, uint16_t* l, int g) {
      scan_rows<N, 32>(f, R, N + 1, K, 0, N - 1, m, l, g, 1); });"""
SEG = """
    bad += run<N, N / 2>(levels, K, [](Found& f, const float* R, const uint32_t* m, uint16_t* l, int g) {
      seg_scan_rows<N>(f, R, K, m, l, g, true); });"""


def _function(header, name):
    """The text of a function template of a header."""
    with open(os.path.join(CSRC, header)) as f:
        text = f.read()
    m = re.search(r"template <[^;{}]*?\b%s\(.*?\n}\n" % name, text, re.S)
    start = text.rindex("\ntemplate", 0, m.end()) if m.group(0).count("\ntemplate") else m.start()
    return text[start:m.end()]


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
@pytest.mark.parametrize("header,names,call,sizes", [
    pytest.param("hh_corr_peaks.cuh", ["scan_rows"], ROWS, (24, 48), id="warps"),
    pytest.param("hh_corr_seg.cuh", ["seg_max", "seg_scan_rows"], SEG, (16, 32), id="segments")])
def test_list_accesses_are_ordered(tmp_path, header, names, call, sizes):
    empty = tmp_path / "empty.cpp"
    empty.write_text("int main() { return 0; }\n")
    tsan = ["g++", "-std=c++17", "-O1", "-g", "-fsanitize=thread"]
    probe = subprocess.run(tsan + [str(empty), "-o", str(tmp_path / "empty")], capture_output=True)
    if probe.returncode or subprocess.run([str(tmp_path / "empty")], capture_output=True).returncode:
        pytest.skip("no working ThreadSanitizer")
    cases = "".join("{ constexpr int N = %d; %s }" % (n, call) for n in sizes)
    src, exe = tmp_path / "scan.cpp", tmp_path / "scan"
    src.write_text(SHIM + "\n".join(_function(header, n) for n in names) + MAIN.replace("CASES", cases))
    subprocess.check_call(tsan + ["-Wno-unknown-pragmas", str(src), "-o", str(exe), "-lpthread"])
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert "ThreadSanitizer" not in r.stderr, r.stderr[:3000]
    assert r.returncode == 0 and r.stdout.strip() == "0"
