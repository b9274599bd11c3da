"""Substitution and replacement update the vector grid in place, a thread per
cell: a cell may read the cells that count (neither flagged nor masked), which
nobody writes, and no other. The per-cell functions of the kernels' header run
here on host threads, and ThreadSanitizer reports a read of a cell that another
thread writes."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "hammerhead.jl_b200", "csrc", "hh_grid.cuh")

SHIM = r"""
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <thread>
#include <vector>
using std::isfinite; using std::isnan; using std::max; using std::min;
#define __device__
#define __forceinline__ inline
#define INF_ __int_as_float(0x7f800000)
static float __int_as_float(int x) { float f; memcpy(&f, &x, 4); return f; }
static double __longlong_as_double(long long x) { double d; memcpy(&d, &x, 8); return d; }
static float __uint_as_float(unsigned x) { return __int_as_float((int)x); }
static unsigned __float_as_uint(float f) { unsigned u; memcpy(&u, &f, 4); return u; }
static int __popc(unsigned x) { return __builtin_popcount(x); }
#define __fadd_rn(a, b) ((float)(a) + (float)(b))
#define __fsub_rn(a, b) ((float)(a) - (float)(b))
#define __fmul_rn(a, b) ((float)(a) * (float)(b))
#define __dadd_rn(a, b) ((double)(a) + (double)(b))
#define __dsub_rn(a, b) ((double)(a) - (double)(b))
#define __dmul_rn(a, b) ((double)(a) * (double)(b))
"""

LOAD = """
inline float ld_present(const float* p, bool on) { return on ? *p : INF_; }
"""

MAIN = r"""
static unsigned rnd = 7;
static float noise() { rnd = rnd * 1664525u + 1013904223u; return (float)(rnd >> 8) / 16777216.f; }
int main() {
  int bad = 0;
  for (int er = 1; er <= 4; ++er)
    for (int masked = 0; masked < 2; ++masked) {
      const int ny = 37, nx = 41, G = ny * nx, nt = 8;
      std::vector<float> u(G), v(G), au(G), av(G);
      std::vector<uint8_t> flags(G), gm(G);
      for (int k = 0; k < G; ++k) {
        u[k] = noise(), v[k] = noise(), au[k] = 0.5f * noise() + 0.25f, av[k] = 0.5f * noise() + 0.25f;
        flags[k] = noise() < 0.35f, gm[k] = masked && noise() < 0.2f;
        if (gm[k]) flags[k] = 0;
      }
      const uint8_t* m = masked ? gm.data() : nullptr;
      std::vector<float> got[2][2];
      std::vector<uint8_t> out[2];
      for (int par = 0; par < 2; ++par) {
        auto uu = u, vv = v;
        std::vector<uint8_t> o(G);
        auto cells = [&](auto f) {
          std::vector<std::thread> t;
          for (int w = 0; w < (par ? nt : 1); ++w)
            t.emplace_back([&, w] { for (int k = w; k < G; k += par ? nt : 1) f(k); });
          for (auto& x : t) x.join();
        };
        cells([&](int k) {
          auto cell = er > 2 ? hh::substitute_cell<true> : hh::substitute_cell<false>;
          o[k] = cell(uu.data(), vv.data(), flags.data(), m, au.data(), av.data(), 1, ny, nx, k % ny, k / ny, er, 2.0);
        });
        cells([&](int k) {
          if (!hh::repl_invalid(o.data(), m, k)) return;
          float a = uu[k], b = vv[k];
          if (m && m[k]) a = b = hh::f_nan();
          else hh::replace_cell(uu.data(), vv.data(), o.data(), m, ny, nx, k % ny, k / ny, a, b);
          uu[k] = a;
          vv[k] = b;
        });
        got[par][0] = uu, got[par][1] = vv, out[par] = o;
      }
      bad += out[0] != out[1] || memcmp(got[0][0].data(), got[1][0].data(), 4 * G) || memcmp(got[0][1].data(), got[1][1].data(), 4 * G);
    }
  printf("%d\n", bad);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_only_cells_that_count_are_read(tmp_path):
    empty = tmp_path / "empty.cpp"
    empty.write_text("int main() { return 0; }\n")
    tsan = ["g++", "-std=c++17", "-O1", "-g", "-fsanitize=thread", "-ffp-contract=off"]
    probe = subprocess.run(tsan + [str(empty), "-o", str(tmp_path / "empty")], capture_output=True)
    if probe.returncode or subprocess.run([str(tmp_path / "empty")], capture_output=True).returncode:
        pytest.skip("no working ThreadSanitizer")
    with open(HEADER) as f:
        text = f.read()
    # the cells' functions: all but the cluster's norm at the end, with the
    # predicated load restated
    text = text[:text.index("constexpr int FC_CLUSTER")] + "}\n"
    text = re.sub(r"#include <cooperative_groups.h>\n|#pragma \w+\n", "", text)
    text = re.sub(r"__device__ __forceinline__ float ld_present\(.*?\n}\n", LOAD, text, flags=re.S)
    src, exe = tmp_path / "cells.cpp", tmp_path / "cells"
    src.write_text(SHIM + text + MAIN)
    subprocess.check_call(tsan + [str(src), "-o", str(exe), "-lpthread"])
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert "ThreadSanitizer" not in r.stderr, r.stderr[:3000]
    assert r.returncode == 0 and r.stdout.strip() == "0"
