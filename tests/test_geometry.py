"""The divisors that a geometry carries beside the counts they are derived from, on the host."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG_DIR

PROGRAM = r"""
#include <cstdio>
#include "dn_common.cuh"
namespace dn { bool force_simt() { return false; } }
using namespace dn;

static int bad = 0;
static void same(const char* what, long long a, long long b) {
  if (a != b) { std::printf("%s: %lld, not %lld\n", what, a, b); ++bad; }
}
static void check(const Geo& g) {
  same("by_BH", g.by_BH.d, g.B * g.H);
  same("by_H", g.by_H.d, g.H);
  same("by_q", g.by_q.d, g.qk_div);
  for (int h = 0; h < g.H; ++h) {
    same("qk_head", g.qk_head(h), h / g.qk_div);
    same("g_head", g.g_head(h), g.gate_head(h, g.gH));
    same("b_head", g.b_head(h), g.gate_head(h, g.bH));
  }
  for (int hv = 0; hv < g.Hv; ++hv) same("w_of", g.w_of(hv), g.w_head(hv));
}

int main() {
  for (int Hk = 1; Hk <= 3; ++Hk)
    for (int group = 1; group <= 4; ++group)
      for (int gates = 0; gates < 27; ++gates) {
        const int heads[3] = {1, Hk, Hk * group};
        dn_shape s{};
        s.B = 5; s.L = 300; s.Hk = Hk; s.Hv = Hk * group; s.K = s.V = 128; s.chunk = 128;
        s.g_heads = heads[gates % 3]; s.b_heads = heads[gates / 3 % 3]; s.w_heads = heads[gates / 9];
        s.g_cols = s.b_cols = s.w_cols = 1;
        s.qkv_dtype = DN_BF16; s.gate_dtype = DN_F32; s.precision = DN_PREC_BF16; s.scale = 1.f;
        Geo g;
        same("make_geo", make_geo(&s, &g), DN_OK);
        check(g);
        check(transition_geo(g));
      }
  unsigned long long r = 1;
  for (int i = 0; i < 200000; ++i) {             // divisors of every size; quotients either side of each multiple
    r = r * 6364136223846793005ull + 1442695040888963407ull;
    const int d = (int)((r >> 33) >> (r >> 8 & 31)) | 1, k = (int)((r >> 20 & 0x7fffffff) % (0x7fffffff / d + 1u));
    for (int e = d; e <= d + 1 && e > 0; ++e) {
      FastDiv f;
      f.set(e);
      for (long long n = (long long)k * e - 1; n <= (long long)k * e + 1; ++n)
        if (n >= 0 && n <= 0x7fffffff) same("div", f.div((int)n), n / e);
      same("div", f.div(0x7fffffff), 0x7fffffff / e);
    }
  }
  return bad != 0;
}
"""


def test_divisors_follow_the_counts(tmp_path):
    """Every geometry, and the copy that a shard's transition matrix is computed with: the kernels divide by these."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("needs nvcc")
    src, exe = tmp_path / "geometry.cu", tmp_path / "geometry"
    src.write_text(PROGRAM)
    csrc = os.path.join(PKG_DIR, "csrc")
    subprocess.run([nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-extended-lambda", "-I" + csrc,
                    "-I" + os.path.join(os.path.dirname(PKG_DIR), "include"), str(src), "-o", str(exe)], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout[-2000:]
