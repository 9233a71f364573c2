"""Host-compilable parts of the device headers, checked on the CPU: the layout of the crystals' cells, and
the float-pair functions, whose results are those of the FP64 functions rounded to float."""
import json
import os
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "fgrain_gb300" / "csrc"


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    """Compiles and runs a program (nvcc, host code only, no contraction); its output is JSON."""
    nvcc = os.environ.get("NVCC") or "/usr/local/cuda/bin/nvcc"

    def go(name, text):
        d = tmp_path_factory.mktemp(name)
        (d / "main.cu").write_text(text)
        subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-O2", "-Xcompiler", "-ffp-contract=off",
                        "-I", str(CSRC), "-o", str(d / "main"), str(d / "main.cu")], check=True, capture_output=True)
        return json.loads(subprocess.run([str(d / "main")], check=True, capture_output=True, text=True).stdout)

    return go


def test_every_coordinate_names_a_cell_of_its_axis(run):
    """cells_layout over boxes from a cube to a thread a million times as long as wide: the last cell's
    number is exact in float (a coordinate is clamped to it), the box's cells and one more are counted in
    31 bits, and there are at most 8 n + 64 of them."""
    r = run("cells", r"""
#include <cstdio>
#include "fg_cells.cuh"
int main() {
  int bad = 0, boxes = 0;
  for (double len : {1e0, 1e2, 1e4, 1e6, 3e6, 1e7, 1e8})
    for (double side : {1.0, 7.0, 300.0})
      for (double n : {1.0, 1e3, 1e5, 3e6, 4.1e6, 2e7, 2.1e9})
        for (int axis = 0; axis < 3; ++axis) {
          fg::CellGrid g{};
          const double b[3] = {axis == 0 ? len : side, axis == 1 ? len : side, axis == 2 ? len : side};
          if (!fg::cells_layout(b[0], b[1], b[2], n, g)) { ++bad; continue; }
          ++boxes;
          const double cells = 1.0 * g.x.n * g.y.n * g.z.n;
          for (const fg::CellAxis* a : {&g.x, &g.y, &g.z})
            if (a->n < 1 || static_cast<double>(a->last) != a->n - 1.0) ++bad;
          if (cells > 8.0 * n + 64.0 || cells + 1.0 >= 2147483648.0) ++bad;
        }
  std::printf("{\"bad\": %d, \"boxes\": %d}\n", bad, boxes);
}
""")
    assert r["boxes"] == 7 * 3 * 7 * 3 and r["bad"] == 0


PAIR = r"""
#include <cstdio>
#include <random>
#include "fg_pair.cuh"
using fg::Pair;
static std::mt19937_64 rng(7);
static double uniform(double a, double b) { return std::uniform_real_distribution<double>(a, b)(rng); }
static float near_by(float x, int ulps) { return fg::pair_float(fg::pair_bits(x) + static_cast<uint32_t>(ulps)); }
struct Stat {
  double worst = 0;  // relative error of the pair
  long n = 0, wrong = 0, unsettled = 0;
  void pair(Pair p, long double want) {
    const double e = static_cast<double>(fabsl((static_cast<long double>(p.h) + p.l - want) / want));
    if (want != 0 && !(e <= worst)) worst = e;
    float r;
    if (!fg::pair_round(p, r)) ++unsettled;
  }
  void value(float got, double want) {
    ++n;
    if (fg::pair_bits(got) != fg::pair_bits(static_cast<float>(want))) ++wrong;
  }
  void print(const char* name, bool last = false) {
    std::printf("\"%s\": {\"n\": %ld, \"wrong\": %ld, \"unsettled\": %ld, \"log2\": %.3f}%s", name, n, wrong, unsettled,
                std::log2(worst > 0 ? worst : 1e-300), last ? "}\n" : ", ");
  }
};
"""


def test_pair_functions_are_the_fp64_ones_rounded(run):
    """Each function's pair within 2^-40 of its value (the rounding is trusted from 2^-38 on) over its range,
    near its zeros and at its limits, and every result, settled or not, the FP64 one rounded to float."""
    r = run("pair", PAIR + r"""
int main() {
  const int N = 1500000;
  Stat lg, ex, sn, cs, qt, dn;
  auto log1 = [&](float x) {
    if (x >= 1.17549435e-38f && x < 2.4e38f) lg.pair(fg::pair_log(x), logl(static_cast<long double>(x)));
    lg.value(fg::pair_logf(x), std::log(static_cast<double>(x)));
  };
  auto exp1 = [&](float x) {
    if (fabsf(x) <= 70.0f) ex.pair(fg::pair_exp(x), expl(static_cast<long double>(x)));
    ex.value(fg::pair_expf(x), std::exp(static_cast<double>(x)));
  };
  auto sincos1 = [&](float x) {
    if (fabsf(x) <= 8.0f) {
      Pair s, c;
      fg::pair_sincos(x, s, c);
      if (x != 0.0f) sn.pair(s, sinl(static_cast<long double>(x)));
      cs.pair(c, cosl(static_cast<long double>(x)));
    }
    float s, c;
    fg::pair_sincosf(x, s, c);
    if (x != 0.0f) sn.value(s, std::sin(static_cast<double>(x)));
    cs.value(c, std::cos(static_cast<double>(x)));
  };
  auto quot1 = [&](double n, double d) {
    Pair a, b;
    fg::split64(n, a.h, a.l);
    fg::split64(d, b.h, b.l);
    qt.value(fg::pair_quotf(n, d, a, b), n / d);
  };
  auto density1 = [&](float T) {
    const double tc = std::fmin(std::fmax(static_cast<double>(T), 1e-4), 1.0);
    dn.value(fg::pair_densityf(T), -std::log10(tc) + 0.05);
  };
  for (int i = 0; i < N; ++i) {
    log1(static_cast<float>(std::exp2(uniform(-126.0, 128.0))));
    log1(static_cast<float>(uniform(0.5, 2.0)));
    exp1(static_cast<float>(uniform(-71.0, 71.0)));
    exp1(static_cast<float>(uniform(-1.0, 1.0)));
    sincos1(static_cast<float>(uniform(-8.5, 8.5)));
    quot1(std::exp2(uniform(-70.0, 70.0)) * (i & 1 ? 1 : -1), std::exp2(uniform(-70.0, 70.0)));
    quot1(uniform(-1.0, 1.0), uniform(0.05, 2.0));
    density1(static_cast<float>(uniform(0.0, 1.0)));
    density1(static_cast<float>(std::exp2(uniform(-14.0, 0.0))));
  }
  for (int u = -3000; u <= 3000; ++u) {
    log1(near_by(1.0f, u));
    log1(near_by(3.4028235e38f, u < 0 ? u : 0));
    exp1(near_by(70.0f, u));
    for (int k = 1; k <= 5; ++k) sincos1(near_by(static_cast<float>(k * 1.5707963267948966), u));
    sincos1(near_by(8.0f, u));
    sincos1(static_cast<float>(u) * 1e-9f);
    quot1(std::exp2(60.0) * (1.0 + u * 1e-9), 3.0);
    quot1(7.0, std::exp2(-60.0) * (1.0 + u * 1e-9));
    quot1(1.0 + u * 0x1p-23, 1.0);
    density1(near_by(1.0f, u));
    density1(near_by(1e-4f, u));
    density1(near_by(1.0001e-4f, u));
  }
  quot1(0.0, 2.0);
  quot1(1.0, INFINITY);
  density1(0.0f);
  std::printf("{");
  lg.print("log"), ex.print("exp"), sn.print("sin"), cs.print("cos"), qt.print("quotient"), dn.print("density", true);
}
""")
    for name, s in r.items():
        assert s["n"] > 1_000_000 and s["wrong"] == 0, (name, s)
    for name in ("log", "exp", "sin", "cos"):
        assert r[name]["log2"] < -40.0, (name, r[name])
        # The values within PAIR_ERR of one that rounds the other way: 2 * 2^-38 of 2^-24 on average.
        assert r[name]["unsettled"] < 3e-4 * r[name]["n"], (name, r[name])


def test_split64_rounds_as_the_conversion(run):
    """hi = v rounded to float (ties to even), lo = v - hi rounded, bit for bit, over all exponents."""
    r = run("split", PAIR + r"""
int main() {
  long n = 0, wrong = 0;
  auto one = [&](uint64_t b) {
    double v;
    std::memcpy(&v, &b, sizeof(v));
    float h, l;
    fg::split64(v, h, l);
    const float wh = static_cast<float>(v), wl = static_cast<float>(v - static_cast<double>(wh));
    ++n;
    if (fg::pair_bits(h) != fg::pair_bits(wh) || fg::pair_bits(l) != fg::pair_bits(wl)) ++wrong;
  };
  for (uint64_t e = 0; e < 2047; ++e)
    for (int i = 0; i < 300; ++i)
      for (uint64_t sign = 0; sign < 2; ++sign) {
        const uint64_t m = rng() & ((1ull << 52) - 1), top = m & ~((1ull << 29) - 1), at = sign << 63 | e << 52;
        one(at | m);
        one(at | top);
        one(at | top | 1ull << 28);         // ties
        one(at | top | ((1ull << 28) + 1));
        one(at | top | ((1ull << 28) - 1));
        one(at | ((1ull << 52) - 1 - (m & 0xff)));  // carries into the exponent
      }
  std::printf("{\"n\": %ld, \"wrong\": %ld}\n", n, wrong);
}
""")
    assert r["n"] == 2047 * 300 * 2 * 6 and r["wrong"] == 0
