"""The order, neighbour words and messages of the pipelined LU-SGS sweeps
(aero_pipe.cu, aero_topology.cpp), compiled here as plain C++: for boxes of
every shape and cut, each updated node has one position, every neighbour index
stays inside its plane (or message), and a sweep that follows the tables and
passes values across the cuts by message number gives the serial sweep's
values in both directions."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <vector>
using std::fabs; using std::fma; using std::max; using std::min; using std::sqrt;
struct double2 { double x, y; };
#define __host__
#define __device__
#define __global__
#define __forceinline__ inline
#define __noinline__
struct D3 { unsigned x = 0, y = 0; };
static D3 blockIdx, blockDim, threadIdx;
static double __longlong_as_double(long long v) { double d; std::memcpy(&d, &v, 8); return d; }
static long long __double_as_longlong(double d) { long long v; std::memcpy(&v, &d, 8); return v; }
#include "aero_topology.cpp"
#include "aero_pipe.cu"
using namespace aero;
#define REQUIRE(x) do { if (!(x)) { std::printf("failed: %s (%d x %d x %d, dir %d, ce %d)\n", #x, nx, ny, nz, dir, ce); return 1; } } while (0)

static int check(int nx, int ny, int nz, int dir, int want) {
  BlockView B{};
  B.b1 = Box{2, nx + 1, 2, ny + 1, 2, nz + 1};
  B.b = Box{1, nx + 2, 1, ny + 2, 1, nz + 2};
  B.nx = nx + 2; B.ny = ny + 2;
  PipeTables t = pipe_tables(B.b1, dir, want);
  const int ce = t.ce;
  const long N1 = B.b1.size();
  REQUIRE(ce <= kPipeSlabs);
  std::vector<int> nat(N1, -1), at(N1, -1);
  std::vector<double> rec((size_t)N1 * kPipeRec, 0.0), sa_rec((size_t)N1 * kPipeSaRec, 0.0);
  B.pipe = PipeView{t.dir, t.ce, t.slab.data(), t.plane.data(), at.data(), rec.data(), sa_rec.data()};
  blockDim.x = 1;
  for (long u = 0; u < N1; ++u) { blockIdx.x = (unsigned)u; k_pipe_index(&B); }
  // bijection: every node has a position of its own
  for (long u = 0; u < N1; ++u) {
    REQUIRE(at[u] >= 0 && at[u] < N1 && nat[at[u]] < 0);
    nat[at[u]] = (int)box_node(B, (int)u);
    REQUIRE(nat[at[u]] == B.at(2 + u % nx, 2 + u / nx % ny, 2 + u / nx / ny));
  }
  // serial sweeps of one scalar per node with three coefficients
  auto coef = [&](long n, int d) { return 0.1 + 0.01 * (double)((n * 7 + d * 13) % 17); };
  std::vector<double> x(N1), y(N1);
  const long st[3] = {1, nx, (long)nx * ny};
  for (long u = 0; u < N1; ++u) {
    const int o[3] = {(int)(u % nx), (int)(u / nx % ny), (int)(u / nx / ny)};
    double s = 1.0 + 0.001 * (double)(u % 101);
    for (int d = 0; d < 3; ++d) if (o[d] > 0) s += coef(u - st[d], d) * x[u - st[d]];
    x[u] = s;
  }
  for (long u = N1 - 1; u >= 0; --u) {
    const int o[3] = {(int)(u % nx), (int)(u / nx % ny), (int)(u / nx / ny)}, n1[3] = {nx, ny, nz};
    double s = x[u];
    for (int d = 0; d < 3; ++d) if (o[d] < n1[d] - 1) s -= 0.5 * coef(u + st[d], d) * y[u + st[d]];
    y[u] = s;
  }
  // the same by the tables; messages per receiving CTA: (number, index) -> value
  std::vector<std::map<std::pair<int, int>, double>> inbox(ce);
  std::vector<double> v(N1, 0.0);
  for (int pass = 0; pass < 2; ++pass) {
    const bool fwd = pass == 0;
    for (int k = 0; k < ce; ++k) {
      const int me = fwd ? k : ce - 1 - k;
      const SlabBox box = slab_box(B, me);
      const Cuts cut(box, dir, me, ce);
      const int H = box.n[0] + box.n[1] + box.n[2] - 2;
      REQUIRE(H == t.slab[me + 1] - t.slab[me] && H <= t.hmax);
      std::vector<double> prev, cur;
      int last_in = fwd ? -1 : cut.Mf - 1;
      for (int gs = 0; gs < H; ++gs) {
        const int h = fwd ? gs : H - 1 - gs;
        const PipePlane q = t.plane[t.slab[me] + h];
        REQUIRE(q.cnt >= 1 && q.cnt <= t.pmax && q.pos + q.cnt <= N1);
        cur.assign(3 * t.pmax, 0.0);
        const int m_in = cut.in(fwd, h);
        if (m_in >= 0) { REQUIRE(m_in == last_in + 1 && m_in < cut.Mall); last_in = m_in; REQUIRE(cut.count(m_in) <= t.lmax); }
        int reads = 0;
        for (int n = 0; n < q.cnt; ++n) {
          const unsigned long long w = (unsigned long long)__double_as_longlong(rec[(size_t)kPipeRec * (q.pos + n) + PW_NBR]);
          REQUIRE(std::memcmp(&rec[(size_t)kPipeRec * (q.pos + n) + PW_NBR], &sa_rec[(size_t)kPipeSaRec * (q.pos + n) + SW_NBR], 8) == 0);
          const long N = nat[q.pos + n];
          const long u = (N % B.nx - 1) + nx * ((N / B.nx % B.ny - 1) + (long)ny * (N / B.nx / B.ny - 1));
          const unsigned half = (unsigned)(fwd ? w : w >> 32), other = (unsigned)(fwd ? w >> 32 : w);
          const bool edge_in = (half & (fwd ? kLoBit : kHiBit)) != 0, edge_out = (half & (fwd ? kHiBit : kLoBit)) != 0;
          double s = fwd ? 1.0 + 0.001 * (double)(u % 101) : v[q.pos + n];
          for (int d = 0; d < 3; ++d) {
            const int i = nbr_index(half, d);
            if (i == kNoNbr) continue;
            if (edge_in && d == dir) {
              REQUIRE(m_in >= 0 && i < cut.count(m_in));
              auto it = inbox[me].find({m_in, i});
              REQUIRE(it != inbox[me].end());
              s += it->second;
              inbox[me].erase(it);
              ++reads;
            } else {
              REQUIRE(gs > 0 && i < (int)t.pmax);
              s += prev[d * t.pmax + i];
            }
          }
          v[q.pos + n] = s;
          for (int d = 0; d < 3; ++d) {
            const double out = fwd ? coef(u, d) * s : -0.5 * coef(u, d) * s;
            if (edge_out && d == dir) {
              const int to = fwd ? me + 1 : me - 1;
              const int i = nbr_index(other, d);
              const std::pair<int, int> key{cut.out(fwd, h, me), i};
              REQUIRE(to >= 0 && to < ce && i < t.lmax && !inbox[to].count(key));
              inbox[to][key] = out;
            } else cur[d * t.pmax + n] = out;
          }
        }
        REQUIRE(m_in < 0 || reads == cut.count(m_in));
        prev = cur;
      }
      REQUIRE(last_in == (fwd ? cut.Mf : cut.Mall) - 1 && inbox[me].empty());
    }
    for (int p = 0; p < N1; ++p) {
      const long N = nat[p];
      const long u = (N % B.nx - 1) + nx * ((N / B.nx % B.ny - 1) + (long)ny * (N / B.nx / B.ny - 1));
      const double want_v = fwd ? x[u] : y[u];
      REQUIRE(fabs(v[p] - want_v) <= 1e-12 * fabs(want_v));
    }
  }
  return 0;
}

int main() {
  const int boxes[][3] = {{1, 1, 1}, {3, 1, 1}, {1, 9, 2}, {31, 15, 3}, {129, 63, 1}, {25, 127, 31}, {2, 3, 40},
                          {17, 16, 15}, {7, 5, 7}, {95, 47, 3}, {5, 33, 8}};
  for (auto& n : boxes)
    for (int dir = 0; dir < 3; ++dir)
      for (int ce : {1, 2, 3, 4, 8, 16})
        if (check(n[0], n[1], n[2], dir, ce)) return 1;
  for (auto& n : boxes) {
    const int d = pipe_direction(Box{1, n[0], 1, n[1], 1, n[2]}, 8);
    if (d < 0 || d > 2) return 1;
  }
  std::puts("ok");
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_pipelined_order_and_messages(tmp_path):
    src = tmp_path / "order.cpp"
    src.write_text(SRC)
    exe = tmp_path / "order"
    csrc = os.path.join(ROOT, "aerocfd_b200", "csrc")
    subprocess.run(["g++", "-x", "c++", "-std=c++17", "-O2", "-ffp-contract=off", "-w", "-I" + csrc, str(src), "-o",
                    str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip().endswith("ok"), out.stdout


DIV = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
using std::fabs; using std::fma;
#define __host__
#define __device__
#define __forceinline__ inline
#define __noinline__
#include "aero_device.cuh"
int main() {
  std::mt19937_64 g(5);
  std::uniform_real_distribution<double> u(1.0, 2.0);
  long bad = 0;
  auto num = [&](int e) { return std::ldexp(u(g), e) * ((g() & 1) ? -1 : 1); };
  auto same = [&](double q, double t) { if (std::memcmp(&q, &t, 8) && !(std::isnan(q) && std::isnan(t)) && !(q == 0 && t == 0)) ++bad; };
  auto one = [&](double a, double b) { const double r = 1.0 / b; same(aero::div_pair(a, b, r, aero::recip_lo(b, r)), a / b); };
  auto two = [&](double a, double b, double c) {
    const double r = 1.0 / b, s = 1.0 / c;
    same(aero::div2_pair(a, b, r, aero::recip_lo(b, r), c, s, aero::recip_lo(c, s), aero::divisors_ok(b, c)), a / b / c);
  };
  for (int ea = -750; ea <= 750; ea += 11)
    for (int eb = -199; eb <= 199; eb += 9)
      for (int x = 0; x < 20; ++x) one(num(ea), std::ldexp(u(g), eb));
  for (long x = 0; x < 2000000; ++x) {  // quotients next to a rounding midpoint
    const double q = u(g), b = std::ldexp(u(g), (int)(g() % 60) - 30);
    double a = (double)((long double)(q + std::ldexp(1.0, -53)) * (long double)b);
    for (int k = (int)(g() % 3); k > 0; --k) a = std::nextafter(a, (g() & 1) ? INFINITY : -INFINITY);
    one(a, b);
  }
  one(0.0, 3.0);
  for (int ea = -1000; ea <= 1000; ea += 37)
    for (int e1 = -260; e1 <= 260; e1 += 20)
      for (int e2 = -260; e2 <= 260; e2 += 20) two(num(ea), num(e1), num(e2));
  for (int ea : {-501, -500, -499, 499, 500, 501})
    for (int e1 : {-201, -200, -199, 199, 200, 201}) two(num(ea), num(e1), num(-e1));
  for (long x = 0; x < 1000000; ++x) two(num((int)(g() % 80) - 40), num((int)(g() % 60) - 30), num((int)(g() % 60) - 30));
  two(0.0, 3.0, 5.0); two(-0.0, 3.0, -5.0); two(1.0, 0.0, 2.0); two(NAN, 2.0, 3.0); two(INFINITY, 2.0, 3.0);
  two(1.0, 1e-300, 1e-300); two(0.0, 0.0, 1.0);
  std::printf("bad=%ld\n", bad);
  return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_division_by_a_reciprocal_in_two_words(tmp_path):
    """div_pair and div2_pair equal IEEE division to the bit (zeros: in value)
    over the ranges their callers keep to, at their bounds and past them."""
    src = tmp_path / "div.cpp"
    src.write_text(DIV)
    exe = tmp_path / "div"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "aerocfd_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_division_by_a_rounded_reciprocal(tmp_path):
    """div_rn_lean equals IEEE division to the bit (zeros: in value) inside its
    operand range, at the range's bounds, outside it and for special values."""
    head, _ = DIV.split("int main() {")
    src = tmp_path / "lean.cpp"
    src.write_text(head + r"""
int main() {
  std::mt19937_64 g(7);
  std::uniform_real_distribution<double> u(1.0, 2.0);
  long bad = 0;
  auto num = [&](int e) { return std::ldexp(u(g), e) * ((g() & 1) ? -1 : 1); };
  auto one = [&](double a, double b) {
    const double q = aero::div_rn_lean(a, b, 1.0 / b), t = a / b;
    if (std::memcmp(&q, &t, 8) && !(std::isnan(q) && std::isnan(t)) && !(q == 0 && t == 0)) ++bad;
  };
  for (int ea = -1060; ea <= 1020; ea += 13)
    for (int eb = -1060; eb <= 1020; eb += 17)
      for (int x = 0; x < 20; ++x) one(num(ea), num(eb));
  const int edge[] = {-481, -480, -479, 479, 480, 481};
  for (int ea : edge)
    for (int eb : edge) {
      for (int x = 0; x < 50; ++x) one(num(ea), num(eb));
      one(std::ldexp(1.0, ea), std::ldexp(-1.0, eb));
    }
  for (long x = 0; x < 2000000; ++x) {  // quotients next to a rounding midpoint
    const double q = u(g), b = num((int)(g() % 60) - 30);
    double a = (double)((long double)(q + std::ldexp(1.0, -53)) * (long double)b);
    for (int k = (int)(g() % 3); k > 0; --k) a = std::nextafter(a, (g() & 1) ? INFINITY : -INFINITY);
    one(a, b);
  }
  for (double b : {3.0, -3.0, 0.0, -0.0, 1e-300, 1e300, (double)INFINITY, (double)NAN})
    for (double a : {0.0, -0.0, 1.0, 1e-310, 1e308, (double)INFINITY, (double)-INFINITY, (double)NAN}) one(a, b);
  std::printf("bad=%ld\n", bad);
  return bad != 0;
}
""")
    exe = tmp_path / "lean"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "aerocfd_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
