// 2nd-order Crank-Nicolson dual-time advance (crank2nd,
// sub_timeadvancement_2ndcrank.f90:1-466, 3-D) and update_q0 (main.f90:692-711).
//
// crank2nd is an approximately factorised point-implicit update: a forward
// and a backward recurrence along every i line, then every j line, then every
// k line of the updated box.  Lines of one direction are independent, so each
// is one thread walking its line; the per-point arithmetic is the
// reference's.  dq lives in the first five planes of the FVH scratch field
// (natural order, zero outside the updated box).  q0 holds the two earlier
// time levels: component plane (l+1) + 2*(c-1) is q0(l, c), l = -1, 0.
#include <cmath>
#include <type_traits>

#include "aero_device.cuh"
#include "aero_kernels.h"

namespace aero {

namespace {

constexpr double kAlph = 0.5;

__device__ __forceinline__ double& q0v(const BlockView& B, int l, int c, long n) {
  return B.v(F_Q0, 1 + (l + 1) + 2 * (c - 1), n);
}
__device__ __forceinline__ double& dqv(const BlockView& B, int c, long n) {
  return B.f[F_FVH][(long)(c - 1) * B.plane + n];
}

// rou = |U| + c|grad| along the direction whose metric row starts at cb (:92-106)
__device__ __forceinline__ double crank_rou(const BlockView& B, int cb, long n) {
  double u = B.v(F_PRI, 2, n), v = B.v(F_PRI, 3, n), w = B.v(F_PRI, 4, n), c = B.v(F_PRI, 7, n);
  double x0 = B.v(F_DXIDX, cb, n), y0 = B.v(F_DXIDX, cb + 1, n), z0 = B.v(F_DXIDX, cb + 2, n);
  double temp = p2(x0) + p2(y0) + p2(z0);
  temp = sqrt(temp);
  double cu = u * x0 + v * y0 + w * z0;
  return fabs(cu) + fabs(c * temp);
}

// The neighbour term of one recurrence step (:107-161): the flux-Jacobian
// product of neighbour nb with its dq, with +rou (forward) or -rou (backward).
__device__ __forceinline__ void crank_a(const BlockView& B, int cb, long nb, double r, double hdv, double gamma,
                                        bool fwd, double a[5]) {
  double u = B.v(F_PRI, 2, nb), v = B.v(F_PRI, 3, nb), w = B.v(F_PRI, 4, nb), c = B.v(F_PRI, 7, nb);
  double dxidx0 = B.v(F_DXIDX, cb, nb), dxidy0 = B.v(F_DXIDX, cb + 1, nb), dxidz0 = B.v(F_DXIDX, cb + 2, nb);
  double q2 = 0.5 * (p2(u) + p2(v) + p2(w));
  double h = p2(c) / (gamma - 1.0) + q2;
  double cu = dxidx0 * u + dxidy0 * v + dxidz0 * w;
  double s1 = dqv(B, 1, nb), s2 = dqv(B, 2, nb), s3 = dqv(B, 3, nb), s4 = dqv(B, 4, nb), s5 = dqv(B, 5, nb);
  double b1 = hdv * (-(cu * s1) + dxidx0 * s2 + dxidy0 * s3 + dxidz0 * s4);
  double b2 = hdv * (q2 * s1 - u * s2 - v * s3 - w * s4 + s5) * (gamma - 1.0);
  double b3 = fwd ? hdv * (cu + r) : hdv * (cu - r);
  a[0] = b1 + b3 * s1;
  a[1] = b1 * u + b2 * dxidx0 + b3 * s2;
  a[2] = b1 * v + b2 * dxidy0 + b3 * s3;
  a[3] = b1 * w + b2 * dxidz0 + b3 * s4;
  a[4] = b1 * h + b2 * cu + b3 * s5;
}

}  // namespace

// :62-87: rhs = rhsi + rhsv, then the dual-time form with alph = 1/2, on the
// updated nodes.
__global__ void k_crank_rhs(const BlockView* __restrict__ blocks) {
  const BlockView& B = blocks[blockIdx.y];
  if (B.retired()) return;
  const Box& b1 = B.b1;
  long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= b1.size()) return;
  int i = b1.is + (int)(t % b1.nx());
  long r = t / b1.nx();
  int j = b1.js + (int)(r % b1.ny());
  int k = b1.ks + (int)(r / b1.ny());
  long n = B.at(i, j, k);
  const double alph_i = 1.0 / (1.0 + kAlph);
  double dt = B.s(F_DT, n), ij = B.s(F_INVJ, n);
#pragma unroll
  for (int c = 1; c <= 5; ++c) {
    double rhs = B.v(F_RHSI, c, n) + B.v(F_RHSV, c, n);
    B.v(F_RHS, c, n) = alph_i * (rhs * dt - ((1.0 + kAlph) * B.v(F_Q, c, n) - (1.0 + 2.0 * kAlph) * q0v(B, 0, c, n) +
                                             kAlph * q0v(B, -1, c, n)) * ij);
  }
}

// One direction's recurrences with the lines in shared memory: a CTA takes
// `lpc` lines of direction d (0: i, 1: j, 2: k).  All its threads form what the
// recurrences read of every node (the neighbour term's factors, the radius,
// the pivot), one warp then walks the lines, a lane per line, and all threads
// store the result.  Walking the lines through global memory, as
// k_crank_sweep does, takes a memory latency per node; from shared memory a node
// costs its chain of about ten dependent FP64 operations (97 x 49 x 5 channel: i
// lines 555 -> 56 us, j lines 200 -> 31, k lines 15 -> 13).  The i lines form
// the dual-time rhs on the way (:62-87), the last direction adds dq/inv_j to q
// (:455-462).  The forward recurrence of the k lines starts at ks1+1 and the
// backward one at ke1-1 (:352, :398), as in the reference; along i and j they
// cover the whole line.  A neighbour outside the updated box has dq = 0.
namespace {
enum LineWord { LW_CU = 0, LW_X, LW_Y, LW_Z, LW_Q2, LW_U, LW_V, LW_W, LW_H, LW_R, LW_HDV, LW_DIV, LW_DQ, LW_NUM = LW_DQ + 5 };
}
__global__ void __launch_bounds__(256) k_crank_lines(const BlockView* __restrict__ blocks, int d, int lpc, double gamma,
                                                     int last) {
  extern __shared__ double sm[];
  const BlockView& B = blocks[blockIdx.y];
  if (B.retired()) return;
  const Box& b1 = B.b1;
  const int n1[3] = {b1.nx(), b1.ny(), b1.nz()};
  const int lo[3] = {b1.is, b1.js, b1.ks};
  const int u1 = d == 0 ? 1 : 0, u2 = d == 2 ? 1 : 2;  // the two other directions
  const int len = n1[d], lines = n1[u1] * n1[u2];
  const int line0 = blockIdx.x * lpc;
  if (line0 >= lines) return;
  const int nl = min(lpc, lines - line0);
  const int cb = 3 * d + 1;
  const double inv1 = 1.0 + kAlph;
  // word w of node x (-1 .. len) of line l; the row stride is odd, so threads on
  // neighbouring nodes of one line write different banks
  const int row = LW_NUM * lpc + 1 - (LW_NUM * lpc & 1);
  auto at = [&](int x, int w, int l) -> double& { return sm[(x + 1) * row + w * lpc + l]; };
  auto node = [&](int l, int x) {
    int ijk[3];
    ijk[u1] = lo[u1] + (line0 + l) % n1[u1];
    ijk[u2] = lo[u2] + (line0 + l) / n1[u1];
    ijk[d] = lo[d] + x;
    return B.at(ijk[0], ijk[1], ijk[2]);
  };
  // threads run along the lines for i, across them (along i) otherwise
  for (int t = threadIdx.x; t < (len + 2) * nl; t += blockDim.x) {
    const int l = d == 0 ? t / (len + 2) : t % nl, x = (d == 0 ? t % (len + 2) : t / nl) - 1;
    const long n = node(l, x);
    const double u = B.v(F_PRI, 2, n), v = B.v(F_PRI, 3, n), w = B.v(F_PRI, 4, n), c = B.v(F_PRI, 7, n);
    const double x0 = B.v(F_DXIDX, cb, n), y0 = B.v(F_DXIDX, cb + 1, n), z0 = B.v(F_DXIDX, cb + 2, n);
    const double q2 = 0.5 * (p2(u) + p2(v) + p2(w));
    const double r = crank_rou(B, cb, n);
    at(x, LW_CU, l) = x0 * u + y0 * v + z0 * w;
    at(x, LW_X, l) = x0;
    at(x, LW_Y, l) = y0;
    at(x, LW_Z, l) = z0;
    at(x, LW_Q2, l) = q2;
    at(x, LW_U, l) = u;
    at(x, LW_V, l) = v;
    at(x, LW_W, l) = w;
    at(x, LW_H, l) = p2(c) / (gamma - 1.0) + q2;
    at(x, LW_R, l) = r;
    const bool inside = x >= 0 && x < len;
    const double dt = inside ? B.s(F_DT, n) : 0.0;
    const double dtsub = dt / inv1;
    at(x, LW_HDV, l) = 0.5 * dtsub;
    at(x, LW_DIV, l) = 1.0 / (1.0 + dtsub * r);
    const double alph_i = 1.0 / (1.0 + kAlph), ij = d == 0 && inside ? B.s(F_INVJ, n) : 0.0;
#pragma unroll
    for (int k = 1; k <= 5; ++k) {
      double base = 0.0;
      if (inside && d == 0) {
        const double rhs = B.v(F_RHSI, k, n) + B.v(F_RHSV, k, n);
        base = alph_i * (rhs * dt - ((1.0 + kAlph) * B.v(F_Q, k, n) - (1.0 + 2.0 * kAlph) * q0v(B, 0, k, n) +
                                     kAlph * q0v(B, -1, k, n)) * ij);
        B.v(F_RHS, k, n) = base;
      } else if (inside) {
        base = dqv(B, k, n);
      }
      at(x, LW_DQ + k - 1, l) = base;
    }
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const int l = min((int)threadIdx.x, nl - 1);  // further lanes repeat the last line
    auto walk = [&](auto forward, int from, int to, int by) {
      constexpr bool F = decltype(forward)::value;
      if (F ? from >= to : from <= to) return;
      // the neighbour's dq, and its factors one node ahead of their use
      double s[5], f[10], hdv, div, base[5];
#pragma unroll
      for (int k = 0; k < 5; ++k) s[k] = at(from - by, LW_DQ + k, l);
      auto fetch = [&](int x) {
#pragma unroll
        for (int k = 0; k < 10; ++k) f[k] = at(x - by, k, l);
        hdv = at(x, LW_HDV, l);
        div = at(x, LW_DIV, l);
#pragma unroll
        for (int k = 0; k < 5; ++k) base[k] = at(x, LW_DQ + k, l);
      };
      fetch(from);
      for (int x = from; x != to; x += by) {
        const double b1 = hdv * (-(f[LW_CU] * s[0]) + f[LW_X] * s[1] + f[LW_Y] * s[2] + f[LW_Z] * s[3]);
        const double b2 = hdv * (f[LW_Q2] * s[0] - f[LW_U] * s[1] - f[LW_V] * s[2] - f[LW_W] * s[3] + s[4]) * (gamma - 1.0);
        const double b3 = F ? hdv * (f[LW_CU] + f[LW_R]) : hdv * (f[LW_CU] - f[LW_R]);
        double a[5];
        a[0] = b1 + b3 * s[0];
        a[1] = b1 * f[LW_U] + b2 * f[LW_X] + b3 * s[1];
        a[2] = b1 * f[LW_V] + b2 * f[LW_Y] + b3 * s[2];
        a[3] = b1 * f[LW_W] + b2 * f[LW_Z] + b3 * s[3];
        a[4] = b1 * f[LW_H] + b2 * f[LW_CU] + b3 * s[4];
#pragma unroll
        for (int k = 0; k < 5; ++k) s[k] = F ? div * (base[k] + a[k]) : base[k] - div * a[k];
        if (x + by != to) fetch(x + by);
        if ((int)threadIdx.x < nl) {
#pragma unroll
          for (int k = 0; k < 5; ++k) at(x, LW_DQ + k, l) = s[k];
        }
      }
    };
    const int end = d == 2 ? 1 : 0;
    walk(std::true_type{}, end, len, 1);
    __syncwarp();
    walk(std::false_type{}, len - 1 - end, -1, -1);
  }
  __syncthreads();
  for (int t = threadIdx.x; t < len * nl; t += blockDim.x) {
    const int l = d == 0 ? t / len : t % nl, x = d == 0 ? t % len : t / nl;
    const long n = node(l, x);
    const double ij = last ? B.s(F_INVJ, n) : 1.0;
#pragma unroll
    for (int k = 1; k <= 5; ++k) {
      const double dq = at(x, LW_DQ + k - 1, l);
      if (last)
        B.v(F_Q, k, n) = B.v(F_Q, k, n) + dq / ij;
      else
        dqv(B, k, n) = dq;
    }
  }
}
// Dynamic shared memory of k_crank_lines for lines of `len` nodes.
size_t crank_lines_smem(int len, int lpc) {
  return (size_t)(len + 2) * (LW_NUM * lpc + 1 - (LW_NUM * lpc & 1)) * sizeof(double);
}

// The same through global memory, for lines that do not fit shared memory:
// thread = one line of the updated box along
// direction d (0: i, 1: j, 2: k).  The forward recurrence of the k lines
// starts at ks1+1 and the backward one at ke1-1 (:352, :398), as in the
// reference; along i and j they cover the whole line.
__global__ void k_crank_sweep(const BlockView* __restrict__ blocks, int d, double gamma) {
  const BlockView& B = blocks[blockIdx.y];
  if (B.retired()) return;
  const Box& b1 = B.b1;
  const int n1[3] = {b1.nx(), b1.ny(), b1.nz()};
  const int lo[3] = {b1.is, b1.js, b1.ks};
  const int u1 = d == 0 ? 1 : 0, u2 = d == 2 ? 1 : 2;  // the two other directions
  long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long)n1[u1] * n1[u2]) return;
  int ijk[3];
  ijk[u1] = lo[u1] + (int)(t % n1[u1]);
  ijk[u2] = lo[u2] + (int)(t / n1[u1]);
  ijk[d] = lo[d];
  const long st = d == 0 ? 1 : (d == 1 ? (long)B.nx : (long)B.nx * B.ny);
  const long n0 = B.at(ijk[0], ijk[1], ijk[2]);  // first updated node of the line
  const int len = n1[d];
  const int cb = 3 * d + 1;
  const double inv1 = 1.0 + kAlph;
  double a[5];
  // forward
  int f0 = d == 2 ? 1 : 0;
  double rprev = crank_rou(B, cb, n0 + (f0 - 1) * st);
  for (int x = f0; x < len; ++x) {
    long n = n0 + x * st, nb = n - st;
    double r = crank_rou(B, cb, n);
    double dtsub = B.s(F_DT, n) / inv1;
    crank_a(B, cb, nb, rprev, 0.5 * dtsub, gamma, true, a);
    double div = 1.0 / (1.0 + dtsub * r);
#pragma unroll
    for (int c = 1; c <= 5; ++c) {
      double base = d == 0 ? B.v(F_RHS, c, n) : dqv(B, c, n);
      dqv(B, c, n) = div * (base + a[c - 1]);
    }
    rprev = r;
  }
  // backward
  int b0 = d == 2 ? len - 2 : len - 1;
  if (b0 < 0) return;
  rprev = crank_rou(B, cb, n0 + (b0 + 1) * st);
  for (int x = b0; x >= 0; --x) {
    long n = n0 + x * st, nb = n + st;
    double r = crank_rou(B, cb, n);
    double dtsub = B.s(F_DT, n) / inv1;
    crank_a(B, cb, nb, rprev, 0.5 * dtsub, gamma, false, a);
    double div = 1.0 / (1.0 + dtsub * r);
#pragma unroll
    for (int c = 1; c <= 5; ++c) dqv(B, c, n) = dqv(B, c, n) - div * a[c - 1];
    rprev = r;
  }
}

// :455-462: q += dq / inv_j on the updated nodes.
__global__ void k_crank_update(const BlockView* __restrict__ blocks) {
  const BlockView& B = blocks[blockIdx.y];
  if (B.retired()) return;
  const Box& b1 = B.b1;
  long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= b1.size()) return;
  int i = b1.is + (int)(t % b1.nx());
  long r = t / b1.nx();
  int j = b1.js + (int)(r % b1.ny());
  int k = b1.ks + (int)(r / b1.ny());
  long n = B.at(i, j, k);
  double ij = B.s(F_INVJ, n);
#pragma unroll
  for (int c = 1; c <= 5; ++c) B.v(F_Q, c, n) = B.v(F_Q, c, n) + dqv(B, c, n) / ij;
}

// main.f90:692-711 on the physical nodes.
__global__ void k_update_q0(const BlockView* __restrict__ blocks) {
  const BlockView& B = blocks[blockIdx.y];
  if (B.retired()) return;
  const Box& b0 = B.b0;
  long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= b0.size()) return;
  int i = b0.is + (int)(t % b0.nx());
  long r = t / b0.nx();
  int j = b0.js + (int)(r % b0.ny());
  int k = b0.ks + (int)(r / b0.ny());
  long n = B.at(i, j, k);
#pragma unroll
  for (int c = 1; c <= 5; ++c) {
    q0v(B, -1, c, n) = q0v(B, 0, c, n);
    q0v(B, 0, c, n) = B.v(F_Q, c, n);
  }
}

}  // namespace aero
