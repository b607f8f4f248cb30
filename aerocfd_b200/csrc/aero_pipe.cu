// The LU-SGS update (sub_timeadvancement_1stimplicit.f90 and
// sub_timeadvancement_jac.f90) as a pipeline of slabs that forms its blocks on
// the way.
//
// The forward sweep's node (i,j,k) depends on its three lower neighbours, so
// the nodes of one hyperplane run together (the backward sweep likewise from
// the other corner).  A block's updated box is cut into slabs along one
// direction, one CTA of a thread-block cluster per slab.  Inside a slab the CTA
// walks the slab's own hyperplanes; the only values it needs from outside are
// what the last layer of the slab before it passes on, so the CTAs run one
// behind the other and no plane ends with an exchange over the whole cluster.
//
// A node passes on three products, its off-diagonal block of each direction
// S = 0.5*(A +- r*I)*inv_j times its own dq.  S needs only the node's own q,
// metrics, radius and inv_j (25 words, kPipeRec, in place of the 150 that both
// passes' blocks take), so it is formed in registers right where it is used:
// thread (node, direction) computes its 25 entries ahead of the plane's turn.
// With the blocks read from memory instead, one plane step moved 76 words per
// node through shared memory twice and through HBM once, which bounded it.
// What bounds it now is the FP64 rate, about 780 operations per node and pass,
// or, for small planes, the step from plane to plane.  Its chain of dependent
// operations (two divisions, two products, a barrier) adds up to about 340
// cycles; measured are 576 a step for aerofoil blocks of 129 x 65 x 3 on 8 CTAs
// (112 us over 382 steps at 1965 MHz, the start behind the cuts included), 670 for a
// channel of 97 x 49 x 5 on 16 and 870 for one of 33 x 17 x 5 on 8 (both with about 8
// us of launch): the rest is the other groups' block formation, which shares
// the chain's FP64 pipe, and the hand-over between the groups.
//
// The arithmetic per node is the reference's, operation by operation (calc_jm,
// the products summed column by column, the three directions added in their
// order, the two divisions), so the result is the serial sweep's to the bit.
#include <cmath>
#include <type_traits>

#include "aero_device.cuh"
#include "aero_kernels.h"

namespace aero {

namespace {

// Updated-box dimensions of one slab and the offset of its first layer.
struct SlabBox {
  int n[3];
  int c0, c1;
};
__device__ __forceinline__ SlabBox slab_box(const BlockView& B, int r) {
  SlabBox s;
  s.n[0] = B.b1.nx();
  s.n[1] = B.b1.ny();
  s.n[2] = B.b1.nz();
  const int X = B.pipe.dir, nX = X == 0 ? s.n[0] : X == 1 ? s.n[1] : s.n[2];
  s.c0 = (int)((long)r * nX / B.pipe.ce);
  s.c1 = (int)((long)(r + 1) * nX / B.pipe.ce);
  if (X == 0) s.n[0] = s.c1 - s.c0;
  if (X == 1) s.n[1] = s.c1 - s.c0;
  if (X == 2) s.n[2] = s.c1 - s.c0;
  return s;
}
// Index of offsets (a, b, c) in its hyperplane of an n[0] x n[1] x n[2] box.
__device__ int index_in_plane(const int n[3], int a, int b, int c) {
  const int h = a + b + c;
  int idx = 0;
  for (int cc = max(0, h - (n[0] - 1) - (n[1] - 1)); cc < c; ++cc) {
    const int bmin = max(0, h - cc - (n[0] - 1)), bmax = min(n[1] - 1, h - cc);
    if (bmax >= bmin) idx += bmax - bmin + 1;
  }
  return idx + b - max(0, h - c - (n[0] - 1));
}
// Layer nodes (u, v) of a slab's first or last layer, u + v = s: how many, and
// the index of v among them.
__device__ __forceinline__ int layer_count(int s, int nu, int nv) {
  return min(s, nu - 1) - max(0, s - (nv - 1)) + 1;
}
__device__ __forceinline__ int layer_index(int s, int v, int nu) { return v - max(0, s - (nu - 1)); }

// Messages across the cuts of one CTA's slab (see pipe_body): numbers by plane.
struct Cuts {
  int nu, nv, thick, M, Mf, Mall;
  bool has_lo, has_hi;
  __device__ Cuts(const SlabBox& s, int X, int me, int ce) {
    nu = X == 0 ? s.n[1] : s.n[0];
    nv = X == 2 ? s.n[1] : s.n[2];
    thick = s.c1 - s.c0;
    has_lo = me > 0 && me < ce;
    has_hi = me + 1 < ce;
    M = nu + nv - 1;           // messages per pass across a cut
    Mf = has_lo ? M : 0;       // messages received in the forward pass
    Mall = Mf + (has_hi ? M : 0);
  }
  // values of message m
  __device__ int count(int m) const { return layer_count(m < Mf ? m : M - 1 - (m - Mf), nu, nv); }
  // the message the edge nodes of local plane h read (-1: it has none of them)
  __device__ int in(bool fwd, int h) const {
    const int s = fwd ? h : h - (thick - 1);
    if (!(fwd ? has_lo : has_hi) || s < 0 || s >= M) return -1;
    return fwd ? s : Mf + M - 1 - s;
  }
  // the same without the check (for planes with such nodes)
  __device__ int in_number(bool fwd, int h) const { return fwd ? h : Mf + M - 1 - (h - (thick - 1)); }
  // the message, numbered as its receiver counts, that local plane h of CTA
  // `me` sends (for planes with nodes in the layer that sends)
  __device__ int out(bool fwd, int h, int me) const {
    const int s = fwd ? h - (thick - 1) : h;
    return fwd ? s : (me > 1 ? M : 0) + M - 1 - s;
  }
};

// Natural (box) index of the u-th updated node.
__device__ __forceinline__ long box_node(const BlockView& B, int u) {
  const int nx = B.b1.nx(), ny = B.b1.ny();
  const int r = u / nx, i = u - r * nx, k = r / ny, j = r - k * ny;
  return B.at(B.b1.is + i, B.b1.js + j, B.b1.ks + k);
}

// The neighbour word: its low half holds the 10-bit indices of i-1, j-1, k-1 (what
// the forward pass reads), its high half those of i+1, j+1, k+1, each the
// neighbour's index in its plane, or for the neighbour across a cut its index in
// that layer (an inbox index); kNoNbr outside the updated box.  Bits 30 / 31 of
// both halves: the node is in the slab's first / last layer and a slab lies
// beyond it.
constexpr int kNoNbr = 1023;
constexpr unsigned kLoBit = 1u << 30, kHiBit = 1u << 31;
__device__ __forceinline__ int nbr_index(unsigned half, int e) { return (int)(half >> (10 * e)) & 1023; }

}  // namespace

// The order's tables and the neighbour words of every updated node, once per
// case (and set of slabs).
__global__ void k_pipe_index(const BlockView* __restrict__ blocks) {
  const BlockView& B = blocks[blockIdx.y];
  const Box& b1 = B.b1;
  const long u = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= b1.size()) return;
  const int nx1 = b1.nx(), ny1 = b1.ny(), nz1 = b1.nz();
  const int o[3] = {(int)(u % nx1), (int)(u / nx1 % ny1), (int)(u / nx1 / ny1)};
  const int lim[3] = {nx1, ny1, nz1};
  const PipeView& P = B.pipe;
  const int X = P.dir;
  const int r = (int)((((long)o[X] + 1) * P.ce - 1) / lim[X]);
  const SlabBox s = slab_box(B, r);
  int l[3] = {o[0], o[1], o[2]};
  l[X] -= s.c0;
  const int entry = P.slab[r] + l[0] + l[1] + l[2];
  const PipePlane pl = P.plane[entry];
  const int pos = pl.pos + index_in_plane(s.n, l[0], l[1], l[2]);
  P.at[u] = pos;
  // the two directions of a layer, and the node's index in its layer
  const int U = X == 0 ? 1 : 0, V = X == 2 ? 1 : 2;
  const int in_layer = layer_index(l[U] + l[V], l[V], s.n[U]);
  unsigned wl = 0, wh = 0, flags = 0;
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    int lo[3] = {l[0], l[1], l[2]}, hi[3] = {l[0], l[1], l[2]};
    lo[e] -= 1;
    hi[e] += 1;
    int fl = kNoNbr, fh = kNoNbr;
    if (l[e] > 0)
      fl = index_in_plane(s.n, lo[0], lo[1], lo[2]);
    else if (e == X && r > 0) {
      fl = in_layer;
      flags |= kLoBit;
    }
    if (l[e] < s.n[e] - 1)
      fh = index_in_plane(s.n, hi[0], hi[1], hi[2]);
    else if (e == X && r + 1 < P.ce) {
      fh = in_layer;
      flags |= kHiBit;
    }
    wl |= (unsigned)fl << (10 * e);
    wh |= (unsigned)fh << (10 * e);
  }
  const double word = __longlong_as_double((long long)((unsigned long long)(wh | flags) << 32 | (wl | flags)));
  if (P.rec) P.rec[(long)kPipeRec * pos + PW_NBR] = word;  // (a view holds the records of its own sweeps only)
  if (P.sa_rec) P.sa_rec[(long)kPipeSaRec * pos + SW_NBR] = word;
}

#ifdef __CUDACC__  // (the order's tables above also build as host code, for their test)
// A warp's 32 records from shared memory to their places, CHUNKS 16-byte chunks
// from word `word` on, chunk c of lane r's record at sm[r * CHUNKS + c]; p is the
// lane's position, or -1.  Consecutive lanes store consecutive chunks, so a store
// covers whole runs of records instead of 16 bytes in each of 32 (which the L2
// counted as 17.4 million sectors on the plate, 2.5 times the bytes).  A chunk
// `half` keeps its upper word.
template <int CHUNKS>
__device__ __forceinline__ void store_records(const double2* sm, double* base, int words, int word, int p, int half) {
  __syncwarp();
  const int lane = (int)(threadIdx.x & 31);
#pragma unroll
  for (int x = lane; x < 32 * CHUNKS; x += 32) {
    const int r = x / CHUNKS, c = x - r * CHUNKS;
    const int pr = __shfl_sync(0xffffffffu, p, r);
    if (pr < 0) continue;
    double* to = base + (long)words * pr + word + 2 * c;
    if (c == half)
      to[0] = sm[x].x;
    else
      *reinterpret_cast<double2*>(to) = sm[x];
  }
}

// Per updated node what its blocks are made of: the
// spectral radii (sub_timeadvancement_1stimplicit.f90:108-156) and calc_jm's
// common terms (sub_timeadvancement_jac.f90:17-62).  It reads q, the primitives
// and the metrics only, so it runs beside the flux and time-step kernels.  The
// nodes are taken in box order: the loads run along the rows of the box, and a
// warp writes its records one after another (store_records), wherever they lie.
// Plate (0.72 million nodes): 95 us for 320 MB, 138 with each thread storing its
// own record.
__global__ void k_pipe_recs(const BlockView* __restrict__ blocks, CaseConsts cc_launch) {
  const BlockView& B = blocks[blockIdx.y];
  if (B.retired()) return;
  const CaseConsts& cc = B.ccb ? *B.ccb : cc_launch;
  const int u = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (u - (int)threadIdx.x >= B.b1.size()) return;  // the whole CTA
  constexpr int CH = PW_NBR / 2;
  __shared__ double2 sm[128 * CH];
  const bool act = u < B.b1.size();
  const long n = box_node(B, act ? u : 0);
  const int p = act ? B.pipe.at[u] : -1;
  double2* rec = sm + threadIdx.x * CH;
  double k[9];
#pragma unroll
  for (int x = 0; x < 9; ++x) k[x] = B.v(F_DXIDX, x + 1, n);
  const double rho = B.v(F_Q, 1, n), mu = B.v(F_Q, 2, n), mv = B.v(F_Q, 3, n), mw = B.v(F_Q, 4, n);
  const double e0 = B.v(F_Q, 5, n), gamma = cc.gamma, a2 = gamma - 1.0;
  const double rrho = 1.0 / rho, hj = 0.5 * B.s(F_INVJ, n);
  const double phi = 0.5 * a2 * (p2(mu) + p2(mv) + p2(mw)) / p2(rho);
  const double a1 = div_rn_lean(gamma * e0, rho, rrho) - phi;
  // Every quotient of calc_jm is a product of two or three of these over rho.
  // With rho in (2^-200, 2^200) and each factor zero or in (2^-250, 2^250),
  // div_pair's conditions hold for all of them; any other node is marked (a NaN
  // in place of 1/rho) and takes the IEEE divisions.
  bool fast = rho > 0x1p-200 && rho < 0x1p200;
  auto in = [](double x) { return x == 0.0 || (fabs(x) > 0x1p-250 && fabs(x) < 0x1p250); };
  fast = fast && in(mu) && in(mv) && in(mw);
  const double vx = B.v(F_PRI, 2, n), vy = B.v(F_PRI, 3, n), vz = B.v(F_PRI, 4, n), c = B.v(F_PRI, 7, n);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double x = k[3 * d], y = k[3 * d + 1], z = k[3 * d + 2];
    const double temp = sqrt(p2(x) + p2(y) + p2(z));
    const double cu = x * vx + y * vy + z * vz, rad = fabs(cu) + fabs(c * temp);
    const double uu = div_rn_lean(x * mu + y * mv + z * mw, rho, rrho);
    fast = fast && in(x) && in(y) && in(z) && in(uu);
    rec[PW_DIR / 2 + 3 * d] = double2{uu, x};
    rec[PW_DIR / 2 + 3 * d + 1] = double2{y, z};
    rec[PW_DIR / 2 + 3 * d + 2] = double2{rad, hj};
    if (act) B.s(F_RA + d, n) = rad;
  }
  rec[PW_M / 2] = double2{mu, mv};
  rec[PW_M / 2 + 1] = double2{mw, rho};
  rec[PW_RCP / 2] = double2{fast ? rrho : __longlong_as_double(0x7ff8000000000000ll), recip_lo(rho, rrho)};
  rec[PW_PHI / 2] = double2{phi, a1};
  store_records<CH>(sm + (threadIdx.x & ~31u) * CH, B.pipe.rec, kPipeRec, 0, p, -1);
}

// rhs = rhsi + rhsv and the diagonal phi/dt + ra + rb + rc of every updated
// node (sub_timeadvancement_1stimplicit.f90:72-156; 2-D: no zeta radius), rhs in
// its place of the box too (the residual norm reads it there).  Plate: 73 us, 89
// with each thread storing its own record.
__global__ void k_pipe_sca(const BlockView* __restrict__ blocks, CaseConsts cc_launch) {
  const BlockView& B = blocks[blockIdx.y];
  if (B.retired()) return;
  const CaseConsts& cc = B.ccb ? *B.ccb : cc_launch;
  const int u = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (u - (int)threadIdx.x >= B.b1.size()) return;  // the whole CTA
  constexpr int CH = (PW_OK + 1 - PW_DIV) / 2;
  __shared__ double2 sm[128 * CH];
  const bool act = u < B.b1.size();
  const long n = box_node(B, act ? u : 0);
  const int p = act ? B.pipe.at[u] : -1;
  double2* rec = sm + threadIdx.x * CH;
  // every load before the first store and division, so that all are in flight at once
  const double dt = B.s(F_DT, n), ra = B.s(F_RA, n), rb = B.s(F_RB, n), rc = B.s(F_RC, n), invj = B.s(F_INVJ, n);
  double ri5[5], r[5];
#pragma unroll
  for (int c = 0; c < 5; ++c) {
    ri5[c] = B.v(F_RHSI, c + 1, n);
    r[c] = B.v(F_RHSV, c + 1, n);
  }
#pragma unroll
  for (int c = 0; c < 5; ++c) {
    r[c] = ri5[c] + r[c];
    if (act) B.v(F_RHS, c + 1, n) = r[c];
  }
  const double phi = cc.cfl >= 1.0e3 ? 0.0 : 1.0;
  double diag = phi * 1.0 / dt + ra + rb;
  if (!B.planar()) diag = diag + rc;
  const double rd = 1.0 / diag, ri = 1.0 / invj;
  rec[0] = double2{diag, invj};
  rec[1] = double2{rd, ri};
  rec[2] = double2{recip_lo(diag, rd), recip_lo(invj, ri)};
  rec[3] = double2{r[0], r[1]};
  rec[4] = double2{r[2], r[3]};
  rec[5] = double2{r[4], divisors_ok(diag, invj) ? 1.0 : 0.0};
  store_records<CH>(sm + (threadIdx.x & ~31u) * CH, B.pipe.rec, kPipeRec, PW_DIV, p, -1);
}

// The SA sweeps' records (sub_tur_sa.f90:676-750, :762-778): the upwind
// coefficients 0.5*(U + |U|) and 0.5*(U - |U|) per direction, sa_rhs and the
// diagonal.  Plate: 57 us, 78 with each thread storing its own record.
__global__ void k_pipe_sa_recs(const BlockView* __restrict__ blocks, CaseConsts cc_launch) {
  const BlockView& B = blocks[blockIdx.y];
  if (B.retired()) return;
  const CaseConsts& cc = B.ccb ? *B.ccb : cc_launch;
  const int u0 = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (u0 - (int)threadIdx.x >= B.b1.size()) return;  // the whole CTA
  constexpr int CH = kPipeSaRec / 2;
  __shared__ double2 sm[128 * CH];
  const bool act = u0 < B.b1.size();
  const long n = box_node(B, act ? u0 : 0);
  const int p = act ? B.pipe.at[u0] : -1;
  const double phi = (cc.cfl >= 1.0e3 && cc.time == IFLAG_STEADY) ? 0.0 : 1.0;
  const double u = B.v(F_PRI, 2, n), v = B.v(F_PRI, 3, n), w = B.v(F_PRI, 4, n), nut = B.s(F_NUT, n);
  const double dt = B.s(F_DT, n), diasd = B.s(F_DIASD, n), rhs = B.s(F_SARHS, n);
  double c[3], d2 = 0.0;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double x = B.v(F_DXIDX, 3 * d + 1, n), y = B.v(F_DXIDX, 3 * d + 2, n), z = B.v(F_DXIDX, 3 * d + 3, n);
    d2 = d == 0 ? x * x + y * y + z * z : d2 + x * x + y * y + z * z;
    c[d] = x * u + y * v + z * w;
  }
  const double tm = 4.0 * d2 * nut / cc.re;
  const double diag = 1.0 / dt * phi + fabs(c[0]) + fabs(c[1]) + fabs(c[2]) + tm - diasd;
  const double rd = 1.0 / diag;
  double2* rec2 = sm + threadIdx.x * CH;
  rec2[SW_A / 2] = double2{0.5 * (c[0] + fabs(c[0])), 0.5 * (c[1] + fabs(c[1]))};
  rec2[SW_A / 2 + 1] = double2{0.5 * (c[2] + fabs(c[2])), 0.0};
  rec2[SW_B / 2] = double2{0.5 * (c[0] - fabs(c[0])), 0.5 * (c[1] - fabs(c[1]))};
  rec2[SW_B / 2 + 1] = double2{0.5 * (c[2] - fabs(c[2])), __longlong_as_double((long long)n)};
  rec2[SW_RHS / 2] = double2{rhs, diag};
  rec2[SW_RHS / 2 + 1] = double2{rd, recip_lo(diag, rd)};
  rec2[SW_NUT / 2] = double2{nut, divisors_ok(diag, 1.0) ? 1.0 : 0.0};
  // (the neighbour word beside the third coefficient stays)
  store_records<CH>(sm + (threadIdx.x & ~31u) * CH, B.pipe.sa_rec, kPipeSaRec, 0, p, SW_NBR / 2);
}

// q += dq over the updated box (sub_timeadvancement_1stimplicit.f90:568-574), in
// box order so that q is read and written along its rows.
__global__ void k_pipe_update(const BlockView* __restrict__ blocks) {
  const BlockView& B = blocks[blockIdx.y];
  if (B.retired()) return;
  const int u = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (u >= B.b1.size()) return;
  const long n = box_node(B, u);
  const double* dq = B.pipe.rec + (long)kPipeRec * B.pipe.at[u] + PW_RHS;
#pragma unroll
  for (int x = 0; x < 5; ++x) B.v(F_Q, x + 1, n) = B.v(F_Q, x + 1, n) + dq[x];
}

// ------------------------------------------------------------------ the sweeps
namespace {

// The 25 entries of calc_jm's A with rs on the diagonal, times hj, by IEEE
// divisions (nodes outside div_pair's range).
__device__ __noinline__ void entries_ieee(const double* w, double* s) {
  const double rho = w[3], phi = w[6], a1 = w[7], uu = w[8], gamma = w[14], rs = w[12], hj = w[13];
  const double a2 = gamma - 1.0, a3 = gamma - 2.0;
  s[0] = 0.0;
  for (int c = 0; c < 3; ++c) s[1 + c] = w[9 + c];
  s[4] = 0.0;
  for (int r = 0; r < 3; ++r) {
    const double kr = w[9 + r], mr = w[r];
    double* a = s + 5 * (r + 1);
    a[0] = phi * kr - uu * mr / rho;
    for (int c = 0; c < 3; ++c)
      a[1 + c] = c == r ? uu - a3 * kr * mr / rho : w[9 + c] * mr / rho - a2 * kr * w[c] / rho;
    a[4] = a2 * kr;
  }
  s[20] = (phi - a1) * uu;
  for (int c = 0; c < 3; ++c) s[21 + c] = a1 * w[9 + c] - a2 * uu * w[c] / rho;
  s[24] = gamma * uu;
  for (int x = 0; x < 25; ++x) s[x] = (x % 6 == 0 ? s[x] + rs : s[x]) * hj;
}

__device__ __forceinline__ void arrive(unsigned long long* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(slab::local(bar)) : "memory");
}
// Bulk copy global -> this CTA's shared memory, counted in bytes on `bar`
// (addresses 16-byte aligned, bytes a multiple of 16).
__device__ __forceinline__ void copy_in(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   slab::local(dst)),
               "l"(src), "r"(bytes), "r"(slab::local(bar))
               : "memory");
}
// (double)(float)x for |x| in the normal range of a float, by integer
// operations: a thread rounds 24 entries per plane, and the two conversions
// would take the slow pipe beside the FP64 one (plate: 683 us a sweep with
// them, 665 so, 590 without any rounding).  Below that range the value keeps its 24
// bits.
__device__ __forceinline__ double round_to_float(double x) {
  unsigned long long u = (unsigned long long)__double_as_longlong(x);
  u += 0x0fffffffull + ((u >> 29) & 1ull);
  return __longlong_as_double((long long)(u & ~0x1fffffffull));
}
__device__ __forceinline__ double load_s(unsigned at) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(at) : "memory");
  return v;
}
__device__ __forceinline__ void store_s(unsigned at, double v) {
  asm volatile("st.shared.f64 [%0], %1;" ::"r"(at), "d"(v) : "memory");
}

// |a| in (2^-500, 2^500) or a = 0, by its bits: div2_pair's range.
__device__ __forceinline__ bool div2_fast(double a) {
  const unsigned hi = (unsigned)__double2hiint(a) & 0x7fffffffu;
  return (hi - ((1023u - 500u) << 20) < (1000u << 20)) | ((hi | (unsigned)__double2loint(a)) == 0u);
}

// Waits for the phase of `bar` with this parity until it completes, the CTA's
// abort flag rises or (polls < 0) the time bound of the cluster waits or (else)
// so many polls are over; whether it has completed.
__device__ __noinline__ bool wait_phase(unsigned long long* bar, unsigned parity, volatile int* abort, long polls) {
  if (polls < 0) {
    wait_bounded([&] { return *abort != 0 || slab::bar_try(bar, parity); });
  } else {
    for (long n = 0; n < polls; ++n)
      if (*abort != 0 || slab::bar_try(bar, parity)) break;
  }
  return slab::bar_try(bar, parity);
}

// One value into another CTA's shared memory, its 8 bytes counted on that
// CTA's mbarrier.
__device__ __forceinline__ void send(unsigned dst, double v, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(dst),
               "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}

}  // namespace

// One cluster of CTAs per block (grid x = blocks x cluster size), CTA r the
// slab r (CTAs beyond the block's slabs only take the cluster barriers).
//  * The last warp is the producer: one lane brings the records and scalars of
//    the next planes into NST stages with bulk copies (a `full` mbarrier per
//    stage counts the bytes, an `empty` one the warps that have read it).
//  * The other warps form NG groups of W warps; group g takes the planes g,
//    g + NG, ...  A warp covers 10 nodes x 3 directions.  Ahead of its plane's
//    turn a thread forms its 25 entries of S and loads the node's scalars; then
//    the group waits for the plane before (a named barrier, which that plane's
//    group arrives on), forms dq row by row from the neighbours' products, hands
//    it round the node's three threads by shuffles, and writes the products
//    S*dq to the ring (or, across a cut, into the next CTA's inbox with
//    st.async).  So one group's blocks are formed while another group has the
//    chain.
//  * Values across a cut are messages: number s is the layer's nodes (u, v)
//    with u + v = s, in that order forward and the reverse order backward,
//    counted on through both passes.  Message m lies in inbox slot m % D; its
//    mbarrier is armed with its bytes before the slot's reader count (posted
//    to both neighbours) allows the sender to reach m, so no slot is
//    overwritten while it is read and no phase is armed twice.
// Waits: for a stage's records by polls (spin_limit; the default budget: by
// time), all others by time; a wait that gives up raises the abort flag of every CTA of the cluster,
// which ends every other wait.  The threads then run on through the barriers
// without reading stages, and slab::finish keeps all CTAs resident until no
// store can still be on its way.
// What the sweeps solve: words of a record, nodes of a warp, words a node leaves
// for the next plane, words it sends across a cut.
template <bool F32_>
struct MeanFlow {
  static constexpr bool kSa = false, kF32 = F32_;
  static constexpr int kRec = kPipeRec, kNodes = 10, kRing = kPipeProd, kVal = 5;
};
// The SA equation (sub_tur_sa.f90:759-818): one value per node, which the next
// plane's nodes multiply by their own upwind coefficients; a thread per node.
struct SaFlow {
  static constexpr bool kSa = true, kF32 = false;
  static constexpr int kRec = kPipeSaRec, kNodes = 32, kRing = 1, kVal = 1;
};

template <class Eq>
__device__ __forceinline__ void pipe_body(const BlockView* __restrict__ blocks, CaseConsts cc_launch, PipeShape sh,
                                          unsigned* status, long spin_limit, int stall_plane) {
  constexpr int kRec = Eq::kRec, kNodes = Eq::kNodes, kRing = Eq::kRing, kVal = Eq::kVal;
  extern __shared__ __align__(128) double sm[];
  __shared__ int s_read[2];  // messages read by the CTA below / above
  __shared__ int s_fail;
  __shared__ volatile int s_abort;
  const int ncta = (int)slab::size(), me = (int)slab::rank();
  const BlockView& B = blocks[blockIdx.x / ncta];
  if (B.retired()) return;
  const PipeView& V = B.pipe;
  double* const g_rec = Eq::kSa ? V.sa_rec : V.rec;
  const int tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int P = sh.P, W = sh.W, NG = sh.NG, NST = sh.NST, D = sh.D, L = sh.L;
  const PipeSmem at(sh, kRec, kRing, kVal, 0);
  const int sdoubles = P * kRec;
  const int o_stage = at.stage, o_ring = at.ring, o_inbox = at.inbox;
  unsigned long long* const full = (unsigned long long*)(sm + at.bars);
  unsigned long long* const empty = full + NST;
  unsigned long long* const inb = empty + NST;
  unsigned long long* const fdone = inb + D;
  PipePlane* const plane = (PipePlane*)(sm + at.planes);
  const int X = V.dir, ce = V.ce;
  const bool active = me < ce;
  const SlabBox box = slab_box(B, active ? me : 0);
  const int H = box.n[0] + box.n[1] + box.n[2] - 2;
  const Cuts cut(box, X, me, ce);
  const int Dlog = 31 - __clz(D);
  if (tid < 16) sm[tid] = 0.0;
  if (tid == 0) {
    s_read[0] = 0;
    s_read[1] = 0;
    s_fail = 0;
    s_abort = 0;
    for (int x = 0; x < NST; ++x) {
      slab::bar_init(&full[x], 1);
      slab::bar_init(&empty[x], W);
    }
    for (int x = 0; x < D; ++x) slab::bar_init(&inb[x], 1);
    slab::bar_init(fdone, W * NG);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int m = 0; m < min(D, cut.Mall); ++m) slab::bar_expect(&inb[m], 8u * kVal * (unsigned)cut.count(m));
  }
  if (active)
    for (int x = tid; x < H; x += (int)blockDim.x) plane[x] = V.plane[V.slab[me] + x];
  __syncthreads();
  slab::sync();  // every CTA's mbarriers exist (and its first messages are armed) before a neighbour sends

  auto give_up = [&]() {
    s_fail = 1;
    s_abort = 1;
    for (int r = 0; r < ncta; ++r)
      if (r != me) slab::store_relaxed(slab::map(slab::local(const_cast<const int*>(&s_abort)), r), 1);
  };
  auto note = [&](int gs, int wait) {
    if (s_abort == 0) note_timeout(status, Eq::kSa ? TS_SA_SLAB : TS_STAGED, (int)(blockIdx.x / ncta), me, gs, wait);
  };
  auto wait_timed = [&](unsigned long long* bar, unsigned parity) {
    return slab::bar_try(bar, parity) || wait_phase(bar, parity, &s_abort, -1);
  };
  const long stage_polls = spin_limit >= kPipePolls ? -1 : spin_limit;

  if (active && warp == W * NG) {
    // ------------------------------------------------------------- producer
    if (lane == 0) {
      int issued = 0, st = 0;
      unsigned ph = 1;  // parity of the empty phase to wait for (none in the first round)
      for (int gs = 0; gs < 2 * H; ++gs) {
        // fault injection: the first slab's copies of this forward plane are never issued
        if (gs == stall_plane && me == 0) break;
        // a free stage and, before the backward pass, the forward dq* (stored by the warps)
        if ((gs >= NST && !wait_timed(&empty[st], ph)) || (gs == H && !wait_timed(fdone, 0))) {
          note(gs, TW_PROGRESS);
          give_up();
          break;
        }
        if (gs == H) asm volatile("fence.proxy.async.global;" ::: "memory");
        const PipePlane pl = plane[gs < H ? gs : 2 * H - 1 - gs];
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        slab::bar_expect(&full[st], (unsigned)pl.cnt * kRec * 8u);
        copy_in(sm + o_stage + st * sdoubles, g_rec + (long)kRec * pl.pos, (unsigned)pl.cnt * kRec * 8u,
                &full[st]);
        issued = gs + 1;
        if (++st == NST) {
          st = 0;
          ph ^= 1u;
        }
      }
      // the copies in flight land before this CTA leaves (bounded)
      for (int gs = max(0, issued - NST); gs < issued; ++gs)
        wait_bounded([&] { return slab::bar_try(&full[gs % NST], (unsigned)(gs / NST) & 1u); });
    }
    __syncwarp();
  } else if (active && warp < W * NG) {
    // -------------------------------------------------------------- compute
    const CaseConsts& cc = B.ccb ? *B.ccb : cc_launch;
    const double gamma = cc.gamma;
    double* const g_nut = B.f[F_NUT];
    const int g = warp / W, wg = warp - g * W;
    const int d = min(lane / 10, 2), q = lane - 10 * (lane / 10);
    const int n0 = Eq::kSa ? wg * kNodes + lane : wg * kNodes + q;  // this thread's node of a plane
    const int step_b = d < 2 ? 3 : 0;  // from its first row of dq to its second
    const int TG2 = 2 * 32 * W;
    const unsigned read_lo = cut.has_lo ? slab::map(slab::local(&s_read[1]), me - 1) : 0u;
    const unsigned read_hi = cut.has_hi ? slab::map(slab::local(&s_read[0]), me + 1) : 0u;
    const int lot = pipe_lot(D);
    const unsigned sm_at = slab::local(sm), step_b8 = 8u * (unsigned)step_b;
    // Once a stage's wait has run out the warp reads no stage any more (a later
    // phase of a stage whose copies never came would pass for complete) and
    // releases none.
    bool dead = false;
    int gs = g, st = g % NST;  // NG <= NST
    unsigned ph = 0;
    // This thread's node: the 25 entries of its direction's block, r: rhs or dq*
    // of its rows (d and, for d < 2, d + 3), b1 and b2 the divisors in the
    // pass's order with their reciprocals, and where the neighbours' products
    // for its rows lie.
    double s[25];
    double rA, rB, b1, h1, l1, b2, h2, l2;
    unsigned at0 = sm_at, at1 = sm_at, at2 = sm_at;
    int send_to = -1;  // its index in the message it sends, -1: none
    int nat = 0;       // SA: its place in the box
    bool bok = true, edge_in = false;

    auto pass = [&](auto direction) {
      constexpr bool FWD = decltype(direction)::value;
      const int end = FWD ? H : 2 * H;
      // where the neighbours' values lie, and whether some cross a cut
      auto locate = [&](uint2 nb, bool act, int prev, int in_slot) {
        const unsigned half = FWD ? nb.x : nb.y;
        const bool in = act && (half & (FWD ? kLoBit : kHiBit)) != 0;
        const bool out = act && (Eq::kSa || d == X) && (half & (FWD ? kHiBit : kLoBit)) != 0;
        const int row = Eq::kSa ? 0 : d;
        const int near = prev + row, far = o_inbox + in_slot * kVal * L + row;
        auto where = [&](int e) {
          const int w = nbr_index(half, e);
          const bool across = in && e == X;
          const int word = (across ? far : near + (Eq::kSa ? 0 : 5 * e)) + (across ? kVal : kRing) * w;
          return sm_at + (act && w != kNoNbr ? 8u * (unsigned)word : 0u);
        };
        at0 = where(0);
        at1 = where(1);
        at2 = where(2);
        edge_in = in;
        send_to = out ? nbr_index(FWD ? nb.y : nb.x, X) : -1;
      };
      auto load = [&](const double* rec, bool act, int prev, int in_slot) {
        const double2* r = reinterpret_cast<const double2*>(rec);
        if constexpr (Eq::kSa) {
          // the upwind coefficients (s[0..2]), rhs or dnut* (rA), the diagonal
          const double2 c01 = r[(FWD ? SW_A : SW_B) / 2], c2x = r[(FWD ? SW_A : SW_B) / 2 + 1];
          const double2 rd = r[SW_RHS / 2], rc = r[SW_RHS / 2 + 1];
          locate(*reinterpret_cast<const uint2*>(rec + SW_NBR), act, prev, in_slot);
          s[0] = c01.x;
          s[1] = c01.y;
          s[2] = c2x.x;
          rA = rd.x;
          b1 = rd.y;
          h1 = rc.x;
          l1 = rc.y;
          bok = reinterpret_cast<const int*>(rec + SW_OK)[1] != 0;
          if (!FWD) {
            rB = rec[SW_NUT];
            nat = reinterpret_cast<const int*>(rec + SW_NAT)[0];
          }
          return;
        }
        const double2 m01 = r[PW_M / 2], m2r = r[PW_M / 2 + 1], rc = r[PW_RCP / 2], pa = r[PW_PHI / 2];
        const double2 uk = r[PW_DIR / 2 + 3 * d], kk = r[PW_DIR / 2 + 3 * d + 1], rh = r[PW_DIR / 2 + 3 * d + 2];
        locate(*reinterpret_cast<const uint2*>(rec + PW_NBR), act, prev, in_slot);
        const double rho = m2r.y, rr = rc.x, rl = rc.y;
        const double phi = pa.x, a1 = pa.y, uu = uk.x, hj = rh.y, rs = FWD ? rh.x : -rh.x;
        const double m[3] = {m01.x, m01.y, m2r.x}, k[3] = {uk.y, kk.x, kk.y};
        const double a2 = gamma - 1.0, a3 = gamma - 2.0;
        auto dv = [&](double a) { return div_pair(a, rho, rr, rl); };
        s[0] = rs * hj;
        s[4] = 0.0;
#pragma unroll
        for (int c = 0; c < 3; ++c) s[1 + c] = k[c] * hj;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const double a2k = a2 * k[i];
          s[5 * i + 5] = (phi * k[i] - dv(uu * m[i])) * hj;
#pragma unroll
          for (int c = 0; c < 3; ++c)
            s[5 * i + 6 + c] =
                c == i ? (uu - dv(a3 * k[i] * m[i]) + rs) * hj : (dv(k[c] * m[i]) - dv(a2k * m[c])) * hj;
          s[5 * i + 9] = a2k * hj;
        }
        const double a2u = a2 * uu;
        s[20] = (phi - a1) * uu * hj;
#pragma unroll
        for (int c = 0; c < 3; ++c) s[21 + c] = (a1 * k[c] - dv(a2u * m[c])) * hj;
        s[24] = (gamma * uu + rs) * hj;
        if (!(rr == rr)) {
          const double w[15] = {m[0], m[1], m[2], rho, 0.0, 0.0, phi, a1, uu, k[0], k[1], k[2], rs, hj, gamma};
          double t[25];
          entries_ieee(w, t);
#pragma unroll
          for (int x = 0; x < 25; ++x) s[x] = t[x];
        }
        if (Eq::kF32) {
#pragma unroll
          for (int x = 0; x < 25; ++x)
            if (x != 4) s[x] = round_to_float(s[x]);
        }
        const double2 di = r[PW_DIV / 2], rdi = r[PW_DIV / 2 + 1], lo = r[PW_DIV / 2 + 2];
        rA = rec[PW_RHS + d];
        rB = rec[PW_RHS + d + step_b];
        b1 = FWD ? di.x : di.y;
        b2 = FWD ? di.y : di.x;
        h1 = FWD ? rdi.x : rdi.y;
        h2 = FWD ? rdi.y : rdi.x;
        l1 = FWD ? lo.x : lo.y;
        l2 = FWD ? lo.y : lo.x;
        bok = reinterpret_cast<const int*>(rec + PW_OK)[1] != 0;
      };
      for (; gs < end; gs += NG) {
        const int h = FWD ? gs : 2 * H - 1 - gs;
        const PipePlane pl = plane[h];
        const int cnt = pl.cnt;
        const double* const stg = sm + o_stage + st * sdoubles;
        const int prev = o_ring + ((gs - 1) & 1) * kRing * P, cur = o_ring + (gs & 1) * kRing * P;
        const int in_m = cut.in_number(FWD, h);  // the message this plane's edge nodes read (if it has any)
        const bool one = cnt <= kNodes * W, mine = wg * kNodes < cnt;
        const bool have = __all_sync(
            0xffffffffu, !dead && (slab::bar_try(&full[st], ph) || wait_phase(&full[st], ph, &s_abort, stage_polls)));
        int n = n0;
        bool act = have && (Eq::kSa || lane < 30) && n < cnt;
        // the message, where a node of this warp reads one
        auto await_message = [&]() {
          if (__any_sync(0xffffffffu, act && edge_in) &&
              !wait_timed(&inb[in_m & (D - 1)], (unsigned)(in_m >> Dlog) & 1u)) {
            note(gs, TW_LAST_PLANE);
            give_up();
          }
          __syncwarp();
        };
        // dq of the warp's nodes from the products of the plane before, and their
        // own products; nothing here waits or (rare divisions aside) branches
        double vA, vB, prod[5];
        auto chain = [&](unsigned to) {
          if constexpr (Eq::kSa) {
            const double t0 = s[0] * load_s(at0), t1 = s[1] * load_s(at1), t2 = s[2] * load_s(at2);
            const double n = FWD ? rA + (t0 + t1 + t2) : t0 + t1 + t2;
            double v = div_pair(n, b1, h1, l1);
            if (__any_sync(0xffffffffu, !(bok & div2_fast(n))))
              v = bok && div2_fast(n) ? v : div1_ieee(n, b1);
            if (!FWD) v = rA - v;
            store_s(to, v);
            vA = v;
            prod[0] = v;
            return;
          }
          const double A0 = load_s(at0), A1 = load_s(at1), A2 = load_s(at2);
          const double B0 = load_s(at0 + step_b8), B1 = load_s(at1 + step_b8), B2 = load_s(at2 + step_b8);
          const double sA = A0 + A1 + A2, sB = B0 + B1 + B2;
          const double nA = FWD ? rA + sA : sA, nB = FWD ? rB + sB : sB;
          vA = div_pair(div_pair(nA, b1, h1, l1), b2, h2, l2);
          vB = div_pair(div_pair(nB, b1, h1, l1), b2, h2, l2);
          const bool slow = !(bok & div2_fast(nA) & div2_fast(nB));
          if (__any_sync(0xffffffffu, slow)) {
            vA = div2_pair(nA, b1, h1, l1, b2, h2, l2, bok);
            vB = div2_pair(nB, b1, h1, l1, b2, h2, l2, bok);
          }
          if (!FWD) {
            vA = rA - vA;
            vB = rB - vB;
          }
          double x[5];
          x[0] = __shfl_sync(0xffffffffu, vA, q);
          x[1] = __shfl_sync(0xffffffffu, vA, q + 10);
          x[2] = __shfl_sync(0xffffffffu, vA, q + 20);
          x[3] = __shfl_sync(0xffffffffu, vB, q);
          x[4] = __shfl_sync(0xffffffffu, vB, q + 10);
#pragma unroll
          for (int r = 0; r < 5; ++r) {
            prod[r] = s[5 * r] * x[0];
#pragma unroll
            for (int c = 1; c < 5; ++c) prod[r] = prod[r] + s[5 * r + c] * x[c];
          }
#pragma unroll
          for (int r = 0; r < 5; ++r) store_s(to + 8u * r, prod[r]);
        };
        auto target = [&]() { return sm_at + 8u * (unsigned)(act ? cur + kRing * n + (Eq::kSa ? 0 : 5 * d) : 16); };
        // what the chain of this CTA's planes does not wait for: the products that
        // leave the slab, and dq itself
        auto finish_nodes = [&]() {
          if (!act) return;
          if (send_to >= 0) {
            const int to = FWD ? me + 1 : me - 1;
            const int m = cut.out(FWD, h, me);
            const int* count = &s_read[FWD ? 1 : 0];
            // (the groups post their counts in no particular order, so a count may
            // be followed by a smaller one; pipe_groups keeps that one large enough)
            bool room = m < D || slab::load_relaxed(count) > m - D;
            if (!room) wait_bounded([&] { return (room = slab::load_relaxed(count) > m - D) || s_abort != 0; });
            if (room) {
              const unsigned dst =
                  slab::map(slab::local(sm + o_inbox + (m & (D - 1)) * kVal * L + kVal * send_to), (unsigned)to);
              const unsigned bar = slab::map(slab::local(&inb[m & (D - 1)]), (unsigned)to);
#pragma unroll
              for (int r = 0; r < kVal; ++r) send(dst + (unsigned)(r * 8), prod[r], bar);
            } else {
              note(gs, TW_PROGRESS);
              give_up();
            }
          }
          if constexpr (Eq::kSa) {
            if (FWD)
              g_rec[(long)kRec * (pl.pos + n) + SW_RHS] = vA;
            else
              g_nut[nat] = rB + vA;
          } else {
            double* const out = g_rec + (long)kRec * (pl.pos + n) + (PW_RHS + d);
            out[0] = vA;
            if (d < 2) out[3] = vB;
          }
        };
        // the products of the plane before are there / this plane's are
        auto plane_wait = [&]() {
          if (!FWD || gs > 0) asm volatile("bar.sync %0, %1;" ::"r"(1 + ((gs - 1) & 7)), "r"(TG2) : "memory");
        };
        auto plane_done = [&]() {
          if (FWD || gs + 1 < 2 * H) asm volatile("bar.arrive %0, %1;" ::"r"(1 + (gs & 7)), "r"(TG2) : "memory");
        };
        if (have && one && mine) {
          load(stg + kRec * (act ? n : 0), act, prev, in_m & (D - 1));
          __syncwarp();
          if (lane == 0) arrive(&empty[st]);
          await_message();
          const unsigned to = target();
          plane_wait();
          chain(to);
          plane_done();
          finish_nodes();
        } else if (have && !one) {
          // planes wider than the group: the nodes in turn
          load(stg + kRec * (act ? n : 0), act, prev, in_m & (D - 1));
          __syncwarp();
          plane_wait();
          for (int base = 0;;) {
            await_message();
            chain(target());
            finish_nodes();
            __syncwarp();
            base += kNodes * W;
            if (base >= cnt) break;
            n = base + n0;
            act = (Eq::kSa || lane < 30) && n < cnt;
            load(stg + kRec * (act ? n : 0), act, prev, in_m & (D - 1));
          }
          if (lane == 0) arrive(&empty[st]);
          plane_done();
        } else {
          // no node of this plane, or no records
          if (have && lane == 0) arrive(&empty[st]);
          plane_wait();
          if (!have && !dead) {
            // reported in the planes' turn, so that the first plane is the one noted
            if (lane == 0) {
              note(gs, TW_PLANE);
              give_up();
            }
            dead = true;
          }
          __syncwarp();
          plane_done();
        }
        // every `lot` messages: the planes up to the one before this have been
        // read, so arm their slots again and tell the neighbours (a message whose
        // wait ran out raised the abort flag before the barrier)
        if (wg == 0 && cut.Mall > D && lane == 31 && gs > 0) {
          const int p = gs - 1;
          const int m = cut.in(p < H, p < H ? p : 2 * H - 1 - p);
          if (m >= 0 && ((m + 1) & (lot - 1)) == 0 && s_abort == 0) {
            for (int x = m + 1 - lot; x <= m; ++x)
              if (x + D < cut.Mall) slab::bar_expect(&inb[x & (D - 1)], 8u * kVal * (unsigned)cut.count(x + D));
            if (cut.has_lo) slab::store_relaxed(read_lo, m + 1);
            if (cut.has_hi) slab::store_relaxed(read_hi, m + 1);
          }
        }
        __syncwarp();
        st += NG;
        if (st >= NST) {
          st -= NST;
          ph ^= 1u;
        }
      }
    };
    pass(std::true_type{});
    // the forward dq* of this warp, for the copies of the backward pass
    asm volatile("fence.proxy.async.global;" ::: "memory");
    __syncwarp();
    if (lane == 0) arrive(fdone);
    pass(std::false_type{});
  }
  __syncwarp();
  slab::finish(s_fail, ncta, status, B);
}

template <int WARPS, int CTAS, bool F32>
__global__ void __launch_bounds__(32 * WARPS, CTAS)
    k_pipe_sweep(const BlockView* __restrict__ blocks, CaseConsts cc, PipeShape sh, unsigned* status, long spin_limit,
                 int stall_plane) {
  pipe_body<MeanFlow<F32>>(blocks, cc, sh, status, spin_limit, stall_plane);
}
PipeKernel pipe_kernel(int variant, bool f32) {
  static const PipeKernel k[kPipeVariants][2] = {
      {k_pipe_sweep<8, 1, false>, k_pipe_sweep<8, 1, true>},
      {k_pipe_sweep<11, 1, false>, k_pipe_sweep<11, 1, true>},
      {k_pipe_sweep<16, 1, false>, k_pipe_sweep<16, 1, true>},
      {k_pipe_sweep<6, 2, false>, k_pipe_sweep<6, 2, true>},
      {k_pipe_sweep<8, 2, false>, k_pipe_sweep<8, 2, true>}};
  return k[variant][f32 ? 1 : 0];
}

__global__ void __launch_bounds__(512, 1)
    k_pipe_sa_sweep(const BlockView* __restrict__ blocks, CaseConsts cc, PipeShape sh, unsigned* status,
                    long spin_limit, int stall_plane) {
  pipe_body<SaFlow>(blocks, cc, sh, status, spin_limit, stall_plane);
}

#endif

}  // namespace aero
