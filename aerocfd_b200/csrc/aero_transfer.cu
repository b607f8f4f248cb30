// Layout conversion between the reference's host arrays a(nc, is:ie, js:je, ks:ke)
// (column-major, component fastest) and the device's component planes.
#include "aero_device.cuh"
#include "aero_kernels.h"

namespace aero {

__global__ void k_aos_to_soa(const double* __restrict__ src, double* __restrict__ dst, long n,
                             int nc, long plane) {
  long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  for (int c = 0; c < nc; ++c) dst[(long)c * plane + t] = src[t * nc + c];
}

__global__ void k_soa_to_aos(const double* __restrict__ src, double* __restrict__ dst, long n,
                             int nc, long plane) {
  long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  for (int c = 0; c < nc; ++c) dst[t * nc + c] = src[(long)c * plane + t];
}

// The freestream start of every block (sub_init_flowfield.f90:55-111) in one
// launch, a block's values from its own row of `values`: written once per node,
// about 60 words, so bound by the HBM writes of a large set and by the one
// launch of a small one (a fill per component plane was 60 launches a block).
__global__ void k_init_flowfield(const BlockView* __restrict__ blocks, const InitValues* __restrict__ values, int sa) {
  const BlockView& B = blocks[blockIdx.y];
  const InitValues& v = values[blockIdx.y];
  const long n = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= B.b.size()) return;
#pragma unroll
  for (int x = 0; x < 5; ++x) {
    B.v(F_Q, x + 1, n) = v.q[x];
    B.v(F_Q0, 2 * x + 1, n) = v.q[x];  // q0(l, c) = q(c) at both time levels (:78-82)
    B.v(F_Q0, 2 * x + 2, n) = v.q[x];
    B.v(F_RHSV, x + 1, n) = 0.0;
    B.v(F_RHSI, x + 1, n) = 0.0;
    B.v(F_RHS, x + 1, n) = 0.0;
  }
#pragma unroll
  for (int x = 0; x < 7; ++x) B.v(F_PRI, x + 1, n) = v.pri[x];
#pragma unroll
  for (int x = 0; x < 3; ++x) B.v(F_AMU, x + 1, n) = v.amu[x];
  B.s(F_DT, n) = v.dt;
  if (sa) {
    B.s(F_NUT, n) = v.nut;
    B.s(F_SARHS, n) = 0.0;
  }
#pragma unroll
  for (int x = 1; x <= 9; ++x) B.v(F_DUDX, x, n) = 0.0;
  B.s(F_VOR, n) = 0.0;
#pragma unroll
  for (int x = 1; x <= 6; ++x) B.v(F_TAO, x, n) = 0.0;
}

}  // namespace aero
