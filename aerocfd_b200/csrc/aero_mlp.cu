// Warm-start network of the solver (no counterpart in the reference): an MLP
// with BF16 weights and activations and FP32 accumulation whose forward and
// backward contractions run on the tcgen05 GEMM of aero_mlp_gemm.cuh.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <vector>

#include "../../include/aerocfd_gpu.h"
#include "aero_mlp_gemm.cuh"

namespace aero {
int set_last_error(int code, const char* msg);  // aero_runtime.cu

namespace mlp {
namespace {

#define MCK(call)                                                                      \
  do {                                                                                 \
    cudaError_t e_ = (call);                                                           \
    if (e_ != cudaSuccess) {                                                           \
      cudaGetLastError(); /* reported here, not by the next call's check */            \
      char b_[200];                                                                    \
      std::snprintf(b_, sizeof b_, "%s: %s", #call, cudaGetErrorString(e_));           \
      return set_last_error(e_ == cudaErrorMemoryAllocation ? AERO_ERR_NOMEM : AERO_ERR_CUDA, b_); \
    }                                                                                  \
  } while (0)

// Fixed-order sum of the split-K partial tiles: out[i] = sum_s part[s][i].
__global__ void k_splitk_reduce(const float* __restrict__ part, int splits, long n, float* __restrict__ out) {
  long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float s = 0.f;
  for (int x = 0; x < splits; ++x) s += part[(long)x * n + i];
  out[i] = s;
}

__device__ __forceinline__ uint16_t to_bf16(float f) {  // round to nearest even
  uint32_t u = __float_as_uint(f);
  if ((u & 0x7F800000u) == 0x7F800000u) return (uint16_t)(u >> 16);  // inf / nan
  u += 0x7FFFu + ((u >> 16) & 1u);
  return (uint16_t)(u >> 16);
}
__device__ __forceinline__ float sigmoid(float z) { return 1.0f / (1.0f + expf(-z)); }

// One batch of the network's inputs: rows idx[0 .. n) of src (idx null: rows 0 ..
// n) in BF16 into h (rows x ld) and its transpose ht (ld x rows); rows past n are
// zero, and the padding columns are zero from the start and never written.
__global__ void k_load_inputs(const float* __restrict__ src, const int* __restrict__ idx, int n, int cols, int rows,
                              int ld, uint16_t* __restrict__ h, uint16_t* __restrict__ ht) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long)rows * cols) return;
  const int r = (int)(i / cols), c = (int)(i % cols);
  const uint16_t v = r < n ? to_bf16(src[(long)(idx ? idx[r] : r) * cols + c]) : (uint16_t)0;
  h[(long)r * ld + c] = v;
  ht[(long)c * rows + r] = v;
}

// y = c + b, the real rows and columns only.
__global__ void k_outputs(const float* __restrict__ c, const float* __restrict__ b, int n, int n_out, int ld,
                          float* __restrict__ y) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long)n * n_out) return;
  const int r = (int)(i / n_out), j = (int)(i % n_out);
  y[i] = c[(long)r * ld + j] + b[j];
}

// Rows and columns of an elementwise CTA's tile, and its threads: 32 columns by
// kTileRows rows, 32 x 32 threads, so that 32 warps hide the loads' and the
// exponentials' latency.
constexpr int kTileRows = 512;
constexpr dim3 kTileThreads(32, 32);
constexpr size_t kTileSmem = (size_t)kTileRows * 33 * sizeof(float);
// Stores a tile's 32 columns (f[row][33]) in BF16 as rows of out (cols x rows).
__device__ __forceinline__ void store_transposed(const float* f, int rows, uint16_t* __restrict__ out) {
  const int lane = threadIdx.x;
  for (int c = threadIdx.y; c < 32; c += 32)
    for (int r = 2 * lane; r < kTileRows; r += 64) {
      const uint32_t pair = (uint32_t)to_bf16(f[r * 33 + c]) | (uint32_t)to_bf16(f[(r + 1) * 33 + c]) << 16;
      *(uint32_t*)(out + (long)(blockIdx.x * 32 + c) * rows + (long)blockIdx.y * kTileRows + r) = pair;
    }
}

// Hidden layer, forward: z += b per column, h = bf16(silu(z)) and, for the weight
// gradients (ht not null), its transpose.
__global__ void __launch_bounds__(1024) k_activate(float* __restrict__ z, const float* __restrict__ b, int rows,
                                                   int cols, uint16_t* __restrict__ h, uint16_t* __restrict__ ht) {
  extern __shared__ float f[];
  const int tx = threadIdx.x, col = blockIdx.x * 32 + tx;
  const float bias = b[col];
#pragma unroll 4
  for (int r = threadIdx.y; r < kTileRows; r += 32) {
    const long i = (long)(blockIdx.y * kTileRows + r) * cols + col;
    const float v = z[i] + bias;
    z[i] = v;
    const float a = v * sigmoid(v);
    h[i] = to_bf16(a);
    f[r * 33 + tx] = a;
  }
  if (!ht) return;
  __syncthreads();
  store_transposed(f, rows, ht);
}

// The elementwise parts of the backward pass: a CTA takes 32 columns of kTileRows
// rows and forms the gradient g(row, column) there, its BF16 value row-major (the
// GEMM for the layer below) and transposed (the weight gradient's GEMM), and its
// column sums for the bias, summed over every eighth row, then over the eight,
// in that order; the tiles' sums are added in order by the update.  One pass
// over the inputs in place of four (silu', transpose, column sums and the FP32
// copy they read: 52 us a layer of 8192 x 256).
template <class G>
__device__ __forceinline__ void column_pass(int rows, int cols, uint16_t* __restrict__ d, uint16_t* __restrict__ dt,
                                            float* __restrict__ part, G g) {
  extern __shared__ float f[];
  __shared__ float sm[8][33];
  const int tx = threadIdx.x, ty = threadIdx.y, col = blockIdx.x * 32 + tx, r0 = blockIdx.y * kTileRows;
#pragma unroll 4
  for (int r = ty; r < kTileRows; r += 32) {
    const float v = g(r0 + r, col);
    d[(long)(r0 + r) * cols + col] = to_bf16(v);
    f[r * 33 + tx] = v;
  }
  __syncthreads();
  if (ty < 8) {
    float s = 0.f;
#pragma unroll 16
    for (int r = ty; r < kTileRows; r += 8) s += f[r * 33 + tx];
    sm[ty][tx] = s;
  }
  store_transposed(f, rows, dt);
  __syncthreads();
  if (ty == 0) {
    float t = 0.f;
    for (int y = 0; y < 8; ++y) t += sm[y][tx];
    part[(long)blockIdx.y * cols + col] = t;
  }
}

// Hidden layer: dz = dh * silu'(z).
__global__ void __launch_bounds__(1024) k_back_hidden(const float* __restrict__ dh, const float* __restrict__ z,
                                                     int rows, int cols, uint16_t* __restrict__ dz,
                                                     uint16_t* __restrict__ dzt, float* __restrict__ part) {
  column_pass(rows, cols, dz, dzt, part, [&](int r, int c) {
    const float zz = z[(long)r * cols + c], s = sigmoid(zz);
    return dh[(long)r * cols + c] * (s * (1.f + zz * (1.f - s)));
  });
}

// Output layer: y = c + b, the masked difference to the target and its gradient;
// per-CTA sums of the squared differences.
__global__ void __launch_bounds__(1024) k_back_output(const float* __restrict__ c, const float* __restrict__ b,
                                                     const float* __restrict__ t, const int* __restrict__ idx,
                                                     int n_real, int n_out, int rows, int cols, float inv_count,
                                                     uint16_t* __restrict__ dy, uint16_t* __restrict__ dyt,
                                                     float* __restrict__ part, float* __restrict__ loss_part) {
  float l = 0.f;
  column_pass(rows, cols, dy, dyt, part, [&](int r, int j) {
    const float v = c[(long)r * cols + j] + b[j];
    const float d = (r < n_real && j < n_out) ? v - t[(long)(idx ? idx[r] : r) * n_out + j] : 0.f;
    l += d * d;
    return 2.f * d * inv_count;
  });
  __shared__ float sm[1024];
  const int tid = threadIdx.y * 32 + threadIdx.x;
  sm[tid] = l;
  __syncthreads();
  for (int o = 512; o > 0; o >>= 1) {
    if (tid < o) sm[tid] += sm[tid + o];
    __syncthreads();
  }
  if (tid == 0) loss_part[blockIdx.y * gridDim.x + blockIdx.x] = sm[0];
}

// Sum of the loss parts of a step (one warp).
__global__ void k_loss_sum(const float* __restrict__ part, int n, float* __restrict__ out) {
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += 32) s += part[i];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (threadIdx.x == 0) *out = (float)s;
}

// out[c][r] = in[r][c] for a rows x cols BF16 matrix (32 x 32 tiles).
__global__ void k_transpose_bf16(const uint16_t* __restrict__ in, int rows, int cols, uint16_t* __restrict__ out) {
  __shared__ uint16_t tile[32][33];
  int c = blockIdx.x * 32 + threadIdx.x, r0 = blockIdx.y * 32;
  for (int y = threadIdx.y; y < 32; y += blockDim.y) {
    int r = r0 + y;
    if (r < rows && c < cols) tile[y][threadIdx.x] = in[(long)r * cols + c];
  }
  __syncthreads();
  int r = r0 + threadIdx.x, cc0 = blockIdx.x * 32;
  for (int y = threadIdx.y; y < 32; y += blockDim.y) {
    int cc = cc0 + y;
    if (cc < cols && r < rows) out[(long)cc * rows + r] = tile[threadIdx.x][y];
  }
}

// One layer's parameters (weights, then biases).
struct LayerParams {
  float *w, *mw, *vw, *gw, *b, *mb, *vb, *gb;
  uint16_t *wb, *wt;  // BF16 copy of the weights and its transpose
  int nin, nout;
};
// The layer's gradients from the weight GEMM's split-K partial tiles and the bias
// column sums, each added in a fixed order: stored (train = 0), or (train = 1)
// used by Adam (Kingma & Ba 2015) on the FP32 master parameters, which also
// renews the BF16 weights and their transpose; one launch a layer in place of
// five.
__global__ void k_update_layer(LayerParams p, const float* __restrict__ wpart, int splits,
                               const float* __restrict__ bpart, int chunks, int train, float lr, float b1, float b2,
                               float c1, float c2, float eps) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x, nw = (long)p.nin * p.nout;
  if (i >= nw + p.nout) return;
  const bool weight = i < nw;
  const long j = weight ? i : i - nw, n = weight ? nw : p.nout;
  const float* part = weight ? wpart : bpart;
  float g = 0.f;
#pragma unroll 8
  for (int x = 0; x < (weight ? splits : chunks); ++x) g += part[(long)x * n + j];
  if (!train) {
    (weight ? p.gw : p.gb)[j] = g;
    return;
  }
  float *w = weight ? p.w : p.b, *m = weight ? p.mw : p.mb, *v = weight ? p.vw : p.vb;
  const float mi = b1 * m[j] + (1.f - b1) * g;
  const float vi = b2 * v[j] + (1.f - b2) * g * g;
  m[j] = mi;
  v[j] = vi;
  const float wi = w[j] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  w[j] = wi;
  if (weight) {
    const uint16_t b = to_bf16(wi);
    p.wb[j] = b;
    p.wt[(j % p.nin) * p.nout + j / p.nin] = b;
  }
}

}  // namespace

// The product C = A * B^T in `splits` partial tiles (changed to the number made),
// one after another in C.
int gemm_problem(GemmProblem& p, const uint16_t* A, const uint16_t* B, float* C, int M, int N, int K, int& splits) {
  if (M % kBM || N % kBN || K % kBK || splits < 1)
    return set_last_error(AERO_ERR_ARG, "tensor-core GEMM needs M, N multiples of 128 and K a multiple of 64");
  const int ktiles = K / kBK;
  if (splits > ktiles) splits = ktiles;
  const int klen = ((ktiles + splits - 1) / splits) * kBK;
  splits = (K + klen - 1) / klen;
  p = GemmProblem{A, B, C, M, N, K, klen, N / kBN * (M / kBM) * splits};
  return AERO_OK;
}
int launch_gemms(const GemmProblem& p0, const GemmProblem& p1, unsigned* status, cudaStream_t st) {
  static int smem_dev = -1;  // device whose limit was raised (one device per process)
  int dev = 0;
  MCK(cudaGetDevice(&dev));
  if (smem_dev != dev) {
    MCK(cudaFuncSetAttribute(k_gemm_bf16, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemmSmem));
    smem_dev = dev;
  }
  k_gemm_bf16<<<p0.tiles + p1.tiles, kGemmThreads, kGemmSmem, st>>>(p0, p1, status);
  MCK(cudaGetLastError());
  return AERO_OK;
}
int gemm_parts(const uint16_t* A, const uint16_t* B, float* C, int M, int N, int K, int& splits, unsigned* status,
               cudaStream_t st) {
  GemmProblem p;
  int rc = gemm_problem(p, A, B, C, M, N, K, splits);
  return rc ? rc : launch_gemms(p, GemmProblem{}, status, st);
}
// The same into C; splits > 1 adds the partial tiles from `scratch` (splits * M *
// N floats).
int gemm(const uint16_t* A, const uint16_t* B, float* C, int M, int N, int K, int splits, float* scratch,
         unsigned* status, cudaStream_t st) {
  int rc = gemm_parts(A, B, splits > 1 ? scratch : C, M, N, K, splits, status, st);
  if (rc) return rc;
  if (splits > 1) {
    long n = (long)M * N;
    k_splitk_reduce<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(scratch, splits, n, C);
    MCK(cudaGetLastError());
  }
  return AERO_OK;
}

}  // namespace mlp
}  // namespace aero

using namespace aero;

extern "C" int aero_mlp_gemm_timed(int M, int N, int K, int reps, double* ms_per_gemm) {
  if (M <= 0 || N <= 0 || K <= 0 || M % 128 || N % 128 || K % 64 || reps < 1 || !ms_per_gemm)
    return set_last_error(AERO_ERR_ARG, "aero_mlp_gemm_timed: M, N multiples of 128, K a multiple of 64, reps >= 1");
  uint16_t *dA = nullptr, *dB = nullptr;
  float* dC = nullptr;
  unsigned* dst = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  auto cleanup = [&] {
    cudaFree(dA); cudaFree(dB); cudaFree(dC); cudaFree(dst);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
  };
  size_t na = (size_t)M * K, nb = (size_t)N * K, nc = (size_t)M * N;
  if (cudaMalloc(&dA, na * 2) || cudaMalloc(&dB, nb * 2) || cudaMalloc(&dC, nc * 4) || cudaMalloc(&dst, 4)) {
    cleanup();
    return set_last_error(AERO_ERR_NOMEM, "aero_mlp_gemm_timed: device allocation failed");
  }
  // operands: every byte 0x3c, i.e. BF16 0x3c3c (about 0.0115) everywhere; the
  // values do not change the time
  cudaMemset(dA, 0x3c, na * 2);
  cudaMemset(dB, 0x3c, nb * 2);
  cudaMemset(dst, 0, 4);
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  int rc = mlp::gemm(dA, dB, dC, M, N, K, 1, nullptr, dst, 0);  // warm-up
  if (!rc) {
    cudaEventRecord(e0, 0);
    for (int r = 0; r < reps && !rc; ++r) rc = mlp::gemm(dA, dB, dC, M, N, K, 1, nullptr, dst, 0);
    cudaEventRecord(e1, 0);
  }
  unsigned st = 0;
  if (!rc) {
    cudaError_t e = cudaEventSynchronize(e1);
    float ms = 0.f;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
    if (e == cudaSuccess) e = cudaMemcpy(&st, dst, 4, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) rc = set_last_error(AERO_ERR_CUDA, cudaGetErrorString(e));
    else if (st) rc = set_last_error(AERO_ERR_DEVICE, "aero_mlp_gemm_timed: a tensor-core wait timed out");
    *ms_per_gemm = ms / reps;
  }
  cleanup();
  return rc;
}

extern "C" int aero_mlp_gemm(const uint16_t* a, const uint16_t* b, float* c, int M, int N, int K, int splits) {
  if (M <= 0 || N <= 0 || K <= 0 || M % 128 || N % 128 || K % 64 || splits < 1)
    return set_last_error(AERO_ERR_ARG, "aero_mlp_gemm: M, N multiples of 128, K a multiple of 64, splits >= 1");
  uint16_t *dA = nullptr, *dB = nullptr;
  float *dC = nullptr, *dS = nullptr;
  unsigned* dst = nullptr;
  int rc = AERO_OK;
  auto cleanup = [&] {
    cudaFree(dA); cudaFree(dB); cudaFree(dC); cudaFree(dS); cudaFree(dst);
  };
  size_t na = (size_t)M * K, nb = (size_t)N * K, nc = (size_t)M * N;
  if (cudaMalloc(&dA, na * 2) || cudaMalloc(&dB, nb * 2) || cudaMalloc(&dC, nc * 4) ||
      cudaMalloc(&dS, nc * 4 * (size_t)splits) || cudaMalloc(&dst, 4)) {
    cleanup();
    return set_last_error(AERO_ERR_NOMEM, "aero_mlp_gemm: device allocation failed");
  }
  cudaMemcpy(dA, a, na * 2, cudaMemcpyHostToDevice);
  cudaMemcpy(dB, b, nb * 2, cudaMemcpyHostToDevice);
  cudaMemset(dst, 0, 4);
  rc = mlp::gemm(dA, dB, dC, M, N, K, splits, dS, dst, 0);
  unsigned st = 0;
  if (!rc) {
    cudaError_t e = cudaMemcpy(c, dC, nc * 4, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(&st, dst, 4, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) rc = set_last_error(AERO_ERR_CUDA, cudaGetErrorString(e));
    else if (st) rc = set_last_error(AERO_ERR_DEVICE, "aero_mlp_gemm: a tensor-core wait timed out");
  }
  cleanup();
  return rc;
}

// ---------------------------------------------------------------- the network
namespace aero {
namespace mlp {
namespace {

// Layer l maps nin inputs to nout outputs (padded sizes: multiples of 128).
struct Layer {
  int nin = 0, nout = 0;
  float *w = nullptr, *b = nullptr;                        // FP32 master
  float *mw = nullptr, *vw = nullptr, *mb = nullptr, *vb = nullptr;  // Adam moments
  float *gw = nullptr, *gb = nullptr;                      // gradients
  uint16_t *wb = nullptr, *wt = nullptr;                   // BF16 copy and its transpose
};

struct Net {
  bool ok = false;
  int n_in = 0, n_out = 0, width = 0, depth = 0, batch = 0;
  int kin = 128, nout = 128;  // padded input and output widths
  std::vector<Layer> L;       // depth hidden layers, then the output layer
  std::vector<uint16_t*> h;   // h[0] input, h[l] = silu(z[l-1]); BF16 batch x width
  std::vector<uint16_t*> ht;  // their transposes
  std::vector<float*> z;      // pre-activations, FP32
  float *c_out = nullptr, *y = nullptr, *dh = nullptr;
  uint16_t *d = nullptr, *dt = nullptr;  // a layer's gradient and its transpose
  float *scratch = nullptr, *cpart = nullptr, *lpart = nullptr;
  float *xb = nullptr, *tb = nullptr, *xall = nullptr, *tall = nullptr;
  int* perm[2] = {nullptr, nullptr};  // row order of an epoch and of the next
  unsigned* status = nullptr;
  long n_all = 0;
  int adam_t = 0;
  char* arena = nullptr;  // the arrays above but xall, tall and perm
  size_t arena_bytes = 0;
} g_net;

constexpr int kSplitMax = 32;

// Elements of the largest layer's side.
size_t widest() { return (size_t)std::max(g_net.width, 128); }

// The next n elements of the network's one device allocation, from a 256-byte
// boundary on (null while the bytes are only counted).
template <class T>
void take(T*& p, size_t n) {
  p = g_net.arena ? (T*)(g_net.arena + g_net.arena_bytes) : nullptr;
  g_net.arena_bytes += (n * sizeof(T) + 255) / 256 * 256;
}
int loss_parts() { return g_net.nout / 32 * (g_net.batch / kTileRows); }
void lay_out() {
  Net& N = g_net;
  const size_t B = N.batch, W = widest();
  N.arena_bytes = 0;
  for (Layer& y : N.L) {
    const size_t nw = (size_t)y.nin * y.nout, nb = y.nout;
    take(y.w, nw); take(y.b, nb); take(y.mw, nw); take(y.vw, nw); take(y.mb, nb);
    take(y.vb, nb); take(y.gw, nw); take(y.gb, nb); take(y.wb, nw); take(y.wt, nw);
  }
  for (int l = 0; l <= N.depth; ++l) {
    const size_t n = B * (l == 0 ? N.kin : N.width);
    take(N.h[l], n);
    take(N.ht[l], n);
  }
  for (int l = 0; l < N.depth; ++l) take(N.z[l], B * N.width);
  take(N.c_out, B * N.nout);
  take(N.y, B * N.n_out);
  take(N.dh, B * N.width);
  take(N.d, B * W);
  take(N.dt, B * W);
  take(N.scratch, kSplitMax * W * W);
  take(N.cpart, B / kTileRows * W);
  take(N.lpart, (size_t)loss_parts());
  take(N.xb, B * N.n_in);
  take(N.tb, B * N.n_out);
  take(N.status, (size_t)1);
}

void release() {
  cudaFree(g_net.arena);
  cudaFree(g_net.xall);
  cudaFree(g_net.tall);
  cudaFree(g_net.perm[0]);
  cudaFree(g_net.perm[1]);
  g_net = Net{};
}

unsigned cdiv(long a, long b) { return (unsigned)((a + b - 1) / b); }

int transpose(const uint16_t* in, int rows, int cols, uint16_t* out) {
  k_transpose_bf16<<<dim3(cols / 32, rows / 32), dim3(32, 8)>>>(in, rows, cols, out);
  MCK(cudaGetLastError());
  return AERO_OK;
}
int refresh_transposes() {
  for (Layer& l : g_net.L) {
    int rc = transpose(l.wb, l.nout, l.nin, l.wt);
    if (rc) return rc;
  }
  return AERO_OK;
}

// Forward pass of the rows idx[0 .. n) (null: 0 .. n) of x, to c_out (without the
// output layer's bias); with_back also leaves what backward reads.
int forward(const float* x, const int* idx, int n, bool with_back) {
  Net& N = g_net;
  const int B = N.batch;
  int rc, one = 1;
  k_load_inputs<<<cdiv((long)B * N.n_in, 256), 256>>>(x, idx, n, N.n_in, B, N.kin, N.h[0], N.ht[0]);
  MCK(cudaGetLastError());
  for (int l = 0; l < N.depth; ++l) {
    if ((rc = gemm_parts(N.h[l], N.L[l].wb, N.z[l], B, N.width, N.L[l].nin, one, N.status, 0))) return rc;
    k_activate<<<dim3(N.width / 32, B / kTileRows), kTileThreads, kTileSmem>>>(N.z[l], N.L[l].b, B, N.width, N.h[l + 1],
                                                                               with_back ? N.ht[l + 1] : nullptr);
    MCK(cudaGetLastError());
  }
  return gemm_parts(N.h[N.depth], N.L[N.depth].wb, N.c_out, B, N.nout, N.width, one, N.status, 0);
}

// Backward pass of the last forward with the targets t (rows as forward's): the
// loss parts and, layer by layer, the gradients into gw, gb or (train) an Adam
// step with them.
int backward(const float* t, const int* idx, int n, bool train, float lr) {
  Net& N = g_net;
  const int B = N.batch, chunks = B / kTileRows;
  int rc, one = 1;
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  float c1 = 1.f, c2 = 1.f;
  if (train) {
    ++N.adam_t;
    c1 = 1.f - std::pow(b1, (float)N.adam_t);
    c2 = 1.f - std::pow(b2, (float)N.adam_t);
  }
  for (int l = N.depth; l >= 0; --l) {
    Layer& y = N.L[l];
    const dim3 grid(y.nout / 32, chunks);
    if (l == N.depth)
      k_back_output<<<grid, kTileThreads, kTileSmem>>>(N.c_out, y.b, t, idx, n, N.n_out, B, y.nout, 1.0f / ((float)n * (float)N.n_out),
                                     N.d, N.dt, N.cpart, N.lpart);
    else
      k_back_hidden<<<grid, kTileThreads, kTileSmem>>>(N.dh, N.z[l], B, y.nout, N.d, N.dt, N.cpart);
    MCK(cudaGetLastError());
    // the weight gradient and, by this layer's weights before their update, the
    // gradient of the layer below
    int splits = std::min(kSplitMax, B / 512);
    GemmProblem gw, dh;
    if ((rc = gemm_problem(gw, N.dt, N.ht[l], N.scratch, y.nout, y.nin, B, splits))) return rc;
    if (l > 0 && (rc = gemm_problem(dh, N.d, y.wt, N.dh, B, y.nin, y.nout, one))) return rc;
    if ((rc = launch_gemms(gw, dh, N.status, 0))) return rc;
    const LayerParams p{y.w, y.mw, y.vw, y.gw, y.b, y.mb, y.vb, y.gb, y.wb, y.wt, y.nin, y.nout};
    k_update_layer<<<cdiv((long)y.nin * y.nout + y.nout, 256), 256>>>(p, N.scratch, splits, N.cpart, chunks, train,
                                                                     lr, b1, b2, c1, c2, eps);
    MCK(cudaGetLastError());
  }
  return AERO_OK;
}

int check_status() {
  unsigned st = 0;
  MCK(cudaMemcpy(&st, g_net.status, 4, cudaMemcpyDeviceToHost));
  if (st) return set_last_error(AERO_ERR_DEVICE, "warm-start network: a tensor-core wait timed out");
  return AERO_OK;
}

// splitmix64 for reproducible initial weights and batch order
uint64_t mix(uint64_t& s) {
  uint64_t z = (s += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
double unit(uint64_t& s) { return (mix(s) >> 11) * (1.0 / 9007199254740992.0); }

}  // namespace
}  // namespace mlp
}  // namespace aero

// ------------------------------------------------------------------- C ABI
extern "C" {

int aero_mlp_create(int n_in, int n_out, int width, int depth, int batch, unsigned long long seed) {
  using namespace aero::mlp;
  release();
  if (n_in < 1 || n_in > 128 || n_out < 1 || n_out > 128 || width < 128 || width % 128 || width > 1024 ||
      depth < 1 || depth > 32 || batch < 512 || batch % 512)
    return set_last_error(AERO_ERR_ARG,
                          "aero_mlp_create: n_in, n_out in 1..128, width a multiple of 128 up to 1024, depth 1..32, "
                          "batch a multiple of 512");
  Net& N = g_net;
  N.n_in = n_in; N.n_out = n_out; N.width = width; N.depth = depth; N.batch = batch;
  int rc;
  N.L.resize(depth + 1);
  N.h.resize(depth + 1);
  N.ht.resize(depth + 1);
  N.z.resize(depth);
  for (int l = 0; l <= depth; ++l) {
    N.L[l].nin = l == 0 ? N.kin : width;
    N.L[l].nout = l == depth ? N.nout : width;
  }
  lay_out();
  if (cudaMalloc(&N.arena, N.arena_bytes) != cudaSuccess) {
    cudaGetLastError();
    release();
    return set_last_error(AERO_ERR_NOMEM, "warm-start network: device allocation failed");
  }
  MCK(cudaMemset(N.arena, 0, N.arena_bytes));
  lay_out();
  uint64_t s = seed;
  for (int l = 0; l <= depth; ++l) {
    const Layer& y = N.L[l];
    const size_t nw = (size_t)y.nin * y.nout;
    // Glorot-uniform over the real fan-in / fan-out; padded rows/columns stay 0
    int fin = l == 0 ? n_in : width, fout = l == depth ? n_out : width;
    double a = std::sqrt(6.0 / (fin + fout));
    std::vector<float> w(nw, 0.f);
    std::vector<uint16_t> wb(nw, 0);
    for (int r = 0; r < fout; ++r)
      for (int c = 0; c < fin; ++c) {
        float v = (float)((2.0 * unit(s) - 1.0) * a);
        w[(size_t)r * y.nin + c] = v;
      }
    for (size_t i = 0; i < nw; ++i) {  // round to BF16 (nearest even) on the host
      uint32_t u;
      std::memcpy(&u, &w[i], 4);
      u += 0x7FFFu + ((u >> 16) & 1u);
      wb[i] = (uint16_t)(u >> 16);
    }
    MCK(cudaMemcpy(y.w, w.data(), nw * 4, cudaMemcpyHostToDevice));
    MCK(cudaMemcpy(y.wb, wb.data(), nw * 2, cudaMemcpyHostToDevice));
  }
  for (auto k : {(const void*)k_activate, (const void*)k_back_hidden, (const void*)k_back_output})
    MCK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTileSmem));
  if ((rc = refresh_transposes())) return rc;
  MCK(cudaDeviceSynchronize());
  N.ok = true;
  return AERO_OK;
}

int aero_mlp_destroy(void) {
  aero::mlp::release();
  return AERO_OK;
}

int aero_mlp_param_count(long long* count) {
  using namespace aero::mlp;
  if (!g_net.ok) return set_last_error(AERO_ERR_STATE, "aero_mlp_create has not been called");
  long long n = 0;
  for (Layer& l : g_net.L) n += (long long)l.nin * l.nout + l.nout;
  *count = n;
  return AERO_OK;
}

int aero_mlp_get_params(float* out) {
  using namespace aero::mlp;
  if (!g_net.ok) return set_last_error(AERO_ERR_STATE, "aero_mlp_create has not been called");
  for (Layer& l : g_net.L) {
    size_t nw = (size_t)l.nin * l.nout;
    MCK(cudaMemcpy(out, l.w, nw * 4, cudaMemcpyDeviceToHost));
    out += nw;
    MCK(cudaMemcpy(out, l.b, (size_t)l.nout * 4, cudaMemcpyDeviceToHost));
    out += l.nout;
  }
  return AERO_OK;
}

int aero_mlp_gradients(const float* x, const float* t, int n, float* loss, float* grad) {
  using namespace aero::mlp;
  Net& N = g_net;
  if (!N.ok) return set_last_error(AERO_ERR_STATE, "aero_mlp_create has not been called");
  if (n < 1 || n > N.batch) return set_last_error(AERO_ERR_ARG, "aero_mlp_gradients: 1 <= n <= batch");
  MCK(cudaMemcpy(N.xb, x, (size_t)n * N.n_in * 4, cudaMemcpyHostToDevice));
  MCK(cudaMemcpy(N.tb, t, (size_t)n * N.n_out * 4, cudaMemcpyHostToDevice));
  int rc;
  if ((rc = forward(N.xb, nullptr, n, true)) || (rc = backward(N.tb, nullptr, n, false, 0.f))) return rc;
  int np = loss_parts();
  std::vector<float> lp(np);
  MCK(cudaMemcpy(lp.data(), N.lpart, np * 4, cudaMemcpyDeviceToHost));
  double sum = 0;
  for (float v : lp) sum += v;
  *loss = (float)(sum / ((double)n * N.n_out));
  for (Layer& l : N.L) {
    size_t nw = (size_t)l.nin * l.nout;
    MCK(cudaMemcpy(grad, l.gw, nw * 4, cudaMemcpyDeviceToHost));
    grad += nw;
    MCK(cudaMemcpy(grad, l.gb, (size_t)l.nout * 4, cudaMemcpyDeviceToHost));
    grad += l.nout;
  }
  return check_status();
}

int aero_mlp_train(const float* x, const float* t, long long n, int steps, float lr, unsigned long long seed,
                   float* loss_hist) {
  using namespace aero::mlp;
  Net& N = g_net;
  if (!N.ok) return set_last_error(AERO_ERR_STATE, "aero_mlp_create has not been called");
  if (n < N.batch || steps < 1) return set_last_error(AERO_ERR_ARG, "aero_mlp_train: n >= batch and steps >= 1");
  int rc = AERO_OK;
  if (N.n_all != n) {
    cudaFree(N.xall); cudaFree(N.tall); cudaFree(N.perm[0]); cudaFree(N.perm[1]);
    N.xall = N.tall = nullptr;
    N.perm[0] = N.perm[1] = nullptr;
    N.n_all = 0;
    MCK(cudaMalloc(&N.xall, (size_t)n * N.n_in * 4));
    MCK(cudaMalloc(&N.tall, (size_t)n * N.n_out * 4));
    for (int k = 0; k < 2; ++k) MCK(cudaMalloc(&N.perm[k], (size_t)n * sizeof(int)));
    N.n_all = n;
  }
  MCK(cudaMemcpy(N.xall, x, (size_t)n * N.n_in * 4, cudaMemcpyHostToDevice));
  MCK(cudaMemcpy(N.tall, t, (size_t)n * N.n_out * 4, cudaMemcpyHostToDevice));
  float* dhist = nullptr;
  MCK(cudaMalloc(&dhist, (size_t)steps * 4));
  uint64_t s = seed;
  std::vector<int> perm(n);
  for (long long i = 0; i < n; ++i) perm[i] = (int)i;
  long long pos = n;
  // An epoch's row order crosses the bus once, in stream order, into the buffer
  // of the epoch before last, whose steps are over by then; nothing in the loop
  // waits for the device, so the host shuffles and launches ahead of it.
  int epoch = -1;
  for (int step = 0; step < steps && !rc; ++step) {
    if (pos + N.batch > n) {  // new epoch: Fisher-Yates shuffle
      for (long long i = n - 1; i > 0; --i) {
        long long j = (long long)(mix(s) % (uint64_t)(i + 1));
        std::swap(perm[i], perm[j]);
      }
      pos = 0;
      ++epoch;
      if (cudaMemcpyAsync(N.perm[epoch & 1], perm.data(), (size_t)n * sizeof(int), cudaMemcpyHostToDevice, 0) !=
          cudaSuccess) {
        rc = set_last_error(AERO_ERR_CUDA, "aero_mlp_train: copy of the row order failed");
        break;
      }
    }
    const int* idx = N.perm[epoch & 1] + pos;
    pos += N.batch;
    if ((rc = forward(N.xall, idx, N.batch, true)) || (rc = backward(N.tall, idx, N.batch, true, lr))) break;
    k_loss_sum<<<1, 32>>>(N.lpart, loss_parts(), dhist + step);  // sum of squared errors of the step
  }
  if (!rc && cudaDeviceSynchronize() != cudaSuccess) rc = set_last_error(AERO_ERR_CUDA, "aero_mlp_train failed");
  if (!rc && loss_hist) {
    if (cudaMemcpy(loss_hist, dhist, (size_t)steps * 4, cudaMemcpyDeviceToHost) != cudaSuccess)
      rc = set_last_error(AERO_ERR_CUDA, "aero_mlp_train: copy of the loss history failed");
    for (int i = 0; i < steps; ++i) loss_hist[i] /= (float)((double)N.batch * N.n_out);
  }
  cudaFree(dhist);
  if (!rc) rc = check_status();
  return rc;
}

int aero_mlp_predict(const float* x, long long n, float* y) {
  using namespace aero::mlp;
  Net& N = g_net;
  if (!N.ok) return set_last_error(AERO_ERR_STATE, "aero_mlp_create has not been called");
  int rc;
  for (long long r0 = 0; r0 < n; r0 += N.batch) {
    int m = (int)std::min<long long>(N.batch, n - r0);
    MCK(cudaMemcpy(N.xb, x + r0 * N.n_in, (size_t)m * N.n_in * 4, cudaMemcpyHostToDevice));
    if ((rc = forward(N.xb, nullptr, m, false))) return rc;
    k_outputs<<<cdiv((long)m * N.n_out, 256), 256>>>(N.c_out, N.L[N.depth].b, m, N.n_out, N.nout, N.y);
    MCK(cudaGetLastError());
    MCK(cudaMemcpy(y + r0 * N.n_out, N.y, (size_t)m * N.n_out * 4, cudaMemcpyDeviceToHost));
  }
  return check_status();
}

}  // extern "C"
