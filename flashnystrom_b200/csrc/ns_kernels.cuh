// Newton-Schulz pseudoinverse, forward and exact backward, entirely in shared memory (FP32, CUDA
// cores, no cuBLAS) for num_landmarks <= 64.  One CTA of 256 threads per (b,h) slice; every
// (m x m) matrix lives in a zero-padded 64 x 64 shared buffer with row stride 68, so all loops
// have compile-time bounds and every operand access is a conflict-free 16-byte load.
// Larger landmark counts use mid_tc.cuh (mid_kernels.cuh on the CUDA cores).
#pragma once
#include "common.cuh"
#include "mid_kernels.cuh"

namespace fnb {
namespace ns {

constexpr int kN = 64;          // padded matrix size
constexpr int kLd = 68;         // row stride (floats): 16-byte aligned rows, rows 8 apart hit distinct banks
constexpr int kBuf = kN * kLd;  // floats per buffer

enum { NN = 0, NT = 1, TN = 2 };

// Barrier over the 256 threads that run the code of this file.  In the kernels of this file that
// is the whole CTA; the tensor-core kernels add a ninth warp that only issues MMAs and must not
// be counted, so a named barrier is used instead of __syncthreads().
__device__ __forceinline__ void ns_sync() { asm volatile("bar.sync 7, 256;" ::: "memory"); }

// C-tile of this thread for op(A) * op(B), all operands 64 x 64 in shared memory.
//   NN: C = A B      rows ty+16i, cols 4tx+j
//   NT: C = A B^T    rows ty+16i, cols tx+16j
//   TN: C = A^T B    rows 4ty+i,  cols 4tx+j
// epi(r, c, acc) is called once per owned element after a barrier, so outputs may alias inputs;
// a second barrier follows the stores.
// Packed FP32 FMA (two independent IEEE fused multiply-adds per instruction on sm_100).
__device__ __forceinline__ void fma2(float2& acc, float a, float2 b) {
  acc = __ffma2_rn(make_float2(a, a), b, acc);
}
__device__ __forceinline__ void fma2v(float2& acc, float2 a, float2 b) { acc = __ffma2_rn(a, b, acc); }

template <int MODE, class Epi>
__device__ __forceinline__ void mm(const float* __restrict__ A, const float* __restrict__ B, Epi epi) {
  const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
  // NN / TN: acc[i][0] = columns (0,1), acc[i][1] = columns (2,3) of the 4x4 tile.
  // NT: acc[i][j] holds the even-k and odd-k partial sums of element (i, j).
  float2 acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
  if (MODE == NN) {
#pragma unroll 4
    for (int k = 0; k < kN; k += 4) {
      float4 a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(A + (ty + 16 * i) * kLd + k);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) b[kk] = *reinterpret_cast<const float4*>(B + (k + kk) * kLd + 4 * tx);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float av[4] = {a[i].x, a[i].y, a[i].z, a[i].w};
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          fma2(acc[i][0], av[kk], make_float2(b[kk].x, b[kk].y));
          fma2(acc[i][1], av[kk], make_float2(b[kk].z, b[kk].w));
        }
      }
    }
  } else if (MODE == NT) {
#pragma unroll 4
    for (int k = 0; k < kN; k += 4) {
      float4 a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(A + (ty + 16 * i) * kLd + k);
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(B + (tx + 16 * j) * kLd + k);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          fma2v(acc[i][j], make_float2(a[i].x, a[i].y), make_float2(b[j].x, b[j].y));
          fma2v(acc[i][j], make_float2(a[i].z, a[i].w), make_float2(b[j].z, b[j].w));
        }
    }
  } else {
#pragma unroll 8
    for (int k = 0; k < kN; ++k) {
      const float4 a = *reinterpret_cast<const float4*>(A + k * kLd + 4 * ty);
      const float4 b = *reinterpret_cast<const float4*>(B + k * kLd + 4 * tx);
      const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        fma2(acc[i][0], av[i], make_float2(b.x, b.y));
        fma2(acc[i][1], av[i], make_float2(b.z, b.w));
      }
    }
  }
  ns_sync();
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int r = (MODE == TN) ? 4 * ty + i : ty + 16 * i;
      const int c = (MODE == NT) ? tx + 16 * j : 4 * tx + j;
      float val;
      if (MODE == NT) val = acc[i][j].x + acc[i][j].y;
      else val = (j & 1) ? acc[i][j >> 1].y : acc[i][j >> 1].x;
      epi(r, c, val);
    }
  ns_sync();
}

__device__ __forceinline__ void zero_buf(float* X) {
  for (int idx = threadIdx.x; idx < kBuf; idx += kThreads) X[idx] = 0.f;
}
// global (m x m, dense) -> padded shared buffer
__device__ __forceinline__ void load_mat(float* X, const float* g, int m) {
  for (int idx = threadIdx.x; idx < kN * kN; idx += kThreads) {
    int r = idx >> 6, c = idx & 63;
    X[r * kLd + c] = (r < m && c < m) ? g[r * m + c] : 0.f;
  }
}
__device__ __forceinline__ void store_mat(float* g, const float* X, int m) {
  for (int idx = threadIdx.x; idx < m * m; idx += kThreads) {
    int r = idx / m, c = idx - r * m;
    g[idx] = X[r * kLd + c];
  }
}

struct Norms { float n1, ninf; int jc, ir; };
constexpr int kRedFloats = 6 * kN;   // shared scratch of norms()
// Max column / row abs-sum of the padded buffer X (zero outside the leading m x m block) with
// first-occurrence argmax.  All 256 threads take part; red: kRedFloats floats of shared scratch.
__device__ inline Norms norms(const float* X, int m, float* red) {
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  {
    // row sums: thread = (row, 16-column quarter); the four quarters sit in adjacent lanes
    const int r = t >> 2, q = t & 3;
    float rs = 0.f;
#pragma unroll
    for (int i = 0; i < 16; i += 4) {
      const float4 x = *reinterpret_cast<const float4*>(X + r * kLd + 16 * q + i);
      rs += fabsf(x.x) + fabsf(x.y) + fabsf(x.z) + fabsf(x.w);
    }
    rs += __shfl_xor_sync(0xffffffffu, rs, 1);
    rs += __shfl_xor_sync(0xffffffffu, rs, 2);
    if (q == 0) red[kN + r] = rs;
    // column sums: thread = (column, 16-row block), partial sums combined below
    const int c = t & 63, blk = t >> 6;
    float cs = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) cs += fabsf(X[(16 * blk + i) * kLd + c]);
    red[2 * kN + blk * kN + c] = cs;
  }
  ns_sync();
  if (w < 2) {
    // warp 0: columns, warp 1: rows; each lane owns entries lane and lane + 32
    float v0, v1;
    if (w == 0) {
      v0 = red[2 * kN + lane] + red[3 * kN + lane] + red[4 * kN + lane] + red[5 * kN + lane];
      v1 = red[2 * kN + lane + 32] + red[3 * kN + lane + 32] + red[4 * kN + lane + 32] + red[5 * kN + lane + 32];
    } else {
      v0 = red[kN + lane];
      v1 = red[kN + lane + 32];
    }
    float best = (lane < m) ? v0 : -1.f;
    int bi = lane;
    if (lane + 32 < m && v1 > best) { best = v1; bi = lane + 32; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    if (lane == 0) { red[2 * w] = best; red[2 * w + 1] = __int_as_float(bi); }
  }
  ns_sync();
  Norms out;
  out.n1 = red[0]; out.jc = __float_as_int(red[1]);
  out.ninf = red[2]; out.ir = __float_as_int(red[3]);
  ns_sync();
  return out;
}

constexpr int kFwdBufs = 7;
constexpr size_t kFwdSmem = (size_t)kFwdBufs * kBuf * sizeof(float) + 1024;

// K2 (in shared buffer bK2, already softmaxed, padded) -> iterates / k2inv in global memory.
__device__ inline void pinv_forward_smem(float* sm, float* red, float* iterates, float* k2inv, int m, int J,
                                         float kappa) {
  float* bK2 = sm;
  float* bA = sm + 1 * kBuf;
  float* bZ = sm + 2 * kBuf;
  float* bM = sm + 3 * kBuf;
  float* bU = sm + 4 * kBuf;
  float* bV = sm + 5 * kBuf;
  float* bT = sm + 6 * kBuf;
  const int mm_ = m * m;
  const float* A = bK2;
  if (kappa > 0.f) {
    Norms nk = norms(bK2, m, red);
    const float lam = nk.n1 * nk.ninf / kappa;
    mm<TN>(bK2, bK2, [&](int r, int c, float acc) { bA[r * kLd + c] = acc + ((r == c && r < m) ? lam : 0.f); });
    A = bA;
  }
  Norms na = norms(A, m, red);
  const float cden = fmaxf(na.n1 * na.ninf, 1e-12f);
  for (int idx = threadIdx.x; idx < kN * kN; idx += kThreads) {
    int r = idx >> 6, c = idx & 63;
    float z = A[c * kLd + r] / cden;
    bZ[r * kLd + c] = z;
    if (r < m && c < m) iterates[r * m + c] = z;
  }
  ns_sync();
  for (int j = 0; j < J; ++j) {
    float* Zn = iterates + (size_t)(j + 1) * mm_;
    mm<NN>(A, bZ, [&](int r, int c, float acc) {
      bM[r * kLd + c] = acc;
      bU[r * kLd + c] = ((r == c && r < m) ? 7.f : 0.f) - acc;
    });
    mm<NN>(bM, bU, [&](int r, int c, float acc) { bV[r * kLd + c] = ((r == c && r < m) ? 15.f : 0.f) - acc; });
    mm<NN>(bM, bV, [&](int r, int c, float acc) { bT[r * kLd + c] = ((r == c && r < m) ? 13.f : 0.f) - acc; });
    mm<NN>(bZ, bT, [&](int r, int c, float acc) {
      const float z = 0.25f * acc;
      bZ[r * kLd + c] = z;
      if (r < m && c < m) Zn[r * m + c] = z;
    });
  }
  if (kappa > 0.f) {
    mm<NT>(bZ, bK2, [&](int r, int c, float acc) { if (r < m && c < m) k2inv[r * m + c] = acc; });
  } else {
    store_mat(k2inv, bZ, m);
    ns_sync();
  }
}

// ------------------------------------------------------------------------------------------
// Forward: S2 = Qt Kt^T, softmax (K2, lse2), pseudoinverse.
struct NsFwdParams {
  const float* qt; const float* kt;         // [BH][m][D] (scaled landmarks)
  float* k2; float* lse2; float* iterates; float* k2inv;
  int m, D, J;
  float kappa;
  // Optional (tensor-core kernel, head_dim 64): form the landmarks here from the raw segment sums
  // of the pooling pass, land [2][BH][m][C][D], and write them to qt_out / kt_out.
  const float* land; int C; int64_t BH; int64_t seg_N; float scale;
  float* qt_out; float* kt_out;
};

__device__ inline void softmax_rows(float* bK2, const NsFwdParams& p, int64_t bh);

// S2 = Qt Kt^T straight from global memory, row softmax -> K2 (padded, in bK2 and in global), lse2.
__device__ inline void s2_softmax(float* bK2, const NsFwdParams& p, int64_t bh) {
  const int m = p.m, D = p.D, t = threadIdx.x, tx = t & 15, ty = t >> 4;
  const float* qt = p.qt + bh * m * D;
  const float* kt = p.kt + bh * m * D;
  // S2 tile straight from global (L2): rows ty+16i, cols tx+16j
  {
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    for (int d = 0; d < D; d += 4) {
      float4 a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = ty + 16 * i;
        a[i] = (r < m) ? *reinterpret_cast<const float4*>(qt + r * D + d) : make_float4(0, 0, 0, 0);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = tx + 16 * j;
        b[j] = (c < m) ? *reinterpret_cast<const float4*>(kt + c * D + d) : make_float4(0, 0, 0, 0);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          acc[i][j] += a[i].x * b[j].x + a[i].y * b[j].y + a[i].z * b[j].z + a[i].w * b[j].w;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) bK2[(ty + 16 * i) * kLd + tx + 16 * j] = acc[i][j];
  }
  ns_sync();
  softmax_rows(bK2, p, bh);
}

// Row softmax of the scores in bK2 (one warp per row; padded rows / columns become zero)
// -> K2 in bK2 and in global memory, lse2.
__device__ inline void softmax_rows(float* bK2, const NsFwdParams& p, int64_t bh) {
  const int m = p.m, t = threadIdx.x;
  const int w = t >> 5, lane = t & 31;
  float* k2g = p.k2 + bh * m * m;
  for (int r = w; r < kN; r += kThreads / 32) {
    float v0 = (r < m && lane < m) ? bK2[r * kLd + lane] : -INFINITY;
    float v1 = (r < m && lane + 32 < m) ? bK2[r * kLd + lane + 32] : -INFINITY;
    float mx = fmaxf(v0, v1);
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float e0 = (r < m && lane < m) ? expf(v0 - mx) : 0.f;
    float e1 = (r < m && lane + 32 < m) ? expf(v1 - mx) : 0.f;
    float sum = e0 + e1;
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float p0 = (r < m) ? e0 / sum : 0.f, p1 = (r < m) ? e1 / sum : 0.f;
    bK2[r * kLd + lane] = p0;
    bK2[r * kLd + lane + 32] = p1;
    if (r < m) {
      if (lane < m) k2g[r * m + lane] = p0;
      if (lane + 32 < m) k2g[r * m + lane + 32] = p1;
      if (lane == 0) p.lse2[bh * m + r] = mx + logf(sum);
    }
  }
  ns_sync();
}

__global__ void __launch_bounds__(kThreads, 1) ns_fwd_kernel(NsFwdParams p) {
  extern __shared__ float sm[];
  __shared__ float red[kRedFloats];
  const int64_t bh = blockIdx.x;
  const int m = p.m;
  s2_softmax(sm, p, bh);
  pinv_forward_smem(sm, red, p.iterates + bh * (size_t)(p.J + 1) * m * m, p.k2inv + bh * m * m, m, p.J,
                    p.kappa);
}

__global__ void __launch_bounds__(kThreads, 1)
ns_pinv_fwd_debug_kernel(const float* k2, float* iterates, float* k2inv, int m, int J, float kappa) {
  extern __shared__ float sm[];
  __shared__ float red[kRedFloats];
  const int64_t bh = blockIdx.x;
  load_mat(sm, k2 + bh * m * m, m);
  ns_sync();
  pinv_forward_smem(sm, red, iterates + bh * (size_t)(J + 1) * m * m, k2inv + bh * m * m, m, J, kappa);
}

// ------------------------------------------------------------------------------------------
constexpr int kBwdBufs = 12;
constexpr size_t kBwdSmem = (size_t)kBwdBufs * kBuf * sizeof(float) + 1024;

// Tail of the pseudoinverse backward, shared by the CUDA-core and the tensor-core loop: gradient
// through Z0 = A^T / (||A||_1 ||A||_inf) (norm terms at the first-occurrence argmax), then through
// the ridge wrap.  In: bdZ = dL/dZ_0, bdA = dL/dA accumulated over the iterations.  Out: dK2 in bdA.
// bdM, bdT: scratch buffers.
__device__ inline float* pinv_backward_tail(const float* bK2, const float* A, float* bdZ, float* bdA, float* bdM,
                                            float* bdT, float* red, const float* spill, int m, float kappa) {
  // Z0 = A^T / c,  c = ||A||_1 ||A||_inf
  Norms na = norms(A, m, red);
  const float craw = na.n1 * na.ninf;
  const float cden = fmaxf(craw, 1e-12f);
  float part = 0.f;
  for (int idx = threadIdx.x; idx < kN * kN; idx += kThreads) {
    int a = idx >> 6, b = idx & 63;
    part += bdZ[a * kLd + b] * A[b * kLd + a];
  }
  for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = part;
  ns_sync();
  float S = 0.f;
  for (int w = 0; w < kThreads / 32; ++w) S += red[w];
  ns_sync();
  const bool clamped = !(craw > 1e-12f);
  const float col_term = clamped ? 0.f : -S * na.ninf / (cden * cden);
  const float row_term = clamped ? 0.f : -S * na.n1 / (cden * cden);
  for (int idx = threadIdx.x; idx < kN * kN; idx += kThreads) {
    int r = idx >> 6, c = idx & 63;
    if (r < m && c < m) {
      const float a = A[r * kLd + c];
      const float sg = a > 0.f ? 1.f : (a < 0.f ? -1.f : 0.f);
      float g = bdA[r * kLd + c] + bdZ[c * kLd + r] / cden;
      if (c == na.jc) g += sg * col_term;
      if (r == na.ir) g += sg * row_term;
      bdM[r * kLd + c] = g;              // dA complete (staged in bdM to avoid the transpose hazard)
    } else {
      bdM[r * kLd + c] = 0.f;
    }
  }
  ns_sync();
  if (kappa > 0.f) {
    // dK2 = dK2_a + K2 (dA + dA^T)
    for (int idx = threadIdx.x; idx < kN * kN; idx += kThreads) {
      int r = idx >> 6, c = idx & 63;
      bdT[r * kLd + c] = bdM[r * kLd + c] + bdM[c * kLd + r];
    }
    ns_sync();
    mm<NN>(bK2, bdT, [&](int r, int c, float acc) {
      bdA[r * kLd + c] = (r < m && c < m) ? acc + spill[r * m + c] : 0.f;
    });
  } else {
    for (int idx = threadIdx.x; idx < kBuf; idx += kThreads) bdA[idx] = bdM[idx];
    ns_sync();
  }
  return bdA;
}

// G = dL/d k2inv (global) -> dK2 = dL/d K2 left in shared buffer bdA (returned pointer).
// spill: (m x m) floats of global scratch, used only with the ridge.
__device__ inline float* pinv_backward_smem(float* sm, float* red, const float* k2g, const float* iterates,
                                            const float* G, float* spill, int m, int J, float kappa) {
  float* bK2 = sm;
  float* bA = sm + 1 * kBuf;
  float* bZ = sm + 2 * kBuf;
  float* bM = sm + 3 * kBuf;
  float* bU = sm + 4 * kBuf;
  float* bV = sm + 5 * kBuf;
  float* bT = sm + 6 * kBuf;     // T, then dZ_outer
  float* bdZ = sm + 7 * kBuf;
  float* bdT = sm + 8 * kBuf;
  float* bdV = sm + 9 * kBuf;
  float* bdM = sm + 10 * kBuf;
  float* bdA = sm + 11 * kBuf;
  const int mm_ = m * m;
  load_mat(bK2, k2g, m);
  load_mat(bdZ, G, m);          // holds G until dZ_J is formed
  zero_buf(bdA);
  ns_sync();
  const float* A = bK2;
  if (kappa > 0.f) {
    Norms nk = norms(bK2, m, red);
    const float lam = nk.n1 * nk.ninf / kappa;
    mm<TN>(bK2, bK2, [&](int r, int c, float acc) { bA[r * kLd + c] = acc + ((r == c && r < m) ? lam : 0.f); });
    A = bA;
    load_mat(bZ, iterates + (size_t)J * mm_, m);
    ns_sync();
    // dK2_a = G^T Z_J -> global spill; dZ_J = G K2
    mm<TN>(bdZ, bZ, [&](int r, int c, float acc) { if (r < m && c < m) spill[r * m + c] = acc; });
    mm<NN>(bdZ, bK2, [&](int r, int c, float acc) { bdZ[r * kLd + c] = acc; });
  }
  for (int j = J - 1; j >= 0; --j) {
    load_mat(bZ, iterates + (size_t)j * mm_, m);
    ns_sync();
    mm<NN>(A, bZ, [&](int r, int c, float acc) {
      bM[r * kLd + c] = acc;
      bU[r * kLd + c] = ((r == c && r < m) ? 7.f : 0.f) - acc;
    });
    mm<NN>(bM, bU, [&](int r, int c, float acc) { bV[r * kLd + c] = ((r == c && r < m) ? 15.f : 0.f) - acc; });
    mm<NN>(bM, bV, [&](int r, int c, float acc) { bT[r * kLd + c] = ((r == c && r < m) ? 13.f : 0.f) - acc; });
    mm<TN>(bZ, bdZ, [&](int r, int c, float acc) { bdT[r * kLd + c] = 0.25f * acc; });           // dT = Z^T dZ / 4
    mm<NT>(bdZ, bT, [&](int r, int c, float acc) { bT[r * kLd + c] = 0.25f * acc; });            // dZ_outer
    mm<NT>(bdT, bV, [&](int r, int c, float acc) { bdM[r * kLd + c] = -acc; });                  // -dT V^T
    mm<TN>(bM, bdT, [&](int r, int c, float acc) { bdV[r * kLd + c] = -acc; });                  // dV = -M^T dT
    mm<NT>(bdV, bU, [&](int r, int c, float acc) { bdM[r * kLd + c] -= acc; });                  // -= dV U^T
    mm<TN>(bM, bdV, [&](int r, int c, float acc) { bdM[r * kLd + c] += acc; });                  // += M^T dV
    mm<NT>(bdM, bZ, [&](int r, int c, float acc) { bdA[r * kLd + c] += acc; });                  // dA += dM Z^T
    mm<TN>(A, bdM, [&](int r, int c, float acc) { bdZ[r * kLd + c] = bT[r * kLd + c] + acc; });  // dZ_outer + A^T dM
  }
  return pinv_backward_tail(bK2, A, bdZ, bdA, bdM, bdT, red, spill, m, kappa);
}

__global__ void __launch_bounds__(kThreads, 1)
ns_pinv_bwd_debug_kernel(const float* k2, const float* iterates, const float* G, float* dK2, float* spill,
                         int m, int J, float kappa) {
  extern __shared__ float sm[];
  __shared__ float red[kRedFloats];
  const int64_t bh = blockIdx.x;
  float* out = pinv_backward_smem(sm, red, k2 + bh * m * m, iterates + bh * (size_t)(J + 1) * m * m,
                                  G + bh * m * m, spill + bh * m * m, m, J, kappa);
  store_mat(dK2 + bh * m * m, out, m);
}

// Backward middle stage 2: pseudoinverse backward, softmax-2 Jacobian, landmark gradients.
struct NsBwdParams {
  const float* k2; const float* iterates; const float* G;   // G = dK2inv [BH][m][m]
  const float* qt; const float* kt; const float* dkt_a;     // [BH][m][D]
  float* dqt_ns; float* dkt_tot;                            // [BH][m][D]
  float* spill;                                             // [BH][m][m]
  float* rows_k;                                            // optional [BH][m][D]: scale * dkt_tot / len
  int64_t N;
  float scale;
  int m, D, J;
  float kappa;
};

// After the pseudoinverse backward: softmax-2 Jacobian and the landmark gradients.
// bK2: K2 (padded shared buffer); dK2: dL/dK2 (padded shared buffer, overwritten with dS2).
__device__ inline void ns_bwd_finish(const NsBwdParams& p, int64_t bh, const float* bK2, float* dK2) {
  const int m = p.m, D = p.D, t = threadIdx.x, md = m * D;
  // softmax-2 Jacobian in place: dS2 = K2 o (dK2 - rowsum(dK2 o K2))
  const int w = t >> 5, lane = t & 31;
  for (int r = w; r < kN; r += kThreads / 32) {
    float a0 = dK2[r * kLd + lane], a1 = dK2[r * kLd + lane + 32];
    float k0 = bK2[r * kLd + lane], k1 = bK2[r * kLd + lane + 32];
    float s = a0 * k0 + a1 * k1;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    dK2[r * kLd + lane] = k0 * (a0 - s);
    dK2[r * kLd + lane + 32] = k1 * (a1 - s);
  }
  ns_sync();
  // dqt_ns = dS2 Kt ; dkt_tot = dkt_a + dS2^T Qt.  Thread owns 4 consecutive d of one landmark row.
  const float* kt = p.kt + bh * md;
  const float* qt = p.qt + bh * md;
  const float* dkt_a = p.dkt_a + bh * md;
  float* dqt_ns = p.dqt_ns + bh * md;
  float* dkt_tot = p.dkt_tot + bh * md;
  const int vec_per_row = D >> 2;
  for (int v = t; v < m * vec_per_row; v += kThreads) {
    const int l = v / vec_per_row, d = (v - l * vec_per_row) << 2;
    float4 a = make_float4(0, 0, 0, 0);
    float4 b = *reinterpret_cast<const float4*>(dkt_a + l * D + d);
    for (int k = 0; k < m; ++k) {
      const float s1 = dK2[l * kLd + k];     // dS2[l][k]
      const float s2 = dK2[k * kLd + l];     // dS2[k][l]
      const float4 kv = *reinterpret_cast<const float4*>(kt + k * D + d);
      const float4 qv = *reinterpret_cast<const float4*>(qt + k * D + d);
      a.x = fmaf(s1, kv.x, a.x); a.y = fmaf(s1, kv.y, a.y); a.z = fmaf(s1, kv.z, a.z); a.w = fmaf(s1, kv.w, a.w);
      b.x = fmaf(s2, qv.x, b.x); b.y = fmaf(s2, qv.y, b.y); b.z = fmaf(s2, qv.z, b.z); b.w = fmaf(s2, qv.w, b.w);
    }
    *reinterpret_cast<float4*>(dqt_ns + l * D + d) = a;
    *reinterpret_cast<float4*>(dkt_tot + l * D + d) = b;
    if (p.rows_k) {
      Segments sg(p.N, m);
      const float f = p.scale / (float)sg.len(l);
      *reinterpret_cast<float4*>(p.rows_k + bh * md + l * D + d) = make_float4(b.x * f, b.y * f, b.z * f, b.w * f);
    }
  }
}


__global__ void __launch_bounds__(kThreads, 1) ns_bwd_kernel(NsBwdParams p) {
  extern __shared__ float sm[];
  __shared__ float red[kRedFloats];
  const int64_t bh = blockIdx.x;
  const int m = p.m, mm_ = m * m;
  float* dK2 = pinv_backward_smem(sm, red, p.k2 + bh * mm_, p.iterates + bh * (size_t)(p.J + 1) * mm_,
                                  p.G + bh * mm_, p.spill + bh * mm_, m, p.J, p.kappa);
  ns_bwd_finish(p, bh, sm, dK2);
}

// Isolation hook for the tail of the backward (the role of the reference's debug_ns_bwd_final,
// csrc/flash_nystrom.cu:474-520, without the ridge): from dL/dZ_0 and the dL/dK2 accumulated over the
// iterations to the complete dL/dK2 (Z0 = K2^T / (||K2||_1 ||K2||_inf) with its norm terms), then
// through the softmax-2 Jacobian to the landmark gradients dQt = dS2 Kt, dKt = dS2^T Qt.
// zeros: [m][D] floats of zeros (stands in for the softmax-1 contribution the product path adds).
__global__ void __launch_bounds__(kThreads, 1)
ns_bwd_final_debug_kernel(const float* qt, const float* kt, const float* k2, const float* dz0, const float* dk2_in,
                          const float* zeros, float* dqt, float* dkt, float* dk2_out, int m, int D) {
  extern __shared__ float sm[];
  __shared__ float red[kRedFloats];
  const int64_t bh = blockIdx.x;
  const int mm_ = m * m;
  float* bK2 = sm;
  float* bdZ = sm + 1 * kBuf;
  float* bdA = sm + 2 * kBuf;
  float* bdM = sm + 3 * kBuf;
  float* bdT = sm + 4 * kBuf;
  load_mat(bK2, k2 + bh * mm_, m);
  load_mat(bdZ, dz0 + bh * mm_, m);
  load_mat(bdA, dk2_in + bh * mm_, m);
  ns_sync();
  float* dK2 = pinv_backward_tail(bK2, bK2, bdZ, bdA, bdM, bdT, red, nullptr, m, 0.f);
  store_mat(dk2_out + bh * mm_, dK2, m);
  ns_sync();
  NsBwdParams p;
  p.k2 = k2; p.iterates = nullptr; p.G = nullptr; p.qt = qt; p.kt = kt; p.dkt_a = zeros - bh * (int64_t)m * D;
  p.dqt_ns = dqt; p.dkt_tot = dkt; p.spill = nullptr; p.rows_k = nullptr; p.N = m; p.scale = 1.f;
  p.m = m; p.D = D; p.J = 0; p.kappa = 0.f;
  ns_bwd_finish(p, bh, bK2, dK2);
}

}  // namespace ns
}  // namespace fnb
