// Newton-Schulz pseudoinverse on the sm_100a tensor cores with FP32-equivalent arithmetic (up to 64 landmarks).
//
// Arithmetic.  The iteration Z' = Z (13 I - M (15 I - M (7 I - M))) / 4, M = A Z, is run in its residual form: with
// R = I - M the polynomial is 4 (I + R (I + R / 2)^2), so
//     R = I - A Z,   Y = Z R,   W = I + R + R^2 / 4,   Z' = Z + Y W.
// That is four products as before, but three dependent steps in place of four (Y and W go side by side), and
// nothing cancels near convergence: the error of K2inv against 64 bits is 0.57 to 1.04 times the nested form's,
// 0.79 in the mean (16 to 128 landmarks, J = 4 to 8, three ridges).  The backward is that of this form (below); gradients do not depend on which form is differentiated.
//
// Products.  Every 64 x 64 FP32 matrix is kept in shared memory as three bf16 tiles x = x0 + x1 + x2 (each term the
// bf16 rounding of what the previous terms left over: 24 significant bits together, the FP32 exponent range), stored in
// the order (x1, x0, x2) so that (x1, x0) and (x0, x2) are both contiguous.  A product needs the partial products x_i y_j with
// i + j <= 2 (the others are below 2^-24 relative).  The terms are stacked along M and N, two MMAs of 128 x 128 per
// 16-wide K step into the SAME 128 accumulator columns:
//     [x1; x0] * [y1 | y0], then [x0; x2] * [y0 | y2]
//     lanes  0..63:  columns 0..63 = x1 y1 + x0 y0,  columns 64..127 = x1 y0 + x0 y2
//     lanes 64..127: columns 0..63 = x0 y1 + x2 y0,  columns 64..127 = not used (x0 y0 once more)
// All K steps of the first pair come first, so the leading partial product is added to four times, onto a
// small value.  An epilogue thread reads 32 (lanes 64..127) or 64 columns, and the two lane halves are added through
// shared memory between partner warps.  The tiles use the 128-byte swizzle ([64 rows x 128 B]); a matrix stored row-major
// serves as either operand, plain or transposed, through the K-major or the MN-major descriptor.
//
// Roles.  One CTA per (b,h) slice: 8 compute warps and a ninth warp that issues the MMAs (warp-uniform code, one elected lane;
// with a single lane in the role every descriptor went through vector registers and the kernels were slower than
// what they replaced).  After the
// exchange every compute thread owns 16 consecutive columns of one row, applies the step's affine map and writes
// the next operand tiles, then arrives on a "ready" mbarrier that the issuing thread waits on; groups of MMAs are
// committed to "done" mbarriers.  A wait that gives up (bounded, 1.5 s) marks the call failed in the status word;
// control flow never depends on it, so no barrier is missed.
//
// With m <= 48 the K steps past m are left out, with m <= 32 also the epilogues of the warps whose 32 x 32 block is empty:
// what lies there in the tiles is never read.
//
// What bounds it: the latency of a step (issue and eight MMAs about 1000 cycles, accumulator out, lane halves added, split and
// stored about 1000), three of them per iteration in the forward; in the backward, where eight products run beside the
// chain, shared-memory bandwidth (an MMA reads 8 KB per 65 cycles, an epilogue moves 56 KB).  Instructions come from a cold
// cache the first time round: 5 us of the forward, 15 of the backward.  Measured (us, nested form with one accumulator per
// partial product / this, J = 6): 32 slices, m = 64 forward 45 / 43, backward 76 / 66; m = 32 43 / 33 and 66 / 48;
// 512 slices 162 / 107 and 310 / 275; 64 slices of head_dim 128 with the ridge (then on the CUDA cores) 74 / 50 and 121 / 86.
#pragma once
#include "ns_kernels.cuh"
#include "small_kernels.cuh"
#include "tc_common.cuh"

namespace fnb {
namespace nstc {

using namespace tc;
using ns::kBuf;
using ns::kLd;
using ns::kN;
using ns::Norms;

constexpr int kTileBytes = kN * 128;        // one bf16 term of a matrix
constexpr int kSet = 3 * kTileBytes;        // the three terms of a matrix, order (x1, x0, x2)
constexpr int kTerm0 = kTileBytes, kTerm1 = 0, kTerm2 = 2 * kTileBytes;
constexpr int kFwdSlots = 4, kBwdSlots = 9;
constexpr size_t kFwdSmem = (size_t)kFwdSlots * kSet + 1024;   // 97 KB: two slices per SM
constexpr size_t kBwdSmem = (size_t)kBwdSlots * kSet + 1024;
static_assert(kBuf * (int)sizeof(float) <= kSet, "an FP32 staging buffer has to fit a slot");
constexpr uint32_t kAccCols = 128;
constexpr uint32_t kFwdTmemCols = 2 * kAccCols, kBwdTmemCols = 4 * kAccCols;
constexpr int kMaxBars = 8;

constexpr int kComputeThreads = 256;
constexpr int kNsTcThreads = kComputeThreads + 32;
__device__ __forceinline__ bool is_compute() { return threadIdx.x < kComputeThreads; }

struct Shared {
  uint64_t done[kMaxBars];    // MMA groups complete (issuing warp -> compute warps)
  uint64_t ready[kMaxBars];   // operand tiles written, accumulators read (one arrival per compute warp -> issuing warp)
  uint32_t tmem_slot;
  int abort_word;
};

struct Ctx {
  uint8_t* base;        // 1024-byte aligned start of the tile slots
  uint32_t smem;        // the same as a shared-memory address
  Shared* sh;
  uint32_t parity;      // bit b: parity of the next wait on done[b] (compute) or ready[b] (issuer)
  bool failed;          // a wait of this thread gave up
  uint32_t tmem;        // base address of the allocated tensor memory
  Abort ab;
  // epilogue role of this thread: TMEM lane 32 * quarter + lane holds row `row` of the lane half `part`; after
  // the exchange the thread owns columns col0 .. col0 + 15 of that row
  int row, part, col0, c32, pair_bar;
  uint32_t lane_addr;   // TMEM offset of the thread's 32 columns
  float trunc;          // see fetch()
  bool mm16, md16;      // (m x m) (forward), (m x head_dim) matrices go sixteen bytes at a time
  bool act;             // this warp's 32 x 32 block of an m x m matrix has something in it (it is never read otherwise)
  __device__ __forceinline__ uint32_t slot(int i) const { return smem + i * kSet; }
  __device__ __forceinline__ float* stage(int i) const { return reinterpret_cast<float*>(base + i * kSet); }
};

// common set-up / teardown of the kernels below (called by all 288 threads)
__device__ __forceinline__ void ctx_open(Ctx& c, Shared& sh, uint8_t* dyn, int* status, uint32_t cols, int m) {
  c.base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(dyn) + 1023) & ~(uintptr_t)1023);
  c.smem = smem_u32(c.base);
  c.sh = &sh;
  c.parity = 0;
  c.failed = false;
  c.ab.flag = &sh.abort_word;
  c.ab.status = status;
  const int warp = (threadIdx.x >> 5) & 7, lane = threadIdx.x & 31, quarter = warp & 3, half = warp >> 2;
  c.part = quarter >> 1;
  c.row = (quarter & 1) * 32 + lane;
  c.c32 = half * 32;
  c.col0 = c.c32 + 16 * c.part;
  c.pair_bar = 1 + (quarter & 1) + 2 * half;      // warps w and w ^ 2 share a barrier
  c.lane_addr = ((uint32_t)(quarter * 32) << 16) + (uint32_t)c.c32;
  c.act = (quarter & 1) * 32 < m && c.c32 < m;
  c.trunc = (float)((m + 15) / 16) * 0x1p-26f;
  if (threadIdx.x == 0) {
    sh.abort_word = 0;
    for (int i = 0; i < kMaxBars; ++i) {
      mbar_init(&sh.done[i], 1);
      mbar_init(&sh.ready[i], kComputeThreads / 32);
    }
    fence_mbar_init();
  }
  if (threadIdx.x < 32) {
    tmem_alloc(&sh.tmem_slot, cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  c.tmem = sh.tmem_slot;
}
__device__ __forceinline__ void ctx_close(Ctx& c, uint32_t cols) {
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x < 32) tmem_dealloc(c.tmem, cols);
}

// ---- FP32 <-> three bf16 terms ---------------------------------------------------------------
// (Shared memory is accessed by 32-bit addresses: the slots are picked at run time, and generic accesses cost more.)
__device__ __forceinline__ void sts128(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
// 8 consecutive values of row r, columns 8*chunk .. 8*chunk+7 -> one 16-byte chunk per term
__device__ __forceinline__ void split_store8(uint32_t set, int r, int chunk, const float* v) {
  uint32_t w0[4], w1[4], w2[4];
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    float a = v[2 * p], b = v[2 * p + 1];
    w0[p] = pack2<__nv_bfloat16>(a, b);            // low half = a, high half = b
    a -= __uint_as_float(w0[p] << 16);
    b -= __uint_as_float(w0[p] & 0xffff0000u);
    w1[p] = pack2<__nv_bfloat16>(a, b);
    a -= __uint_as_float(w1[p] << 16);
    b -= __uint_as_float(w1[p] & 0xffff0000u);
    w2[p] = pack2<__nv_bfloat16>(a, b);
  }
  const uint32_t at = set + sw128_offset(r, chunk);
  sts128(at + kTerm0, w0[0], w0[1], w0[2], w0[3]);
  sts128(at + kTerm1, w1[0], w1[1], w1[2], w1[3]);
  sts128(at + kTerm2, w2[0], w2[1], w2[2], w2[3]);
}
// this thread's 16 columns of its row
__device__ __forceinline__ void put_row16(const Ctx& c, uint32_t set, const float* v) {
  split_store8(set, c.row, c.col0 >> 3, v);
  split_store8(set, c.row, (c.col0 >> 3) + 1, v + 8);
}
// the sum of the three terms, smallest first (the FP32 value the tile was made from)
__device__ __forceinline__ void get_row16(const Ctx& c, uint32_t set, float* v) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t off = sw128_offset(c.row, (c.col0 >> 3) + h);
    uint32_t w0[4], w1[4], w2[4];
    *reinterpret_cast<uint4*>(w0) = lds128(set + kTerm0 + off);
    *reinterpret_cast<uint4*>(w1) = lds128(set + kTerm1 + off);
    *reinterpret_cast<uint4*>(w2) = lds128(set + kTerm2 + off);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      v[8 * h + 2 * p] = __uint_as_float(w0[p] << 16) + (__uint_as_float(w1[p] << 16) + __uint_as_float(w2[p] << 16));
      v[8 * h + 2 * p + 1] = __uint_as_float(w0[p] & 0xffff0000u) +
                             (__uint_as_float(w1[p] & 0xffff0000u) + __uint_as_float(w2[p] & 0xffff0000u));
    }
  }
}

// ---- global / staging accesses ---------------------------------------------------------------
// `vec`: sixteen bytes at a time; the caller's FP32 tensors need no more than their type's alignment.  The backward has two forms: W
// for matrices that all lie whole on sixteen bytes, rows of (m x m) ones included, which is the usual case and has no other way
// in its code; else (m x m) matrices go four bytes at a time and (m x head_dim) ones by their addresses.  With a look at each address
// in one form it took 1 to 4 % longer than with none, in two forms it takes 0 to 5 % less (us, pseudoinverse alone, J = 6, none /
// look / two forms: m = 32, 4 slices 41.0 / 41.0 / 39.0; m = 64, 32 slices 49.2 / 51.0 / 49.2, 512 slices 203 / 210 / 197).  The forward in two
// forms took longer (m = 64, 32 slices 31.0 / 30.8 / 32.8): it asks Ctx.
template <class... P>
__host__ __device__ __forceinline__ bool whole16(const P*... g) { return ((reinterpret_cast<uintptr_t>(g) | ...) & 15u) == 0; }
// Whole-matrix tile loads: thread t handles row t >> 2 and the 8-column chunks (t & 3) and (t & 3) + 4, so that four
// adjacent lanes cover 128 consecutive bytes.
__device__ __forceinline__ void load_chunk8(const float* g, int r, int chunk, int rows, int cols, int ld, bool vec, float* v) {
  const int c0 = 8 * chunk;
  if (vec) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r < rows && c0 + 4 * q < cols) x = *reinterpret_cast<const float4*>(g + (size_t)r * ld + c0 + 4 * q);
      v[4 * q] = x.x; v[4 * q + 1] = x.y; v[4 * q + 2] = x.z; v[4 * q + 3] = x.w;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = (r < rows && c0 + i < cols) ? g[(size_t)r * ld + c0 + i] : 0.f;
  }
}
// dense global [rows x cols] matrix with row stride ld -> registers, zero beyond rows / cols
__device__ __forceinline__ void load_tile16(const float* g, int rows, int cols, int ld, bool vec, float* v) {
  load_chunk8(g, threadIdx.x >> 2, threadIdx.x & 3, rows, cols, ld, vec, v);
  load_chunk8(g, threadIdx.x >> 2, (threadIdx.x & 3) + 4, rows, cols, ld, vec, v + 8);
}
__device__ __forceinline__ void put_tile16(uint32_t set, const float* v) {
  split_store8(set, threadIdx.x >> 2, threadIdx.x & 3, v);
  split_store8(set, threadIdx.x >> 2, (threadIdx.x & 3) + 4, v + 8);
}
// the same elements -> / <- a padded FP32 staging buffer (row stride kLd)
__device__ __forceinline__ void stage_tile16(float* X, const float* v) {
  float* d = X + (threadIdx.x >> 2) * kLd + (threadIdx.x & 3) * 8;
#pragma unroll
  for (int q = 0; q < 4; ++q)
    *reinterpret_cast<float4*>(d + (q & 1) * 4 + (q >> 1) * 32) = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
}
// this thread's 16 columns of its row: global, staging
__device__ __forceinline__ void load_row16(const Ctx& c, const float* g, int rows, int cols, int ld, bool vec, float* v) {
  load_chunk8(g, c.row, c.col0 >> 3, rows, cols, ld, vec, v);
  load_chunk8(g, c.row, (c.col0 >> 3) + 1, rows, cols, ld, vec, v + 8);
}
__device__ __forceinline__ void store_row16(const Ctx& c, float* g, const float* v, int rows, int cols, int ld, bool vec) {
  if (c.row >= rows) return;
  if (vec) {
#pragma unroll
    for (int i = 0; i < 16; i += 4)
      if (c.col0 + i < cols)
        *reinterpret_cast<float4*>(g + (size_t)c.row * ld + c.col0 + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
  } else {
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (c.col0 + i < cols) g[(size_t)c.row * ld + c.col0 + i] = v[i];
  }
}
__device__ __forceinline__ void stage_row16(const Ctx& c, float* X, const float* v) {
#pragma unroll
  for (int i = 0; i < 16; i += 4)
    *reinterpret_cast<float4*>(X + c.row * kLd + c.col0 + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
}
__device__ __forceinline__ void unstage_row16(const Ctx& c, const float* X, float* v) {
#pragma unroll
  for (int i = 0; i < 16; i += 4) {
    const float4 x = *reinterpret_cast<const float4*>(X + c.row * kLd + c.col0 + i);
    v[i] = x.x; v[i + 1] = x.y; v[i + 2] = x.z; v[i + 3] = x.w;
  }
}
// the same for the transposed matrix
__device__ __forceinline__ void unstage_col16(const Ctx& c, const float* X, float* v) {
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = X[(c.col0 + i) * kLd + c.row];
}
// A staged matrix -> the leading rows x cols block of a dense global matrix, whole sectors per instruction.  (From the
// accumulator layout, 32 rows of 16 bytes per instruction, the store of an iterate kept the warps for 1700 cycles, this takes 400.)
__device__ __forceinline__ void store_staged(const float* X, float* g, int rows, int cols, int ld, bool vec) {
  if (vec) {
    const int r = threadIdx.x >> 2;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int c = 16 * q + 4 * (threadIdx.x & 3);
      if (r < rows && c < cols) *reinterpret_cast<float4*>(g + (size_t)r * ld + c) = *reinterpret_cast<const float4*>(X + r * kLd + c);
    }
  } else {
#pragma unroll 4
    for (int i = 0; i < 8; ++i) {
      const int r = (threadIdx.x >> 5) + 8 * i, c = threadIdx.x & 31;
      if (r < rows && c < cols) g[(size_t)r * ld + c] = X[r * kLd + c];
      if (r < rows && c + 32 < cols) g[(size_t)r * ld + c + 32] = X[r * kLd + c + 32];
    }
  }
}
// x / c with rc = 1 / c: a product and one correction of its remainder (Markstein 1990), correctly rounded but for results near
// the underflow threshold.  The remainder of an infinite x or c is not a number: there the product is the quotient.
__device__ __forceinline__ float div_by(float x, float c, float rc) {
  const float q = x * rc, corrected = fmaf(fmaf(-q, c, x), rc, q);
  return corrected == corrected ? corrected : q;
}
// d on the diagonal of the leading m x m block
__device__ __forceinline__ void add_diag(const Ctx& c, float* v, float d, int m) {
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] += (c.col0 + i == c.row && c.row < m) ? d : 0.f;
}

// ---- products -------------------------------------------------------------------------------
// accumulator at TMEM address d (128 columns) (+)= a * b over nk K steps of 16.  Operands are tile sets:
//   left operand  X (M x K):  plain = K-major,  transposed (X^T as left operand) = MN-major
//   right operand Y (K x N):  plain = MN-major, transposed (Y^T as right operand) = K-major
// Warp-uniform code, one elected lane issues: the eight MMAs are one block of assembly, so that the election happens once
// and the descriptors stay in uniform registers (750 cycles per product when each MMA elected and its strides were run-time
// values).
template <bool AT, bool BT>
__device__ __forceinline__ void issue_product(uint32_t d, uint32_t a, uint32_t b, bool accumulate, uint32_t nk) {
  // K-major: rows 64..127 continue into the next tile, 16 of K are 32 bytes; MN-major: the second 64-wide block is
  // the next tile, 16 of K are 16 rows
  const uint64_t da = smem_desc_sw128(a, AT ? kTileBytes : 16, 1024), db = smem_desc_sw128(b, BT ? 16 : kTileBytes, 1024);
  constexpr uint32_t idesc = make_idesc<__nv_bfloat16>(128, 128, AT, !BT);
  constexpr int sa = AT ? 2048 / 16 : 2, sb = BT ? 2 : 2048 / 16, t = kTileBytes / 16;
  // first the (x1, x0) (y1, y0) tiles over all of K, then (x0, x2) (y0, y2)
  asm volatile(
      "{\n\t.reg .pred e, e1, e2, e3, p, q;\n\t.reg .b64 x, y;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "setp.gt.and.u32 e1, %5, 1, e;\n\tsetp.gt.and.u32 e2, %5, 2, e;\n\tsetp.gt.and.u32 e3, %5, 3, e;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "add.s64 x, %1, %6;\n\tadd.s64 y, %2, %7;\n\t"
      "@e1 tcgen05.mma.cta_group::1.kind::f16 [%0], x, y, %3, q;\n\t"
      "add.s64 x, x, %6;\n\tadd.s64 y, y, %7;\n\t"
      "@e2 tcgen05.mma.cta_group::1.kind::f16 [%0], x, y, %3, q;\n\t"
      "add.s64 x, x, %6;\n\tadd.s64 y, y, %7;\n\t"
      "@e3 tcgen05.mma.cta_group::1.kind::f16 [%0], x, y, %3, q;\n\t"
      "add.s64 x, %1, %8;\n\tadd.s64 y, %2, %8;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], x, y, %3, q;\n\t"
      "add.s64 x, x, %6;\n\tadd.s64 y, y, %7;\n\t"
      "@e1 tcgen05.mma.cta_group::1.kind::f16 [%0], x, y, %3, q;\n\t"
      "add.s64 x, x, %6;\n\tadd.s64 y, y, %7;\n\t"
      "@e2 tcgen05.mma.cta_group::1.kind::f16 [%0], x, y, %3, q;\n\t"
      "add.s64 x, x, %6;\n\tadd.s64 y, y, %7;\n\t"
      "@e3 tcgen05.mma.cta_group::1.kind::f16 [%0], x, y, %3, q;\n\t}"
      ::"r"(d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate ? 1u : 0u), "r"(nk), "n"(sa), "n"(sb), "n"(t)
      : "memory");
}

// compute side: my operand tiles (and my reads of the accumulators) are done
__device__ __forceinline__ void arrive_ready(Ctx& c, int b) {
  fence_proxy_async();
  tc_fence_before();
  mbar_arrive_warp(c.sh->ready + b);
}
// issuing warp (all lanes, so that its control flow and operands stay warp-uniform)
__device__ __forceinline__ void wait_ready(Ctx& c, int b, int where) {
  const bool ok = c.failed || mbar_wait(c.sh->ready + b, (c.parity >> b) & 1u, c.ab, where);
  if (!__all_sync(0xffffffffu, ok)) c.failed = true;
  c.parity ^= 1u << b;
  tc_fence_after();
}
__device__ __forceinline__ void wait_done(Ctx& c, int b, int where) {
  if (!mbar_wait(c.sh->done + b, (c.parity >> b) & 1u, c.ab, where)) c.failed = true;
  c.parity ^= 1u << b;
  tc_fence_after();
}

// The tensor core truncates when it adds to an accumulator; the leading partial product is added to once per K step and
// loses about an eighth of an ulp each time on the average, which `trunc` (a share of the value) gives back on its way to the
// small ones.  Without it K2inv and dQ of fp32 calls were up to 1.28 and 1.24 times as far from the oracle as with an accumulator
// of its own for x1 y1 (one addition fewer per product), with it 0.83 to 0.98 and 0.90 to 0.99 times.
// A product that is added to one before adds its small terms onto the large value as well: two products in an accumulator are three
// times as many truncating additions as one, three five times.  (With one product's share for all, dL/dK2 was 1.6 to 2.2 times as far
// from 64 bits as FP32 sums are, with theirs 1.2 to 1.3 times; mean over 16 to 64 landmarks, J = 4 to 8.)
constexpr float kTruncScores = 0x1p-25f;    // below half an ulp of any value: exact sums stay exact
constexpr float kTruncHead = 4 * 0x1p-26f;  // a sum over 64 columns, however many landmarks
// This thread's share of the accumulator at TMEM column `col`, before the two lane halves are added: 16 columns that it
// keeps and 16 that its partner finalises.  Every thread of a warp must call.
__device__ __forceinline__ void fetch(const Ctx& c, uint32_t col, float trunc, float* keep, float* send) {
  const uint32_t a = c.tmem + col + c.lane_addr, ak = a + 16 * c.part, as = a + 16 - 16 * c.part;
  tmem_ld16(ak, keep);
  tmem_ld16(as, send);
  if (c.part == 0) {
    float x[16], y[16];
    tmem_ld16(ak + kN, x);
    tmem_ld16(as + kN, y);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      keep[i] += fmaf(trunc, keep[i], x[i]);
      send[i] += fmaf(trunc, send[i], y[i]);
    }
  } else {
    tmem_ld_wait();
  }
}
// Adds the two lane halves.  `set`: a slot that no product reads and no thread but this pair's touches in the rows and
// columns of the pair (the slot the result goes to, usually): each half hands over through a term of its own.
__device__ __forceinline__ void exchange(const Ctx& c, uint32_t set, const float* keep, const float* send, float* v) {
  const uint32_t x = set + c.part * kTileBytes, y = set + (1 - c.part) * kTileBytes;
#pragma unroll
  for (int q = 0; q < 4; ++q)
    sts128(x + sw128_offset(c.row, (c.c32 >> 3) + q), __float_as_uint(send[4 * q]), __float_as_uint(send[4 * q + 1]),
           __float_as_uint(send[4 * q + 2]), __float_as_uint(send[4 * q + 3]));
  named_barrier(c.pair_bar, 64);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint4 w = lds128(y + sw128_offset(c.row, (c.c32 >> 3) + q));
    v[4 * q] = keep[4 * q] + __uint_as_float(w.x); v[4 * q + 1] = keep[4 * q + 1] + __uint_as_float(w.y);
    v[4 * q + 2] = keep[4 * q + 2] + __uint_as_float(w.z); v[4 * q + 3] = keep[4 * q + 3] + __uint_as_float(w.w);
  }
  named_barrier(c.pair_bar, 64);
}

// the two together: the accumulator at `col` once done[b] has completed; nothing where `act` is false
__device__ __forceinline__ void take(Ctx& c, int b, uint32_t col, uint32_t set, bool act, float* v, float trunc) {
  wait_done(c, b, 0x2100 + b);
  if (act) {
    float keep[16], send[16];
    fetch(c, col, trunc, keep, send);
    exchange(c, set, keep, send, v);
  }
}

// ---------------------------------------------------------------------------------------------
// Forward.  Products in order (s):
//   -2        scores Qt Kt^T (head_dim 128: two products, 64 columns each)    slots 0, 1 (2, 3)
//   -1        K2^T K2 (ridge only)                                            slot 2
//   4j, ...   R = I - A Z | Y = Z R | W = I + R + R R / 4 | Z' = Z + Y W      A 0, Z 1, R and W 2, Y 3
//   4J        k2inv = Z K2^T (ridge only)                                     K2 in slot 0
// Even s: accumulator 0, odd s: accumulator 1.  Y is formed before W: Z is in registers too, so its slot
// stays free, and W goes over R.  FP32 staging of K2, then A: slot 3.
// Two slices per SM (97 KB, 256 TMEM columns, 96 registers): the epilogues of one run beside the products of the other.
constexpr int kFwdStage = 3;
struct FwdParams {
  ns::NsFwdParams p;
  bool k2_given;        // p.k2 holds the softmaxed matrix: no scores, no softmax
};

__device__ inline void fwd_issue(Ctx& c, const FwdParams& f) {
  const bool ridge = f.p.kappa > 0.f;
  const uint32_t nk = (f.p.m + 15) / 16, acc0 = c.tmem, acc1 = c.tmem + kAccCols;
  if (!f.k2_given) {
    wait_ready(c, 0, 0x2100);
    if (c.failed) return;
    issue_product<false, true>(acc0, c.slot(0), c.slot(1), false, 4);
    if (f.p.D > kN) issue_product<false, true>(acc0, c.slot(2), c.slot(3), true, 4);
    umma_commit_elect(c.sh->done);
  }
  if (ridge) {
    wait_ready(c, 0, 0x2101);
    if (c.failed) return;
    issue_product<true, false>(acc1, c.slot(2), c.slot(2), false, nk);
    umma_commit_elect(c.sh->done + 1);
  }
#pragma unroll 1
  for (int j = 0; j < f.p.J; ++j) {
    wait_ready(c, 0, 0x2102);
    if (c.failed) return;
    issue_product<false, false>(acc0, c.slot(0), c.slot(1), false, nk);    // A Z
    umma_commit_elect(c.sh->done);
    wait_ready(c, 0, 0x2103);
    if (c.failed) return;
    issue_product<false, false>(acc1, c.slot(1), c.slot(2), false, nk);    // Z R
    umma_commit_elect(c.sh->done + 1);
    issue_product<false, false>(acc0, c.slot(2), c.slot(2), false, nk);    // R R
    umma_commit_elect(c.sh->done);
    wait_ready(c, 0, 0x2104);
    if (c.failed) return;
    issue_product<false, false>(acc1, c.slot(3), c.slot(2), false, nk);    // Y W
    umma_commit_elect(c.sh->done + 1);
  }
  if (ridge) {
    wait_ready(c, 0, 0x2105);
    if (c.failed) return;
    issue_product<false, true>(acc0, c.slot(1), c.slot(0), false, nk);     // Z K2^T
    umma_commit_elect(c.sh->done);
  }
}

// Row softmax of the scores in the padded buffer X, in place (rows and columns past m become zero), K2 and lse2 to
// global memory.  Four adjacent lanes share a row, lane k the columns 4 i + k: the row sum is then the tree
// of ns::softmax_rows (columns 32 apart, 16, 8 and 4 in the lane, 2 and 1 by shuffles), bit for bit, with two
// shuffles per reduction in place of five.
__device__ inline void softmax16(float* X, const ns::NsFwdParams& p, int64_t bh) {
  const int m = p.m, r = threadIdx.x >> 2, k = threadIdx.x & 3;
  float* row = X + r * kLd;
  float v[16], mx = -INFINITY, sum;
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = row[4 * i + k];
#pragma unroll
  for (int i = 0; i < 16; ++i) if (4 * i + k < m) mx = fmaxf(mx, v[i]);
  mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
  mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    v[i] = (r < m && 4 * i + k < m) ? expf(v[i] - mx) : 0.f;
  }
  float part[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) part[i] = v[i] + v[i + 8];
#pragma unroll
  for (int o = 4; o > 0; o >>= 1)
#pragma unroll
    for (int i = 0; i < o; ++i) part[i] += part[i + o];
  sum = part[0];
  sum += __shfl_xor_sync(0xffffffffu, sum, 2);
  sum += __shfl_xor_sync(0xffffffffu, sum, 1);
  const float rsum = 1.f / sum;
#pragma unroll
  for (int i = 0; i < 16; ++i) row[4 * i + k] = r < m ? div_by(v[i], sum, rsum) : 0.f;
  __syncwarp();                              // a row's four lanes are in one warp
  if (r < m && k == 0) p.lse2[bh * m + r] = mx + logf(sum);
  ns::ns_sync();
}

// The landmarks as tiles: Qt in slots 0 (and 2 for head_dim 128), Kt in slots 1 (and 3).
__device__ __forceinline__ void fwd_landmarks(Ctx& c, const ns::NsFwdParams& p, int64_t bh) {
  const int m = p.m, D = p.D, r = threadIdx.x >> 2;
  float q[16], k[16];
  if (p.land) {
    // raw segment sums of the pooling pass, [2][BH][m][C][64]: scale * sum / length, and FP32 copies to global memory
#pragma unroll
    for (int i = 0; i < 16; ++i) { q[i] = 0.f; k[i] = 0.f; }
    if (r < m) {
      const size_t off = ((size_t)bh * m + r) * p.C * kN, which = (size_t)p.BH * m * p.C * kN;
      const int c0 = (threadIdx.x & 3) * 8;
      for (int ch = 0; ch < p.C; ++ch) {
        const float* src = p.land + off + (size_t)ch * kN + c0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int o = (j & 1) * 4 + (j >> 1) * 32;
          const float4 x = *reinterpret_cast<const float4*>(src + o), y = *reinterpret_cast<const float4*>(src + which + o);
          q[4 * j] += x.x; q[4 * j + 1] += x.y; q[4 * j + 2] += x.z; q[4 * j + 3] += x.w;
          k[4 * j] += y.x; k[4 * j + 1] += y.y; k[4 * j + 2] += y.z; k[4 * j + 3] += y.w;
        }
      }
      const float f = p.scale / (float)Segments(p.seg_N, m).len(r);
      float* dq = p.qt_out + ((size_t)bh * m + r) * kN + c0;
      float* dk = p.kt_out + ((size_t)bh * m + r) * kN + c0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int o = (j & 1) * 4 + (j >> 1) * 32;
#pragma unroll
        for (int i = 4 * j; i < 4 * j + 4; ++i) { q[i] *= f; k[i] *= f; }
        *reinterpret_cast<float4*>(dq + o) = make_float4(q[4 * j], q[4 * j + 1], q[4 * j + 2], q[4 * j + 3]);
        *reinterpret_cast<float4*>(dk + o) = make_float4(k[4 * j], k[4 * j + 1], k[4 * j + 2], k[4 * j + 3]);
      }
    }
    put_tile16(c.slot(0), q);
    put_tile16(c.slot(1), k);
    return;
  }
#pragma unroll 1
  for (int h = 0; h < (D > kN ? 2 : 1); ++h) {
    const int cols = min(D, kN);
    load_tile16(p.qt + bh * m * D + h * kN, m, cols, D, c.md16, q);
    load_tile16(p.kt + bh * m * D + h * kN, m, cols, D, c.md16, k);
    put_tile16(c.slot(2 * h), q);
    put_tile16(c.slot(2 * h + 1), k);
  }
}

__device__ __forceinline__ void fwd_compute(Ctx& c, float* red, const FwdParams& f, int64_t bh) {
  const ns::NsFwdParams& p = f.p;
  const int m = p.m, J = p.J, mm_ = m * m;
  const bool ridge = p.kappa > 0.f;
  const int last = 4 * J + (ridge ? 1 : 0);
  float* X = c.stage(kFwdStage);
  float* iterates = p.iterates + bh * (size_t)(J + 1) * mm_;
  float* k2 = p.k2 + bh * mm_;
  float z[16], r[16], v[16];       // Z_j, R and the value in hand
#pragma unroll
  for (int i = 0; i < 16; ++i) { r[i] = 0.f; v[i] = 0.f; }       // (inactive warps keep zeros)
  if (f.k2_given) {
    load_tile16(k2, m, m, m, c.mm16, v);
    stage_tile16(X, v);
    ns::ns_sync();
  } else {
    fwd_landmarks(c, p, bh);
    arrive_ready(c, 0);
  }
#pragma unroll 1
  for (int s = f.k2_given ? -1 : -2; s < last; ++s) {
    if (s == -1 && !ridge) continue;                       // A = K2
    if (s == -1 || s == 0) {
      // X = K2 (s = -1) or A: its norms, then K2 as an operand, or A and Z0
      const Norms n = ns::norms(X, m, red);
      unstage_row16(c, X, v);
      if (s == -1) {
        r[0] = n.n1 * n.ninf / p.kappa;                    // lambda
        put_row16(c, c.slot(2), v);
      } else {
        const float cden = fmaxf(n.n1 * n.ninf, 1e-12f), rcden = 1.f / cden;
        put_row16(c, c.slot(0), v);
        unstage_col16(c, X, z);                            // Z0 = A^T / cden
#pragma unroll
        for (int i = 0; i < 16; ++i) z[i] = div_by(z[i], cden, rcden);
        put_row16(c, c.slot(1), z);
      }
      arrive_ready(c, 0);
      // to global memory beside the product: K2 first, Z0 (staged over it) below
      if (!f.k2_given && !c.failed && (s == -1 || !ridge)) store_staged(X, k2, m, m, m, c.mm16);
      if (s == 0) {
        ns::ns_sync();
        stage_row16(c, X, z);
      }
    }
    if (s >= 0 && s < 4 * J) {
      // one iteration; R, then Y and W, then Z'.  Z_j is staged in X (slot 3, free until Y) and leaves while the product runs.
      ns::ns_sync();
      if (!c.failed) store_staged(X, iterates + (size_t)(s >> 2) * mm_, m, m, m, c.mm16);
      take(c, 0, 0, c.slot(2), c.act, v, c.trunc);
      if (c.act) {
#pragma unroll
        for (int i = 0; i < 16; ++i) r[i] = -v[i];
        add_diag(c, r, 1.f, m);
        put_row16(c, c.slot(2), r);
      }
      arrive_ready(c, 0);
      take(c, 1, kAccCols, c.slot(3), c.act, v, c.trunc);
      if (c.act) put_row16(c, c.slot(3), v);
      take(c, 0, 0, c.slot(2), c.act, v, c.trunc);
      if (c.act) {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = fmaf(0.25f, v[i], r[i]);
        add_diag(c, v, 1.f, m);
        put_row16(c, c.slot(2), v);
      }
      arrive_ready(c, 0);
      s += 3;
      const bool end = s == 4 * J - 1;
      if (ridge && end) load_row16(c, k2, m, m, m, c.mm16, r);      // (R is dead; K2 is the last product's operand)
      take(c, 1, kAccCols, c.slot(1), c.act, v, c.trunc);
      if (c.act) {
#pragma unroll
        for (int i = 0; i < 16; ++i) z[i] += v[i];
        put_row16(c, c.slot(1), z);
        if (ridge && end) put_row16(c, c.slot(0), r);
      }
      if (!end || ridge) arrive_ready(c, 0);
      stage_row16(c, X, z);
      if (end) {
        ns::ns_sync();
        if (!c.failed) {
          store_staged(X, iterates + (size_t)J * mm_, m, m, m, c.mm16);
          if (!ridge) store_staged(X, p.k2inv + bh * mm_, m, m, m, c.mm16);
        }
      }
      continue;
    }
    // scores (s = -2), K2^T K2 (s = -1), k2inv (s = 4J)
    take(c, s & 1, (s & 1) * kAccCols, c.slot(s == -1 ? 0 : 2), c.act, v, s == -2 ? kTruncScores : c.trunc);
    if (s == 4 * J) {
      ns::ns_sync();
      stage_row16(c, X, v);
      ns::ns_sync();
      if (!c.failed) store_staged(X, p.k2inv + bh * mm_, m, m, m, c.mm16);
      break;
    }
    if (!c.act) {
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = 0.f;
    }
    if (s == -1) {
      add_diag(c, v, r[0], m);
      ns::ns_sync();                         // K2 leaves X behind its arrival for the product: every warp is through with that
    }
    stage_row16(c, X, v);
    ns::ns_sync();
    if (s == -2) softmax16(X, p, bh);
  }
}

__global__ void __launch_bounds__(kNsTcThreads, 2) ns_fwd_tc_kernel(FwdParams f, int* status) {
  extern __shared__ uint8_t dyn_smem[];
  __shared__ float red[ns::kRedFloats];
  __shared__ Shared sh;
  Ctx c;
  ctx_open(c, sh, dyn_smem, status, kFwdTmemCols, f.p.m);
  c.md16 = whole16(f.p.qt, f.p.kt);
  c.mm16 = (f.p.m & 3) == 0 && whole16(f.p.k2, f.p.iterates, f.p.k2inv);
  if (is_compute()) fwd_compute(c, red, f, blockIdx.x);
  else fwd_issue(c, f);
  ctx_close(c, kFwdTmemCols);
}

// ---------------------------------------------------------------------------------------------
// Backward.  With R = I - A Z, W = I + R + R^2 / 4, Y = Z R, Z' = Z + Y W and G = dL/dZ':
//     dY = G W^T,  H = Y^T G / 4 (= dW / 4),  D = -dL/dR = -(Z^T dY + H R^T + R^T H + 4 H)
//     dL/dZ = G + dY R^T + A^T D,  dL/dA += D Z^T
// Three dependent steps per iteration (four in the nested form), and R, W, Y of the next lower iterate are formed
// beside them.  Slots: A 0, Z_j and Z_{j-1} 1 and 2, R_j and R_{j-1} 3 and 4, G_j (then D) and G_{j-1} 5 and 6, W (then dY) 7,
// Y (then H) 8.  Per iteration, in the order the products are issued (accumulator, done barrier):
//     dY (3, 0) | H (2, 1) | R_{j-1} (1, 2) | D = Z^T dY + H R^T + R^T H (0, 3) | dY R^T (3)
//     | R_{j-1}^2 (1, 4) | + A^T D (3, 5) | Z_{j-1} R_{j-1} (2, 6) | D Z^T (0, 7)
// so that the products (11 of about 520 cycles) keep the tensor core busy while the epilogues run.  dL/dA is
// summed in registers before the lane halves are added.  j = J is a prologue that only forms R, W, Y of Z_{J-1}.
// Before it: dO3 = K2inv^T dstep2 and dK2inv = dstep2 Bmat^T of the fused middle stage, and with the ridge A = K2^T K2 +
// lambda I, dZ_J = dK2inv K2 and dL/dK2 = dK2inv^T Z_J.  After it: the norm terms of Z0, the ridge, the softmax-2
// Jacobian, and dqt_ns = dS2 Kt, dkt_tot = dkt_a + dS2^T Qt, 64 columns at a time.
//
// Head of the fused middle stage (head_dim 64):
struct BwdHeadParams {
  const float* partA;         // [BH][nchunk][2][m][D]: dstep2 partials, dKt partials (null: G is given)
  int nchunk;
  const float* k2inv; const float* bmat;
  float* dkt_a;               // [BH][m][D] out
  // The four outputs below feed the column pass; all are skipped when D3 is null (the column pass
  // then runs beside this kernel and takes them from a separate small kernel).
  float* D3;                  // [BH][m] out
  void* do3n;                 // [BH][MP][D] 16-bit out = dO3 / do3_scale
  float* do3_scale;           // [BH] out
  void* qt16;                 // [BH][MP][D] 16-bit out = qt_mul * Qt
  float qt_mul;
  int dtype, MP;
};
struct BwdParams {
  ns::NsBwdParams p;
  BwdHeadParams h;
  float* dK2;                 // [BH][m][m]: stop there (pseudoinverse alone)
  float* step_dz;             // [BH][m][m] each: stop after the iterations with dL/dZ_0 and dL/dA
  float* step_da;             //   (p.iterates then is Z_0 alone)
};

// Steps outside the iterations, which share one body.  kNorms comes with no accumulator first (K2), with the ridge again for
// the Gram matrix.
enum BwdStep { kNorms, kHeadO3, kHeadG, kRidgeG, kRidgeK2, kSumDA, kTailK2, kDQ, kDK };

// issuing warp.  ready barriers: 0 G and W (also the head's operands, and those of the tail), 1 Y (also K2), 2 Z_{j-1}
// (also A), 3 dY (also dK2inv), 4 H, 5 R_{j-1}, 6 D.
__device__ inline void bwd_issue(Ctx& c, const BwdParams& f, int finish) {
  const bool ridge = f.p.kappa > 0.f, head = f.h.partA != nullptr;
  const int J = f.p.J;
  const uint32_t nk = (f.p.m + 15) / 16, acc0 = c.tmem, acc1 = acc0 + kAccCols, acc2 = acc1 + kAccCols, acc3 = acc2 + kAccCols;
  auto commit = [&](int b) { umma_commit_elect(c.sh->done + b); };
  if (ridge) {
    wait_ready(c, 1, 0x2201);
    if (c.failed) return;
    issue_product<true, false>(acc1, c.slot(4), c.slot(4), false, nk);                 // K2^T K2
    commit(3);
  }
  if (head) {
    wait_ready(c, 0, 0x2200);
    if (c.failed) return;
    issue_product<true, false>(acc3, c.slot(7), c.slot(8), false, nk);                 // K2inv^T dstep2
    commit(0);
    issue_product<false, true>(acc0, c.slot(8), c.slot(6), false, 4);                  // dstep2 Bmat^T (K is the head_dim)
    commit(1);
  }
  if (ridge) {
    wait_ready(c, 3, 0x2203);
    if (c.failed) return;
    issue_product<false, false>(acc3, c.slot(6), c.slot(4), false, nk);                // dK2inv K2
    commit(5);
    issue_product<true, false>(acc0, c.slot(6), c.slot(2), false, nk);                 // dK2inv^T Z_J
    commit(7);
  }
#pragma unroll 1
  for (int j = J; j >= 0; --j) {
    const int par = (J - 1 - j) & 1;
    const bool main_part = j < J, prime = j > 0;
    const uint32_t z = c.slot(1 + par), zn = c.slot(2 - par), r = c.slot(3 + par), rn = c.slot(4 - par), g = c.slot(5 + par);
    if (main_part) {
      wait_ready(c, 0, 0x2210);
      if (c.failed) return;
      issue_product<false, true>(acc3, g, c.slot(7), false, nk);                       // G W^T
      commit(0);
      wait_ready(c, 1, 0x2211);
      if (c.failed) return;
      issue_product<true, false>(acc2, c.slot(8), g, false, nk);                       // Y^T G
      commit(1);
    }
    if (prime) {
      wait_ready(c, 2, 0x2212);
      if (c.failed) return;
      issue_product<false, false>(acc1, c.slot(0), zn, false, nk);                     // A Z'
      commit(2);
    }
    if (main_part) {
      wait_ready(c, 3, 0x2213);
      if (c.failed) return;
      issue_product<true, false>(acc0, z, c.slot(7), false, nk);                       // Z^T dY
      wait_ready(c, 4, 0x2214);
      if (c.failed) return;
      issue_product<false, true>(acc0, c.slot(8), r, true, nk);                        // + H R^T
      issue_product<true, false>(acc0, r, c.slot(8), true, nk);                        // + R^T H
      commit(3);
      issue_product<false, true>(acc3, c.slot(7), r, false, nk);                       // dY R^T
    }
    if (prime) {
      wait_ready(c, 5, 0x2215);
      if (c.failed) return;
      issue_product<false, false>(acc1, rn, rn, false, nk);                            // R'^2
      commit(4);
    }
    if (main_part) {
      wait_ready(c, 6, 0x2216);
      if (c.failed) return;
      issue_product<true, false>(acc3, c.slot(0), g, true, nk);                        // + A^T D
      commit(5);
    }
    if (prime) {
      issue_product<false, false>(acc2, zn, rn, false, nk);                            // Z' R'
      commit(6);
    }
    if (main_part) {
      issue_product<false, true>(acc0, g, z, false, nk);                               // D Z^T
      commit(7);
    }
  }
  if (finish < 0) return;
  if (ridge) {
    wait_ready(c, 0, 0x2220);
    if (c.failed) return;
    issue_product<false, false>(acc3, c.slot(6), c.slot(5), false, nk);                // K2 dA
    issue_product<false, true>(acc3, c.slot(6), c.slot(5), true, nk);                  // + K2 dA^T
    commit(0);
  }
#pragma unroll 1
  for (int half = 0; half < finish; ++half) {
    wait_ready(c, 0, 0x2221);
    if (c.failed) return;
    issue_product<false, false>(acc0, c.slot(5), c.slot(6), false, nk);                // dS2 Kt
    commit(0);
    issue_product<true, false>(acc1, c.slot(5), c.slot(7), false, nk);                 // dS2^T Qt
    commit(1);
  }
}

// compute warps.  finish: batches of 64 columns of the landmark gradients; 0: stop at dL/dK2, -1: after the iterations.
template <bool W>
__device__ __forceinline__ void bwd_compute(Ctx& c, float* red, const BwdParams& f, int64_t bh, int finish) {
  const ns::NsBwdParams& p = f.p;
  const BwdHeadParams& h = f.h;
  const int m = p.m, D = p.D, J = p.J, mm_ = m * m, t = threadIdx.x;
  const int64_t md = (int64_t)m * D;
  const bool ridge = p.kappa > 0.f, head = h.partA != nullptr;
  const float* iterates = p.iterates + bh * (size_t)(f.step_dz ? 1 : J + 1) * mm_;
  float* X = c.stage(3);
  float v[16], g[16], da_keep[16], da_send[16], z[16], hd[16], r[16];
  float lam = 0.f;
  Norms nrm;
  // ---- operands ----
  load_tile16(iterates + (size_t)(J - 1) * mm_, m, m, m, W, z);
  load_tile16(p.k2 + bh * mm_, m, m, m, W, r);
  if (ridge) load_tile16(iterates + (size_t)J * mm_, m, m, m, W, hd);
#pragma unroll
  for (int i = 0; i < 16; ++i) { g[i] = 0.f; da_keep[i] = 0.f; da_send[i] = 0.f; }
  if (!head) load_row16(c, p.G + bh * mm_, m, m, m, W, g);
  put_tile16(c.slot(1), z);
  put_tile16(c.slot(ridge ? 4 : 0), r);
  if (ridge) put_tile16(c.slot(2), hd);
  arrive_ready(c, ridge ? 1 : 2);
  stage_tile16(X, r);
  if (!head) put_row16(c, c.slot(ridge ? 6 : 5), g);
  if (!head && ridge) arrive_ready(c, 3);
  if (ridge) {
#pragma unroll
    for (int i = 0; i < 16; ++i) g[i] = 0.f;       // dL/dZ_J = G K2 is added to it
  }
  if (J > 1) load_tile16(iterates + (size_t)(J - 2) * mm_, m, m, m, W, z);
  if (head) {
    // reduce the partials of the first row pass: dstep2 -> slot 8, dkt_a -> global
    float ds[16], dk[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) { ds[i] = 0.f; dk[i] = 0.f; }
    const int row = t >> 2, c0 = (t & 3) * 8;
    if (row < m) {
      const float* src = h.partA + bh * (int64_t)h.nchunk * 2 * md + (size_t)row * kN + c0;
#pragma unroll 2
      for (int ch = 0; ch < h.nchunk; ++ch, src += 2 * md) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int o = (q & 1) * 4 + (q >> 1) * 32;
          const float4 x = *reinterpret_cast<const float4*>(src + o), y = *reinterpret_cast<const float4*>(src + md + o);
          ds[4 * q] += x.x; ds[4 * q + 1] += x.y; ds[4 * q + 2] += x.z; ds[4 * q + 3] += x.w;
          dk[4 * q] += y.x; dk[4 * q + 1] += y.y; dk[4 * q + 2] += y.z; dk[4 * q + 3] += y.w;
        }
      }
      float* out = h.dkt_a + bh * md + (size_t)row * kN + c0;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        *reinterpret_cast<float4*>(out + (q & 1) * 4 + (q >> 1) * 32) = make_float4(dk[4 * q], dk[4 * q + 1], dk[4 * q + 2], dk[4 * q + 3]);
    }
    put_tile16(c.slot(8), ds);
    load_tile16(h.k2inv + bh * mm_, m, m, m, W, v);
    load_tile16(h.bmat + bh * md, m, kN, kN, W || c.md16, ds);
    put_tile16(c.slot(7), v);
    put_tile16(c.slot(6), ds);
    arrive_ready(c, 0);
  }
  ns::ns_sync();                                     // X is complete

#pragma unroll 1
  for (int phase = 0; phase < 2; ++phase) {
    // ---- before and after the iterations ----
    int step = phase ? kSumDA : kNorms;
    bool first = true;                                 // the first kNorms has no accumulator
    int half = 0;
#pragma unroll 1
    for (;;) {
      // global operands of this step or of the batch after it, ahead of the wait
      if (step == kHeadO3 && h.D3) load_row16(c, p.qt + bh * md, m, kN, kN, W || c.md16, hd);
      if (step == kDQ) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {                    // dkt_a, as store_staged walks a matrix
          const int rr = t >> 2, cc = 16 * q + 4 * (t & 3);
          float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
          if (rr < m && cc < min(D, kN)) x = *reinterpret_cast<const float4*>(p.dkt_a + bh * md + (size_t)rr * D + half * kN + cc);
          z[4 * q] = x.x; z[4 * q + 1] = x.y; z[4 * q + 2] = x.z; z[4 * q + 3] = x.w;
        }
        if (half + 1 < finish) {
          load_tile16(p.kt + bh * md + (half + 1) * kN, m, min(D, kN), D, W || c.md16, hd);
          load_tile16(p.qt + bh * md + (half + 1) * kN, m, min(D, kN), D, W || c.md16, r);
        }
      }
      // slot that the result goes to (or a free one to add the lane halves in), accumulator, done barrier
      int dst, acc, done;
      switch (step) {
        case kNorms: dst = 0; acc = 1; done = 3; break;
        case kHeadO3: dst = 5; acc = 3; done = 0; break;
        case kHeadG: dst = ridge ? 6 : 5; acc = 0; done = 1; break;
        case kRidgeG: dst = 5; acc = 3; done = 5; break;
        case kRidgeK2: dst = 6; acc = 0; done = 7; break;
        case kTailK2: dst = 4; acc = 3; done = 0; break;
        case kDQ: dst = 8; acc = 0; done = 0; break;
        case kDK: dst = 4; acc = 1; done = 1; break;
        default: dst = 7; acc = 0; done = -1; break;   // kSumDA: in registers
      }
      // (results of the head and of the last batch have head_dim columns)
      const bool act = (step == kHeadO3 || step == kDQ || step == kDK) ? (c.row & 32) < m : c.act;
      if (step == kNorms && first) {
      } else {
        if (done >= 0) wait_done(c, done, 0x2210 + step);
        if (act) {
          float keep[16], send[16];
          if (step == kSumDA) {
#pragma unroll
            for (int i = 0; i < 16; ++i) { keep[i] = da_keep[i]; send[i] = da_send[i]; }
          } else {
            fetch(c, acc * kAccCols, step == kHeadG ? kTruncHead : step == kTailK2 ? 3.f * c.trunc : c.trunc, keep, send);
          }
          exchange(c, c.slot(dst), keep, send, v);
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = 0.f;
        }
      }
      int next = -1, arrive = -1;
      bool jacobian = false;
      switch (step) {
        case kNorms:
          if (!first) {
            add_diag(c, v, lam, m);
            put_row16(c, c.slot(0), v);
            stage_row16(c, X, v);
            arrive_ready(c, 2);
            ns::ns_sync();
          }
          nrm = ns::norms(X, m, red);
          if (first && ridge) { lam = nrm.n1 * nrm.ninf / p.kappa; next = kNorms; }
          else next = head ? kHeadO3 : ridge ? kRidgeG : -1;
          first = false;
          break;
        case kHeadO3: {
          next = kHeadG;
          if (!h.D3) break;
          // dO3: its row sums with Bmat, and the 16-bit operands of the column pass, dO3 / scale and qt_mul * Qt (rows
          // past m are zero)
          float b[16], d3 = 0.f, amax = 0.f;
          get_row16(c, c.slot(6), b);
#pragma unroll
          for (int i = 0; i < 16; ++i) { d3 = fmaf(v[i], b[i], d3); amax = fmaxf(amax, fabsf(v[i])); }
          red[c.row * 4 + (c.col0 >> 4)] = d3;
          for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
          if ((t & 31) == 0) red[4 * kN + (t >> 5)] = amax;
          ns::ns_sync();
          float cmax = red[4 * kN];
#pragma unroll
          for (int w = 1; w < kComputeThreads / 32; ++w) cmax = fmaxf(cmax, red[4 * kN + w]);
          const float sc = pow2_scale(cmax), inv_sc = 1.f / sc;
          if (t == 0) h.do3_scale[bh] = sc;
          if (t < m) h.D3[bh * m + t] = (red[4 * t] + red[4 * t + 1]) + (red[4 * t + 2] + red[4 * t + 3]);
          uint32_t w0[8], w1[8];
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            const float x = v[i] * inv_sc, y = v[i + 1] * inv_sc, q0 = hd[i] * h.qt_mul, q1 = hd[i + 1] * h.qt_mul;
            w0[i >> 1] = h.dtype == 1 ? pack2<__half>(x, y) : pack2<__nv_bfloat16>(x, y);
            w1[i >> 1] = h.dtype == 1 ? pack2<__half>(q0, q1) : pack2<__nv_bfloat16>(q0, q1);
          }
          const size_t off = ((size_t)bh * h.MP + c.row) * kN + c.col0;
          uint4* d0 = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(h.do3n) + off);
          uint4* d1 = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(h.qt16) + off);
          d0[0] = make_uint4(w0[0], w0[1], w0[2], w0[3]); d0[1] = make_uint4(w0[4], w0[5], w0[6], w0[7]);
          d1[0] = make_uint4(w1[0], w1[1], w1[2], w1[3]); d1[1] = make_uint4(w1[4], w1[5], w1[6], w1[7]);
          break;
        }
        case kHeadG:
          if (act) put_row16(c, c.slot(dst), v);
          if (ridge) { arrive = 3; next = kRidgeG; }
          else {
#pragma unroll
            for (int i = 0; i < 16; ++i) g[i] = v[i];
          }
          break;
        case kRidgeG:
#pragma unroll
          for (int i = 0; i < 16; ++i) g[i] = v[i];
          if (act) put_row16(c, c.slot(dst), v);
          next = kRidgeK2;
          break;
        case kRidgeK2:
          if (act && !c.failed) store_row16(c, p.spill + bh * mm_, v, m, m, m, W);
          break;
        case kSumDA: {
          if (f.step_dz) {
            if (!c.failed) {
              store_row16(c, f.step_dz + bh * mm_, g, m, m, m, W);
              store_row16(c, f.step_da + bh * mm_, v, m, m, m, W);
            }
            break;
          }
          // Z0 = A^T / c, c = ||A||_1 ||A||_inf (first-occurrence maxima): g = dL/dZ_0, v = dL/dA of the iterations
          float gt[16], a[16], part = 0.f;
          stage_row16(c, X, g);
          if (c.act) get_row16(c, c.slot(0), a);
          else {
#pragma unroll
            for (int i = 0; i < 16; ++i) a[i] = 0.f;
          }
          ns::ns_sync();
          unstage_col16(c, X, gt);
#pragma unroll
          for (int i = 0; i < 16; ++i) part = fmaf(gt[i], a[i], part);
          for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
          if ((t & 31) == 0) red[4 * kN + (t >> 5)] = part;
          ns::ns_sync();
          float S = 0.f;
#pragma unroll
          for (int w = 0; w < kComputeThreads / 32; ++w) S += red[4 * kN + w];
          const float craw = nrm.n1 * nrm.ninf, cden = fmaxf(craw, 1e-12f), rcden = 1.f / cden;
          const bool clamped = !(craw > 1e-12f);
          const float col_term = clamped ? 0.f : -S * nrm.ninf / (cden * cden);
          const float row_term = clamped ? 0.f : -S * nrm.n1 / (cden * cden);
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float sg = a[i] > 0.f ? 1.f : (a[i] < 0.f ? -1.f : 0.f);
            float x = v[i] + div_by(gt[i], cden, rcden);
            if (c.col0 + i == nrm.jc) x += sg * col_term;
            if (c.row == nrm.ir) x += sg * row_term;
            v[i] = (c.row < m && c.col0 + i < m) ? x : 0.f;
            g[i] = a[i];
          }
          if (ridge) {
            // dL/dK2 = (what kRidgeK2 left) + K2 (dA + dA^T)
            put_row16(c, c.slot(5), v);
            load_row16(c, p.k2 + bh * mm_, m, m, m, W, g);
            put_row16(c, c.slot(6), g);
            arrive = 0;
            next = kTailK2;
          } else {
            jacobian = true;
          }
          break;
        }
        case kTailK2: {
          float e[16];
          load_row16(c, p.spill + bh * mm_, m, m, m, W, e);
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = (c.row < m && c.col0 + i < m) ? v[i] + e[i] : 0.f;
          jacobian = true;
          break;
        }
        case kDQ:
          stage_row16(c, c.stage(1), v);
          ns::ns_sync();
          if (!c.failed) store_staged(c.stage(1), p.dqt_ns + bh * md + half * kN, m, min(D, kN), D, W || c.md16);
          next = kDK;
          break;
        default: {                                       // kDK
          stage_row16(c, c.stage(2), v);
          ns::ns_sync();
          const int rr = t >> 2;
          const float fk = p.rows_k ? p.scale / (float)Segments(p.N, m).len(min(rr, m - 1)) : 0.f;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int cc = 16 * q + 4 * (t & 3);
            if (rr < m && cc < min(D, kN) && !c.failed) {
              float4 x = *reinterpret_cast<const float4*>(c.stage(2) + rr * kLd + cc);
              x.x += z[4 * q]; x.y += z[4 * q + 1]; x.z += z[4 * q + 2]; x.w += z[4 * q + 3];
              const size_t off = (size_t)bh * md + (size_t)rr * D + half * kN + cc;
              *reinterpret_cast<float4*>(p.dkt_tot + off) = x;
              if (p.rows_k) *reinterpret_cast<float4*>(p.rows_k + off) = make_float4(x.x * fk, x.y * fk, x.z * fk, x.w * fk);
            }
          }
          ++half;
          break;
        }
      }
      if (jacobian && f.dK2) {
        if (!c.failed) store_row16(c, f.dK2 + bh * mm_, v, m, m, m, W);
        jacobian = false;
      } else if (jacobian) {
        // softmax-2: dS2 = K2 o (dK2 - rowsum(dK2 o K2)); g holds K2
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) s = fmaf(v[i], g[i], s);
        red[c.row * 4 + (c.col0 >> 4)] = s;
        ns::ns_sync();
        s = (red[4 * c.row] + red[4 * c.row + 1]) + (red[4 * c.row + 2] + red[4 * c.row + 3]);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = g[i] * (v[i] - s);
        put_row16(c, c.slot(5), v);
      }
      if (jacobian || (step == kDK && half < finish)) {
        put_tile16(c.slot(6), hd);                       // Kt, Qt
        put_tile16(c.slot(7), r);
        arrive = 0;
        next = kDQ;
      }
      if (arrive >= 0) arrive_ready(c, arrive);
      if (next < 0) break;
      step = next;
    }
    if (phase) break;

    // ---- the iterations; j = J only forms R, W, Y of Z_{J-1}, j = 0 needs none ----
#pragma unroll 1
    for (int j = J; j >= 0; --j) {
      const int par = (J - 1 - j) & 1;
      const bool main_part = j < J, prime = j > 0;
      if (main_part) {
        if (prime) {
          put_tile16(c.slot(2 - par), z);                // Z_{j-1}: every product that read this slot is complete
          arrive_ready(c, 2);
          if (j > 1) load_tile16(iterates + (size_t)(j - 2) * mm_, m, m, m, W, z);
        }
        take(c, 0, 3 * kAccCols, c.slot(7), c.act, v, c.trunc);   // dY
        if (c.act) put_row16(c, c.slot(7), v);
        arrive_ready(c, 3);
        take(c, 1, 2 * kAccCols, c.slot(8), c.act, v, c.trunc);   // H
        if (c.act) {
#pragma unroll
          for (int i = 0; i < 16; ++i) { v[i] *= 0.25f; hd[i] = v[i]; }
          put_row16(c, c.slot(8), v);
        }
        arrive_ready(c, 4);
      }
      if (prime) {
        take(c, 2, kAccCols, c.slot(4 - par), c.act, v, c.trunc); // R of the next lower iterate
        if (c.act) {
#pragma unroll
          for (int i = 0; i < 16; ++i) r[i] = -v[i];
          add_diag(c, r, 1.f, m);
          put_row16(c, c.slot(4 - par), r);
        }
        arrive_ready(c, 5);
      }
      if (main_part) {
        take(c, 3, 0, c.slot(5 + par), c.act, v, 5.f * c.trunc);  // D
        if (c.act) {
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = -fmaf(4.f, hd[i], v[i]);
          put_row16(c, c.slot(5 + par), v);
        }
        arrive_ready(c, 6);
        if (!prime && finish > 0) {                      // the first operands of the landmark gradients, ahead of time
          load_tile16(p.kt + bh * md, m, min(D, kN), D, W || c.md16, hd);
          load_tile16(p.qt + bh * md, m, min(D, kN), D, W || c.md16, r);
        }
      }
      if (prime) {
        take(c, 4, kAccCols, c.slot(7), c.act, v, c.trunc);       // W
        if (c.act) {
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = fmaf(0.25f, v[i], r[i]);
          add_diag(c, v, 1.f, m);
          put_row16(c, c.slot(7), v);
        }
        if (!main_part) arrive_ready(c, 0);
      }
      if (main_part) {
        take(c, 5, 3 * kAccCols, c.slot(6 - par), c.act, v, 3.f * c.trunc);   // G
        if (c.act) {
#pragma unroll
          for (int i = 0; i < 16; ++i) g[i] += v[i];
          if (prime) put_row16(c, c.slot(6 - par), g);
        }
        if (prime) arrive_ready(c, 0);
      }
      if (prime) {
        take(c, 6, 2 * kAccCols, c.slot(8), c.act, v, c.trunc);   // Y
        if (c.act) put_row16(c, c.slot(8), v);
        arrive_ready(c, 1);
      }
      if (main_part) {
        wait_done(c, 7, 0x2107);                         // dL/dA
        if (c.act) {
          float keep[16], send[16];
          fetch(c, 0, c.trunc, keep, send);
#pragma unroll
          for (int i = 0; i < 16; ++i) { da_keep[i] += keep[i]; da_send[i] += send[i]; }
        }
      }
    }
  }
}

template <bool W>
__global__ void __launch_bounds__(kNsTcThreads, 1) ns_bwd_tc_kernel(BwdParams f, int finish, int* status) {
  extern __shared__ uint8_t dyn_smem[];
  __shared__ float red[ns::kRedFloats];
  __shared__ Shared sh;
  Ctx c;
  pdl_trigger();
  ctx_open(c, sh, dyn_smem, status, kBwdTmemCols, f.p.m);
  c.md16 = whole16(f.p.qt, f.p.kt, f.h.bmat);
  pdl_wait();
  if (is_compute()) bwd_compute<W>(c, red, f, blockIdx.x, finish);
  else bwd_issue(c, f, finish);
  ctx_close(c, kBwdTmemCols);
}

// the form for a call
inline auto bwd_kernel(const BwdParams& f) {
  const ns::NsBwdParams& p = f.p;
  return (p.m & 3) == 0 && whole16(p.qt, p.kt, p.k2, p.iterates, p.G, p.spill, f.h.k2inv, f.h.bmat, f.dK2, f.step_dz, f.step_da)
             ? ns_bwd_tc_kernel<true> : ns_bwd_tc_kernel<false>;
}

}  // namespace nstc
}  // namespace fnb
