// Landmark-sized stages for 64 < num_landmarks <= 128 on the sm_100a tensor cores, FP32-equivalent: a
// thread-block cluster of two CTAs per (b,h) slice works through the softmax-2, ridge and Newton-Schulz
// products (forward and exact backward).
//
// Outside the forward iteration, which keeps its operands on the chip (fwd_program), every matrix that is an operand exists
// once as an "image" in global memory (it stays in L2): three bf16
// terms x = x0 + x1 + x2 (24 significant bits), padded with zeros to 128 x 128, already in the 128-byte
// swizzle the tensor core reads, [64-column block][term][128 rows x 128 B].  The epilogue that forms a result
// splits it once and writes its image; a consumer's operands are plain bulk copies into a ring of shared-
// memory stages, K in chunks of 64, in whichever orientation the product needs (an image serves as left or
// right operand, plain or transposed, by the pieces that are copied and the descriptor they are read
// with).  CTA `rank` of the pair forms the 64 output columns [64 rank, 64 rank + 64) of every product; the
// terms of the right operand are stacked along N, so a K step of 16 is three MMAs (four in the second chunk),
//     x0 [y0 | y1 | y2],  x1 [y0 | y1],  x2 [y0],
// into column groups by weight that the epilogue adds, small ones first.  x0 y0 has one group per chunk: the
// tensor core truncates when it adds, and with a single group fp32 dQ and dK were up to 30 % less precise
// than with the products added up one by one in FP32.
// 16 compute warps (epilogues and element-wise phases), one warp that copies, one that issues MMAs; all run
// through the same program.  A phase ends with an arrival of all warps of both CTAs on both CTAs'
// `ready` barriers; operands that are older than the last phase are copied ahead of it.  All waits are
// bounded; control flow never depends on them.
//
// The iteration runs in its residual form (ns_tc_kernels.cuh): with R = I - A Z three dependent phases in place of four.
//
// What bounds it: forward, the products of an iteration (four, 2400 cycles each: shared-memory bandwidth, an MMA set of a K step
// reads 24 KB) and between them the way of a result through registers, split and shared memory (2500 cycles, three times);
// backward, the same with what a phase waits for: copies out of L2 (9 KB per K step), the result block out to it (put 1600,
// publish 2300), the peer, the first chunk in (1550).  Measured at B=2, H=8, m=128 (us): forward D=128, J=8 with
// ridge 222 with four products in a row, 205 in residual form through L2, 136 with the operands on the chip (121 of it behind the
// softmax); D=64, J=6 without 164, 152, 100; backward 447 / 406 and 318 / 287.
#pragma once
#include "common.cuh"
#include "small_kernels.cuh"
#include "split_stream.cuh"
#include "tc_common.cuh"

namespace fnb {
namespace mx {

using namespace tc;

constexpr int kTermBytes = 128 * 128;          // 128 rows x 64 columns of one term
constexpr int kBlockBytes = 3 * kTermBytes;    // a 64-column block of an image
constexpr int kImg = 2 * kBlockBytes;
constexpr int kStages = 2;
constexpr int kStageBytes = kBlockBytes + kBlockBytes / 2;   // left chunk (128 x 64) and right chunk (64 x 64), all terms
constexpr int kComputeWarps = 16;
constexpr int kThr = 32 * (kComputeWarps + 2);
constexpr int kRedFloats = 64 * kMaxM;          // 17 kMaxM for norms(); the forward iteration stages 64 columns of an iterate
constexpr size_t kSmem = (size_t)kStages * kStageBytes + kBlockBytes + kRedFloats * sizeof(float) + 256 + 1024;
constexpr int kAccCols = 256;                  // tensor-memory columns of one accumulator
constexpr int kF32 = kMaxM * kMaxM;            // floats of one FP32 scratch matrix

// scratch of a cluster: images, then FP32 matrices.  A launch has at most as many clusters as run at once; each walks slices
// gridDim.x / 2 apart and works in one scratch area, so that the scratch stays in L2 and does not grow with the slices.
enum FwdImg { kFK2, kFA, kFR, kFW, kFwdImgs };
constexpr size_t kFwdScratchBytes = (size_t)kFwdImgs * kImg + kF32 * sizeof(float);
enum BwdImg { kBK2, kBA, kBZ0, kBZ1, kBZ2, kBG0, kBG1, kBR0, kBR1, kBW, kBY, kBdY, kBH, kBwdImgs };
enum BwdF32 { kGA, kGdZ, kGdK, kGg, kBwdF32s };
constexpr size_t kBwdScratchBytes = (size_t)kBwdImgs * kImg + (size_t)kBwdF32s * kF32 * sizeof(float);

// Share of a leading partial product that its truncating additions (three per group of four K steps) have lost on the average.
// Given back, K2inv is 0.45 to 0.98 times as far from the oracle as in the nested form, without it up to 1.17 times.
constexpr float kTrunc = 0x1.8p-25f;
// Two and three products in one accumulator: four additions more for each (dL/dK2 1.0 times as far from 64 bits as FP32 sums are, 1.2 to
// 1.3 times with one product's share for all).
constexpr float kTrunc2 = 7 * kTrunc / 3, kTrunc3 = 11 * kTrunc / 3;

enum { kProducer = 0, kIssuer = 1, kCompute = 2 };

struct Shared {
  uint64_t full[kStages], empty[kStages], done[2], released[2], ready, drain;
  // forward iteration: products complete in both CTAs; result blocks written here; blocks that came from the peer; slots loaded
  uint64_t both[2], put, came[3], loaded[2];
  uint32_t tmem_slot;
  uint32_t loads[2];        // loads of each slot, written when the issuing warp is through
  uint32_t inbound[4][3];   // copies that the peer has sent here, likewise
  uint32_t fills;           // stages filled by the copying warp, written when it is through
  int abort_word;
};

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// One arrival on this CTA's barrier and one on the peer's.  The remote one is relaxed: whoever has written
// something the peer reads has fenced it before.
__device__ __forceinline__ void arrive_both(uint64_t* bar, int rank) {
  uint32_t ra;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(smem_u32(bar)), "r"(rank ^ 1));
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(ra) : "memory");
  mbar_arrive(bar);
}
__device__ __forceinline__ bool wait_cluster(uint64_t* bar, uint32_t parity, const Abort& ab, int where) {
  uint64_t t0 = 0;
  for (uint32_t spin = 0;; ++spin) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    if (ok) return true;
    if ((spin & 63u) == 63u) {
      if (ab.raised()) return false;
      const uint64_t now = global_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > g_wait_limit_ns) break;
    }
  }
  ab.raise(where);
  return false;
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const uint8_t* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
               "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void bulk_store(uint8_t* dst, uint32_t src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }
__device__ __forceinline__ void compute_sync() { named_barrier(1, 32 * kComputeWarps); }

// 16 values, columns 16 seg .. 16 seg + 15 of row r (seg counts over both column blocks) -> image
__device__ __forceinline__ void put16(uint8_t* img, int r, int seg, const float* v) {
  uint4 a[3], b[3];
  sx::split8<3>(v, a);
  sx::split8<3>(v + 8, b);
  const int cg = seg & 3, odd = r & 1;
  uint8_t* p = img + (seg >> 2) * kBlockBytes + r * 128 + (((2 * cg) ^ (r & 6)) << 4);
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    const uint4 lo = odd ? b[t] : a[t], hi = odd ? a[t] : b[t];
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p + t * kTermBytes), "r"(lo.x), "r"(lo.y),
                 "r"(lo.z), "r"(lo.w), "r"(hi.x), "r"(hi.y), "r"(hi.z), "r"(hi.w)
                 : "memory");
  }
}
// 4 values, columns 4 lane .. 4 lane + 3 of row r -> image (a warp writes a whole row)
__device__ __forceinline__ void put_row(uint8_t* img, int r, int lane, const float* v) {
  uint8_t* p = img + (lane >> 4) * kBlockBytes + sw128_offset(r, (lane >> 1) & 7) + (lane & 1) * 8;
  float a[4] = {v[0], v[1], v[2], v[3]};
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    const uint32_t w0 = pack2<__nv_bfloat16>(a[0], a[1]), w1 = pack2<__nv_bfloat16>(a[2], a[3]);
    *reinterpret_cast<uint2*>(p + t * kTermBytes) = make_uint2(w0, w1);
    a[0] -= __uint_as_float(w0 << 16); a[1] -= __uint_as_float(w0 & 0xffff0000u);
    a[2] -= __uint_as_float(w1 << 16); a[3] -= __uint_as_float(w1 & 0xffff0000u);
  }
}
// n consecutive values of an FP32 row (zero past `cols`); n a multiple of 4
template <int n>
__device__ __forceinline__ void get_row(const float* g, int c0, int cols, bool row_ok, float* v) {
  const float* src = g + c0;
  if ((reinterpret_cast<uintptr_t>(src) & 15u) == 0 && (cols & 3) == 0) {
#pragma unroll
    for (int q = 0; q < n; q += 4) {
      const float4 x = (row_ok && c0 + q < cols) ? __ldcg(reinterpret_cast<const float4*>(src + q)) : make_float4(0.f, 0.f, 0.f, 0.f);
      v[q] = x.x; v[q + 1] = x.y; v[q + 2] = x.z; v[q + 3] = x.w;
    }
  } else {
#pragma unroll
    for (int i = 0; i < n; ++i) v[i] = (row_ok && c0 + i < cols) ? __ldcg(src + i) : 0.f;
  }
}
template <int n>
__device__ __forceinline__ void set_row(float* g, int c0, int cols, bool row_ok, const float* v) {
  if (!row_ok) return;
  float* dst = g + c0;
  if ((reinterpret_cast<uintptr_t>(dst) & 15u) == 0 && (cols & 3) == 0) {
#pragma unroll
    for (int q = 0; q < n; q += 4)
      if (c0 + q < cols) *reinterpret_cast<float4*>(dst + q) = make_float4(v[q], v[q + 1], v[q + 2], v[q + 3]);
  } else {
#pragma unroll
    for (int i = 0; i < n; ++i)
      if (c0 + i < cols) dst[i] = v[i];
  }
}

// The MMAs of one K chunk (64): warp-uniform code, one elected lane issues.  One block of assembly, so that the election
// happens once and the descriptors stay in uniform registers: issued from a single lane an MMA took 103 cycles, a product
// 2900, and the issuing warp bounded the backward.  d: accumulator, l: left chunk, r: right chunk.
// RS: bytes between the terms of the right chunk.
template <bool LT, bool RT, int RS = kTermBytes / 2>
__device__ __forceinline__ void issue_chunk(uint32_t d, uint32_t l, uint32_t r, bool second, bool accumulate) {
  const uint64_t a = LT ? smem_desc_sw128(l, kTermBytes / 2, 1024) : smem_desc_sw128(l, 16, 1024);
  const uint64_t b = RT ? smem_desc_sw128(r, 16, 1024) : smem_desc_sw128(r, RS, 1024);
  static_assert(!RT || RS == 64 * 128, "the rows of all terms are one operand");
  constexpr uint32_t i192 = make_idesc<__nv_bfloat16>(128, 192, LT, !RT), i128 = make_idesc<__nv_bfloat16>(128, 128, LT, !RT),
                     i64 = make_idesc<__nv_bfloat16>(128, 64, LT, !RT);
  constexpr int sa = LT ? 2048 / 16 : 2, sb = RT ? 2 : 2048 / 16, ta = kTermBytes / 16, tb = RS / 16;
  if (!second) {
    asm volatile(
          "{\n\t.reg .pred e, p, q;\n\t.reg .b64 a0, a1, a2, b, b1;\n\t.reg .b32 d1, d2, d3;\n\t"
          "elect.sync _|e, 0xffffffff;\n\t"
          "setp.ne.b32 p, %3, 0;\n\t"
          "setp.eq.b32 q, %3, %3;\n\t"
          "add.u32 d1, %0, 64;\n\tadd.u32 d2, %0, 128;\n\tadd.u32 d3, %0, 192;\n\t"
          "mov.b64 a0, %1;\n\tadd.s64 a1, %1, %9;\n\tadd.s64 a2, a1, %9;\n\tmov.b64 b, %2;\n\tadd.s64 b1, %2, %10;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a0, b, %4, p;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [d1], a1, b, %5, q;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [d2], a2, b, %6, q;\n\t"
          "add.s64 a0, a0, %7;\n\tadd.s64 a1, a1, %7;\n\tadd.s64 a2, a2, %7;\n\tadd.s64 b, b, %8;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a0, b, %4, q;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [d1], a1, b, %5, q;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [d2], a2, b, %6, q;\n\t"
          "add.s64 a0, a0, %7;\n\tadd.s64 a1, a1, %7;\n\tadd.s64 a2, a2, %7;\n\tadd.s64 b, b, %8;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a0, b, %4, q;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [d1], a1, b, %5, q;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [d2], a2, b, %6, q;\n\t"
          "add.s64 a0, a0, %7;\n\tadd.s64 a1, a1, %7;\n\tadd.s64 a2, a2, %7;\n\tadd.s64 b, b, %8;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a0, b, %4, q;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [d1], a1, b, %5, q;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [d2], a2, b, %6, q;\n\t"
          "}"
          ::"r"(d), "l"(a), "l"(b), "r"(accumulate ? 1u : 0u), "r"(i192), "r"(i128), "r"(i64), "n"(sa), "n"(sb), "n"(ta), "n"(tb)
          : "memory");
  } else {
    // b1: the second term of the right operand, its columns 0..127 then being y1 | y2
    asm volatile(
          "{\n\t.reg .pred e, p, q;\n\t.reg .b64 a0, a1, a2, b, b1;\n\t.reg .b32 d1, d2, d3;\n\t"
          "elect.sync _|e, 0xffffffff;\n\t"
          "setp.ne.b32 p, %3, 0;\n\t"
          "setp.eq.b32 q, %3, %3;\n\t"
          "add.u32 d1, %0, 64;\n\tadd.u32 d2, %0, 128;\n\tadd.u32 d3, %0, 192;\n\t"
          "mov.b64 a0, %1;\n\tadd.s64 a1, %1, %9;\n\tadd.s64 a2, a1, %9;\n\tmov.b64 b, %2;\n\tadd.s64 b1, %2, %10;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [d3], a0, b, %6, p;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [d1], a0, b1, %5, q;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [d1], a1, b, %5, q;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [d2], a2, b, %6, q;\n\t"
          "add.s64 a0, a0, %7;\n\tadd.s64 a1, a1, %7;\n\tadd.s64 a2, a2, %7;\n\tadd.s64 b, b, %8;\n\tadd.s64 b1, b1, %8;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [d3], a0, b, %6, q;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [d1], a0, b1, %5, q;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [d1], a1, b, %5, q;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [d2], a2, b, %6, q;\n\t"
          "add.s64 a0, a0, %7;\n\tadd.s64 a1, a1, %7;\n\tadd.s64 a2, a2, %7;\n\tadd.s64 b, b, %8;\n\tadd.s64 b1, b1, %8;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [d3], a0, b, %6, q;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [d1], a0, b1, %5, q;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [d1], a1, b, %5, q;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [d2], a2, b, %6, q;\n\t"
          "add.s64 a0, a0, %7;\n\tadd.s64 a1, a1, %7;\n\tadd.s64 a2, a2, %7;\n\tadd.s64 b, b, %8;\n\tadd.s64 b1, b1, %8;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [d3], a0, b, %6, q;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [d1], a0, b1, %5, q;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [d1], a1, b, %5, q;\n\t"
          "@e tcgen05.mma.cta_group::1.kind::f16 [d2], a2, b, %6, q;\n\t"
          "}"
          ::"r"(d), "l"(a), "l"(b), "r"(accumulate ? 1u : 0u), "r"(i192), "r"(i128), "r"(i64), "n"(sa), "n"(sb), "n"(ta), "n"(tb)
          : "memory");
  }
}

// One role's walk through the program.
template <int R>
struct Role {
  Shared* sh;
  uint8_t* ring;
  uint8_t* out;       // compute: staging of one result block, [term][128 rows x 128 B]
  float* red;
  uint32_t tmem;
  Abort ab;
  int rank, lane;
  bool failed, pend;
  uint32_t rphase;
  // copy / issue: position in the ring
  int stage;
  uint32_t sphase, fills;   // fills: stages filled so far, in ring order
  bool drop;                // test only: this CTA never issues one of its fills, so that a wait runs out
  // compute: accumulator row, column segment of 16 (over both blocks), completion parities
  int row, seg;
  uint32_t dphase[2];
  uint32_t relphase[2];     // issue: parity of the next wait on released[]
  uint32_t bphase[2], pphase, cphase[3], lphase[2], loads[2], sent[3];     // forward iteration: parities, loads and copies issued

  __device__ void open(Shared* s, uint8_t* r, float* rd, int rk, int* status, bool drop_fill) {
    drop = drop_fill;
    sh = s; ring = r; out = r + (size_t)kStages * kStageBytes; red = rd; rank = rk; lane = threadIdx.x & 31;
    tmem = s->tmem_slot;
    ab = Abort{&s->abort_word, status};
    failed = pend = false;
    rphase = sphase = fills = 0; stage = 0;
    dphase[0] = dphase[1] = relphase[0] = relphase[1] = bphase[0] = bphase[1] = pphase = 0;
    lphase[0] = lphase[1] = loads[0] = loads[1] = 0;
    for (int i = 0; i < 3; ++i) cphase[i] = sent[i] = 0;
    const int w = threadIdx.x >> 5;
    row = (w & 3) * 32 + lane;
    seg = rank * 4 + (w >> 2);
  }
  // the phase published last is complete in both CTAs (and, for a compute warp that asks, what the peer's
  // compute warps wrote with ordinary stores can be read)
  __device__ __forceinline__ void ensure(bool read_peer = true) {
    if (R == kCompute && read_peer && !pend) __threadfence();
    if (!pend) return;
    pend = false;
    if (R == kIssuer) {
      settle(wait_cluster(&sh->ready, rphase, ab, 0x6000 + R));
    } else if (R == kCompute || lane == 0) {
      if (!wait_cluster(&sh->ready, rphase, ab, 0x6000 + R)) failed = true;
      if (R == kProducer) fence_proxy_async_all();
      if (R == kCompute && read_peer) __threadfence();
    }
    if (R == kIssuer) tc_fence_after();
    rphase ^= 1u;
  }
  // This warp's part of the phase is done.  Images written through put() are complete; with `plain` so are the
  // ordinary global stores of the phase, for readers of either kind.
  __device__ __forceinline__ void publish(bool plain) {
    ensure(false);
    if (R == kCompute) {
      if (threadIdx.x < 128 && lane == 0) tma_store_wait_all();
      if (plain || (threadIdx.x < 128 && lane == 0)) {
        fence_proxy_async_all();
        __threadfence();
      }
      tc_fence_before();
    }
    __syncwarp();
    if (lane == 0) arrive_both(&sh->ready, rank);
    pend = true;
  }
  // The result block of this CTA (this thread: row, 16 columns) -> image.  The four warps that hold the same 32
  // rows stage their 4 KB per term, which one thread stores in bulk: stored straight from the accumulator layout
  // (32 rows x 32 B per instruction) the block took 3300 cycles and its fence 2000.
  __device__ __forceinline__ void put(uint8_t* img, const float* v) {
    const int q = (threadIdx.x >> 5) & 3;
    const bool storing = threadIdx.x < 128 && lane == 0;
    if (storing) tma_store_wait_read();
    named_barrier(2 + q, 128);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      uint4 a[3];
      sx::split8<3>(v + 8 * c, a);
      uint8_t* p = out + sw128_offset(row, (seg & 3) * 2 + c);
#pragma unroll
      for (int t = 0; t < 3; ++t) *reinterpret_cast<uint4*>(p + t * kTermBytes) = a[t];
    }
    fence_proxy_async();
    named_barrier(2 + q, 128);
    if (storing) {
      uint8_t* dst = img + rank * kBlockBytes + q * 4096;
#pragma unroll
      for (int t = 0; t < 3; ++t) bulk_store(dst + t * kTermBytes, smem_u32(out) + t * kTermBytes + q * 4096, 4096);
      tma_store_commit();
    }
  }
  // accumulator `acc` (+)= op(X) op(Y)[:, own columns].  fx, fy: the operand was written in the last phase.
  template <bool LT, bool RT>
  __device__ __forceinline__ void product(const uint8_t* X, bool fx, const uint8_t* Y, bool fy, int kchunks, int acc, bool accumulate) {
    if (R == kProducer) {
      if (lane == 0) {
        for (int kc = 0; kc < kchunks; ++kc) {
          if (!failed && !mbar_wait(&sh->empty[stage], sphase ^ 1u, ab, 0x6010)) failed = true;
          if (drop && fills == 2) failed = true;         // fault injection on the host's request
          const bool fill = !failed, meet = pend && (fx || fy);
          const uint32_t l = smem_u32(ring) + stage * kStageBytes, r = l + kBlockBytes;
          if (fill) {
            mbar_expect_tx(&sh->full[stage], kStageBytes);
            ++fills;
            if (!fx) load_left<LT>(l, X, kc);
            if (!fy) load_right<RT>(r, Y, kc);
          }
          if (meet) {
            if (!failed && !wait_cluster(&sh->ready, rphase, ab, 0x6011)) failed = true;
            fence_proxy_async_all();
            rphase ^= 1u;
            pend = false;
          }
          // (also after that wait has given up: the stage's barrier counts on all of its bytes, and the drain on the barrier)
          if (fill) {
            if (fx) load_left<LT>(l, X, kc);
            if (fy) load_right<RT>(r, Y, kc);
          }
          advance();
        }
      }
    } else if (R == kIssuer) {
      ensure();
      const uint32_t d = tmem + acc * kAccCols;
      for (int kc = 0; kc < kchunks; ++kc) {
        settle(failed || mbar_wait(&sh->full[stage], sphase, ab, 0x6020));
        if (!failed) {
          tc_fence_after();
          const uint32_t l = smem_u32(ring) + stage * kStageBytes;
          issue_chunk<LT, RT>(d, l, l + kBlockBytes, kc > 0, accumulate);
          umma_commit_elect(&sh->empty[stage]);
        }
        advance();
      }
    }
  }
  // issue: the warp goes on as one
  __device__ __forceinline__ void settle(bool ok) {
    if (!__all_sync(0xffffffffu, ok)) failed = true;
  }
  __device__ __forceinline__ void advance() {
    if (++stage == kStages) { stage = 0; sphase ^= 1u; }
  }
  template <bool LT>
  __device__ __forceinline__ void load_left(uint32_t dst, const uint8_t* X, int kc) {
    if (!LT) {
      bulk_load(dst, X + (size_t)kc * kBlockBytes, kBlockBytes, &sh->full[stage]);
    } else {
#pragma unroll
      for (int t = 0; t < 3; ++t)
#pragma unroll
        for (int cb = 0; cb < 2; ++cb)
          bulk_load(dst + t * kTermBytes + cb * (kTermBytes / 2), X + (size_t)cb * kBlockBytes + t * kTermBytes + kc * (kTermBytes / 2),
                    kTermBytes / 2, &sh->full[stage]);
    }
  }
  template <bool RT>
  __device__ __forceinline__ void load_right(uint32_t dst, const uint8_t* Y, int kc) {
    const uint8_t* src = RT ? Y + (size_t)kc * kBlockBytes + rank * (kTermBytes / 2) : Y + (size_t)rank * kBlockBytes + kc * (kTermBytes / 2);
#pragma unroll
    for (int t = 0; t < 3; ++t) bulk_load(dst + t * (kTermBytes / 2), src + t * kTermBytes, kTermBytes / 2, &sh->full[stage]);
  }
  __device__ __forceinline__ void commit(int g) {
    if (R == kIssuer && !failed) umma_commit_elect(&sh->done[g]);
  }
  // compute: the 16 values of this thread (row, columns 16 seg ..) of accumulator acc once group g is complete;
  // kchunks as in product()
  __device__ __forceinline__ void result(int g, int acc, float* v, int kchunks = 2, float trunc = kTrunc) {
    if (!mbar_wait(&sh->done[g], dphase[g], ab, 0x6030 + g)) failed = true;
    dphase[g] ^= 1u;
    take(acc, v, kchunks, trunc);
  }
  __device__ __forceinline__ void take(int acc, float* v, int kchunks = 2, float trunc = kTrunc) const {
    __syncwarp();
    tc_fence_after();
    const uint32_t a = tmem + (uint32_t)acc * kAccCols + ((uint32_t)(row & ~31) << 16) + (uint32_t)((seg & 3) * 16);
    float x[16], y[16];
    sx::ld<16>(a + 128, x);
    sx::ld<16>(a + 64, y);
    sx::ld<16>(a, v);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] += y[i];
    if (kchunks > 1) {
      sx::ld<16>(a + 192, y);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] += y[i];
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] += fmaf(trunc, v[i], x[i]);
  }
  // An accumulator that is used again within a phase: the compute warps release it once it has been read, the issuing
  // warp waits for that (as often as it is released).
  __device__ __forceinline__ void release(int acc) {
    if (R == kCompute) {
      tc_fence_before();
      mbar_arrive_warp(&sh->released[acc]);
    }
  }
  __device__ __forceinline__ void reuse(int acc) {
    if (R == kIssuer) {
      settle(failed || mbar_wait(&sh->released[acc], relphase[acc], ab, 0x6040 + acc));
      relphase[acc] ^= 1u;
      tc_fence_after();
    }
  }
  // ---- forward iteration: operands stay in four blocks of shared memory ("slots", where ring and staging are otherwise)
  __device__ __forceinline__ uint32_t slot(int i) const { return smem_u32(ring) + i * kBlockBytes; }
  // every product issued before is complete in both CTAs
  __device__ __forceinline__ void wait_both(int g) {
    const bool ok = mbar_wait(&sh->both[g], bphase[g], ab, 0x6050 + g);
    if (R == kIssuer) settle(failed || ok);
    else if (!ok) failed = true;
    bphase[g] ^= 1u;
  }
  __device__ __forceinline__ void commit_both(int g) {
    if (!failed)
      asm volatile(
          "{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
          "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}"
          ::"r"(smem_u32(&sh->both[g])), "h"((uint16_t)3)
          : "memory");
  }
  // compute: this thread's 16 values -> its place in slot i
  __device__ __forceinline__ void put_slot(int i, const float* v) {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      uint4 w[3];
      sx::split8<3>(v + 8 * c, w);
      uint8_t* p = ring + (size_t)i * kBlockBytes + sw128_offset(row, (seg & 3) * 2 + c);
#pragma unroll
      for (int t = 0; t < 3; ++t) *reinterpret_cast<uint4*>(p + t * kTermBytes) = w[t];
    }
    fence_proxy_async();
  }
  // for the issuing warp: the blocks put so far are there
  __device__ __forceinline__ void announce() {
    tc_fence_before();
    mbar_arrive_warp(&sh->put);
  }
  // the block put into slot `from` -> slot `to` of the peer.  The four warps that hold the same 32 rows have them copied in bulk
  // by one thread: stored from the registers (32 rows x 16 B per instruction) a block took 3000 cycles.
  __device__ __forceinline__ void send(int from, int to, int what) {
    const int q = (threadIdx.x >> 5) & 3;
    named_barrier(2 + q, 128);
    if (threadIdx.x < 128 && lane == 0 && !failed) {
      uint32_t dst, bar;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(slot(to) + q * 4096), "r"(rank ^ 1));
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(bar) : "r"(smem_u32(&sh->came[what])), "r"(rank ^ 1));
      asm volatile("mbarrier.arrive.expect_tx.relaxed.cluster.shared::cluster.b64 _, [%0], %1;" ::"r"(bar), "r"(3 * 4096) : "memory");
#pragma unroll
      for (int t = 0; t < 3; ++t)
        asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(dst + t * kTermBytes), "r"(slot(from) + q * 4096 + t * kTermBytes), "r"(4096), "r"(bar) : "memory");
      ++sent[what];
    }
  }
  // this thread's 16 values -> staged row (64 columns, 16-byte words swizzled); after a barrier of the four warps of these
  // rows (send() has one), the staged rows -> an (m x m) matrix.  Stored from the accumulator layout (32 rows x 16 B per
  // instruction) an iterate took 3500 cycles, and everything behind it waited.
  __device__ __forceinline__ void stage_rows(const float* v) {
    float4* dst = reinterpret_cast<float4*>(red) + row * 16;
#pragma unroll
    for (int q = 0; q < 4; ++q) dst[((seg & 3) * 4 + q) ^ (row & 15)] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
  }
  __device__ __forceinline__ void store_rows(float* g, int m) const {
    const int w = threadIdx.x >> 5, c = lane & 15;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int rr = (w & 3) * 32 + (w >> 2) * 8 + 2 * i + (lane >> 4);
      const float4 x = reinterpret_cast<const float4*>(red)[rr * 16 + (c ^ (rr & 15))];
      const float v[4] = {x.x, x.y, x.z, x.w};
      set_row<4>(g + (size_t)rr * m, rank * 64 + 4 * c, m, rr < m && !failed, v);
    }
  }
  __device__ __forceinline__ void row_sync() { named_barrier(2 + ((threadIdx.x >> 5) & 3), 128); }
  // issue
  __device__ __forceinline__ void wait_put() {
    settle(failed || mbar_wait(&sh->put, pphase, ab, 0x6060));
    pphase ^= 1u;
    tc_fence_after();
  }
  __device__ __forceinline__ void wait_came(int what) {
    settle(failed || wait_cluster(&sh->came[what], cphase[what], ab, 0x6070 + what));
    cphase[what] ^= 1u;
  }
  __device__ __forceinline__ void wait_loaded(int l) {
    settle(failed || mbar_wait(&sh->loaded[l], lphase[l], ab, 0x6080 + l));
    lphase[l] ^= 1u;
  }
  // may the next load be issued?  (lane 0 issues it)
  __device__ __forceinline__ bool begin_load(int l, uint32_t bytes) {
    if (drop && loads[0] + loads[1] == 2) failed = true;     // fault injection on the host's request
    if (failed) return false;
    ++loads[l];
    if (lane == 0) mbar_expect_tx(&sh->loaded[l], bytes);
    return lane == 0;
  }
  template <bool RT = false, int RS = kTermBytes>
  __device__ __forceinline__ void chunk(int acc, uint32_t left, uint32_t right, bool second) {
    if (!failed) issue_chunk<false, RT, RS>(tmem + acc * kAccCols, left, right, second, false);
  }
  __device__ __forceinline__ int col0() const { return 16 * seg; }
  __device__ __forceinline__ void add_diag(float* v, float d, int m) const {
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] += (col0() + i == row && row < m) ? d : 0.f;
  }
  // (rows x cols) FP32 matrix -> this CTA's half of the rows of its image
  __device__ __forceinline__ void convert(const float* g, int rows, int cols, uint8_t* img) {
    const int r = rank * 64 + (threadIdx.x >> 3), s = threadIdx.x & 7;
    if (16 * s >= 64 && cols <= 64) return;      // the second block of such an operand is never copied
    float v[16];
    get_row<16>(g + (size_t)r * cols, 16 * s, cols, r < rows, v);
    put16(img, r, s, v);
  }
  __device__ void close() {
    ensure();
    if (R == kProducer && lane == 0) sh->fills = fills;
    if (R == kIssuer && lane == 0)
      for (int i = 0; i < 2; ++i) sh->loads[i] = loads[i];
    if (R == kCompute && threadIdx.x < 128 && lane == 0)       // (the peer counts on these copies until they have arrived)
      for (int i = 0; i < 3; ++i) {
        uint32_t at;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_u32(&sh->inbound[threadIdx.x >> 5][i])), "r"(rank ^ 1));
        asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(at), "r"(sent[i]) : "memory");
      }
  }
};

// ||A||_1, ||A||_inf and their first-occurrence argmax positions (compute warps; A: m x m in global memory)
struct Norms { float n1, ninf; int jc, ir; };
__device__ inline Norms norms(const float* A, int m, float* red) {
  const int t = threadIdx.x, w = t >> 5, lane = t & 31;
  float* rowsum = red;
  float* colpart = red + kMaxM;
  float cs[4] = {0.f, 0.f, 0.f, 0.f};
  float x[kMaxM / kComputeWarps][4];      // every load in flight at once
#pragma unroll
  for (int i = 0; i < kMaxM / kComputeWarps; ++i) {
    const int r = w + i * kComputeWarps;
#pragma unroll
    for (int q = 0; q < 4; ++q) x[i][q] = (r < m && lane + 32 * q < m) ? fabsf(__ldcg(A + (size_t)r * m + lane + 32 * q)) : 0.f;
  }
#pragma unroll
  for (int i = 0; i < kMaxM / kComputeWarps; ++i) {
    float rs = 0.f;
#pragma unroll
    for (int q = 0; q < 4; ++q) { cs[q] += x[i][q]; rs += x[i][q]; }
    for (int o = 16; o > 0; o >>= 1) rs += __shfl_xor_sync(0xffffffffu, rs, o);
    if (lane == 0) rowsum[w + i * kComputeWarps] = rs;
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) colpart[w * kMaxM + lane + 32 * q] = cs[q];
  compute_sync();
  if (t < m) {
    float s = 0.f;
#pragma unroll
    for (int ww = 0; ww < kComputeWarps; ++ww) s += colpart[ww * kMaxM + t];
    colpart[t] = s;           // (column t of the first partial row is read by this thread alone)
  }
  compute_sync();
  // every warp finds both maxima for itself
  float b[2];
  int bi[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const float* src = k ? rowsum : colpart;
    float best = -1.f;
    int at = 0;
    for (int c = lane; c < m; c += 32)
      if (src[c] > best) { best = src[c]; at = c; }
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, at, o);
      if (ob > best || (ob == best && oi < at)) { best = ob; at = oi; }
    }
    b[k] = best; bi[k] = at;
  }
  compute_sync();
  return Norms{b[0], b[1], bi[0], bi[1]};
}

// ---- forward ------------------------------------------------------------------------------------------
struct FwdParams {
  const float* qt; const float* kt;       // [BH][m][D]; null: k2 is given (softmaxed)
  float* k2; float* lse2; float* iterates; float* k2inv;
  uint8_t* scratch;                       // [gridDim.x / 2][kFwdScratchBytes]
  int64_t BH;
  int m, D, J;
  float kappa;
  int* status;
  int test_drop;                          // test only: CTA 0 never issues one fill
};

template <int R>
__device__ __forceinline__ void fwd_program(Role<R>& r, const FwdParams& p, int64_t bh) {
  constexpr bool C = R == kCompute;
  const int m = p.m, D = p.D, mm = m * m;
  uint8_t* base = p.scratch + (int64_t)(blockIdx.x >> 1) * kFwdScratchBytes;
  auto img = [&](int i) { return base + (size_t)i * kImg; };
  float* a32 = reinterpret_cast<float*>(base + (size_t)kFwdImgs * kImg);
  float* k2 = p.k2 + bh * mm;
  float* iterates = p.iterates + bh * (int64_t)(p.J + 1) * mm;
  float* k2inv = p.k2inv + bh * mm;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float v[16];
  if (p.qt) {
    if (C) {
      r.convert(p.qt + bh * m * D, m, D, img(kFR));
      r.convert(p.kt + bh * m * D, m, D, img(kFW));
    }
    r.publish(true);
    r.template product<false, true>(img(kFR), true, img(kFW), true, (D + 63) / 64, 0, false);
    r.commit(0);
    if (C) {
      r.result(0, 0, v, (D + 63) / 64, 0.f);
      r.stage_rows(v);
      r.row_sync();
      r.store_rows(k2, m);
    }
    r.publish(true);
  }
  if (C) {
    r.ensure();
    // row softmax (this CTA's half of the rows, one warp per row, four columns per lane)
    for (int i = 0; i < 4; ++i) {
      const int row = r.rank * 64 + 4 * w + i;
      float x[4];
      get_row<4>(k2 + (size_t)row * m, 4 * lane, m, row < m, x);
      if (p.qt && row < m) {
        float mx = -INFINITY;
#pragma unroll
        for (int q = 0; q < 4; ++q) if (4 * lane + q < m) mx = fmaxf(mx, x[q]);
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        float sum = 0.f;
#pragma unroll
        for (int q = 0; q < 4; ++q) { x[q] = 4 * lane + q < m ? expf(x[q] - mx) : 0.f; sum += x[q]; }
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
#pragma unroll
        for (int q = 0; q < 4; ++q) x[q] /= sum;
        if (!r.failed) set_row<4>(k2 + (size_t)row * m, 4 * lane, m, true, x);
        if (lane == 0) p.lse2[bh * m + row] = mx + logf(sum);
      }
      put_row(img(kFK2), row, lane, x);
    }
  }
  r.publish(true);
  const uint8_t* A = img(kFK2);
  const float* A32 = k2;
  if (p.kappa > 0.f) {
    r.template product<true, false>(img(kFK2), true, img(kFK2), true, 2, 0, false);
    r.commit(0);
    if (C) {
      r.ensure();
      const Norms nk = norms(k2, m, r.red);
      r.result(0, 0, v);
      r.add_diag(v, nk.n1 * nk.ninf / p.kappa, m);
      r.put(img(kFA), v);
      r.stage_rows(v);
      r.row_sync();
      r.store_rows(a32, m);
    }
    r.publish(true);
    A = img(kFA);
    A32 = a32;
  }
  // R = I - A Z, then Y = Z R and W = I + R + R^2 / 4 side by side, then Z' = Z + Y W.  All operands are on the chip: a
  // block of 64 columns is left operand (K) and right operand (columns) from the same place, a CTA's own block needs no
  // exchange, and the products begin with it; the peer's block, needed on the left only, arrives behind them from the peer's
  // shared memory.  So no phase waits for the L2.  Slots: 0, 1 hold Z, then Y (own block, peer's); 2, 3 hold R
  // (W in 2), and before that the two blocks of A, which come from its image while Z' is formed.  A slot is written again
  // after the products that read it are complete in BOTH CTAs (commits arrive in both).
  constexpr bool I = R == kIssuer;
  const bool ridge = p.kappa > 0.f;
  const int own = r.rank, peer = r.rank ^ 1;
  enum { kFromR, kFromY, kFromZ };
  constexpr uint32_t half = kTermBytes / 2;       // 64 rows of a block
  float z[16], rv[16];
  r.ensure();
  auto load_A = [&](int b) {
    if (r.begin_load(b, kBlockBytes)) bulk_load(r.slot(2 + b), A + (size_t)b * kBlockBytes, kBlockBytes, &r.sh->loaded[b]);
  };
  if (I) {
    fence_proxy_async_all();
    load_A(1);
    load_A(0);
  }
  if (C) {
    // Z0 = A^T / c, lanes along the rows of Z0 (the columns of A)
    const Norms na = norms(A32, m, r.red);
    const float c = fmaxf(na.n1 * na.ninf, 1e-12f);
#pragma unroll
    for (int i = 0; i < 16; ++i) z[i] = (r.row < m && r.col0() + i < m) ? __ldcg(A32 + (size_t)(r.col0() + i) * m + r.row) / c : 0.f;
    r.put_slot(0, z);
    r.announce();
    r.stage_rows(z);
    r.send(0, 1, kFromZ);
    r.store_rows(iterates, m);
  }
  for (int j = 0; j < p.J; ++j) {
    const bool more = j + 1 < p.J;
    if (I) {
      r.wait_put();                                  // Z
      r.wait_loaded(1);
      tc_fence_after();
      r.chunk(0, r.slot(3), r.slot(0) + half, false);
      r.wait_loaded(0);
      r.chunk(0, r.slot(2), r.slot(0), true);
      r.commit_both(0);
      r.wait_put();                                  // R
      r.wait_both(0);
      r.wait_came(kFromZ);
      r.chunk(0, r.slot(0), r.slot(2) + own * half, false);
      r.chunk(0, r.slot(1), r.slot(2) + peer * half, true);
      r.commit_both(0);
      r.chunk(1, r.slot(2), r.slot(2) + own * half, false);
      r.wait_came(kFromR);
      r.chunk(1, r.slot(3), r.slot(2) + peer * half, true);
      r.commit_both(1);
      r.wait_put();                                  // Y and W
      r.wait_both(0);
      r.wait_both(1);
      r.chunk(0, r.slot(0), r.slot(2) + own * half, false);
      if (more) load_A(1);
      r.wait_came(kFromY);
      r.chunk(0, r.slot(1), r.slot(2) + peer * half, true);
      r.commit_both(0);
      r.wait_both(0);
      if (more) {
        load_A(0);
      } else if (ridge && r.begin_load(0, kBlockBytes)) {
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
          for (int x = 0; x < 3; ++x)
            bulk_load(r.slot(2) + (b * 3 + x) * half, img(kFK2) + (size_t)b * kBlockBytes + x * kTermBytes + own * half, half, &r.sh->loaded[0]);
      }
    }
    if (C) {
      r.wait_both(0);
      r.take(0, rv);
#pragma unroll
      for (int i = 0; i < 16; ++i) rv[i] = -rv[i];
      r.add_diag(rv, 1.f, m);
      r.put_slot(2, rv);
      r.announce();
      r.send(2, 3, kFromR);
      r.wait_both(0);
      r.take(0, v);
      r.put_slot(0, v);
      r.send(0, 1, kFromY);
      r.wait_both(1);
      r.take(1, v);
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = fmaf(0.25f, v[i], rv[i]);
      r.add_diag(v, 1.f, m);
      r.put_slot(2, v);
      r.announce();
      r.wait_both(0);
      r.take(0, v);
#pragma unroll
      for (int i = 0; i < 16; ++i) z[i] += v[i];
      if (more || ridge) {
        r.put_slot(0, z);
        r.announce();
        r.stage_rows(z);
        r.send(0, 1, kFromZ);
      } else {
        r.stage_rows(z);
        r.row_sync();
        r.store_rows(k2inv, m);
      }
      r.store_rows(iterates + (size_t)(j + 1) * mm, m);
    }
  }
  if (ridge) {                                       // K2inv = Z_J K2^T
    if (I) {
      r.wait_put();
      r.wait_loaded(0);
      tc_fence_after();
      r.template chunk<true, kTermBytes / 2>(0, r.slot(0), r.slot(2) + own * 3 * half, false);
      r.wait_came(kFromZ);
      r.template chunk<true, kTermBytes / 2>(0, r.slot(1), r.slot(2) + peer * 3 * half, true);
      r.commit_both(0);
      r.wait_both(0);
    }
    if (C) {
      r.wait_both(0);
      r.take(0, v);
      r.row_sync();                                  // the staged rows of Z_J have left
      r.stage_rows(v);
      r.row_sync();
      r.store_rows(k2inv, m);
    }
  }
  r.close();
}

// ---- backward -----------------------------------------------------------------------------------------
struct BwdParams {
  const float* sums;          // [BH][2][m][D]: dstep2, dKt sums of the row pass
  const float* qt; const float* kt; const float* k2; const float* iterates; const float* k2inv; const float* bmat;
  float* dO3; float* D3;      // [BH][m][D], [BH][m]
  float* dqt_ns; float* dkt_tot; float* rows_k;   // [BH][m][D]; rows_k (scale * dkt_tot / segment length) may be null
  const float* G;             // debug entry: dL/dk2inv given, dK2 wanted
  float* dK2;
  uint8_t* scratch;           // [gridDim.x / 2][kBwdScratchBytes]
  int64_t BH;
  int m, D, J;
  float kappa, scale;
  int64_t N;
  int head, tail;             // run dO3 / D3 / dK2inv; run the pseudoinverse backward and what follows
  int* status;
  int test_drop;
};

template <int R>
__device__ __forceinline__ void bwd_program(Role<R>& r, const BwdParams& p, int64_t bh) {
  constexpr bool C = R == kCompute;
  const int m = p.m, D = p.D, mm = m * m, md = m * D, J = p.J;
  const bool ridge = p.kappa > 0.f;
  uint8_t* base = p.scratch + (int64_t)(blockIdx.x >> 1) * kBwdScratchBytes;
  auto img = [&](int i) { return base + (size_t)i * kImg; };
  auto f32 = [&](int i) { return reinterpret_cast<float*>(base + (size_t)kBwdImgs * kImg) + (size_t)i * kF32; };
  const float* k2 = p.k2 + bh * mm;
  const float* iterates = p.iterates + bh * (int64_t)(J + 1) * mm;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool own_d = r.rank * 64 < D;          // this CTA has columns of an (m x D) result
  uint8_t* Gi = ridge ? img(kBH) : img(kBG0 + (J & 1));     // dL/dk2inv; without the ridge it is dL/dZ_J
  float v[16];
  if (p.head) {
    const float* dstep2 = p.sums + bh * 2 * md;
    float* dO3 = p.dO3 + bh * md;
    if (C) {
      r.convert(p.k2inv + bh * mm, m, m, img(kBR0));
      r.convert(dstep2, m, D, img(kBR1));
      r.convert(p.bmat + bh * md, m, D, img(kBW));
    }
    r.publish(true);
    if (own_d) {
      r.template product<true, false>(img(kBR0), true, img(kBR1), true, 2, 0, false);     // dO3 = K2inv^T dstep2
      r.commit(0);
    }
    r.template product<false, true>(img(kBR1), true, img(kBW), true, (D + 63) / 64, 1, false);  // dK2inv = dstep2 Bmat^T
    r.commit(1);
    if (C) {
      if (own_d) {
        r.result(0, 0, v);
        set_row<16>(dO3 + (size_t)r.row * D, r.col0(), D, r.row < m && !r.failed, v);
      }
      r.result(1, 1, v, (D + 63) / 64);
      r.put(Gi, v);
      set_row<16>(f32(kGdZ) + (size_t)r.row * m, r.col0(), m, r.row < m, v);     // (read back by this thread, maybe in a launch of its own)
    }
    r.publish(true);
    if (C) {
      r.ensure();
      for (int i = 0; i < 4; ++i) {
        const int row = r.rank * 64 + 4 * w + i;
        if (row >= m) continue;
        float s = 0.f;
        for (int d = lane; d < D; d += 32) s = fmaf(p.bmat[bh * md + row * D + d], __ldcg(dO3 + row * D + d), s);
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) p.D3[bh * m + row] = s;
      }
    }
  }
  if (!p.tail) { r.close(); return; }
  float* out32 = p.G ? p.dK2 + bh * mm : f32(kGg);
  if (C) {
    if (p.G) r.convert(p.G + bh * mm, m, m, Gi);
    r.convert(k2, m, m, img(kBK2));
    r.convert(iterates + (size_t)(J - 1) * mm, m, m, img(kBZ0 + (J - 1) % 3));
    if (J > 1) r.convert(iterates + (size_t)(J - 2) * mm, m, m, img(kBZ0 + (J - 2) % 3));
    if (ridge) r.convert(iterates + (size_t)J * mm, m, m, img(kBY));
  }
  r.publish(true);
  const uint8_t* A = img(kBK2);
  const float* A32 = k2;
  float g[16];                                    // dL/dZ of the iterate above
  if (C && !ridge) get_row<16>((p.G ? p.G + bh * mm : f32(kGdZ)) + (size_t)r.row * m, r.col0(), m, r.row < m, g);
  if (ridge) {
    r.template product<true, false>(img(kBK2), true, img(kBK2), true, 2, 0, false);
    r.commit(0);
    r.template product<true, false>(Gi, true, img(kBY), true, 2, 1, false);          // G^T Z_J
    r.commit(1);
    if (C) {
      const Norms nk = norms(k2, m, r.red);
      r.result(0, 0, v);
      r.add_diag(v, nk.n1 * nk.ninf / p.kappa, m);
      r.put(img(kBA), v);
      set_row<16>(f32(kGA) + (size_t)r.row * m, r.col0(), m, r.row < m, v);
      r.result(1, 1, v);
      set_row<16>(f32(kGdK) + (size_t)r.row * m, r.col0(), m, r.row < m, v);
    }
    r.publish(true);
    r.template product<false, false>(Gi, false, img(kBK2), false, 2, 0, false);      // dL/dZ_J = G K2
    r.commit(0);
    if (C) {
      r.result(0, 0, g);
      r.put(img(kBG0 + (J & 1)), g);
    }
    r.publish(false);
    A = img(kBA);
    A32 = f32(kGA);
  }
  // Per iteration, with R = I - A Z, W = I + R + R^2 / 4, Y = Z R, Z' = Z + Y W and G = dL/dZ':
  //   1:  dY = G W^T | H = Y^T G / 4 | R of the next lower iterate
  //   2:  D = -(Z^T dY + H R^T + R^T H + 4 H) (over G) | its R^2, for W
  //   3:  its Y | dL/dZ = G + dY R^T + A^T D | dL/dA += D Z^T (registers, read in the next phase)
  // j = J only forms R, W, Y of Z_{J-1}.  Z_{j-2} is converted in phase 2: three images, since the one it goes to was last
  // copied in the phase before.
  float dA[16], rv[16], hd[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) dA[i] = 0.f;
  for (int j = J; j >= 0; --j) {
    const bool main_part = j < J, prime = j > 0;
    uint8_t *Z = img(kBZ0 + j % 3), *Zn = img(kBZ0 + (j + 2) % 3);
    uint8_t *Rj = img(kBR0 + (j & 1)), *Rn = img(kBR0 + ((j + 1) & 1)), *G = img(kBG0 + ((j + 1) & 1)), *Gn = img(kBG0 + (j & 1));
    if (main_part) {
      r.template product<false, true>(G, true, img(kBW), true, 2, 1, false);
      r.commit(1);
      if (j < J - 1) r.reuse(0);
      r.template product<true, false>(img(kBY), true, G, true, 2, 0, false);
      r.commit(0);
      if (prime) r.reuse(1);
    }
    if (prime) {
      r.template product<false, false>(A, !main_part, Zn, true, 2, 1, false);
      r.commit(1);
    }
    if (C) {
      if (main_part) {
        if (j < J - 1) {
          r.result(0, 0, v);
          r.release(0);
#pragma unroll
          for (int i = 0; i < 16; ++i) dA[i] += v[i];
        }
        r.result(1, 1, v);
        if (prime) r.release(1);
        r.put(img(kBdY), v);
        r.result(0, 0, hd);
#pragma unroll
        for (int i = 0; i < 16; ++i) hd[i] *= 0.25f;
        r.put(img(kBH), hd);
      }
      if (prime) {
        r.result(1, 1, rv);
#pragma unroll
        for (int i = 0; i < 16; ++i) rv[i] = -rv[i];
        r.add_diag(rv, 1.f, m);
        r.put(Rn, rv);
      }
    }
    r.publish(false);
    if (main_part) {
      r.template product<true, false>(Z, false, img(kBdY), true, 2, 0, false);
      r.template product<false, true>(img(kBH), true, Rj, false, 2, 0, true);
      r.template product<true, false>(Rj, false, img(kBH), true, 2, 0, true);
      r.commit(0);
    }
    if (prime) {
      r.template product<false, false>(Rn, true, Rn, true, 2, 1, false);
      r.commit(1);
    }
    if (main_part) {
      if (C) {
        r.ensure(false);
        if (j > 1) r.convert(iterates + (size_t)(j - 2) * mm, m, m, img(kBZ0 + (j + 1) % 3));
        r.result(0, 0, v, 2, kTrunc3);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = -fmaf(4.f, hd[i], v[i]);
        r.put(G, v);
      }
      r.publish(false);
    }
    if (C && prime) {
      r.result(1, 1, v);
      if (main_part) r.release(1);
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = fmaf(0.25f, v[i], rv[i]);
      r.add_diag(v, 1.f, m);
      r.put(img(kBW), v);
    }
    if (prime) {
      r.template product<false, false>(Zn, false, Rn, !main_part, 2, 0, false);
      r.commit(0);
    }
    if (main_part) {
      if (prime) r.reuse(1);
      r.template product<false, true>(img(kBdY), false, Rj, false, 2, 1, false);
      r.template product<true, false>(A, false, G, true, 2, 1, true);
      r.commit(1);
      if (prime) r.reuse(0);
      r.template product<false, true>(G, true, Z, false, 2, 0, false);
      r.commit(0);
    }
    if (C) {
      if (prime) {
        r.result(0, 0, v);
        if (main_part) r.release(0);
        r.put(img(kBY), v);
      }
      if (main_part) {
        r.result(1, 1, v, 2, kTrunc2);
#pragma unroll
        for (int i = 0; i < 16; ++i) g[i] += v[i];
        if (prime) r.put(Gn, g);
        else {
          set_row<16>(f32(kGdZ) + (size_t)r.row * m, r.col0(), m, r.row < m, g);
          r.result(0, 0, v);
#pragma unroll
          for (int i = 0; i < 16; ++i) dA[i] += v[i];
        }
      }
    }
    r.publish(j > 1 || j == 0);
  }
  // Z0 = A^T / c with c = ||A||_1 ||A||_inf; S = sum_{a,b} dZ0[a,b] A[b,a]
  if (C) {
    r.ensure();
    const float* dZ0 = f32(kGdZ);
    const Norms na = norms(A32, m, r.red);
    const float craw = na.n1 * na.ninf, c = fmaxf(craw, 1e-12f);
    // this thread's row of A against the same column of dZ0, in both blocks (each CTA forms the whole sum)
    float part = 0.f, z[16];
#pragma unroll
    for (int b = 1; b >= 0; --b) {
      const int c0 = (b ? (r.rank ^ 1) : r.rank) * 64 + (r.seg & 3) * 16;      // the own block last: v and z stay
      get_row<16>(A32 + (size_t)r.row * m, c0, m, r.row < m, v);
#pragma unroll
      for (int i = 0; i < 16; ++i) z[i] = (r.row < m && c0 + i < m) ? __ldcg(dZ0 + (size_t)(c0 + i) * m + r.row) : 0.f;
#pragma unroll
      for (int i = 0; i < 16; ++i) part = fmaf(z[i], v[i], part);
    }
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if (lane == 0) r.red[w] = part;
    compute_sync();
    float S = 0.f;
    for (int i = 0; i < kComputeWarps; ++i) S += r.red[i];
    const bool clamped = !(craw > 1e-12f);
    const float col_term = clamped ? 0.f : -S * na.ninf / (c * c);
    const float row_term = clamped ? 0.f : -S * na.n1 / (c * c);
    if (r.row < m) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int cc = r.col0() + i;
        if (cc < m) {
          const float sg = v[i] > 0.f ? 1.f : (v[i] < 0.f ? -1.f : 0.f);
          float g = dA[i] + z[i] / c;
          if (cc == na.jc) g += sg * col_term;
          if (r.row == na.ir) g += sg * row_term;
          dA[i] = g;
        }
      }
      set_row<16>(out32 + (size_t)r.row * m, r.col0(), m, !r.failed, dA);
    }
  }
  r.publish(true);
  if (ridge) {
    // dK2 = G^T Z_J + K2 (dA + dA^T)
    if (C) {
      r.ensure();
      const int row = r.rank * 64 + (threadIdx.x & 63), s = threadIdx.x >> 6;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int cc = 16 * s + i;
        v[i] = (row < m && cc < m) ? __ldcg(out32 + (size_t)row * m + cc) + __ldcg(out32 + (size_t)cc * m + row) : 0.f;
      }
      put16(img(kBY), row, s, v);
    }
    r.publish(true);
    r.template product<false, false>(img(kBK2), false, img(kBY), true, 2, 0, false);
    r.commit(0);
    if (C) {
      r.result(0, 0, v);
      float x[16];
      get_row<16>(f32(kGdK) + (size_t)r.row * m, r.col0(), m, r.row < m, x);
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] += x[i];
      set_row<16>(out32 + (size_t)r.row * m, r.col0(), m, r.row < m && !r.failed, v);
    }
    r.publish(true);
  }
  if (p.G) { r.close(); return; }
  // softmax-2 Jacobian dS2 = K2 o (dK2 - rowsum(dK2 o K2)), then dqt_ns = dS2 Kt, dkt_tot = dkt_a + dS2^T Qt
  if (C) {
    r.ensure();
    for (int i = 0; i < 4; ++i) {
      const int row = r.rank * 64 + 4 * w + i;
      float x[4], k[4], s = 0.f;
      get_row<4>(out32 + (size_t)row * m, 4 * lane, m, row < m, x);
      get_row<4>(k2 + (size_t)row * m, 4 * lane, m, row < m, k);
#pragma unroll
      for (int q = 0; q < 4; ++q) s = fmaf(x[q], k[q], s);
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
#pragma unroll
      for (int q = 0; q < 4; ++q) x[q] = k[q] * (x[q] - s);
      put_row(img(kBR0), row, lane, x);
    }
    r.convert(p.kt + bh * md, m, D, img(kBW));
    r.convert(p.qt + bh * md, m, D, img(kBdY));
  }
  r.publish(true);
  if (own_d) {
    r.template product<false, false>(img(kBR0), true, img(kBW), true, 2, 0, false);
    r.commit(0);
    r.template product<true, false>(img(kBR0), true, img(kBdY), true, 2, 1, false);
    r.commit(1);
    if (C) {
      const size_t off = (size_t)bh * md + (size_t)r.row * D;
      const bool row_ok = r.row < m;
      float da[16];
      get_row<16>(p.sums + bh * 2 * md + md + (size_t)r.row * D, r.col0(), D, row_ok, da);
      r.result(0, 0, v);
      set_row<16>(p.dqt_ns + off, r.col0(), D, row_ok && !r.failed, v);
      r.result(1, 1, v);
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] += da[i];
      set_row<16>(p.dkt_tot + off, r.col0(), D, row_ok && !r.failed, v);
      if (p.rows_k && row_ok) {
        Segments sg(p.N, m);
        const float f = p.scale / (float)sg.len(r.row);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] *= f;
        set_row<16>(p.rows_k + off, r.col0(), D, !r.failed, v);
      }
    }
  }
  r.close();
}

// ---- kernels --------------------------------------------------------------------------------------------
template <int R, class P, class Prog>
__device__ __forceinline__ void run_role(Shared* sh, uint8_t* ring, float* red, const P& p, Prog prog) {
  Role<R> r;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  r.open(sh, ring, red, (int)rank, p.status, p.test_drop && blockIdx.x == 0);
  for (int64_t bh = blockIdx.x >> 1;;) {
    prog(r, p, bh);
    bh += gridDim.x >> 1;
    if (bh >= p.BH) break;
    __syncwarp();
    __syncthreads();
    cluster_sync_all();        // neither CTA copies from this slice's images any more
  }
}
template <class P, class Prog>
__device__ __forceinline__ void run_kernel(uint8_t* dyn, const P& p, Prog prog) {
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(dyn) + 1023) & ~(uintptr_t)1023);
  float* red = reinterpret_cast<float*>(ring + (size_t)kStages * kStageBytes + kBlockBytes);
  Shared* sh = reinterpret_cast<Shared*>(red + kRedFloats);
  static_assert(sizeof(Shared) <= 256, "barriers");
  const int warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&sh->full[s], 1); mbar_init(&sh->empty[s], 1); }
    mbar_init(&sh->done[0], 1);
    mbar_init(&sh->done[1], 1);
    mbar_init(&sh->released[0], kComputeWarps);
    mbar_init(&sh->released[1], kComputeWarps);
    mbar_init(&sh->drain, 1);
    for (int i = 0; i < 2; ++i) mbar_init(&sh->both[i], 2);
    mbar_init(&sh->put, kComputeWarps);
    for (int i = 0; i < 3; ++i) {
      mbar_init(&sh->came[i], 4);
      if (i < 2) { mbar_init(&sh->loaded[i], 1); sh->loads[i] = 0; }
      for (int q = 0; q < 4; ++q) sh->inbound[q][i] = 0;
    }
    mbar_init(&sh->ready, 2 * (kComputeWarps + 2));
    sh->abort_word = 0;
    fence_mbar_init();
  }
  if (warp == 0) {
    tmem_alloc(&sh->tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();          // the peer's barriers exist
  tc_fence_after();
  pdl_wait();
  if (warp < kComputeWarps) run_role<kCompute>(sh, ring, red, p, prog);
  else if (warp == kComputeWarps) run_role<kProducer>(sh, ring, red, p, prog);
  else run_role<kIssuer>(sh, ring, red, p, prog);
  __syncwarp();
  const uint32_t tmem = sh->tmem_slot;
  tc_fence_before();
  __syncthreads();
  // After a wait gave up, in whichever role, copies and products may still be running.  They end before the memory they
  // write is given back; nothing is issued any more, so each stage's last fill and one more commit cover them.
  if (sh->abort_word) {
    if (threadIdx.x == 0) {
      for (uint32_t s = 0; s < kStages; ++s) {
        const uint32_t n = (sh->fills + kStages - 1 - s) / kStages;    // fills of stage s
        if (n) mbar_drain(&sh->full[s], (n - 1) & 1u);
      }
      for (int i = 0; i < 2; ++i)
        if (sh->loads[i]) mbar_drain(&sh->loaded[i], (sh->loads[i] - 1) & 1u);
    }
    if (warp == kComputeWarps + 1) {
      umma_commit_elect(&sh->drain);       // (from the lane that issued)
      mbar_drain(&sh->drain, 0);
    }
    __syncthreads();
  }
  cluster_sync_all();          // nobody arrives on this CTA's barriers any more, or copies into its memory
  if (sh->abort_word && threadIdx.x == 0)      // (copies on their way: their last phase, with the arrivals of those who gave up before)
    for (int i = 0; i < 3; ++i) {
      uint32_t n = 0;
      for (int q = 0; q < 4; ++q) n = max(n, sh->inbound[q][i]);
      for (int q = 0; q < 4; ++q)
        if (sh->inbound[q][i] < n) mbar_arrive(&sh->came[i]);
      if (n) mbar_drain(&sh->came[i], (n - 1) & 1u);
    }
  __syncwarp();
  cluster_sync_all();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

__global__ void __launch_bounds__(kThr, 1) __cluster_dims__(2, 1, 1) mx_fwd_kernel(FwdParams p) {
  extern __shared__ uint8_t mx_dyn[];
  run_kernel(mx_dyn, p, [](auto& r, const FwdParams& q, int64_t bh) { fwd_program(r, q, bh); });
}
__global__ void __launch_bounds__(kThr, 1) __cluster_dims__(2, 1, 1) mx_bwd_kernel(BwdParams p) {
  extern __shared__ uint8_t mx_dyn[];
  run_kernel(mx_dyn, p, [](auto& r, const BwdParams& q, int64_t bh) { bwd_program(r, q, bh); });
}

}  // namespace mx
}  // namespace fnb
