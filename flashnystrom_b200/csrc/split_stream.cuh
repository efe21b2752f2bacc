// Streaming passes at FP32-equivalent precision on the sm_100a tensor cores: full-precision inputs, and
// the 16-bit shapes whose landmark matrices, probabilities and softmax Jacobians stay in FP32 (head_dim 64
// with more than 64 landmarks, head_dim 16 and 32).
//
// Every FP32 operand is a short sum of bf16 terms (x = x0 + x1 + ..., each term the bf16 rounding of
// what the previous ones left over), and a product is the sum of the partial products whose weight
// matters.  bf16 has the FP32 exponent range, so no operand needs scaling.
//   inputs           bf16: 1 term, fp16: 2, fp32: 3 (exact in all three cases)
//   landmark matrices, probabilities, softmax Jacobians: 3 terms (24 bits)
// Of a product, the partial products of weight 2^-16 and up are formed: six MMAs per K step for fp32 operands,
// five and three for fp16 and bf16 inputs; what is dropped is below 2^-25 of the sum of the products' magnitudes.
//
// One CTA of 16 warps per SM walks 128-row tiles of one (b,h) slice.  All warps stage the tile (global ->
// registers -> terms -> swizzled shared memory), warp 0 issues the MMAs, all warps take the scores out
// of tensor memory (thread = one row x 16 columns of each block of 64 landmarks) and write the probabilities
// back as operand tiles: K-major when they are contracted over landmarks, MN-major when over rows.
// The next tile's rows are in flight in registers meanwhile, and its scores are issued together with
// the products of the current tile wherever the buffers allow.  Exponentials and logarithms are expf and logf, as
// in the CUDA-core kernels: ex2.approx of scores in units of log 2 is faster, but with the roundings of that scaling the
// saved lse1 and the outputs were 25 to 50 % less exact.  With more than 64 landmarks a probability tile
// is 96 KB; where that leaves no room for the rest, its two blocks take turns in one of 48 KB.
//
// What bounds it: no unit, but the phases of a tile in turn (input split, score MMAs, exponentials and split of the
// probabilities, MMAs, results out), which one CTA per SM cannot overlap much for want of room for a second set of buffers.
// fp32, shape below: tensor pipe active 17 to 26 % (about 36 cycles per 128 x 64 x 16 MMA, whose operands come out of
// shared memory; the column pass of the backward issues 128 of them per tile), issue slots 35 to 43 %, DRAM 14 to 20 %.
// Measured on a B200, us per launch, against the CUDA-core kernels of generic_kernels.cuh (fwd_b, fwd_c, bwd_a, bwd_b, bwd_c):
//   fp32, B=1, H=16, N=16384, D=64, m=64    1135, 574, 1996, 1948, 863  ->  95, 70, 129, 143, 103
//   bf16, B=2, H=8,  N=8192,  D=64, m=128    727, 431, 1319, 1379, 713  ->  60, 50,  69, 101,  64
#pragma once
#include <type_traits>
#include "common.cuh"
#include "tc_common.cuh"
#include "tc_stream.cuh"

namespace fnb {
namespace sx {

using namespace tc;
typedef __nv_bfloat16 bf16;

constexpr int kThr = 512;
constexpr int kBlk = kTile * 128;   // bytes of a [128 rows x 64] bf16 block, rows 128 bytes apart

template <class T> struct InTerms { static constexpr int n = 3; };
template <> struct InTerms<__half> { static constexpr int n = 2; };
template <> struct InTerms<bf16> { static constexpr int n = 1; };
constexpr int kTerms = 3;           // of landmark matrices, probabilities and softmax Jacobians
constexpr int kSmemMax = 232448;

// Shared-memory plan of one instantiation (bytes).  X: an input tile, P: a probability tile of one block of 64
// landmarks, L: a landmark operand.  head_dim below 64 leaves the tail of the 128-byte rows unused.
// H*: blocks of a probability tile that are held at once.
template <class T, int D, int MP>
struct Plan {
  static constexpr int NX = InTerms<T>::n, NB = MP / 64;
  static constexpr int kX = NX * kBlk, kP = kTerms * kBlk, kL = kTerms * MP * 128;
  static constexpr int kPitch = D * (int)sizeof(T) + 16;      // staged output row
  static_assert(kTile * kPitch <= kP, "outputs are staged in a probability buffer");
  static constexpr int kRed = 4 * kTile * 4, kVec = 2 * MP * 4, kBars = 256;   // exchange words, per-landmark vectors, barriers
  static constexpr int fit(int rest) { return rest + NB * kP <= kSmemMax ? NB : 1; }
  static constexpr int kFwdB0 = kL + 2 * kX + kRed + kVec + kBars, kHFwdB = fit(kFwdB0), kFwdB = kFwdB0 + kHFwdB * kP;
  static constexpr int kRow0 = 2 * kL + kX + kRed + kBars;
  static constexpr int kHFwdC = fit(kRow0), kFwdC = kRow0 + kHFwdC * kP;
  static constexpr int kHBwdA = fit(kRow0 + kX), kBwdA = kRow0 + kX + kHBwdA * kP, kHBwdC = kHBwdA, kBwdC = kBwdA;
  static constexpr int kHBwdB = 1, kBwdB = 2 * kL + kX + 2 * kP + kVec + kBars;    // V tile, then P tile; dS tile
  static_assert(kX <= kP, "V takes the place of a probability tile");
  static_assert(kHFwdB == NB && kHFwdC == NB, "the forward passes hold whole probability tiles");
  static_assert(kFwdB <= kSmemMax && kFwdC <= kSmemMax && kBwdA <= kSmemMax && kBwdB <= kSmemMax, "shared memory");
};

// ---- terms ---------------------------------------------------------------------------------
// kSat: values past the largest bf16 (3.39e38; an fp32 value may be up to 3.40e38) take it as their first term and stay finite;
// infinities and NaN become NaN in the later terms.
template <int NT, bool kSat = false>
__device__ __forceinline__ void split8(const float* v, uint4* w) {
  uint32_t* o = reinterpret_cast<uint32_t*>(w);
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    float a = v[2 * p], b = v[2 * p + 1];
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      uint32_t x;
      if (kSat && t == 0) asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;" : "=r"(x) : "f"(b), "f"(a));
      else x = pack2<bf16>(a, b);
      o[4 * t + p] = x;
      if (t + 1 < NT) {
        a -= __uint_as_float(x << 16);
        b -= __uint_as_float(x & 0xffff0000u);
      }
    }
  }
}
// Order of the three terms of a probability tile: (x1, x0, x2), so that both (x1, x0) and (x0, x2) are
// neighbours and can be stacked along M (see issue_contract()).
__device__ __forceinline__ constexpr int slot_of(int term) { return term == 0 ? 1 : term == 1 ? 0 : 2; }

// ---- input tiles: global -> registers -> terms in shared memory -----------------------------------
template <class T, int D>
struct InTile {
  static constexpr int kVec = (int)sizeof(T) / 2;            // 16-byte words per eight elements
  static constexpr int kChunks = kTile * D / 8;
  static constexpr int kPer = (kChunks + kThr - 1) / kThr;
  uint4 raw[kPer][kVec];
  __device__ __forceinline__ void fetch(const T* slice, int64_t r0, int64_t N) {
#pragma unroll
    for (int c = 0; c < kPer; ++c) {
      const int idx = threadIdx.x + c * kThr, row = idx / (D / 8), ch = idx % (D / 8);
      const bool ok = (kChunks % kThr == 0 || idx < kChunks) && r0 + row < N;
      const uint4* src = reinterpret_cast<const uint4*>(slice + (r0 + row) * D + ch * 8);
#pragma unroll
      for (int v = 0; v < kVec; ++v) raw[c][v] = ok ? __ldg(src + v) : make_uint4(0, 0, 0, 0);
    }
  }
  __device__ __forceinline__ void put(uint8_t* tile) const {
#pragma unroll
    for (int c = 0; c < kPer; ++c) {
      const int idx = threadIdx.x + c * kThr;
      if (kChunks % kThr != 0 && idx >= kChunks) return;
      const uint32_t off = sw128_offset(idx / (D / 8), idx % (D / 8));
      if constexpr (std::is_same<T, bf16>::value) {
        *reinterpret_cast<uint4*>(tile + off) = raw[c][0];
      } else {
        constexpr int NX = InTerms<T>::n;
        const T* e = reinterpret_cast<const T*>(raw[c]);
        float x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = to_f<T>(e[i]);
        uint4 w[NX];
        split8<NX, std::is_same<T, float>::value>(x, w);
#pragma unroll
        for (int t = 0; t < NX; ++t) *reinterpret_cast<uint4*>(tile + t * kBlk + off) = w[t];
      }
    }
  }
};

// (m x D) FP32 landmark matrix times mul -> three term tiles of [MP rows x 128 B], rows >= m zero
template <int D, int MP>
__device__ __forceinline__ void put_landmarks(uint8_t* op, const float* src, int m, float mul) {
  const bool aligned = (reinterpret_cast<uintptr_t>(src) & 15u) == 0;
  for (int idx = threadIdx.x; idx < MP * D / 8; idx += kThr) {
    const int r = idx / (D / 8), ch = idx % (D / 8);
    float x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = 0.f;
    if (r < m) {
      const float* e = src + r * D + ch * 8;
      if (aligned) {
        const float4 a = *reinterpret_cast<const float4*>(e), b = *reinterpret_cast<const float4*>(e + 4);
        x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
        x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
      } else {                               // (the caller's saved tensors need no more than their type's alignment)
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = e[i];
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] *= mul;
    }
    uint4 w[kTerms];
    split8<kTerms, true>(x, w);
#pragma unroll
    for (int t = 0; t < kTerms; ++t) *reinterpret_cast<uint4*>(op + t * (MP * 128) + sw128_offset(r, ch)) = w[t];
  }
}

// 16 values, columns 16 group .. of block b of row r, -> a probability tile of HB blocks ([term][block][128 rows x 128 B])
template <int HB>
__device__ __forceinline__ void put_probs(uint8_t* tile, int r, int b, int group, const float* v) {
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    uint4 w[kTerms];
    split8<kTerms>(v + 8 * c, w);
    const uint32_t off = (uint32_t)b * kBlk + sw128_offset(r, group * 2 + c);
#pragma unroll
    for (int t = 0; t < kTerms; ++t) *reinterpret_cast<uint4*>(tile + slot_of(t) * (HB * kBlk) + off) = w[t];
  }
}

// ---- products (warp-uniform; one elected lane issues) ------------------------------------------------
// The tensor core truncates when it adds to an accumulator.  So the small partial products go first, and where it
// shows, the K steps of the leading one are spread over G accumulators of their own (column groups 64 apart), which the
// epilogue adds in FP32.  With everything in one accumulator the output and dV of fp32 calls were 1.2 to 1.4 times as far
// from the oracle as with the CUDA-core kernels, with the groups below 0.5 to 1.03 times, for 3 % of the passes'
// time.  The scores have two groups in the forward passes of more than 64 landmarks, where lse3 was 1.2 times as far off
// at scores of about 10 without; elsewhere that changed nothing but the time (680 -> 695 us for a training pass,
// fp32, B=1, H=16, N=16384, D=64, m=64).
// scores (128 x MP) = X (128 x D) L^T, groups MP columns apart
template <int D, int MP, int NX, int G = 1>
__device__ __forceinline__ void issue_scores(uint32_t d, uint32_t x, uint32_t l) {
  constexpr uint32_t idesc = make_idesc<bf16>(kTile, MP, false, false);
  constexpr int K = D / 16;
  static_assert(G <= K, "a group has a K step at least");
  bool acc = false;
#pragma unroll
  for (int s = kTerms - 1; s >= 0; --s)
#pragma unroll
    for (int i = 0; i < NX; ++i) {
      const int j = s - i;
      if (j < 0 || j >= kTerms) continue;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int g = s == 0 ? k * G / K : 0;
        const bool first = g > 0 && (k - 1) * G / K != g;
        umma_elect(d + g * MP, smem_desc_sw128(x + i * kBlk + k * 32, 16, 1024), smem_desc_sw128(l + j * (MP * 128) + k * 32, 16, 1024), idesc,
                   g > 0 ? !first : acc);
        acc = true;
      }
    }
}
// rows (128 x D) = P L over the HB blocks of landmarks from blk on, which the tile p holds.
// This product and the next always run with N = 64, the width of a swizzled block: for a smaller head_dim the columns
// past D hold nothing and are never read.
template <int MP, int HB, int G>
__device__ __forceinline__ void issue_rows(uint32_t d, uint32_t p, uint32_t l, int blk) {
  constexpr uint32_t idesc = make_idesc<bf16>(kTile, 64, false, true);
  constexpr int K = HB * 4;
  bool acc = false;
#pragma unroll
  for (int s = kTerms - 1; s >= 0; --s)
#pragma unroll
    for (int i = 0; i <= s; ++i) {
      const uint32_t pt = p + slot_of(i) * (HB * kBlk), lt = l + (s - i) * (MP * 128) + blk * (64 * 128);
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int g = s == 0 ? k * G / K : 0;
        const bool first = g > 0 && (k - 1) * G / K != g;
        umma_elect(d + g * 64, smem_desc_sw128(pt + (k >> 2) * kBlk + (k & 3) * 32, 16, 1024), smem_desc_sw128(lt + k * 2048, MP * 128, 1024), idesc,
                   g > 0 ? !first : acc);
        acc = true;
      }
    }
}
// tile sum (landmarks x D) = P^T X (128 x D).
// A tile of one block: two terms of P are stacked along M (lanes 0..63 and 64..127, added when the sum is read); the
// one partial product that this cannot place, x2 * X0, goes to the 64 columns behind the groups, lanes 64..127.
// A tile of two blocks: the lanes are the landmarks.
// A run of additions at full magnitude drifts by about 2^-25 each (bmat was off by 5e-5 after 128 tiles in one accumulator),
// so the tile sums are added up over tiles with ordinary FP32 additions (add_tile_sum).
template <int HB, int NX, int G>
__device__ __forceinline__ void issue_contract(uint32_t d, uint32_t p, uint32_t x) {
  constexpr uint32_t idesc = make_idesc<bf16>(128, 64, true, true);
  constexpr int K = kTile / 16;
  bool acc = false;
  if (HB == 1) {
#pragma unroll
    for (int j = NX - 1; j >= 0; --j)
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int g = j == 0 ? k * G / K : 0;
        const bool first = g > 0 && (k - 1) * G / K != g;
        umma_elect(d + g * 64, smem_desc_sw128(p + k * 2048, kBlk, 1024), smem_desc_sw128(x + j * kBlk + k * 2048, kBlk, 1024), idesc,
                   g > 0 ? !first : acc);
        acc = true;
      }
#pragma unroll
    for (int k = 0; k < K; ++k)
      umma_elect(d + G * 64, smem_desc_sw128(p + kBlk + k * 2048, kBlk, 1024), smem_desc_sw128(x + k * 2048, kBlk, 1024), idesc, k > 0);
  } else {
#pragma unroll
    for (int s = kTerms - 1; s >= 0; --s)
#pragma unroll
      for (int j = 0; j < NX; ++j) {
        const int i = s - j;
        if (i < 0 || i >= kTerms) continue;
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const int g = s == 0 ? k * G / K : 0;
          const bool first = g > 0 && (k - 1) * G / K != g;
          umma_elect(d + g * 64, smem_desc_sw128(p + slot_of(i) * (HB * kBlk) + k * 2048, kBlk, 1024),
                     smem_desc_sw128(x + j * kBlk + k * 2048, kBlk, 1024), idesc, g > 0 ? !first : acc);
          acc = true;
        }
      }
  }
}
// tensor-memory columns of a tile sum, and of the running sums of MP landmarks
template <int HB, int G> __host__ __device__ constexpr int tile_cols() { return 64 * (HB == 1 ? G + 1 : G); }
template <int MP, int HB> __host__ __device__ constexpr int sum_cols() { return HB == 1 ? MP : 64; }
__host__ __device__ constexpr uint32_t pow2_cols(int c) { return c <= 64 ? 64u : c <= 128 ? 128u : c <= 256 ? 256u : 512u; }

// ---- tensor memory -> registers, NC columns of this warp's 32 lanes ------------------------------------
template <int NC>
__device__ __forceinline__ void ld(uint32_t a, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  if constexpr (NC == 32) {
    tmem_ld32(a, v);
  } else if constexpr (NC == 16) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(a)
        : "memory");
  } else if constexpr (NC == 8) {
    tmem_ld8(a, v);
  } else {
    static_assert(NC == 4, "columns");
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
  }
}

template <int NC>
__device__ __forceinline__ void st(uint32_t a, const float* v) {
  const uint32_t* r = reinterpret_cast<const uint32_t*>(v);
  if constexpr (NC == 8) {
    tmem_st8(a, v);
  } else {
    static_assert(NC == 4, "columns");
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3])
                 : "memory");
  }
}

// ---- common frame of the kernels --------------------------------------------------------------------
struct Frame {
  uint64_t* bars;          // [3] completion barriers, [1] used on the way out after a wait gave up
  uint32_t tmem;
  Abort ab;
  uint32_t phase[3];
  int warp, row, group;    // row = tile row = tensor-memory lane of this thread; group = its quarter of the columns
  uint32_t lane_base;
  int64_t bh;
  int chunk, first, count;
  __device__ __forceinline__ void wait(int b, int where) {
    mbar_wait(bars + b, phase[b], ab, where);
    phase[b] ^= 1u;
    __syncwarp();
    tc_fence_after();
  }
  // this thread's shared-memory stores and tensor-memory accesses are done; then every thread's are
  __device__ __forceinline__ void publish() const {
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
  }
};
__device__ __forceinline__ bool open_frame(Frame& f, uint8_t* smem, uint8_t* tail, const TcSched& sch, uint32_t cols, int* status, int where) {
  f.bars = reinterpret_cast<uint64_t*>(tail);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(f.bars + 4);
  int* abort_word = reinterpret_cast<int*>(tmem_slot + 1);
  if (smem_u32(smem) & 1023u) {
    if (threadIdx.x == 0 && status) atomicCAS(status, 0, (kStatusSmemAlign << 24) | where);
    return false;
  }
  f.warp = threadIdx.x >> 5;
  f.row = (f.warp & 3) * 32 + (threadIdx.x & 31);
  f.group = f.warp >> 2;
  f.lane_base = (uint32_t)((f.warp & 3) * 32) << 16;
  f.phase[0] = f.phase[1] = f.phase[2] = 0;
  f.bh = blockIdx.x / sch.nchunk;
  f.chunk = (int)(blockIdx.x - f.bh * sch.nchunk);
  const int tiles = (int)((sch.N + kTile - 1) / kTile);
  f.first = f.chunk * sch.tiles_per_chunk;
  f.count = max(0, min(sch.tiles_per_chunk, tiles - f.first));
  if (threadIdx.x == 0) {
    for (int b = 0; b < 4; ++b) mbar_init(f.bars + b, 1);
    *abort_word = 0;
    fence_mbar_init();
  }
  if (f.warp == 0) {
    tmem_alloc(tmem_slot, cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  f.tmem = *tmem_slot;
  f.ab = Abort{abort_word, status};
  return true;
}
__device__ __forceinline__ void close_frame(const Frame& f, uint32_t cols) {
  tc_fence_before();
  __syncthreads();
  if (f.warp == 0 && f.ab.raised()) {      // products may still be running: they end before their memory is given back
    umma_commit_elect(f.bars + 3);
    mbar_drain(f.bars + 3, 0);
    __syncwarp();
  }
  if (f.warp == 0) tmem_dealloc(f.tmem, cols);
}

// D / 4 result columns of this thread's row -> staged row of the output type; then the staged tile -> global rows
template <class T, int D>
__device__ __forceinline__ void stage_row(uint8_t* stage, int pitch, int row, int col0, const float* o) {
  T* dst = reinterpret_cast<T*>(stage + row * pitch) + col0;
  constexpr int NC = D / 4;
  if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int j = 0; j < NC; j += 4) *reinterpret_cast<float4*>(dst + j) = make_float4(o[j], o[j + 1], o[j + 2], o[j + 3]);
  } else {
#pragma unroll
    for (int j = 0; j < NC; j += 4) *reinterpret_cast<uint2*>(dst + j) = make_uint2(pack2<T>(o[j], o[j + 1]), pack2<T>(o[j + 2], o[j + 3]));
  }
}
template <class T, int D>
__device__ __forceinline__ void copy_out(T* slice, const uint8_t* stage, int pitch, int64_t r0, int64_t N) {
  constexpr int VPR = D * (int)sizeof(T) / 16;
  for (int idx = threadIdx.x; idx < kTile * VPR; idx += kThr) {
    const int row = idx / VPR, v = idx % VPR;
    if (r0 + row < N)
      *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(slice + (r0 + row) * D) + v * 16) = *reinterpret_cast<const uint4*>(stage + row * pitch + v * 16);
  }
}
// the scores of this thread's row, 16 columns of each of NB blocks of 64, the sum of G column groups
template <int NB, int G = 1>
__device__ __forceinline__ void ld_scores(const Frame& f, uint32_t at, float* v) {
  const uint32_t a = f.tmem + at + f.lane_base + f.group * 16;
#pragma unroll
  for (int b = 0; b < NB; ++b) ld<16>(a + b * 64, v + 16 * b);
#pragma unroll
  for (int g = 1; g < G; ++g)
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      float x[16];
      ld<16>(a + g * (NB * 64) + b * 64, x);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; ++j) v[16 * b + j] += x[j];
    }
}
// the sum of G column groups (64 apart) of this thread's row, its quarter of the D result columns
template <int D, int G>
__device__ __forceinline__ void ld_rows(const Frame& f, uint32_t at, float* o) {
  constexpr int ND = D / 4;
  const uint32_t a = f.tmem + at + f.lane_base + f.group * ND;
  ld<ND>(a, o);
#pragma unroll
  for (int g = 1; g < G; ++g) {
    float x[ND];
    ld<ND>(a + g * 64, x);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < ND; ++j) o[j] += x[j];
  }
  tmem_ld_wait();
}
// running sum (64 columns at `sum`) += tile sum (at `tile`, see issue_contract), FP32; with `first` the running sum
// starts at zero.  Each thread handles its lane and a quarter of the columns.
template <int D, int HB, int G>
__device__ __forceinline__ void add_tile_sum(const Frame& f, uint32_t tile, uint32_t sum, bool first) {
  constexpr int NC = D / 4, ST = NC < 8 ? NC : 8;
  const uint32_t off = f.tmem + f.lane_base + f.group * NC;
#pragma unroll
  for (int c = 0; c < NC; c += ST) {
    float v[ST], x[G][ST], r[ST];
    ld<ST>(off + tile + c, v);
#pragma unroll
    for (int g = 1; g < G; ++g) ld<ST>(off + tile + g * 64 + c, x[g]);
    if (HB == 1) ld<ST>(off + tile + G * 64 + c, x[0]);
    if (!first) ld<ST>(off + sum + c, r);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < ST; ++j) {
      if (HB == 1) v[j] += f.row >= 64 ? x[0][j] : 0.f;
#pragma unroll
      for (int g = 1; g < G; ++g) v[j] += x[g][j];
      if (!first) v[j] += r[j];
    }
    st<ST>(off + sum + c, v);
  }
  tmem_st_wait();
}
template <int D>
__device__ __forceinline__ void scale_sum(const Frame& f, uint32_t sum, float factor) {
  constexpr int NC = D / 4, ST = NC < 8 ? NC : 8;
  const uint32_t off = f.tmem + f.lane_base + f.group * NC + sum;
#pragma unroll
  for (int c = 0; c < NC; c += ST) {
    float v[ST];
    ld<ST>(off + c, v);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < ST; ++j) v[j] *= factor;
    st<ST>(off + c, v);
  }
  tmem_st_wait();
}
// running sums of MP landmarks -> global (m x D) times mul; scratch: [64][D + 4] floats of shared memory
template <int D, int MP, int HB>
__device__ __forceinline__ void store_sum(const Frame& f, uint32_t sum, float* scratch, float* dst, int m, float mul) {
  constexpr int NC = D / 4, LD = D + 4;
  const int c0 = f.group * NC;
#pragma unroll
  for (int b = 0; b < (HB == 1 ? MP / 64 : 1); ++b) {
    float v[NC];
    ld<NC>(f.tmem + sum + 64 * b + f.lane_base + c0, v);
    tmem_ld_wait();
    if constexpr (HB == 1) {
      __syncthreads();
      if (f.row >= 64) {
#pragma unroll
        for (int j = 0; j < NC; ++j) scratch[(f.row - 64) * LD + c0 + j] = v[j];
      }
      __syncthreads();
      if (f.row < 64) {
#pragma unroll
        for (int j = 0; j < NC; ++j) v[j] += scratch[f.row * LD + c0 + j];
      }
    }
    const int l = 64 * b + f.row;
    if (l < m && f.row < HB * 64) {
#pragma unroll
      for (int j = 0; j < NC; j += 4)
        *reinterpret_cast<float4*>(dst + l * D + c0 + j) = make_float4(v[j] * mul, v[j + 1] * mul, v[j + 2] * mul, v[j + 3] * mul);
    }
  }
}

// ------------------------------------------------------------------------------------------
// Forward column pass: partial Bmat = softmax(Qt (sK)^T) V over this CTA's rows with per-landmark
// maximum and sum.  The exponent's reference moves only when a score exceeds it by kMove (one compare
// per element and one OR-barrier per tile decide it), so the accumulator is rarely rescaled.
template <class T, int D, int MP>
__global__ void __launch_bounds__(kThr, 1)
sx_fwd_b_kernel(const T* __restrict__ k, const T* __restrict__ v, const float* __restrict__ q_landmarks,
                float* __restrict__ part_acc, float* __restrict__ part_max, float* __restrict__ part_sum, TcSched sch,
                int m, float scale, int* status) {
  using L = Plan<T, D, MP>;
  constexpr int NX = L::NX, NB = L::NB, HB = L::kHFwdB, NC = 16 * NB, GS = NB == 2 && D > 16 ? 2 : 1, GT = 2;
  constexpr uint32_t kS = 0, kTileSum = GS * MP, kSum = kTileSum + tile_cols<HB, GT>(), kCols = pow2_cols(kSum + 64);
  static_assert(kSum + 64 <= 512, "tensor memory");
  constexpr float kMove = 6.f;                 // probabilities stay below e^6 = 403
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* s_qt = smem;
  uint8_t* s_k = s_qt + L::kL;
  uint8_t* s_v = s_k + L::kX;
  uint8_t* s_p = s_v + L::kX;
  float* s_red = reinterpret_cast<float*>(s_p + HB * L::kP);      // [4][128]
  float* s_ref = s_red + 4 * kTile;                          // [MP] reference
  float* s_alpha = s_ref + MP;
  pdl_trigger();
  Frame f;
  if (!open_frame(f, smem, reinterpret_cast<uint8_t*>(s_alpha + MP), sch, kCols, status, 0x4000)) return;
  const T* kk = k + f.bh * sch.N * D;
  const T* vv = v + f.bh * sch.N * D;
  const uint32_t a_qt = smem_u32(s_qt), a_k = smem_u32(s_k), a_v = smem_u32(s_v), a_p = smem_u32(s_p);
  InTile<T, D> rk, rv;
  auto row0 = [&](int i) { return (int64_t)(f.first + i) * kTile; };
  auto col = [&](int j) { return (j >> 4) * 64 + f.group * 16 + (j & 15); };   // landmark of this thread's value j
  rk.fetch(kk, row0(0), sch.N);
  rv.fetch(vv, row0(0), sch.N);
  put_landmarks<D, MP>(s_qt, q_landmarks + f.bh * m * D, m, scale);
  if (threadIdx.x < MP) s_ref[threadIdx.x] = -INFINITY;
  rk.put(s_k);
  rk.fetch(kk, row0(1), sch.N);
  f.publish();
  if (f.warp == 0) {
    issue_scores<D, MP, NX, GS>(f.tmem + kS, a_k, a_qt);
    umma_commit_elect(f.bars + 0);
  }
  float sum[NC];
#pragma unroll
  for (int j = 0; j < NC; ++j) sum[j] = 0.f;
  for (int i = 0; i < f.count; ++i) {
    const bool valid = row0(i) + f.row < sch.N;
    f.wait(0, 0x4100);
    float s[NC];
    ld_scores<NB, GS>(f, kS, s);
    tmem_ld_wait();
    bool over = false;
#pragma unroll
    for (int j = 0; j < NC; ++j) over = over || (s[j] - s_ref[col(j)] > kMove);   // (a NaN score never raises it)
    over = over && valid;
    if (i > 0) {
      f.wait(1, 0x4200);                     // the product of the previous tile is done: P and V are free
      add_tile_sum<D, HB, GT>(f, kTileSum, kSum, i == 1);
    }
    if (__syncthreads_or(over)) {
      // tile maximum of every landmark, the new reference and the factor for what has been summed so far
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        float x = valid ? s[j] : -INFINITY;
        for (int o = 16; o > 0; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
        if ((threadIdx.x & 31) == 0) s_red[(f.warp & 3) * kTile + col(j)] = x;
      }
      __syncthreads();
      if (threadIdx.x < MP) {
        const int l = threadIdx.x;
        const float old = s_ref[l];
        const float mx = fmaxf(fmaxf(fmaxf(s_red[l], s_red[kTile + l]), fmaxf(s_red[2 * kTile + l], s_red[3 * kTile + l])), old);
        s_alpha[l] = old == mx ? 1.f : expf(old - mx);
        s_ref[l] = mx;
      }
      __syncthreads();
#pragma unroll
      for (int j = 0; j < NC; ++j) sum[j] *= s_alpha[col(j)];
      if (i > 0) scale_sum<D>(f, kSum, s_alpha[HB == 1 ? (f.row & 63) : f.row]);
    }
#pragma unroll
    for (int j = 0; j < NC; ++j) {
      s[j] = valid ? expf(s[j] - s_ref[col(j)]) : 0.f;
      sum[j] += s[j];
    }
#pragma unroll
    for (int b = 0; b < NB; ++b) put_probs<HB>(s_p, f.row, b, f.group, s + 16 * b);
    rk.put(s_k);
    rv.put(s_v);
    f.publish();
    if (f.warp == 0) {
      issue_contract<HB, NX, GT>(f.tmem + kTileSum, a_p, a_v);
      umma_commit_elect(f.bars + 1);
      if (i + 1 < f.count) {
        issue_scores<D, MP, NX, GS>(f.tmem + kS, a_k, a_qt);
        umma_commit_elect(f.bars + 0);
      }
    }
    if (i + 1 < f.count) {
      rv.fetch(vv, row0(i + 1), sch.N);
      if (i + 2 < f.count) rk.fetch(kk, row0(i + 2), sch.N);
    }
  }
  const int64_t slot = blockIdx.x;
  if (f.count > 0) {
    f.wait(1, 0x4300);
    add_tile_sum<D, HB, GT>(f, kTileSum, kSum, f.count == 1);
    store_sum<D, MP, HB>(f, kSum, reinterpret_cast<float*>(s_k), part_acc + slot * m * D, m, 1.f);
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < NC; ++j) {
    float x = sum[j];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) == 0) s_red[(f.warp & 3) * kTile + col(j)] = x;
  }
  __syncthreads();
  if (threadIdx.x < m) {
    const int l = threadIdx.x;
    part_max[slot * m + l] = s_ref[l];
    part_sum[slot * m + l] = (s_red[l] + s_red[kTile + l]) + (s_red[2 * kTile + l] + s_red[3 * kTile + l]);
  }
  close_frame(f, kCols);
}

// ------------------------------------------------------------------------------------------
// Forward output pass: O = softmax(sQ Kt^T) step2 and lse1.
template <class T, int D, int MP>
__global__ void __launch_bounds__(kThr, 1)
sx_fwd_c_kernel(const T* __restrict__ q, T* __restrict__ out, float* __restrict__ lse1, const float* __restrict__ k_landmarks,
                const float* __restrict__ step2, TcSched sch, int m, float scale, int* status) {
  using L = Plan<T, D, MP>;
  constexpr int NX = L::NX, NB = L::NB, HB = L::kHFwdC, NC = 16 * NB, ND = D / 4, GS = NB == 2 && D > 16 ? 2 : 1, GO = 4;
  constexpr uint32_t kS = 0, kO = GS * MP, kCols = pow2_cols(kO + GO * 64);
  static_assert(kO + GO * 64 <= 512, "tensor memory");
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* s_kt = smem;
  uint8_t* s_st = s_kt + L::kL;
  uint8_t* s_q = s_st + L::kL;
  uint8_t* s_p = s_q + L::kX;               // probabilities, then the staged output tile
  float* s_max = reinterpret_cast<float*>(s_p + HB * L::kP);      // [4][128]: row maxima, then row sums
  pdl_trigger();
  Frame f;
  if (!open_frame(f, smem, reinterpret_cast<uint8_t*>(s_max + 4 * kTile), sch, kCols, status, 0x4400)) return;
  const T* qq = q + f.bh * sch.N * D;
  T* oo = out + f.bh * sch.N * D;
  const uint32_t a_kt = smem_u32(s_kt), a_st = smem_u32(s_st), a_q = smem_u32(s_q), a_p = smem_u32(s_p);
  InTile<T, D> rq;
  auto row0 = [&](int i) { return (int64_t)(f.first + i) * kTile; };
  auto col = [&](int j) { return (j >> 4) * 64 + f.group * 16 + (j & 15); };
  rq.fetch(qq, row0(0), sch.N);
  put_landmarks<D, MP>(s_kt, k_landmarks + f.bh * m * D, m, scale);
  put_landmarks<D, MP>(s_st, step2 + f.bh * m * D, m, 1.f);
  rq.put(s_q);
  rq.fetch(qq, row0(1), sch.N);
  f.publish();
  if (f.warp == 0) {
    issue_scores<D, MP, NX, GS>(f.tmem + kS, a_q, a_kt);
    umma_commit_elect(f.bars + 0);
  }
  for (int i = 0; i < f.count; ++i) {
    const int64_t row = row0(i) + f.row;
    f.wait(0, 0x4500);
    float s[NC];
    ld_scores<NB, GS>(f, kS, s);
    tmem_ld_wait();
    float mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < NC; ++j) {
      if (col(j) >= m) s[j] = -INFINITY;
      mx = fmaxf(mx, s[j]);
    }
    s_max[f.group * kTile + f.row] = mx;
    __syncthreads();                         // (also: the previous output tile has left the staging buffer)
    mx = fmaxf(fmaxf(s_max[f.row], s_max[kTile + f.row]), fmaxf(s_max[2 * kTile + f.row], s_max[3 * kTile + f.row]));
    float part[4] = {0.f, 0.f, 0.f, 0.f};    // (four short chains: less rounding, and less latency)
#pragma unroll
    for (int j = 0; j < NC; ++j) {
      s[j] = expf(s[j] - mx);
      part[j & 3] += s[j];
    }
    float sum = (part[0] + part[1]) + (part[2] + part[3]);
#pragma unroll
    for (int b = 0; b < NB; ++b) put_probs<HB>(s_p, f.row, b, f.group, s + 16 * b);
    rq.put(s_q);
    __syncthreads();                         // every thread has read the maxima
    s_max[f.group * kTile + f.row] = sum;
    f.publish();
    if (f.warp == 0) {
      issue_rows<MP, HB, GO>(f.tmem + kO, a_p, a_st, 0);
      if (!(sch.test_drop && blockIdx.x == 0 && i + 1 == f.count)) umma_commit_elect(f.bars + 1);   // fault injection on the host's request
      if (i + 1 < f.count) {
        issue_scores<D, MP, NX, GS>(f.tmem + kS, a_q, a_kt);
        umma_commit_elect(f.bars + 0);
      }
    }
    if (i + 2 < f.count) rq.fetch(qq, row0(i + 2), sch.N);
    sum = (s_max[f.row] + s_max[kTile + f.row]) + (s_max[2 * kTile + f.row] + s_max[3 * kTile + f.row]);
    if (f.group == 0 && row < sch.N) lse1[f.bh * sch.N + row] = mx + logf(sum);
    const float inv = 1.f / sum;
    f.wait(1, 0x4600);
    float o[ND];
    ld_rows<D, GO>(f, kO, o);
#pragma unroll
    for (int j = 0; j < ND; ++j) o[j] *= inv;
    stage_row<T, D>(s_p, L::kPitch, f.row, f.group * ND, o);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    copy_out<T, D>(oo, s_p, L::kPitch, row0(i), sch.N);
  }
  close_frame(f, kCols);
}

// The softmax-1 Jacobian of a tile from its scores s and dP1 = dO step2^T (both in registers; s becomes
// P1 and g becomes dS1): P1 = exp(S - lse1), D1 = rowsum(P1 o dP1), dS1 = P1 o (dP1 - D1).
template <int NC>
__device__ __forceinline__ void softmax1_jacobian(const Frame& f, float* s_red, float* s, float* g, float lse, bool valid, int m) {
  float part[4] = {0.f, 0.f, 0.f, 0.f};      // (four short chains: less rounding, and less latency)
#pragma unroll
  for (int j = 0; j < NC; ++j) {
    s[j] = (valid && (j >> 4) * 64 + f.group * 16 + (j & 15) < m) ? expf(s[j] - lse) : 0.f;
    part[j & 3] = fmaf(s[j], g[j], part[j & 3]);
  }
  float d1 = (part[0] + part[1]) + (part[2] + part[3]);
  s_red[f.group * kTile + f.row] = d1;
  __syncthreads();
  d1 = (s_red[f.row] + s_red[kTile + f.row]) + (s_red[2 * kTile + f.row] + s_red[3 * kTile + f.row]);
#pragma unroll
  for (int j = 0; j < NC; ++j) g[j] = s[j] * (g[j] - d1);
}

// ------------------------------------------------------------------------------------------
// First backward row pass: per-CTA partials of dstep2 = P1^T dO and dKt = dS1^T (sQ).  P1 and dS1 take
// turns in one buffer: Q, dO, both landmark operands and one probability tile fill the SM.
// kAlias: where only one of two blocks fits, their sums fill tensor memory, the tile sums lie where the scores were,
// and the next scores wait for the last of them.
template <class T, int D, int MP>
__global__ void __launch_bounds__(kThr, 1)
sx_bwd_a_kernel(const T* __restrict__ q, const T* __restrict__ d_out, const float* __restrict__ lse1,
                const float* __restrict__ k_landmarks, const float* __restrict__ step2, float* __restrict__ partA, TcSched sch,
                int m, float scale, int* status) {
  using L = Plan<T, D, MP>;
  constexpr int NX = L::NX, NB = L::NB, HB = L::kHBwdA, NC = 16 * NB, GT = NB == 1 ? 3 : 2;
  constexpr bool kAlias = HB < NB;
  constexpr uint32_t kS = 0, kG = MP, kTileSum = kAlias ? 0 : 2 * MP, kTileCols = tile_cols<HB, GT>();
  constexpr uint32_t kSum1 = 512 - 2 * sum_cols<MP, HB>(), kSum2 = kSum1 + sum_cols<MP, HB>(), kCols = 512;
  static_assert(kTileSum + kTileCols <= kSum1 && 2 * MP <= kSum1, "tensor memory");
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* s_kt = smem;
  uint8_t* s_st = s_kt + L::kL;
  uint8_t* s_q = s_st + L::kL;
  uint8_t* s_g = s_q + L::kX;
  uint8_t* s_p = s_g + L::kX;
  float* s_red = reinterpret_cast<float*>(s_p + HB * L::kP);
  pdl_trigger();
  Frame f;
  if (!open_frame(f, smem, reinterpret_cast<uint8_t*>(s_red + 4 * kTile), sch, kCols, status, 0x4800)) return;
  const T* qq = q + f.bh * sch.N * D;
  const T* gg = d_out + f.bh * sch.N * D;
  const uint32_t a_kt = smem_u32(s_kt), a_st = smem_u32(s_st), a_q = smem_u32(s_q), a_g = smem_u32(s_g), a_p = smem_u32(s_p);
  InTile<T, D> rq, rg;
  auto row0 = [&](int i) { return (int64_t)(f.first + i) * kTile; };
  rq.fetch(qq, row0(0), sch.N);
  rg.fetch(gg, row0(0), sch.N);
  put_landmarks<D, MP>(s_kt, k_landmarks + f.bh * m * D, m, scale);
  put_landmarks<D, MP>(s_st, step2 + f.bh * m * D, m, 1.f);
  rq.put(s_q);
  rg.put(s_g);
  rq.fetch(qq, row0(1), sch.N);
  rg.fetch(gg, row0(1), sch.N);
  f.publish();
  if (f.warp == 0) {
    issue_scores<D, MP, NX>(f.tmem + kS, a_q, a_kt);
    issue_scores<D, MP, NX>(f.tmem + kG, a_g, a_st);
    umma_commit_elect(f.bars + 0);
  }
  for (int i = 0; i < f.count; ++i) {
    const int64_t row = row0(i) + f.row;
    const bool valid = row < sch.N, more = i + 1 < f.count;
    const float lse = valid ? lse1[f.bh * sch.N + row] : 0.f;
    f.wait(0, 0x4900);
    float s[NC], g[NC];
    ld_scores<NB>(f, kS, s);
    ld_scores<NB>(f, kG, g);
    tmem_ld_wait();
    softmax1_jacobian<NC>(f, s_red, s, g, lse, valid, m);
#pragma unroll
    for (int b0 = 0; b0 < NB; b0 += HB) {
#pragma unroll
      for (int b = 0; b < HB; ++b) put_probs<HB>(s_p, f.row, b, f.group, s + 16 * (b0 + b));
      f.publish();
      if (f.warp == 0) {
        issue_contract<HB, NX, GT>(f.tmem + kTileSum, a_p, a_g);
        umma_commit_elect(f.bars + 1);
      }
      f.wait(1, 0x4a00);                     // P1 (and, after the last block, dO) have been used
      add_tile_sum<D, HB, GT>(f, kTileSum, kSum1 + 64 * b0, i == 0);
    }
    if (more) rg.put(s_g);
#pragma unroll
    for (int b0 = 0; b0 < NB; b0 += HB) {
#pragma unroll
      for (int b = 0; b < HB; ++b) put_probs<HB>(s_p, f.row, b, f.group, g + 16 * (b0 + b));
      f.publish();
      if (f.warp == 0) {
        issue_contract<HB, NX, GT>(f.tmem + kTileSum, a_p, a_q);
        umma_commit_elect(f.bars + 2);
        if (more && !kAlias) issue_scores<D, MP, NX>(f.tmem + kG, a_g, a_st);
      }
      if (b0 == 0 && i + 2 < f.count) rg.fetch(gg, row0(i + 2), sch.N);
      f.wait(2, 0x4b00);                     // dS1 (and, after the last block, Q) have been used
      if (kAlias || b0 + HB < NB) add_tile_sum<D, HB, GT>(f, kTileSum, kSum2 + 64 * b0, i == 0);
    }
    if (more) {
      rq.put(s_q);
      if (i + 2 < f.count) rq.fetch(qq, row0(i + 2), sch.N);
      f.publish();
      if (f.warp == 0) {
        issue_scores<D, MP, NX>(f.tmem + kS, a_q, a_kt);
        if (kAlias) issue_scores<D, MP, NX>(f.tmem + kG, a_g, a_st);
        umma_commit_elect(f.bars + 0);
      }
    }
    if (!kAlias) add_tile_sum<D, HB, GT>(f, kTileSum, kSum2, i == 0);
  }
  float* pa = partA + (int64_t)blockIdx.x * 2 * m * D;
  store_sum<D, MP, HB>(f, kSum1, reinterpret_cast<float*>(s_q), pa, m, 1.f);
  store_sum<D, MP, HB>(f, kSum2, reinterpret_cast<float*>(s_q), pa + m * D, m, scale);
  close_frame(f, kCols);
}

// ------------------------------------------------------------------------------------------
// Backward column pass: dV = P3^T dO3, dK = s (dS3^T Qt + dKt_tot[l(n)] / len_l), per-CTA partials of
// dQt = dS3 (sK).  P3 takes V's place once the scores are formed; dV and dK leave through the
// probability buffers.  Two blocks of landmarks take turns in them.  The products lie where the scores were: the next
// scores are issued after everything has been read.
template <class T, int D, int MP>
__global__ void __launch_bounds__(kThr, 1)
sx_bwd_b_kernel(const T* __restrict__ k, const T* __restrict__ v, T* __restrict__ dk, T* __restrict__ dv,
                const float* __restrict__ lse3, const float* __restrict__ D3, const float* __restrict__ q_landmarks,
                const float* __restrict__ dO3, const float* __restrict__ dkt_tot, float* __restrict__ partB, TcSched sch, int m,
                float scale, int* status) {
  using L = Plan<T, D, MP>;
  constexpr int NX = L::NX, NB = L::NB, NC = 16 * NB, ND = D / 4, GV = 4 / NB / NB;   // GV: column groups of dV
  constexpr uint32_t kS = 0, kG = MP, kDv = 0, kDk = kDv + NB * GV * 64, kTileSum = kDk + NB * 64, kSum = 512 - MP, kCols = 512;
  static_assert(L::kHBwdB == 1 && 2 * MP <= kSum && kTileSum + tile_cols<1, 1>() <= kSum, "tensor memory");
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* s_qt = smem;
  uint8_t* s_g3 = s_qt + L::kL;
  uint8_t* s_k = s_g3 + L::kL;
  uint8_t* s_p = s_k + L::kX;               // V, then P3, then the staged dV tile
  uint8_t* s_ds = s_p + L::kP;              // dS3, then the staged dK tile
  float* s_l3 = reinterpret_cast<float*>(s_ds + L::kP);
  float* s_d3 = s_l3 + MP;
  pdl_trigger();
  Frame f;
  if (!open_frame(f, smem, reinterpret_cast<uint8_t*>(s_d3 + MP), sch, kCols, status, 0x5000)) return;
  const T* kk = k + f.bh * sch.N * D;
  const T* vv = v + f.bh * sch.N * D;
  const uint32_t a_qt = smem_u32(s_qt), a_g3 = smem_u32(s_g3), a_k = smem_u32(s_k), a_p = smem_u32(s_p), a_ds = smem_u32(s_ds);
  InTile<T, D> rk, rv;
  auto row0 = [&](int i) { return (int64_t)(f.first + i) * kTile; };
  auto col = [&](int j) { return (j >> 4) * 64 + f.group * 16 + (j & 15); };
  rk.fetch(kk, row0(0), sch.N);
  rv.fetch(vv, row0(0), sch.N);
  put_landmarks<D, MP>(s_qt, q_landmarks + f.bh * m * D, m, scale);
  put_landmarks<D, MP>(s_g3, dO3 + f.bh * m * D, m, 1.f);
  if (threadIdx.x < MP) {
    s_l3[threadIdx.x] = threadIdx.x < m ? lse3[f.bh * m + threadIdx.x] : INFINITY;   // exp(S - inf) = 0
    s_d3[threadIdx.x] = threadIdx.x < m ? D3[f.bh * m + threadIdx.x] : 0.f;
  }
  Segments sg(sch.seg_N, m);
  const float* rows = dkt_tot + f.bh * m * D;
  const int d0 = f.group * ND;
  rk.put(s_k);
  rv.put(s_p);
  f.publish();
  if (f.warp == 0) {
    issue_scores<D, MP, NX>(f.tmem + kS, a_k, a_qt);
    issue_scores<D, MP, NX>(f.tmem + kG, a_p, a_g3);
    umma_commit_elect(f.bars + 0);
  }
  for (int i = 0; i < f.count; ++i) {
    const int64_t row = row0(i) + f.row;
    const bool valid = row < sch.N, more = i + 1 < f.count;
    if (more) {
      rk.fetch(kk, row0(i + 1), sch.N);
      rv.fetch(vv, row0(i + 1), sch.N);
    }
    f.wait(0, 0x5100);
    float s[NC], g[NC];
    ld_scores<NB>(f, kS, s);
    ld_scores<NB>(f, kG, g);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < NC; ++j) {
      s[j] = valid ? expf(s[j] - s_l3[col(j)]) : 0.f;
      g[j] = s[j] * (g[j] - s_d3[col(j)]);
    }
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      if (b > 0) {
        f.wait(1, 0x5200);                   // the previous block's products are done: both buffers are free
        add_tile_sum<D, 1, 1>(f, kTileSum, kSum + 64 * (b - 1), i == 0);
      }
      put_probs<1>(s_p, f.row, 0, f.group, s + 16 * b);
      put_probs<1>(s_ds, f.row, 0, f.group, g + 16 * b);
      f.publish();
      if (f.warp == 0) {
        issue_rows<MP, 1, GV>(f.tmem + kDv + b * GV * 64, a_p, a_g3, b);
        issue_rows<MP, 1, 1>(f.tmem + kDk + b * 64, a_ds, a_qt, b);
        issue_contract<1, NX, 1>(f.tmem + kTileSum, a_ds, a_k);
        umma_commit_elect(f.bars + 1);
      }
    }
    const int l = valid ? sg.landmark_of(sch.row_offset + row) : 0;
    const float inv = scale / (float)sg.len(l);
    float add[ND];
#pragma unroll
    for (int j = 0; j < ND; j += 4) {
      const float4 x = *reinterpret_cast<const float4*>(rows + l * D + d0 + j);
      add[j] = x.x * inv; add[j + 1] = x.y * inv; add[j + 2] = x.z * inv; add[j + 3] = x.w * inv;
    }
    f.wait(1, 0x5300);
    float o[ND];
    ld_rows<D, NB * GV>(f, kDv, o);
    stage_row<T, D>(s_p, L::kPitch, f.row, d0, o);
    ld_rows<D, NB>(f, kDk, o);
#pragma unroll
    for (int j = 0; j < ND; ++j) o[j] += add[j];    // (the operand carries s)
    stage_row<T, D>(s_ds, L::kPitch, f.row, d0, o);
    if (more) rk.put(s_k);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    copy_out<T, D>(dv + f.bh * sch.N * D, s_p, L::kPitch, row0(i), sch.N);
    copy_out<T, D>(dk + f.bh * sch.N * D, s_ds, L::kPitch, row0(i), sch.N);
    add_tile_sum<D, 1, 1>(f, kTileSum, kSum + 64 * (NB - 1), i == 0);
    if (more) {
      __syncthreads();                       // the staged tiles have been read
      rv.put(s_p);
      f.publish();
      if (f.warp == 0) {
        issue_scores<D, MP, NX>(f.tmem + kS, a_k, a_qt);
        issue_scores<D, MP, NX>(f.tmem + kG, a_p, a_g3);
        umma_commit_elect(f.bars + 0);
      }
    }
  }
  store_sum<D, MP, 1>(f, kSum, reinterpret_cast<float*>(s_k), partB + (int64_t)blockIdx.x * m * D, m, scale);
  close_frame(f, kCols);
}

// ------------------------------------------------------------------------------------------
// Second backward row pass: dQ = s (dS1 Kt + dQt_tot[l(n)] / len_l), dS1 formed again from Q and dO.
template <class T, int D, int MP>
__global__ void __launch_bounds__(kThr, 1)
sx_bwd_c_kernel(const T* __restrict__ q, const T* __restrict__ d_out, T* __restrict__ dq, const float* __restrict__ lse1,
                const float* __restrict__ k_landmarks, const float* __restrict__ step2, const float* __restrict__ dqt_tot,
                TcSched sch, int m, float scale, int* status) {
  using L = Plan<T, D, MP>;
  constexpr int NX = L::NX, NB = L::NB, HB = L::kHBwdC, NC = 16 * NB, ND = D / 4, GO = 4 * HB / NB;
  constexpr int GA = NB / HB * GO;           // column groups of dQ: GO for each turn
  constexpr uint32_t kS = 0, kG = MP, kO = 2 * MP, kCols = pow2_cols(kO + GA * 64);
  static_assert(kO + GA * 64 <= 512, "tensor memory");
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* s_kt = smem;
  uint8_t* s_st = s_kt + L::kL;
  uint8_t* s_q = s_st + L::kL;
  uint8_t* s_g = s_q + L::kX;
  uint8_t* s_ds = s_g + L::kX;              // dS1, then the staged dQ tile
  float* s_red = reinterpret_cast<float*>(s_ds + HB * L::kP);
  pdl_trigger();
  Frame f;
  if (!open_frame(f, smem, reinterpret_cast<uint8_t*>(s_red + 4 * kTile), sch, kCols, status, 0x5400)) return;
  const T* qq = q + f.bh * sch.N * D;
  const T* gg = d_out + f.bh * sch.N * D;
  const uint32_t a_kt = smem_u32(s_kt), a_st = smem_u32(s_st), a_q = smem_u32(s_q), a_g = smem_u32(s_g), a_ds = smem_u32(s_ds);
  InTile<T, D> rq, rg;
  auto row0 = [&](int i) { return (int64_t)(f.first + i) * kTile; };
  rq.fetch(qq, row0(0), sch.N);
  rg.fetch(gg, row0(0), sch.N);
  put_landmarks<D, MP>(s_kt, k_landmarks + f.bh * m * D, m, scale);
  put_landmarks<D, MP>(s_st, step2 + f.bh * m * D, m, 1.f);
  rq.put(s_q);
  rg.put(s_g);
  rq.fetch(qq, row0(1), sch.N);
  rg.fetch(gg, row0(1), sch.N);
  f.publish();
  if (f.warp == 0) {
    issue_scores<D, MP, NX>(f.tmem + kS, a_q, a_kt);
    issue_scores<D, MP, NX>(f.tmem + kG, a_g, a_st);
    umma_commit_elect(f.bars + 0);
  }
  Segments sg(sch.seg_N, m);
  const float* rows = dqt_tot + f.bh * m * D;
  const int d0 = f.group * ND;
  for (int i = 0; i < f.count; ++i) {
    const int64_t row = row0(i) + f.row;
    const bool valid = row < sch.N, more = i + 1 < f.count;
    const float lse = valid ? lse1[f.bh * sch.N + row] : 0.f;
    f.wait(0, 0x5500);
    float s[NC], g[NC];
    ld_scores<NB>(f, kS, s);
    ld_scores<NB>(f, kG, g);
    tmem_ld_wait();
    softmax1_jacobian<NC>(f, s_red, s, g, lse, valid, m);   // (its barrier: the previous output tile has left s_ds)
#pragma unroll
    for (int b0 = 0; b0 < NB; b0 += HB) {
      if (b0 > 0) f.wait(1, 0x5600);         // the previous block has been used
#pragma unroll
      for (int b = 0; b < HB; ++b) put_probs<HB>(s_ds, f.row, b, f.group, g + 16 * (b0 + b));
      if (b0 == 0 && more) {
        rq.put(s_q);
        rg.put(s_g);
      }
      f.publish();
      if (f.warp == 0) {
        issue_rows<MP, HB, GO>(f.tmem + kO + b0 / HB * GO * 64, a_ds, a_kt, b0);
        umma_commit_elect(f.bars + 1);
        if (b0 == 0 && more) {
          issue_scores<D, MP, NX>(f.tmem + kS, a_q, a_kt);
          issue_scores<D, MP, NX>(f.tmem + kG, a_g, a_st);
          umma_commit_elect(f.bars + 0);
        }
      }
    }
    if (i + 2 < f.count) {
      rq.fetch(qq, row0(i + 2), sch.N);
      rg.fetch(gg, row0(i + 2), sch.N);
    }
    const int l = valid ? sg.landmark_of(sch.row_offset + row) : 0;
    const float inv = scale / (float)sg.len(l);
    float add[ND];
#pragma unroll
    for (int j = 0; j < ND; j += 4) {
      const float4 x = *reinterpret_cast<const float4*>(rows + l * D + d0 + j);
      add[j] = x.x * inv; add[j + 1] = x.y * inv; add[j + 2] = x.z * inv; add[j + 3] = x.w * inv;
    }
    f.wait(1, 0x5700);
    float o[ND];
    ld_rows<D, GA>(f, kO, o);
#pragma unroll
    for (int j = 0; j < ND; ++j) o[j] += add[j];
    stage_row<T, D>(s_ds, L::kPitch, f.row, d0, o);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    copy_out<T, D>(dq + f.bh * sch.N * D, s_ds, L::kPitch, row0(i), sch.N);
  }
  close_frame(f, kCols);
}

// The shapes these kernels take: fp32 with up to 64 landmarks and head_dim 16 .. 64; 16-bit inputs with head_dim
// 16 .. 64 and up to 128 landmarks (head_dim 64 with up to 64 landmarks has 16-bit kernels of its own, which are
// asked first).  The line lies where the term tiles of one 128-row tile and both landmark operands stop fitting into
// shared memory: three terms of a 128-landmark or head_dim-128 operand pair take 96 .. 192 KB alone.  They are
// faster than the CUDA-core kernels from one tile on (B=1, H=4, N=1024, m=32, fp32: 143 -> 79 us for the five).
inline bool supported(int dtype, int D, int m, uint32_t flags) {
  if ((flags & FNB_FLAG_FORCE_GENERIC) || D > 64) return false;
  return dtype == FNB_F32 ? m <= 64 : m <= 128;
}

}  // namespace sx
}  // namespace fnb
