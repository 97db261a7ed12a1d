// Matrix products of few rows (decode steps, short prompts): out[r, n] = epilogue(sum_k A[r, k] W[n, k]).
//
// Such a call is a read of the weights: 2 bytes per weight against at most 64 rows of work. The tile kernel
// (gemm_sm100.cuh) runs it as chains of 128-row tensor-core tiles with barriers, tensor memory and an
// issuing thread between them: 4.9 us before its first result and 0.21 us per 64 elements of K, whatever the
// rows. Here a block takes 16 (or 32) weight rows and its eight warps a share of K each; weights and rows go
// from global memory straight into the fragments of m16n8k16 products (weights as the 16-row operand, tokens
// as the 8-column one), with no staging and no barrier before the one at which the warps' partial sums meet.
//   * K is permuted inside a step of 32 so that a lane's 16-byte load is two steps' worth of one row: both
//     operands use the same permutation, and the four lanes of a row read 64 consecutive bytes.
//   * A block asks for its weights in L2 BEFORE it waits for the kernel ahead of it. A prefetch reads nothing into
//     the program, so it may run ahead of whatever still writes; it takes the DRAM latency out of the step.
//   * The partial sums are added in the order of their shares of K, whose number depends on the weights alone: results depend
//     neither on timing nor on the rows beside a row.
// Row groups (experts) are walked in passes of at most 32 rows of one group; empty groups end at once.
// Bound by: L2 to SM traffic (weights once, the rows once per block: 7 to 9 TB/s) from 16 rows on, before that by
// the launch (2.1 us at K = N = 768, one row; the tile kernel 6.8). The other figures stand at few_rows_taken.
#include <cuda_bf16.h>
#include "../../include/cdeep.h"
#include "checks.cuh"
#include "elem.cuh"
#include "gemm_sm100.cuh"
#include "kernels.h"
#include "mma.cuh"

namespace cdeep {
namespace {

constexpr int kStep = 32;          // elements of K per step: one 16-byte load per lane and row

struct FewParams {
  GemmParams g;                    // shapes and epilogue, as the tile kernel takes them
  const bf16 *a0, *b0, *a1, *b1;   // a1 / b1: second K segment, or b1 the second problem's weights
  long long lda0, ldb0, lda1, ldb1;
  int half, half2;                 // gated units: rows of a gate block, up rows follow (packed layout); the second problem's
  int tiles, tiles2;               // blocks per group, of the second problem
  int prefetch;                    // ask for the block's own weights ahead of the kernel before
  int sms;                         // of the device
};

// Weights and rows may have been written by the kernel ahead, which can still run when this one starts: neither takes the
// read-only path, and the loads keep their place behind the wait as volatile. Zeros where `on` does not hold. Rows stay in
// the L1 for the other blocks of the SM (8 rows, N 32000: 25.2 us, 27.7 without), weights do not.
template <bool kKeep>
__device__ __forceinline__ uint4 load_if(const bf16* p, bool on) {
  uint4 v;
  if constexpr (kKeep)
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %5, 0;\n\t"
        "mov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\tmov.u32 %2, 0;\n\tmov.u32 %3, 0;\n\t"
        "@q ld.global.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
        : "=&r"(v.x), "=&r"(v.y), "=&r"(v.z), "=&r"(v.w) : "l"(p), "r"(static_cast<uint32_t>(on)));
  else
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %5, 0;\n\t"
        "mov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\tmov.u32 %2, 0;\n\tmov.u32 %3, 0;\n\t"
        "@q ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
        : "=&r"(v.x), "=&r"(v.y), "=&r"(v.z), "=&r"(v.w) : "l"(p), "r"(static_cast<uint32_t>(on)));
  return v;
}
__device__ __forceinline__ void prefetch_row(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// A run of steps of one K segment: `n` of them, of which this lane's elements lie inside K for the first `n_lane`.
struct FewRun {
  int first, n, n_lane;
};
// The part of the steps [s_lo, s_hi) of the concatenated K that lies in the segment of K elements from step `off` on.
__device__ __forceinline__ FewRun few_run(int s_lo, int s_hi, int off, int K, int q8) {
  FewRun r;
  r.first = max(s_lo - off, 0);
  r.n = max(min(s_hi - off, (K + kStep - 1) / kStep) - r.first, 0);
  r.n_lane = min(max((K - q8 - r.first * kStep + kStep - 1) / kStep, 0), r.n);
  return r;
}

// acc += tokens x weights over a run of steps. wp: this lane's weight rows at the run's first step, tp: its token rows
// (kA steps in flight). Nothing but the loads and the products is left in the loop: a warp is one chain of a few
// hundred instructions, and with two warps a scheduler each of them costs some eight cycles. us, with bounds and addresses
// found step by step / so (eight warps a block): K = N = 2048, one row 4.4 / 3.9, 64 rows 6.7 / 6.2; K 5632, N 2048, one row
// 11.2 / 8.1; K 768, N 1280 3.3 / 2.9.
template <int MT, int NT, int kU, int kA>
__device__ __forceinline__ void few_walk(float (&acc)[MT][NT][4], const bf16* (&wp)[MT][2], const bf16* (&tp)[NT],
                                         const FewRun& run) {
  static_assert(kU % kA == 0, "a step's slots are known when the loop is unrolled");
  const int n = run.n_lane;
  uint4 w[kU][MT][2], t[kA][NT];
#pragma unroll
  for (int u = 0; u < kA; ++u)
#pragma unroll
    for (int i = 0; i < NT; ++i) t[u][i] = load_if<true>(tp[i] + u * kStep, u < n);
#pragma unroll
  for (int u = 0; u < kU; ++u)
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int h = 0; h < 2; ++h) w[u][m][h] = load_if<false>(wp[m][h] + u * kStep, u < n);
  auto step = [&](int s, int u) {
    uint4 (&x)[NT] = t[u % kA];
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const uint32_t f0[4] = {w[u][m][0].x, w[u][m][1].x, w[u][m][0].y, w[u][m][1].y};
      const uint32_t f1[4] = {w[u][m][0].z, w[u][m][1].z, w[u][m][0].w, w[u][m][1].w};
#pragma unroll
      for (int i = 0; i < NT; ++i) mma16816(acc[m][i], f0, x[i].x, x[i].y);
#pragma unroll
      for (int i = 0; i < NT; ++i) mma16816(acc[m][i], f1, x[i].z, x[i].w);
    }
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int h = 0; h < 2; ++h) w[u][m][h] = load_if<false>(wp[m][h] + (u + kU) * kStep, s + u + kU < n);
#pragma unroll
    for (int i = 0; i < NT; ++i) x[i] = load_if<true>(tp[i] + (u + kA) * kStep, s + u + kA < n);
  };
  int s = 0;
  for (; s + kU <= run.n; s += kU) {
#pragma unroll
    for (int u = 0; u < kU; ++u) step(s, u);
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int h = 0; h < 2; ++h) wp[m][h] += kU * kStep;
#pragma unroll
    for (int i = 0; i < NT; ++i) tp[i] += kU * kStep;
  }
#pragma unroll
  for (int u = 0; u < kU - 1; ++u)
    if (s + u < run.n) step(s, u);
}

// What the epilogue of four columns reads, asked for ahead of the products.
struct FewItem {
  long long at;                    // destination row (or its address), -1: nothing to store
  uint2 hi, lo, r2;
  float4 rf;
};
template <int EPI>
__device__ __forceinline__ FewItem few_fetch(const GemmParams& g, int r, int m_end, int col, int out_cols) {
  constexpr bool kGated = EPI == kEpiSwiGLU || EPI == kEpiGlu;
  constexpr bool kSplit = EPI == kEpiStoreSplit;
  constexpr bool kF32 = EPI == kEpiStoreF32;
  FewItem it;
  it.at = -1;
  it.hi = it.lo = it.r2 = make_uint2(0, 0);
  it.rf = make_float4(0.f, 0.f, 0.f, 0.f);
  if (r >= m_end || col >= out_cols) return it;
  if constexpr (kGated) {
    it.at = r;
  } else {
    if (!kF32 && !kSplit && g.out_row_ptrs) {
      const long long addr = g.out_row_ptrs[r];
      if (row_address_ok(addr, g.status)) it.at = addr;
      return it;
    }
    const int o = g.row_map ? g.row_map[r] : r;
    if (kChecks && g.row_map && g.out_rows > 0 && !index_ok(o, g.out_rows, g.status)) return it;
    it.at = o;
    if constexpr (kF32) {
      if (g.residual) it.rf = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(g.residual) + static_cast<long long>(o) * g.ldr + col);
    } else {
      if (g.residual) it.hi = *reinterpret_cast<const uint2*>(g.residual + static_cast<long long>(o) * g.ldr + col);
      if (kSplit && g.residual_lo) it.lo = *reinterpret_cast<const uint2*>(g.residual_lo + static_cast<long long>(o) * g.ldr + col);
      if (g.residual2) it.r2 = *reinterpret_cast<const uint2*>(g.residual2 + static_cast<long long>(r) * g.ldr2 + col);
    }
  }
  return it;
}
// f (and, for gated units, u) are the sums of the four columns from `col` on.
template <int EPI>
__device__ __forceinline__ void few_store(const GemmParams& g, bool second, const FewItem& it, int col, float (&f)[4], const float (&u)[4]) {
  constexpr bool kGated = EPI == kEpiSwiGLU || EPI == kEpiGlu;
  constexpr bool kSplit = EPI == kEpiStoreSplit;
  constexpr bool kF32 = EPI == kEpiStoreF32;
  if constexpr (kF32) {
#pragma unroll
    for (int j = 0; j < 4; ++j) f[j] *= g.acc_scale;
    if (g.col_scale) {
      const uint2 c = *reinterpret_cast<const uint2*>(g.col_scale + col);
      f[0] *= bf_lo(c.x); f[1] *= bf_hi(c.x); f[2] *= bf_lo(c.y); f[3] *= bf_hi(c.y);
    }
    *reinterpret_cast<float4*>(reinterpret_cast<float*>(g.out) + it.at * g.ldo + col) =
        make_float4(f[0] + it.rf.x, f[1] + it.rf.y, f[2] + it.rf.z, f[3] + it.rf.w);
  } else if constexpr (kGated) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      f[j] = EPI == kEpiGlu ? clamped_glu_f(f[j], u[j], g.glu_alpha, g.glu_limit, g.glu_offset) : silu_f(f[j]) * u[j];
    *reinterpret_cast<uint2*>((second ? g.out2 : g.out) + it.at * (second ? g.ldo2 : g.ldo) + col) =
        make_uint2(bf_pack(f[0], f[1]), bf_pack(f[2], f[3]));
  } else {
    if (!kSplit && g.act == 1) {
#pragma unroll
      for (int j = 0; j < 4; ++j) f[j] = fmaxf(f[j], 0.f) * fmaxf(f[j], 0.f);
    }
    if (g.bias) {
      const uint2 b = *reinterpret_cast<const uint2*>(g.bias + col);
      const float bb[4] = {bf_lo(b.x), bf_hi(b.x), bf_lo(b.y), bf_hi(b.y)};
#pragma unroll
      for (int j = 0; j < 4; ++j) f[j] += fminf(fmaxf(bb[j], g.bias_lo), g.bias_hi);
    }
    auto add = [&](const uint2& v) { f[0] += bf_lo(v.x); f[1] += bf_hi(v.x); f[2] += bf_lo(v.y); f[3] += bf_hi(v.y); };
    if (g.residual) add(it.hi);
    if (kSplit && g.residual_lo) add(it.lo);
    if (g.residual2) add(it.r2);
    if (g.do_clamp) {
#pragma unroll
      for (int j = 0; j < 4; ++j) f[j] = fminf(fmaxf(f[j], g.clamp_lo), g.clamp_hi);
    }
    const uint2 o = make_uint2(bf_pack(f[0], f[1]), bf_pack(f[2], f[3]));
    if (!kSplit && g.out_row_ptrs) {
      *reinterpret_cast<uint2*>(reinterpret_cast<bf16*>(it.at) + col) = o;
    } else {
      if (g.out) *reinterpret_cast<uint2*>(g.out + it.at * g.ldo + col) = o;
      if (kSplit && g.out_lo)
        *reinterpret_cast<uint2*>(g.out_lo + it.at * g.ldo + col) =
            make_uint2(bf_pack(f[0] - bf_lo(o.x), f[1] - bf_hi(o.x)), bf_pack(f[2] - bf_lo(o.y), f[3] - bf_hi(o.y)));
    }
  }
}


struct Weights {                   // of the block's group, one matrix per K segment
  const bf16 *b0, *b1;
  long long ld0, ld1;
};

template <int MT>
constexpr int kRowFloats = 16 * MT + 4;                    // partial sums of a token: the accumulators' writes hit 32 banks

// One pass: the block's weight rows against the tokens [m0, m0 + 8 NT) of a group that ends at m_end. K is cut into WK x SUB shares,
// SUB behind one another for each warp.
template <int EPI, int MT, int NT, int WK, int SUB, bool kDeep>
__device__ __forceinline__ void few_pass(const FewParams& p, float* red, const Weights& wt, const int (&w_row)[MT][2], int n_steps0,
                                         int n_steps, int m0, int m_end, int col0, bool second) {
  constexpr bool kGated = EPI == kEpiSwiGLU || EPI == kEpiGlu;
  constexpr int kRow = kRowFloats<MT>;
  constexpr int kU = (MT == 1 && NT <= 2) || (kDeep && NT == 1) ? 4 : 2;   // steps of weights in flight
  constexpr int kAhead = NT >= 6 ? 1 : 2;                  // steps of tokens in flight
  const GemmParams& g = p.g;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q8 = (lane & 3) * 8;

  // what the epilogue reads, ahead of the products
  constexpr int kQuads = 4 * (kGated ? 1 : MT);            // outputs of a token in fours
  constexpr int kItems = (8 * NT * kQuads + (WK * 32) - 1) / (WK * 32);
  const int out_cols = second ? g.out_cols2 : g.out_cols;
  FewItem items[kItems];
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const int item = threadIdx.x + i * (WK * 32);
    items[i] = few_fetch<EPI>(g, item < 8 * NT * kQuads ? m0 + item / kQuads : m_end, m_end, col0 + (item % kQuads) * 4, out_cols);
  }

#pragma unroll 1
  for (int sub = 0; sub < SUB; ++sub) {
    const int share = warp * SUB + sub;
    float acc[MT][NT][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[m][n][e] = 0.f;
    // this share's steps, segment by segment
    const int s_lo = share * n_steps / (WK * SUB), s_hi = (share + 1) * n_steps / (WK * SUB);
#pragma unroll 1
    for (int seg = 0; seg < (g.K1 > 0 ? 2 : 1); ++seg) {
      const FewRun run = few_run(s_lo, s_hi, seg ? n_steps0 : 0, seg ? g.K1 : g.K0, q8);
      if (run.n == 0) continue;
      const long long k = run.first * kStep + q8;
      const bf16 *wp[MT][2], *tp[NT];
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) wp[m][h] = (seg ? wt.b1 + w_row[m][h] * wt.ld1 : wt.b0 + w_row[m][h] * wt.ld0) + k;
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        const int row = min(m0 + n * 8 + (lane >> 2), m_end - 1);                       // rows past the end are not stored
        tp[n] = (seg ? p.a1 + row * p.lda1 : p.a0 + row * p.lda0) + k;
      }
      few_walk<MT, NT, kU, kAhead>(acc, wp, tp, run);
    }

    // partial sums: [share][token][feature]
    float* mine = red + share * (8 * NT * kRow);
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        float* row = mine + (n * 8 + (lane & 3) * 2) * kRow + m * 16 + (lane >> 2);
        row[0] = acc[m][n][0];
        row[kRow] = acc[m][n][1];
        row[8] = acc[m][n][2];
        row[kRow + 8] = acc[m][n][3];
      }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    if (items[i].at < 0) continue;
    const int item = threadIdx.x + i * (WK * 32);
    const int tok = item / kQuads, quad = item % kQuads, col = col0 + quad * 4;
    float f[4] = {0.f, 0.f, 0.f, 0.f}, u[4] = {0.f, 0.f, 0.f, 0.f};
    const float* src = red + tok * kRow + quad * 4;
#pragma unroll
    for (int w_ = 0; w_ < WK * SUB; ++w_) {
      const float4 v = *reinterpret_cast<const float4*>(src + w_ * (8 * NT * kRow));
      f[0] += v.x; f[1] += v.y; f[2] += v.z; f[3] += v.w;
      if constexpr (kGated) {
        const float4 x = *reinterpret_cast<const float4*>(src + 16 + w_ * (8 * NT * kRow));
        u[0] += x.x; u[1] += x.y; u[2] += x.z; u[3] += x.w;
      }
    }
    few_store<EPI>(g, second, items[i], col, f, u);
  }
}

struct Block {
  int group, col0;                 // row group, first output column
  bool second;                     // dense block against the second problem's weights
};
template <int EPI, int MT>
__device__ __forceinline__ Block locate(const FewParams& p, int block) {
  constexpr bool kGated = EPI == kEpiSwiGLU || EPI == kEpiGlu;
  const int grouped = p.tiles * p.g.num_groups;
  Block b;
  b.second = kGated && block >= grouped;
  b.group = b.second ? 0 : block / p.tiles;
  b.col0 = (b.second ? block - grouped : block - b.group * p.tiles) * 16 * (kGated ? 1 : MT);
  return b;
}
__device__ __forceinline__ Weights weights_of(const FewParams& p, const Block& b) {
  Weights w;
  w.b0 = b.second ? p.b1 : p.b0 + static_cast<long long>(b.group) * p.g.b0_group_rows * p.ldb0;
  w.b1 = p.b1 + static_cast<long long>(b.group) * p.g.b1_group_rows * p.ldb1;
  w.ld0 = b.second ? p.ldb1 : p.ldb0;
  w.ld1 = p.ldb1;
  return w;
}
// Weight row i of the block's m-th 16 (clamped into the group's rows: what a clamped row gives is not stored).
template <int EPI>
__device__ __forceinline__ int weight_row(const FewParams& p, const Block& b, int m, int i) {
  const int last = (b.second ? p.g.N2 : p.g.N) - 1;
  if constexpr (EPI == kEpiSwiGLU || EPI == kEpiGlu) {
    const int half = b.second ? p.half2 : p.half, j = b.col0 + i, blk = j / half;
    return min(blk * 2 * half + m * half + (j - blk * half), last);
  } else {
    return min(b.col0 + m * 16 + i, last);
  }
}
template <int EPI, int MT>
__device__ __forceinline__ void prefetch_block(const FewParams& p, const Block& b) {
  if (threadIdx.x >= 16 * MT) return;
  const Weights w = weights_of(p, b);
  const long long row = weight_row<EPI>(p, b, threadIdx.x >> 4, threadIdx.x & 15);
  prefetch_row(w.b0 + row * w.ld0, static_cast<uint32_t>(p.g.K0) * 2);
  if (p.g.K1 > 0) prefetch_row(w.b1 + row * w.ld1, static_cast<uint32_t>(p.g.K1) * 2);
}

template <int N> struct Int { static constexpr int value = N; };

// kWhole: up to 8 NTMAX rows, all against the same weights. kGroups: row groups of any sizes in passes of up to 32 rows;
// kManyGroups: in several waves of blocks, where nothing is asked for ahead of time and four steps of weights in flight take its
// place (64 experts, 512 rows, both products: steps of the 2048 wide model 25.8 -> 25.3 ms; in one wave they cost 1 %).
enum Kind { kWhole, kGroups, kManyGroups };
template <int EPI, int MT, int NTMAX, int WK, int KIND, int SUB>
__global__ void __launch_bounds__(WK * 32, NTMAX >= 8 ? 8 / WK : 16 / WK) few_rows_kernel(const __grid_constant__ FewParams p) {
  static_assert((EPI != kEpiSwiGLU && EPI != kEpiGlu) || MT == 2, "a gated unit takes its gate rows and its up rows together");
  extern __shared__ float4 smem4[];
  float* red = reinterpret_cast<float*>(smem4);
  const GemmParams& g = p.g;
  const int lane = threadIdx.x & 31;
  const Block at = locate<EPI, MT>(p, blockIdx.x);
  // this lane's weight rows
  int w_row[MT][2];
  const Weights wt = weights_of(p, at);
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) w_row[m][h] = weight_row<EPI>(p, at, m, (lane >> 2) + h * 8);
  if (p.prefetch) prefetch_block<EPI, MT>(p, at);
  pdl_enter();

  int m_lo = 0, m_hi = g.M;
  if (g.seg_offsets && !at.second) {
    m_lo = g.seg_offsets[at.group];
    m_hi = g.seg_offsets[at.group + 1];
  }
  if (kChecks && g.seg_offsets) {
    // checking build: a segment table that is not 0 <= s[0] <= s[1] <= ... <= M stores nothing
    bool bad = false;
    for (int i = 0; i < g.num_groups; ++i) {
      const int lo = g.seg_offsets[i], hi = g.seg_offsets[i + 1];
      bad = bad || lo < 0 || hi < lo || hi > g.M;
    }
    if (bad) {
      if (threadIdx.x == 0 && g.status) atomicMax(g.status, kStatusBounds);
      return;
    }
  }
  const int n_steps0 = (g.K0 + kStep - 1) / kStep;
  const int n_steps = n_steps0 + (g.K1 + kStep - 1) / kStep;
  for (int m0 = m_lo; m0 < m_hi; m0 += 8 * NTMAX) {
    const int left = m_hi - m0;
    if (m0 > m_lo) __syncthreads();                        // the sums of the pass before are read
    auto pass = [&](auto nt) {
      few_pass<EPI, MT, decltype(nt)::value, WK, SUB, KIND == kManyGroups>(p, red, wt, w_row, n_steps0, n_steps, m0, m_hi, at.col0, at.second);
    };
    if constexpr (KIND == kWhole) {
      if constexpr (NTMAX == 8) {
        if (left <= 48) pass(Int<6>());
        else pass(Int<8>());
      } else {
        pass(Int<NTMAX>());
      }
    } else {
      if (left <= 8) pass(Int<1>());
      else if (left <= 16) pass(Int<2>());
      else pass(Int<4>());
    }
  }
}

template <int EPI, int MT, int NTMAX, int WK, int KIND = kWhole, int SUB = 1>
cudaError_t launch_few(const FewParams& p, cudaStream_t stream) {
  constexpr int smem = WK * SUB * 8 * NTMAX * kRowFloats<MT> * 4;
  cudaError_t e = allow_smem<few_rows_kernel<EPI, MT, NTMAX, WK, KIND, SUB>>(smem);
  if (e != cudaSuccess) return e;
  FewParams q = p;
  const unsigned grid = static_cast<unsigned>(p.tiles * p.g.num_groups + p.tiles2);
  // Beyond one wave the asking ahead gets in the way of the reads themselves: 64 experts of 2 x 704 x 2048, 256 rows 100 us
  // with it (each block asking for the next one's as well), 73 without; N 32000, 8 rows 39 / 32.
  if (grid > static_cast<unsigned>(p.sms * (NTMAX >= 8 ? 8 : 16) / WK)) q.prefetch = 0;
  return launch_kernel(few_rows_kernel<EPI, MT, NTMAX, WK, KIND, SUB>, dim3(grid), dim3(WK * 32), smem, stream, q);
}

template <int EPI, int MT, int WK>
cudaError_t launch_warps(const FewParams& p, cudaStream_t stream) {
  if constexpr (WK == 16) {
    // sixteen shares whatever the number of rows, so that a row's bits do not depend on it: 49 and more do not fit the registers
    // of sixteen warps, and eight take two shares each
    if (p.g.M > 32 && p.g.num_groups > 1) return launch_few<EPI, MT, 4, WK, kGroups>(p, stream);
    if (p.g.M > 48) return launch_few<EPI, MT, 8, 8, kWhole, 2>(p, stream);
    if (p.g.M > 32) return launch_few<EPI, MT, 6, WK>(p, stream);
    if (p.g.M > 16) return launch_few<EPI, MT, 4, WK>(p, stream);
    return p.g.M <= 8 ? launch_few<EPI, MT, 1, WK>(p, stream) : launch_few<EPI, MT, 2, WK>(p, stream);
  } else {
    if (p.g.M <= 8) return launch_few<EPI, MT, 1, WK>(p, stream);
    if (p.g.num_groups > 1 || p.tiles2 > 0) {
      const long long blocks = static_cast<long long>(p.tiles) * p.g.num_groups + p.tiles2;
      if (MT == 2 && blocks > p.sms * 16LL / WK) return launch_few<EPI, MT, 4, WK, kManyGroups>(p, stream);
      return launch_few<EPI, MT, 4, WK, kGroups>(p, stream);
    }
    if (p.g.M > 32) return launch_few<EPI, MT, 8, WK>(p, stream);
    return p.g.M <= 16 ? launch_few<EPI, MT, 2, WK>(p, stream) : launch_few<EPI, MT, 4, WK>(p, stream);
  }
}
// More blocks than the two of eight warps that an SM holds: four warps each and four on an SM, since a block is then
// mostly its own start and end (64 experts of 704 x 2048, 8 rows: 14.5 us with eight warps, 9.4 with four). Fewer
// blocks: eight warps, a shorter chain. No more blocks than SMs, and a long K (64 steps of both segments together): sixteen
// shares, since eight warps with four steps in flight do not keep an SM's share of the bandwidth busy (N 2048, one row, us with
// eight / sixteen: K 2048 3.9 / 3.3, 4096 6.2 / 4.8, 5632 8.1 / 6.1; 32 rows 5.5 / 4.7, 8.6 / 7.3, 11.1 / 8.9; replayed, where
// eight shares were faster: 33 rows 4.6 / 4.8, 7.1 / 7.0, 9.0 / 8.7, 64 rows 5.6 / 6.5, 8.6 / 9.4, 11.0 / 11.9). Of a shorter K
// the sixteen sums cost more than they bring (K = N = 1024, 16 rows 2.7 / 3.1), of few blocks as well (N 64, K 2048 3.2 / 3.6).
template <int EPI, int MT>
cudaError_t launch_rows(const FewParams& p, cudaStream_t stream) {
  const long long blocks = static_cast<long long>(p.tiles) * p.g.num_groups + p.tiles2;
  const int n_steps = (p.g.K0 + kStep - 1) / kStep + (p.g.K1 + kStep - 1) / kStep;
  if constexpr (MT == 1)
    if (blocks <= p.sms && 4 * blocks >= p.sms && n_steps >= 64) return launch_warps<EPI, MT, 16>(p, stream);
  return blocks > 2LL * p.sms ? launch_warps<EPI, MT, 4>(p, stream) : launch_warps<EPI, MT, 8>(p, stream);
}

template <int EPI>
cudaError_t launch_store(const FewParams& p, int mt, cudaStream_t stream) {
  return mt == 2 ? launch_rows<EPI, 2>(p, stream) : launch_rows<EPI, 1>(p, stream);
}

}  // namespace

// 32 weight rows per block once that still gives every SM two blocks: half the reads of the tokens.
static int store_mt(long long cols, int num_groups, int sm_count) { return num_groups * ((cols + 31) / 32) >= 2LL * sm_count ? 2 : 1; }

// Which calls stream (us on one B200, this kernel / the tile kernel):
//   row groups: up to 64 rows; up to 8 per group on average where the caller knows that no group has more than 64 (two
//     passes; the sizes themselves are on the device). 64 experts of 2 x 704 x 2048, cold, 512 rows: evenly dealt 69 / 90,
//     64 in each of 8 groups 35 / 39, their down projections 46 / 47 and 23 / 22; 1024 rows 79 / 90. Without a bound on a group a pass
//     per 32 of its rows reads the weights again: half of 512 rows in one group 100 / 90 and 55 / 47, all of them 152 / 31
//     and 80 / 20; 128 experts, 1024 rows in one 174 / 27. 32 experts of 2 x 704 x 1024, 256 rows 27 / 44. 8 experts and a
//     shared one: 32 rows 14 / 26, 64 rows 15 / 26; 65 rows in one group 33 / 39 and 19 / 21.
//   dense: up to 64 rows, unless the tokens, which every block reads again, cost more than the tile kernel's chains.
//     K 2048, N 2048: 32 rows 4.8 / 11.6, 64 rows 7.0 / 11.6; K 4096, N 4096: 32 rows 11.3 / 16.2, 40 rows 19.1 / 16.2;
//     K 2048, N 6272: 32 rows 10.3 / 12.7, 40 rows 17.9 / 12.7; K 2048, N 32000: 16 rows 26 / 37, 32 rows 34 / 30. The
//     estimates below put the line between these: both sides in bytes per ns at the rates that they reach (from 33 rows
//     on a block has an SM to itself, and more blocks than SMs lose), 4.9 us and 0.21 us per 64 of K for a chain.
bool few_rows_taken(int M, int num_groups, int most_rows, bool second, int kind, int cols, int K, int sm_count) {
  if (num_groups > 1 || second) return M <= 64 || (!second && M <= 8 * num_groups && most_rows > 0 && most_rows <= 64);
  if (M > 64) return false;
  const bool gated = kind == kEpiSwiGLU || kind == kEpiGlu;
  const int per_block = gated ? 16 : 16 * store_mt(cols, 1, sm_count);
  const long long weights = 2LL * cols * K * (gated ? 2 : 1);
  const long long tokens = 2LL * M * K * ((cols + per_block - 1) / per_block);
  const long long blocks = (cols + per_block - 1) / per_block;
  const long long stream_ns = M <= 32 ? 1800 + (weights + tokens) / 8400 : 2000 + (weights + tokens) / (blocks > sm_count ? 6500 : 7500);
  const long long chain_ns = 4900 + 210LL * ((K + 63) / 64), read_ns = 4000 + weights / 5800;
  return stream_ns <= (chain_ns > read_ns ? chain_ns : read_ns);
}

cudaError_t launch_few_rows(const GemmParams& g, int kind, const GemmOperand& op0, const GemmOperand* op1, const GemmSecond* second,
                            int block_n, int sm_count, cudaStream_t stream) {
  FewParams p;
  p.g = g;
  p.a0 = static_cast<const bf16*>(op0.a);
  p.b0 = static_cast<const bf16*>(op0.b);
  p.lda0 = op0.lda;
  p.ldb0 = op0.ldb;
  p.a1 = op1 ? static_cast<const bf16*>(op1->a) : p.a0;
  p.b1 = op1 ? static_cast<const bf16*>(op1->b) : second ? static_cast<const bf16*>(second->b) : p.b0;
  p.lda1 = op1 ? op1->lda : op0.lda;
  p.ldb1 = op1 ? op1->ldb : second ? second->ldb : op0.ldb;
  p.half = block_n / 2;
  p.half2 = second ? second->block_n / 2 : p.half;
  p.tiles2 = second ? (second->out_cols + 15) / 16 : 0;
  // of a grouped call only as much is asked for ahead of time as its rows are sure to use
  p.prefetch = g.num_groups == 1 || g.M >= 2 * g.num_groups;
  p.sms = sm_count;
  if (kind == kEpiSwiGLU || kind == kEpiGlu) {
    p.tiles = (g.out_cols + 15) / 16;
    return kind == kEpiSwiGLU ? launch_rows<kEpiSwiGLU, 2>(p, stream) : launch_rows<kEpiGlu, 2>(p, stream);
  }
  const int mt = store_mt(g.out_cols, g.num_groups, sm_count);
  p.tiles = (g.out_cols + 16 * mt - 1) / (16 * mt);
  if (kind == kEpiStoreF32) return launch_store<kEpiStoreF32>(p, mt, stream);
  if (kind == kEpiStoreSplit) return launch_store<kEpiStoreSplit>(p, mt, stream);
  return launch_store<kEpiStore>(p, mt, stream);
}

}  // namespace cdeep
