// out[m, n] = residual[m, n] + scale * col_scale[n] * act(sum_k a[m, k] b[n, k]), all fp32 on the FMA pipe: the 32-bit
// matrix product of models that run entirely in fp32 (no reduced-precision mode anywhere on that path).
//
// With `seg` the grid's third axis is the group: its rows [seg[g], seg[g + 1]) of a meet the g-th N rows of b.
// Every output is one chain of fused multiply-adds over k in ascending order, whatever the tile, and its last factor and
// the residual are one more (written as such, so that no compiler chooses): results depend on neither the number of rows
// nor the tile nor the width of the stores.
//   * Both operands lie transposed in shared memory, two stages; the next stage is on its way in registers while one
//     is multiplied. A thread holds TM x TN outputs; products go in pairs of columns (fma.rn.f32x2: half the
//     instructions; 1303 against 1543 us with single ones for 1018 x 1024 x 32000).
//   * Bound by: the FMA pipe and the shared-memory reads that feed it, which are about as long (128 x 128 tiles,
//     8 x 8 outputs: 71 % of the pipe). 16 x 8 outputs read less but leave two warps a scheduler: 1367 us.
#include "elem.cuh"
#include "kernels.h"

namespace cdeep {

namespace {

struct LinearF32 {
  const float* a;
  long long lda;
  const float* b;
  const float* residual;
  const float* col_scale;
  float scale;
  int act;
  float* out;
  const int* seg;
  int M, K, N;
  int vec;                   // out, residual and col_scale can be read and written four columns at a time
};

// two independent fp32 multiply-adds in one instruction, each rounded as fmaf rounds
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long pair(float lo, float hi) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ void unpair(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

template <int BM, int BN, int TM, int TN, int TK>
struct Tile {
  static constexpr int kRowThreads = BM / TM, kColThreads = BN / TN;
  static constexpr int kThreads = kRowThreads * kColThreads;
  static constexpr int kWarpCols = kColThreads / 8;           // a warp is 4 x 8 threads
  static_assert(kRowThreads % 4 == 0 && kColThreads % 8 == 0 && TM % 4 == 0 && TN % 4 == 0, "warps of 4 x 8 threads");
  static constexpr int kLda = BM + 4, kLdb = BN + 4;
  static constexpr int kLoadsA = (BM * TK / 4 + kThreads - 1) / kThreads, kLoadsB = (BN * TK / 4 + kThreads - 1) / kThreads;
  static constexpr int kStage = TK * (kLda + kLdb), kSmem = 2 * kStage * 4;
};

template <int BM, int BN, int TM, int TN, int TK, int MINB>
__global__ void __launch_bounds__((Tile<BM, BN, TM, TN, TK>::kThreads), MINB)
linear_f32_kernel(const LinearF32 p) {
  using L = Tile<BM, BN, TM, TN, TK>;
  extern __shared__ float4 smem4[];
  float* const smem = reinterpret_cast<float*>(smem4);    // two stages of [k][rows of a], [k][rows of b]
  pdl_enter();
  int m0 = blockIdx.y * BM, M = p.M;
  const int n0 = blockIdx.x * BN, N = p.N, K = p.K;
  const float* b = p.b;
  if (p.seg) {
    m0 += max(p.seg[blockIdx.z], 0);
    M = min(M, p.seg[blockIdx.z + 1]);
    b += static_cast<long long>(blockIdx.z) * N * K;
    if (m0 >= M) return;
  }
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ty = (warp / L::kWarpCols) * 4 + (lane >> 3), tx = (warp % L::kWarpCols) * 8 + (lane & 7);

  float4 ra[L::kLoadsA], rb[L::kLoadsB];
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  auto fetch = [&](int k0) {
#pragma unroll
    for (int i = 0; i < L::kLoadsA; ++i) {
      const int f = tid + i * L::kThreads, r = f / (TK / 4), k = k0 + (f % (TK / 4)) * 4;
      ra[i] = r < BM && m0 + r < M && k < K ? *reinterpret_cast<const float4*>(p.a + (m0 + r) * p.lda + k) : zero;
    }
#pragma unroll
    for (int i = 0; i < L::kLoadsB; ++i) {
      const int f = tid + i * L::kThreads, r = f / (TK / 4), k = k0 + (f % (TK / 4)) * 4;
      rb[i] = r < BN && n0 + r < N && k < K ? *reinterpret_cast<const float4*>(b + static_cast<size_t>(n0 + r) * K + k) : zero;
    }
  };
  auto put = [&](int s) {
    float* const sa = smem + s * L::kStage;
    float* const sb = sa + TK * L::kLda;
#pragma unroll
    for (int i = 0; i < L::kLoadsA; ++i) {
      const int f = tid + i * L::kThreads, r = f / (TK / 4), k = (f % (TK / 4)) * 4;
      if (L::kLoadsA * L::kThreads * 4 == BM * TK || r < BM) {
        float* const at = sa + k * L::kLda + r;
        at[0] = ra[i].x; at[L::kLda] = ra[i].y; at[2 * L::kLda] = ra[i].z; at[3 * L::kLda] = ra[i].w;
      }
    }
#pragma unroll
    for (int i = 0; i < L::kLoadsB; ++i) {
      const int f = tid + i * L::kThreads, r = f / (TK / 4), k = (f % (TK / 4)) * 4;
      if (L::kLoadsB * L::kThreads * 4 == BN * TK || r < BN) {
        float* const at = sb + k * L::kLdb + r;
        at[0] = rb[i].x; at[L::kLdb] = rb[i].y; at[2 * L::kLdb] = rb[i].z; at[3 * L::kLdb] = rb[i].w;
      }
    }
  };
  // thread (ty, tx) owns rows c * 4 * kRowThreads + 4 ty .. + 3 and columns c * 4 * kColThreads + 4 tx .. + 3
  unsigned long long acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;
  fetch(0);
  put(0);
  __syncthreads();
  for (int k0 = 0, s = 0; k0 < K; k0 += TK, s ^= 1) {
    const bool more = k0 + TK < K;
    if (more) fetch(k0 + TK);
    const float* const sa = smem + s * L::kStage + ty * 4;
    const float* const sb = smem + s * L::kStage + TK * L::kLda + tx * 4;
#pragma unroll
    for (int k = 0; k < TK; ++k) {
      float av[TM];
      ulonglong2 bv[TN / 4];
#pragma unroll
      for (int c = 0; c < TM / 4; ++c)
        *reinterpret_cast<float4*>(av + 4 * c) = *reinterpret_cast<const float4*>(sa + k * L::kLda + c * 4 * L::kRowThreads);
#pragma unroll
      for (int c = 0; c < TN / 4; ++c) bv[c] = *reinterpret_cast<const ulonglong2*>(sb + k * L::kLdb + c * 4 * L::kColThreads);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const unsigned long long aa = pair(av[i], av[i]);
#pragma unroll
        for (int c = 0; c < TN / 4; ++c) {
          fma2(acc[i][2 * c], aa, bv[c].x);
          fma2(acc[i][2 * c + 1], aa, bv[c].y);
        }
      }
    }
    if (more) {
      put(s ^ 1);
      __syncthreads();
    }
  }
  // scale and column factor, or the scale alone, then the residual (-0 changes nothing)
  const float first = p.col_scale ? p.scale : 1.f;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + (i >> 2) * 4 * L::kRowThreads + ty * 4 + (i & 3);
    if (m >= M) continue;
#pragma unroll
    for (int c = 0; c < TN / 4; ++c) {
      const int n = n0 + c * 4 * L::kColThreads + tx * 4;
      float v[4];
      unpair(acc[i][2 * c], v[0], v[1]);
      unpair(acc[i][2 * c + 1], v[2], v[3]);
      if (p.act == 1) {
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = fmaxf(v[j], 0.f) * fmaxf(v[j], 0.f);
      }
      const size_t at = static_cast<size_t>(m) * N + n;
      if (p.vec && n + 4 <= N) {
        float4 f = make_float4(p.scale, p.scale, p.scale, p.scale), r = make_float4(-0.f, -0.f, -0.f, -0.f);
        if (p.col_scale) f = *reinterpret_cast<const float4*>(p.col_scale + n);
        if (p.residual) r = *reinterpret_cast<const float4*>(p.residual + at);
        *reinterpret_cast<float4*>(p.out + at) = make_float4(fmaf(v[0] * first, f.x, r.x), fmaf(v[1] * first, f.y, r.y),
                                                             fmaf(v[2] * first, f.z, r.z), fmaf(v[3] * first, f.w, r.w));
        continue;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (n + j >= N) break;
        p.out[at + j] = fmaf(v[j] * first, p.col_scale ? p.col_scale[n + j] : p.scale, p.residual ? p.residual[at + j] : -0.f);
      }
    }
  }
}

template <int BM, int BN, int TM, int TN, int TK, int MINB>
cudaError_t launch_tile(const LinearF32& p, int groups, cudaStream_t st) {
  using L = Tile<BM, BN, TM, TN, TK>;
  const cudaError_t e = allow_smem<linear_f32_kernel<BM, BN, TM, TN, TK, MINB>>(L::kSmem);
  if (e != cudaSuccess) return e;
  return launch_kernel(linear_f32_kernel<BM, BN, TM, TN, TK, MINB>,
                       dim3((p.N + BN - 1) / BN, (p.M + BM - 1) / BM, p.seg ? groups : 1), dim3(L::kThreads), L::kSmem, st, p);
}

// Which tile: the one whose busiest SM is done first. Measured on one B200 per 1024 of K: `chain` us for a tile that has
// an SM to itself (one wave: bound by the latency of its own stages), `each` us per tile of an SM that runs many (bound
// by shared-memory reads, 16 to 32 floats of fragments per 64 products, and the FMA pipe). us, this rule / 64 x 64 tiles of 4 x 4 outputs a
// thread with one stage, as all calls had before: 1018 rows, K x N 1024 x 4128 196 / 288, 1024 x 5632 253 / 359,
// 1536 x 1024 95 / 125, 2816 x 1024 171 / 227, 1024 x 32000 1303 / 1960 (51 TFLOP/s; the pipe's peak is about 73);
// 200 x 1024 x 1024 30 / 56; 37 x 1024 x 1024 26 / 54; 8 x 1024 x 32000 70 / 176.
struct Choice {
  float us;
  int form;
};
Choice cheaper(Choice best, int form, const LinearF32& p, int groups, int sms, int bm, int bn, float chain, float each) {
  const long long rows = (p.M + bm - 1) / bm;
  if (rows > 65535) return best;                              // beyond the grid's second axis
  // of row groups whose sizes only the device knows: every group ends in a partial tile
  const long long tiles = (p.seg && groups > 1 ? rows + groups - 1 : rows) * ((p.N + bn - 1) / bn);
  const float us = fmaxf(chain, each * static_cast<float>((tiles + sms - 1) / sms));
  return us < best.us ? Choice{us, form} : best;
}

}  // namespace

cudaError_t launch_linear_f32(const float* a, long long lda, const float* b, const float* residual,
                              const float* col_scale, float scale, int act, float* out, const int* seg, int groups,
                              int M, int K, int N, cudaStream_t st) {
  if (M == 0) return cudaSuccess;
  const auto at16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  const LinearF32 p{a, lda, b, residual, col_scale, scale, act, out, seg, M, K, N,
                    (N & 3) == 0 && at16(out) && at16(residual) && at16(col_scale)};
  const int sms = current_sm_count();
  Choice best{1e30f, 0};
  best = cheaper(best, 0, p, groups, sms, 128, 128, 102.f, 96.f);
  best = cheaper(best, 1, p, groups, sms, 128, 64, 59.f, 49.f);
  best = cheaper(best, 2, p, groups, sms, 64, 64, 41.f, 29.f);
  best = cheaper(best, 3, p, groups, sms, 32, 64, 27.f, 21.f);
  best = cheaper(best, 4, p, groups, sms, 32, 32, 23.f, 12.f);
  best = cheaper(best, 5, p, groups, sms, 16, 32, 26.f, 8.f);
  switch (best.form) {
    case 0: return launch_tile<128, 128, 8, 8, 16, 2>(p, groups, st);
    case 1: return launch_tile<128, 64, 8, 8, 16, 1>(p, groups, st);
    case 2: return launch_tile<64, 64, 8, 4, 16, 4>(p, groups, st);
    case 3: return launch_tile<32, 64, 4, 4, 32, 4>(p, groups, st);
    case 4: return launch_tile<32, 32, 4, 4, 32, 6>(p, groups, st);
    default: return launch_tile<16, 32, 4, 4, 32, 8>(p, groups, st);
  }
}

}  // namespace cdeep
