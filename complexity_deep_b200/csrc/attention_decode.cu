// Single-query (decode) attention over a KV cache, HBM-bound: every cached K and V row is
// read exactly once, straight from the cache's own layout, for all the query heads that
// share it (grouped-query attention without repeating the KV heads).
//
// Replaces, for q_len == 1, complexity_deep/core/attention.py:163-177 (repeat_interleave of
// K/V + scaled_dot_product_attention): out[b, h] = softmax(q[b, h] . K[b, h / G]^T * scale
// + mask[b]) V[b, h / G].
//
// Split-KV: grid (splits, kv heads, batch); a block owns one chunk of the cache for one
// (batch, kv head) and all G query heads of the group.  8 lanes share a cached row: for
// every 64 dimensions lane s owns dimensions 8 s .. 8 s + 7, so one 16-byte access per lane
// covers 128 contiguous bytes of the row (whole sectors, no re-fetch); a warp streams 4 rows
// per step; every lane group
// keeps an online-softmax state (running max, sum, weighted V) per query head, merged across
// the block through shared memory. The splits of a pair are one thread-block cluster and
// merge through one another's shared memory, each block a share of the columns; long caches of
// few pairs take several clusters a pair and a kernel that adds what they leave in a workspace.
//
// A decode step (kStep) hands over the raw projections: the first warp of every block normalises and
// rotates the query heads of its group (8 lanes a head), and the block
// whose rows include the new token does so for its key, writes key and value into the cache
// and takes the row behind all others, from shared memory.
//
// Bound by HBM for a full device (B 32, 8 kv heads, 2 064 rows of 128: 270 MB), by the launch and the chain of one
// block before that. A step used to be three launches (rotation and append, partial sums to memory, their sum), each
// with its own start, end and round trip through L2. us, cold L2, three launches / this one: 1 sequence x 4 kv heads x 302
// rows of 3 x 64 9.3 / 5.6, 1 x 8 x 2 064 of 2 x 128 11.9 / 10.4, 8 x 8 x 1 000 16.4 / 13.7, 32 x 8 x 2 064 52.0 / 49.9,
// 64 x 8 x 2 064 103 / 91.
#include <cfloat>
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include "decode_split.h"
#include "kernels.h"

namespace cdeep {

namespace {

constexpr int kAttnThreads = 128;
constexpr int kLanesPerRow = 8;
constexpr int kMaxClusters = 4; // of a pair

__device__ __forceinline__ float lo_f(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float hi_f(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

// Blocks that an SM holds at a time, by the registers of G query heads of D dimensions.
__host__ __device__ constexpr int blocks_per_sm(int G, int D) { return G * D > 384 ? 2 : G * D > 256 ? 3 : 4; }

// Clusters of 1 .. 16 blocks that a B200 holds at a time (cudaOccupancyMaxActiveClusters: a cluster lies within one GPC,
// so the SMs that are left over in each go unused), by blocks per SM. Other devices take other sizes better; which of more than
// eight blocks they take at all they are asked (allow_clusters).
constexpr short kActive[3][kMaxSplits] = {{296, 148, 93, 71, 56, 45, 37, 33, 30, 26, 21, 21, 17, 14, 14, 14},
                                          {444, 222, 142, 104, 82, 71, 56, 48, 45, 41, 31, 31, 28, 24, 24, 21},
                                          {592, 296, 187, 142, 112, 93, 78, 71, 60, 56, 45, 42, 38, 35, 31, 31}};
//   Two blocks of every pair fit the device at once: the largest cluster of which one per pair fits, and of more than eight
//   blocks 13 up to 24 pairs (beside other kernels' blocks a large cluster waits for room: steps of the 18-layer model with
//   8 sequences, 32 pairs, 669 us with 13, 617 with eight; 1B-class with 3, 24 pairs, 1 198 / 1 211) and 16 up to eight. us,
//   cold L2, heads of 2 x 128 and 2 064 rows, by the size of the cluster: 8 pairs 8: 14.1, 13: 12.3, 16: 12.1; 16 pairs 8: 16.2,
//   13: 13.9, 16: 14.2; 24 pairs 8: 16.2, 13: 15.0, 16: 16.2; 32 pairs 8: 16.3, 10: 16.3, 13: 16.6, 16: 22.5; another
//   kernel's blocks aside, 64 pairs 7: 18.9, 8: 18.2, 9: 26; 96 pairs 4: 27.3, 5: 23.2, 6: 32.6; 128 pairs 3: 33, 4: 28.3,
//   5: 38.6; 256 pairs 1: 66, 2: 47.7, 3: 60. Down to 48 rows a block: 4 pairs of 302 rows of 3 x 64 4: 8.6, 5: 8.2, 8: 8.0,
//   of 800 rows 8: 10.1, 12: 10.1, 13: 8.1; 8 pairs of 1 000 of 2 x 128 8: 10.9, 16: 10.0; 24 pairs of 800 8: 11.4, 13: 12.0.
//   More pairs: split_of_waves. us, cold L2, 2 x 128, one block / two / three / four a pair: 384 pairs of 300 rows 21 / 29 / 33 / 34,
//   of 2 064 86 / 109 / 105 / 96; 640 of 300 39 / 41 / 47 / 54, of 1 024 100 / 90 / 87 / 94, of 4 096 310 / 262 / 252 / 244; 768 of
//   300 41 / 45 / 55 / 64, of 2 064 188 / 161 / 171 / 171; 2 048 of 300 83 / 103 / 128 / 153, of 4 096 671 / 663 / 687 / 695.
//   Long caches of few pairs: as many clusters of eight as fit, up to four a pair, with a kernel behind them (some 2 us). A block
//   is one chain of row steps, 0.43 us per 16 rows with an SM to itself whatever it has in flight (8 and 16 steps staged for four:
//   no difference; two and four steps side by side 0.29 to 0.38, eight warps a block 0.26 and no gain beyond one block an SM).
//   us of a step, cold L2, one cluster / several (three launches with up to 32 blocks a pair, before that): 4 pairs of 3 x 64,
//   8 192 rows 22.5 / 18.3 (18.5), 32 768 65.7 / 41.1 (41.1); 8 pairs of 2 x 128, 4 096 14.5 / 16.1 (15.9), 8 192 21.1 / 19.5
//   (20.4), 32 768 63.7 / 42.2 (43.3); 8 of 4 x 128, 8 192 34.9 / 27.0 (27.7), 32 768 109 / 64 (67.5); 16 of 2 x 128, 8 192
//   26.5 / 25.8 (26.9), 32 768 80 / 66 (67); 16 of 3 x 64, 4 096 16.8 / 16.5 (18.5), 32 768 86 / 51 (53); 32 of 2 x 128,
//   16 384 68.2 / 66.2 (66.8), 32 768 125 / 113 (112).
inline DecodeSplit choose_split(int B, int hkv, int G, int D) {
  const int per_sm = blocks_per_sm(G, D);
  const long long pairs = static_cast<long long>(B) * hkv;
  const short(&active)[kMaxSplits] = kActive[per_sm - 2];
  if (pairs <= active[1]) {
    int fit = 2;
    while (fit < kMaxSplits && pairs <= active[fit]) ++fit;
    DecodeSplit r;
    r.most = pairs <= 8 && fit == kMaxSplits ? kMaxSplits : pairs <= 24 && fit >= 13 ? 13 : fit > kPortable ? kPortable : fit;
    r.large_from = r.most * (pairs > 16 ? 64 : 48);
    const long long clusters = active[kPortable - 1] / pairs;
    r.many = kPortable * static_cast<int>(clusters < kMaxClusters ? clusters : kMaxClusters);
    if (r.many > r.most) r.many_from = r.most == kMaxSplits ? 2048 + 32 * D : (r.most > kPortable ? 64 : 128) * D;
    return r;
  }
  return split_of_waves(pairs, active);
}

// programmatic dependent launch: wait for the previous kernel of the stream before touching
// memory, then let the next kernel be scheduled (its launch hides under this one)
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// *p of this block, read from the block of rank `rank` of the cluster
__device__ __forceinline__ float peer_load(const float* p, int rank) {
  uint32_t a;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}

// Sums of some rows for one column: the largest score, the weights relative to it, the weighted values.
struct Sums {
  float m = -FLT_MAX, l = 0.f, a = 0.f;
};
template <int N>
__device__ __forceinline__ Sums add_sums(const Sums (&in)[N]) {
  Sums r;
#pragma unroll
  for (int s = 0; s < N; ++s) r.m = fmaxf(r.m, in[s].m);
#pragma unroll
  for (int s = 0; s < N; ++s) {
    const float w = in[s].m > -FLT_MAX ? __expf(in[s].m - r.m) : 0.f;
    r.l += in[s].l * w;
    r.a += in[s].a * w;
  }
  return r;
}
// no visible row: 0; a NaN score stays one
__device__ __forceinline__ __nv_bfloat16 quotient(const Sums& s) { return __float2bfloat16_rn(s.l == 0.f ? 0.f : s.a / s.l); }

// What a decode step brings besides the query: norm weights (or none), rotation tables, where the new row goes.
struct StepArgs {
  const __nv_bfloat16 *q_w, *k_w;
  const float *cos_t, *sin_t;
  float eps;
  __nv_bfloat16 *k_cache, *v_cache;
  const int* pos_dev;
  int capacity;
};

// One head by 8 lanes: RMSNorm and rotation as qk_norm_rope_vec_kernel computes them, rounded to bf16. Lane `sub` holds
// columns j .. j + 7 and D / 2 + j ..; of 64 columns two lanes hold the same ones, and each returns the half that it
// owns in the row layout (dims 8 sub of every 64).
template <int D>
__device__ __forceinline__ int rope_col(int sub) { return (sub & (D / 16 - 1)) * 8; }
struct Halves {
  uint4 a, b;
};
template <int D>
__device__ __forceinline__ Halves load_halves(const __nv_bfloat16* p, int sub) {
  const __nv_bfloat16* x = p + rope_col<D>(sub);
  return {*reinterpret_cast<const uint4*>(x), *reinterpret_cast<const uint4*>(x + D / 2)};
}
struct Angles {                  // cosines and sines of the two halves
  float c1[8], s1[8], c2[8], s2[8];
};
template <int D>
__device__ __forceinline__ void load_angles(Angles& t, const float* cs, const float* sn, int sub) {
  const int j = rope_col<D>(sub);
#pragma unroll
  for (int v = 0; v < 2; ++v) {
    *reinterpret_cast<float4*>(t.c1 + 4 * v) = *reinterpret_cast<const float4*>(cs + j + 4 * v);
    *reinterpret_cast<float4*>(t.s1 + 4 * v) = *reinterpret_cast<const float4*>(sn + j + 4 * v);
    *reinterpret_cast<float4*>(t.c2 + 4 * v) = *reinterpret_cast<const float4*>(cs + D / 2 + j + 4 * v);
    *reinterpret_cast<float4*>(t.s2 + 4 * v) = *reinterpret_cast<const float4*>(sn + D / 2 + j + 4 * v);
  }
}
template <int D>
__device__ __forceinline__ void norm_rope(const Halves& x, const Halves& w, bool normed, const Angles& t, float eps, bool rotate,
                                          int sub, uint4 (&out)[D / 64]) {
  constexpr int kLanes = D / 16;
  const uint32_t aw[4] = {x.a.x, x.a.y, x.a.z, x.a.w}, bw[4] = {x.b.x, x.b.y, x.b.z, x.b.w};
  float x1[8], x2[8], ss = 0.f;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    x1[2 * e] = lo_f(aw[e]); x1[2 * e + 1] = hi_f(aw[e]);
    x2[2 * e] = lo_f(bw[e]); x2[2 * e + 1] = hi_f(bw[e]);
    ss += x1[2 * e] * x1[2 * e] + x1[2 * e + 1] * x1[2 * e + 1] + x2[2 * e] * x2[2 * e] + x2[2 * e + 1] * x2[2 * e + 1];
  }
#pragma unroll
  for (int o = kLanes >> 1; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  uint4 lo = x.a, hi = x.b;
  if (rotate) {
    if (normed) {
      const float rstd = rsqrtf(ss / static_cast<float>(D) + eps);
      const uint32_t w1[4] = {w.a.x, w.a.y, w.a.z, w.a.w}, w2[4] = {w.b.x, w.b.y, w.b.z, w.b.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        x1[2 * e] *= rstd * lo_f(w1[e]); x1[2 * e + 1] *= rstd * hi_f(w1[e]);
        x2[2 * e] *= rstd * lo_f(w2[e]); x2[2 * e + 1] *= rstd * hi_f(w2[e]);
      }
    }
    uint32_t o1[4], o2[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = 2 * e, k = 2 * e + 1;
      const __nv_bfloat162 p1 = __floats2bfloat162_rn(x1[i] * t.c1[i] - x2[i] * t.s1[i], x1[k] * t.c1[k] - x2[k] * t.s1[k]);
      const __nv_bfloat162 p2 = __floats2bfloat162_rn(x2[i] * t.c2[i] + x1[i] * t.s2[i], x2[k] * t.c2[k] + x1[k] * t.s2[k]);
      o1[e] = *reinterpret_cast<const uint32_t*>(&p1);
      o2[e] = *reinterpret_cast<const uint32_t*>(&p2);
    }
    lo = make_uint4(o1[0], o1[1], o1[2], o1[3]);
    hi = make_uint4(o2[0], o2[1], o2[2], o2[3]);
  }
  if constexpr (D == 64) {
    out[0] = sub < kLanes ? lo : hi;
  } else {
    out[0] = lo;
    out[1] = hi;
  }
}

constexpr int kStages = 4;   // row steps staged in shared memory per thread (3 in flight)

// DPL = dimensions per lane = D / 8 (8 or 16 -> D = 64 or 128), G = query heads per KV head.
// len_dev (optional): the number of cached rows is min(L, *len_dev) and the split of the rows
// over blocks is recomputed from it; the grid stays that of L, and blocks beyond the split only
// take part in the cluster's barriers.
//
// A row step = 16 cached rows of the block (4 warps x 4 lane groups), 2 * DPL bytes of K and
// of V per lane.  Every lane copies its own slices of the next kStages - 1 steps into a
// private slot of shared memory with cp.async (bytes in flight without holding registers:
// 4 blocks per SM keep ~100 KB on the way) and reads them back with 16-byte loads, so no
// block-level synchronisation is needed inside the loop.
//
// The kernel ahead may still run when this one starts, and it writes the query: nothing is read on the read-only path, whose
// loads the compiler may move to before the wait.
//
// The blocks of a pair are clusters of `cl`. Several of them (part != NULL) leave their sums there for combine_kernel, which
// adds them as one cluster adds its blocks: eight at a time, so the bits are the same.
template <int DPL, int G, bool kStep>
__global__ void __launch_bounds__(kAttnThreads, blocks_per_sm(G, DPL * kLanesPerRow))
decode_attn_kernel(const __nv_bfloat16* q, long long q_stride_b,
                   const __nv_bfloat16* k, const __nv_bfloat16* v,
                   long long kv_stride_b, long long kv_stride_h, long long kv_stride_t,
                   const __nv_bfloat16* mask, long long mask_stride_b,
                   float scale, int L, DecodeSplit rule, __nv_bfloat16* out,
                   const int* len_dev, StepArgs st, int cl, float* part) {
  constexpr int D = DPL * kLanesPerRow;
  constexpr int kV = DPL / 8;                               // 16-byte pieces of K (and of V) per lane
  constexpr int kStepBytes = kAttnThreads * 2 * kV * 16;    // one row step of the block
  constexpr int kMergeBytes = 16 * G * D * 4;               // the block-level merge re-uses the slots
  constexpr int kSmemBytes = kStages * kStepBytes > kMergeBytes ? kStages * kStepBytes : kMergeBytes;
  __shared__ __align__(16) unsigned char s_raw[kSmemBytes];
  __shared__ float s_m[16][G], s_l[16][G];
  __shared__ float s_part[G * D + 2 * G];                   // this block's sums, then its maxima and sums of weights
  __shared__ uint4 s_new[2 * kV][kStep ? kLanesPerRow : 1];
  __shared__ uint4 s_q[G][kStep ? D / 8 : 1];               // the rotated query heads

  griddep_wait();
  griddep_launch_dependents();
  const int split = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z, hkv = gridDim.y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane & 7;          // which D/8 slice of the row
  const int rgrp = lane >> 3;        // which of the warp's 4 concurrent rows
  // all that a step needs besides the cache is asked for before the first rows, whose copies end the reach of a load
  const __nv_bfloat16* row = q + b * q_stride_b;
  Halves qx, qw = {};
  Angles ang;
  int pos = -1;                      // the row that this step brings
  if constexpr (kStep) {
    pos = *st.pos_dev;
    if (warp == 0) {                 // a head per lane group
      qx = load_halves<D>(row + static_cast<long long>(kvh * G + min(rgrp, G - 1)) * D, sub);
      if (st.q_w) qw = load_halves<D>(st.q_w, sub);
    }
  }
  if (len_dev) L = max(0, min(L, *len_dev));
  const int splits = rule.bound(L);                          // the last of them may have no rows
  const int chunk = rule.chunk(L);
  const int t_begin = min(L, split * chunk);
  const int t_end = min(L, t_begin + chunk);
  bool owner = false;                // of the new row: the warp whose rows include it, or beyond all rows the first
  if constexpr (kStep) {
    if (pos < 0 || pos >= st.capacity) pos = -1;
    owner = pos >= 0 && (pos < L ? pos >= t_begin && pos < t_end && warp == (((pos - t_begin) >> 2) & 3) : split + warp == 0);
    if (warp == 0 || owner)
      load_angles<D>(ang, st.cos_t + static_cast<long long>(max(pos, 0)) * D, st.sin_t + static_cast<long long>(max(pos, 0)) * D, sub);
  }

  float m_run[G], l_run[G], acc[G][DPL];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    m_run[g] = -FLT_MAX;
    l_run[g] = 0.f;
#pragma unroll
    for (int i = 0; i < DPL; ++i) acc[g][i] = 0.f;
  }
  const __nv_bfloat16* kb = k + b * kv_stride_b + kvh * kv_stride_h + sub * 8;
  const __nv_bfloat16* vb = v + b * kv_stride_b + kvh * kv_stride_h + sub * 8;
  const __nv_bfloat16* mb = !kStep && mask ? mask + b * mask_stride_b : nullptr;

  // slot of (stage, piece) for this thread: consecutive threads are 16 bytes apart, so both
  // the asynchronous writes and the reads are free of bank conflicts
  auto slot = [&](int stage, int piece) -> uint4* {
    return reinterpret_cast<uint4*>(s_raw + stage * kStepBytes) + piece * kAttnThreads + threadIdx.x;
  };
  const int t_lane = t_begin + warp * 4 + rgrp;             // this lane's row of step 0
  const int n_steps = (t_end - t_begin + 15) >> 4;          // same for the whole block
  auto issue = [&](int step) {
    const int t = t_lane + step * 16;
    if (step < n_steps && t < t_end && (!kStep || t != pos)) {
      const int stage = step % kStages;
#pragma unroll
      for (int i = 0; i < kV; ++i) {
        cp_async16(slot(stage, i), kb + t * kv_stride_t + i * 64);
        cp_async16(slot(stage, kV + i), vb + t * kv_stride_t + i * 64);
      }
    }
    cp_async_commit();                                      // one group per step, even if empty
  };
#pragma unroll
  for (int s0 = 0; s0 < kStages - 1; ++s0) issue(s0);

  if constexpr (kStep) {
    if (warp == 0) {
      uint4 w[kV];
      norm_rope<D>(qx, qw, st.q_w != nullptr, ang, st.eps, pos >= 0, sub, w);
      if (rgrp < G) {
#pragma unroll
        for (int i = 0; i < kV; ++i) s_q[rgrp][i * 8 + sub] = w[i];
      }
    }
    if (owner) {                       // the new row into the cache; its own step comes behind all others'
      uint4 w[kV];
      Halves kw = {};
      if (st.k_w) kw = load_halves<D>(st.k_w, sub);
      norm_rope<D>(load_halves<D>(row + static_cast<long long>(hkv * G + kvh) * D, sub), kw, st.k_w != nullptr, ang, st.eps, true,
                   sub, w);
      const __nv_bfloat16* vp = row + static_cast<long long>(hkv * (G + 1) + kvh) * D + sub * 8;
      if (rgrp == 0) {
#pragma unroll
        for (int i = 0; i < kV; ++i) {
          const uint4 x = *reinterpret_cast<const uint4*>(vp + i * 64);
          const long long at = b * kv_stride_b + kvh * kv_stride_h + pos * kv_stride_t + i * 64 + sub * 8;
          s_new[i][sub] = w[i];
          s_new[kV + i][sub] = x;
          *reinterpret_cast<uint4*>(st.k_cache + at) = w[i];
          *reinterpret_cast<uint4*>(st.v_cache + at) = x;
        }
      }
    }
    __syncthreads();
  }

  // query fragments of the G heads, pre-scaled
  float qf[G][DPL];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    uint4 w[kV];
#pragma unroll
    for (int i = 0; i < kV; ++i)
      w[i] = kStep ? s_q[g][i * 8 + sub] : *reinterpret_cast<const uint4*>(row + static_cast<long long>(kvh * G + g) * D + i * 64 + sub * 8);
#pragma unroll
    for (int i = 0; i < kV; ++i) {
      const uint32_t ww[4] = {w[i].x, w[i].y, w[i].z, w[i].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        qf[g][i * 8 + 2 * e] = lo_f(ww[e]) * scale;
        qf[g][i * 8 + 2 * e + 1] = hi_f(ww[e]) * scale;
      }
    }
  }

  // Additive mask: once per 8 steps lane l fetches the value of row group (l & 3) of step
  // (window + l / 4) of this warp, one window ahead of its use; a step then takes its value
  // from the owning lane with a shuffle, so no step waits for a global load.
  auto mask_window = [&](int step0) -> float {
    const int t = t_begin + 16 * (step0 + (lane >> 2)) + warp * 4 + (lane & 3);
    return (mb && t < t_end) ? __bfloat162float(mb[t]) : 0.f;
  };
  float mwin = mask_window(0), mwin_next = mask_window(8);

  // one row per lane group: its scores, and its share of the weighted sums
  auto take = [&](const uint4 (&kr)[kV], const uint4 (&vr)[kV], bool valid, float madd) {
    float kf[DPL], vf[DPL];
#pragma unroll
    for (int i = 0; i < kV; ++i) {
      const uint32_t kw[4] = {kr[i].x, kr[i].y, kr[i].z, kr[i].w};
      const uint32_t vw[4] = {vr[i].x, vr[i].y, vr[i].z, vr[i].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        kf[i * 8 + 2 * e] = lo_f(kw[e]); kf[i * 8 + 2 * e + 1] = hi_f(kw[e]);
        vf[i * 8 + 2 * e] = lo_f(vw[e]); vf[i * 8 + 2 * e + 1] = hi_f(vw[e]);
      }
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < DPL; ++i) s += qf[g][i] * kf[i];
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      s += __shfl_xor_sync(0xffffffffu, s, 4);
      if (valid) {
        s += madd;
        if (s > m_run[g]) {            // new running maximum: rescale (rare after the first rows)
          const float corr = __expf(m_run[g] - s);
          l_run[g] *= corr;
#pragma unroll
          for (int i = 0; i < DPL; ++i) acc[g][i] *= corr;
          m_run[g] = s;
        }
        // s = -inf (masked) gives pr = 0 and leaves the state untouched
        const float pr = __expf(s - m_run[g]);
        l_run[g] += pr;
#pragma unroll
        for (int i = 0; i < DPL; ++i) acc[g][i] += pr * vf[i];
      }
    }
  };
  for (int step = 0; step < n_steps; ++step) {
    issue(step + kStages - 1);
    float madd = 0.f;
    if (mb) {                                               // uniform
      const int j = step & 7;
      if (j == 0 && step > 0) {
        mwin = mwin_next;
        mwin_next = mask_window(step + 8);
      }
      madd = __shfl_sync(0xffffffffu, mwin, (j << 2) | rgrp);
    }
    cp_async_wait<kStages - 1>();                           // this step's group has landed
    const int t = t_lane + step * 16, stage = step % kStages;
    const bool valid = t < t_end && (!kStep || t != pos);
    uint4 kr[kV], vr[kV];
#pragma unroll
    for (int i = 0; i < kV; ++i) {
      kr[i] = vr[i] = make_uint4(0, 0, 0, 0);
      if (valid) {
        kr[i] = *slot(stage, i);
        vr[i] = *slot(stage, kV + i);
      }
    }
    take(kr, vr, valid, madd);
  }
  if constexpr (kStep) {
    if (owner && pos < L) {
      uint4 kr[kV], vr[kV];
      __syncwarp();
#pragma unroll
      for (int i = 0; i < kV; ++i) {
        kr[i] = s_new[i][sub];
        vr[i] = s_new[kV + i][sub];
      }
      take(kr, vr, rgrp == ((pos - t_begin) & 3), 0.f);   // as the last row its sums are those of a cache that already holds it
    }
  }
  cp_async_wait<0>();
  __syncthreads();                     // every lane is done with its slots: re-use them

  // merge the 16 row streams of the block (4 warps x 4 lane groups) in shared memory
  float (*s_acc)[G][D] = reinterpret_cast<float (*)[G][D]>(s_raw);
  const int stream = warp * 4 + rgrp;
#pragma unroll
  for (int g = 0; g < G; ++g) {
    if (sub == 0) {
      s_m[stream][g] = m_run[g];
      s_l[stream][g] = l_run[g];
    }
#pragma unroll
    for (int i = 0; i < DPL; ++i) s_acc[stream][g][(i >> 3) * 64 + sub * 8 + (i & 7)] = acc[g][i];
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < G * D; idx += kAttnThreads) {
    const int g = idx / D, d = idx - g * D;
    float m = -FLT_MAX;
#pragma unroll
    for (int s = 0; s < 16; ++s) m = fmaxf(m, s_m[s][g]);
    float l = 0.f, a = 0.f;
#pragma unroll
    for (int s = 0; s < 16; ++s) {
      const float w = (s_m[s][g] > -FLT_MAX) ? __expf(s_m[s][g] - m) : 0.f;
      l += s_l[s][g] * w;
      a += s_acc[s][g][d] * w;
    }
    s_part[idx] = a;
    if (d == 0) {
      s_part[G * D + g] = m;
      s_part[G * D + G + g] = l;
    }
  }

  // the splits of the pair, every block a share of the columns
  if (cl > 1) {
    __syncwarp();
    cluster_arrive();
    cluster_wait();
  } else {
    __syncthreads();
  }
  const int group = part ? split / kPortable : 0, rank = split - group * kPortable;
  const int live = min(cl, splits - group * kPortable);      // blocks of this cluster that may have rows
  // up to eight blocks: a thread a column; more: two, the first eight and the rest by themselves as several clusters do it
  const int two = live > kPortable ? 1 : 0, from = two & threadIdx.x ? kPortable : 0, per = kAttnThreads >> two;
  for (int idx = rank * per + (threadIdx.x >> two); idx < G * D; idx += cl * per) {
    const int g = idx / D;
    Sums in[kPortable];
#pragma unroll
    for (int x = 0; x < kPortable; ++x) {
      const int s = from + x;
      if (s < live) in[x] = {peer_load(&s_part[G * D + g], s), peer_load(&s_part[G * D + G + g], s), peer_load(&s_part[idx], s)};
    }
    Sums total = add_sums(in);
    if (two) {
      const Sums both[2] = {total, {__shfl_down_sync(0xffffffffu, total.m, 1), __shfl_down_sync(0xffffffffu, total.l, 1),
                                    __shfl_down_sync(0xffffffffu, total.a, 1)}};
      total = add_sums(both);
    }
    if (from > 0) continue;
    const long long pair = static_cast<long long>(b) * hkv + kvh;
    if (part) {
      float* dst = part + (pair * (gridDim.x / kPortable) + group) * (G * D + 2 * G);
      dst[idx] = total.a;
      if (idx == g * D) {
        dst[G * D + g] = total.m;
        dst[G * D + G + g] = total.l;
      }
    } else {
      out[pair * G * D + idx] = quotient(total);
    }
  }
  if (cl > 1) {                        // nobody leaves while its sums are being read
    __syncwarp();
    cluster_arrive();
    cluster_wait();
  }
}

// What the clusters of a pair left behind: grid (pairs), a column per thread.
__global__ void __launch_bounds__(kAttnThreads)
combine_kernel(const float* part, int groups, int G, int D, __nv_bfloat16* out) {
  griddep_wait();
  griddep_launch_dependents();
  const float* src = part + static_cast<long long>(blockIdx.x) * groups * (G * D + 2 * G);
  for (int idx = threadIdx.x; idx < G * D; idx += kAttnThreads) {
    const int g = idx / D;
    Sums in[kMaxClusters];
#pragma unroll
    for (int x = 0; x < kMaxClusters; ++x) {
      const float* from = src + x * (G * D + 2 * G);
      if (x < groups) in[x] = {from[G * D + g], from[G * D + G + g], from[idx]};
    }
    out[static_cast<long long>(blockIdx.x) * G * D + idx] = quotient(add_sums(in));
  }
}

// Clusters of more than eight blocks are asked for only where the device holds one.
template <auto kKernel>
cudaError_t allow_clusters(DecodeSplit& rule) {
  static DeviceNumber largest;
  int device = 0;
  const cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  const int most = largest.get(device, [] {
    return largest_cluster([](int blocks) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(blocks);
      cfg.blockDim = dim3(kAttnThreads);
      cudaLaunchAttribute attr;
      attr.id = cudaLaunchAttributeClusterDimension;
      attr.val.clusterDim.x = blocks;
      attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
      cfg.attrs = &attr;
      cfg.numAttrs = 1;
      int clusters = 0;
      if (cudaFuncSetAttribute(kKernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
          cudaOccupancyMaxActiveClusters(&clusters, kKernel, &cfg) != cudaSuccess)
        cudaGetLastError();              // not a size for this device
      return clusters > 0;
    });
  });
  if (rule.most > most) rule.most = most;
  return cudaSuccess;
}

template <int DPL, int G, bool kStep>
cudaError_t launch_one(int B, int hkv, cudaStream_t stream, const __nv_bfloat16* q, long long qsb, const __nv_bfloat16* k,
                       const __nv_bfloat16* v, long long sb, long long sh, long long stt, const __nv_bfloat16* mask,
                       long long msb, float scale, int L, DecodeSplit rule, __nv_bfloat16* out, const int* len_dev,
                       const StepArgs& step, float* ws) {
  constexpr auto kKernel = decode_attn_kernel<DPL, G, kStep>;
  if (rule.most > kPortable) {
    const cudaError_t e = allow_clusters<kKernel>(rule);
    if (e != cudaSuccess) return e;
  }
  const bool many = L >= rule.many_from;
  const int cl = many ? kPortable : len_dev ? rule.bound(L) : rule.blocks(L);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(many ? rule.many : cl, hkv, B);
  cfg.blockDim = dim3(kAttnThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cl;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cl > 1 ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kKernel, q, qsb, k, v, sb, sh, stt, mask, msb, scale, L, rule, out, len_dev, step, cl,
                                           many ? ws : static_cast<float*>(nullptr));
  if (e != cudaSuccess || !many) return e;
  return launch_kernel(combine_kernel, dim3(B * hkv), dim3(kAttnThreads), 0, stream, static_cast<const float*>(ws), rule.many / kPortable, G,
                       DPL * kLanesPerRow, out);
}

template <bool kStep>
cudaError_t launch_any(const void* q, long long qsb, const void* k, const void* v, long long sb, long long sh, long long stt,
                       const void* mask, long long msb, float scale, int B, int hq, int hkv, int L, int D, void* out,
                       cudaStream_t stream, const int* len_dev, const StepArgs& step, void* ws) {
  const int G = hq / hkv;
  DecodeSplit rule = choose_split(B, hkv, G, D);
  if (!ws) rule.many_from = 1 << 30;
  auto b16 = [](const void* p) { return static_cast<const __nv_bfloat16*>(p); };
#define CDEEP_ATTN_CASE(DPL, GG)                                                                                           \
  if (D == 8 * DPL && G == GG)                                                                                             \
    return launch_one<DPL, GG, kStep>(B, hkv, stream, b16(q), qsb, b16(k), b16(v), sb, sh, stt, b16(mask), msb, scale, L,  \
                                      rule, static_cast<__nv_bfloat16*>(out), len_dev, step, static_cast<float*>(ws));
  CDEEP_ATTN_CASE(8, 1) CDEEP_ATTN_CASE(8, 2) CDEEP_ATTN_CASE(8, 3) CDEEP_ATTN_CASE(8, 4)
  CDEEP_ATTN_CASE(16, 1) CDEEP_ATTN_CASE(16, 2) CDEEP_ATTN_CASE(16, 3) CDEEP_ATTN_CASE(16, 4)
#undef CDEEP_ATTN_CASE
  return cudaErrorInvalidValue;
}

}  // namespace

size_t decode_attention_workspace_bytes(int B, int hq, int hkv, int L, int D) {
  const int G = hq / hkv;
  const DecodeSplit rule = choose_split(B, hkv, G, D);
  return L < rule.many_from ? 0 : sizeof(float) * B * hkv * (rule.many / kPortable) * (G * D + 2 * G);
}

cudaError_t launch_decode_attention(const void* q, long long q_stride_b, const void* k, const void* v, long long kv_stride_b,
                                    long long kv_stride_h, long long kv_stride_t, const void* mask, long long mask_stride_b,
                                    float scale, int B, int hq, int hkv, int L, int D, void* out, void* ws, cudaStream_t stream,
                                    const int* kv_len_dev) {
  return launch_any<false>(q, q_stride_b, k, v, kv_stride_b, kv_stride_h, kv_stride_t, mask, mask_stride_b, scale, B, hq, hkv,
                           L, D, out, stream, kv_len_dev, StepArgs{}, ws);
}

cudaError_t launch_decode_step_attention(const void* qkv, const void* q_w, const void* k_w, const float* cos_t, const float* sin_t,
                                         float eps, void* k_cache, void* v_cache, long long kv_stride_b, long long kv_stride_h,
                                         long long kv_stride_t, int capacity, const int* pos_dev, const int* kv_len_dev,
                                         float scale, int B, int hq, int hkv, int D, void* out, void* ws, cudaStream_t stream) {
  StepArgs st;
  st.q_w = static_cast<const __nv_bfloat16*>(q_w);
  st.k_w = static_cast<const __nv_bfloat16*>(k_w);
  st.cos_t = cos_t;
  st.sin_t = sin_t;
  st.eps = eps;
  st.k_cache = static_cast<__nv_bfloat16*>(k_cache);
  st.v_cache = static_cast<__nv_bfloat16*>(v_cache);
  st.pos_dev = pos_dev;
  st.capacity = capacity;
  return launch_any<true>(qkv, static_cast<long long>(hq + 2 * hkv) * D, k_cache, v_cache, kv_stride_b, kv_stride_h, kv_stride_t,
                          nullptr, 0, scale, B, hq, hkv, capacity, D, out, stream, kv_len_dev, st, ws);
}

}  // namespace cdeep
