// Sliding-window attention with kept first tokens, distance bias and head mixing: the per-head
// norm, the ring append, and the kernels that handle one query, or four behind one another, per
// thread-block cluster.  These serve prompts in 32-bit storage and head layouts that the kernels of
// window_attention_prefill.cu (prompts in bf16) and window_attention_decode.cu do not take.
#include <cfloat>
#include <type_traits>
#include <cooperative_groups.h>
#include "kernels.h"
#include "window_attention.cuh"

namespace cg = cooperative_groups;

namespace cdeep {

namespace {

constexpr int kThreads = 256;
constexpr int kRep = 4;          // query heads of a group handled together

// q and k heads of every row in place: x / rms(x) * w, mean over `dim` columns.  LPH lanes per head,
// eight columns per lane and round.
template <typename T, int LPH>
__global__ void __launch_bounds__(256)
head_norm_kernel(const WindowAttnParams p) {
  pdl_enter();
  const int heads = p.H + p.G;
  const long long item = (blockIdx.x * 256ll + threadIdx.x) / LPH;
  const bool ok = item < static_cast<long long>(p.B) * p.S * heads;
  const int sub = threadIdx.x % LPH;
  const long long row = ok ? item / heads : 0;
  const int h = ok ? static_cast<int>(item - row * heads) : 0;
  const bool is_q = h < p.H;
  T* x = static_cast<T*>(is_q ? p.q : p.k) + row * p.ldp + static_cast<long long>(is_q ? h : h - p.H) * p.dp;
  const T* w = static_cast<const T*>(is_q ? p.q_w : p.k_w);
  float ss = 0.f;
  for (int c = sub * 8; c < p.dp; c += LPH * 8) {
    float f[8];
    load8(x + c, f);
#pragma unroll
    for (int e = 0; e < 8; ++e) ss += f[e] * f[e];
  }
#pragma unroll
  for (int d = 1; d < LPH; d <<= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
  const float r = 1.0f / sqrtf(ss / static_cast<float>(p.dim) + p.eps);
  if (!ok) return;
  for (int c = sub * 8; c < p.dp; c += LPH * 8) {
    float f[8], wv[8];
    load8(x + c, f);
    load8(w + c, wv);
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] *= r * wv[e];
    store8(x + c, f);
  }
}

template <typename T>
cudaError_t head_norm_any(const WindowAttnParams& p, cudaStream_t st) {
  const long long items = static_cast<long long>(p.B) * p.S * (p.H + p.G);
  auto grid = [&](int lph) { return dim3(static_cast<unsigned>((items * lph + 255) / 256)); };
  if (p.dp <= 64) return launch_kernel(head_norm_kernel<T, 8>, grid(8), dim3(256), 0, st, p);
  if (p.dp <= 128) return launch_kernel(head_norm_kernel<T, 16>, grid(16), dim3(256), 0, st, p);
  return launch_kernel(head_norm_kernel<T, 32>, grid(32), dim3(256), 0, st, p);
}

// Rows of the call that later queries may see go into the ring: the kept first positions and the
// last `window` ones.  One block per (row, sequence).
template <typename T>
__global__ void __launch_bounds__(128)
window_append_kernel(const WindowAttnParams p) {
  pdl_enter();
  const int t = blockIdx.x, b = blockIdx.y;
  const int pos0 = window_pos0(p);
  const int j = pos0 + t;
  if (j >= p.keep && j + p.window < pos0 + p.S) return;   // overwritten by a later row of this call
  const long long slot = static_cast<long long>(b) * (p.keep + p.window) + window_slot(j, p.window, p.keep);
  const long long row = static_cast<long long>(b) * p.S + t;
  const int nk = p.G * p.dp, nv = p.G * p.vp;
  const T* k = static_cast<const T*>(p.k) + row * p.ldp;
  const T* v = static_cast<const T*>(p.v) + row * p.ldp;
  T* rk = static_cast<T*>(p.ring_k) + slot * nk;
  T* rv = static_cast<T*>(p.ring_v) + slot * nv;
  for (int c = threadIdx.x * 8; c < nk + nv; c += blockDim.x * 8) {
    float f[8];
    if (c < nk) {
      load8(k + c, f);
      store8(rk + c, f);
    } else {
      load8(v + c - nk, f);
      store8(rv + c - nk, f);
    }
  }
}

struct RowsSmem {   // offsets in floats
  int q, s, m, stat, o, red, total;
};
__host__ __device__ inline RowsSmem rows_smem(int H, int dp, int vp, int cap) {
  RowsSmem L;
  L.q = 0;                                  // [H][dp]
  L.s = L.q + H * dp;                       // [H][cap] scores, then weights
  L.m = L.s + H * cap;                      // [H][cap] mixed weights
  L.stat = L.m + H * cap;                   // [2][H] this block's maximum and sum
  L.o = L.stat + ((2 * H + 3) & ~3);        // [H][vp] this block's part of the output
  L.red = L.o + H * vp;                     // [kThreads][kRep * 8]
  L.total = L.red + kThreads * kRep * 8;
  return L;
}

// One query per cluster of `gridDim.x / S` blocks; the blocks share the query's keys and exchange
// their softmax statistics and parts of the output through distributed shared memory.
template <typename T>
__global__ void __launch_bounds__(kThreads)
window_rows_kernel(const WindowAttnParams p, int cap) {
  extern __shared__ float4 smem4[];
  float* sm = reinterpret_cast<float*>(smem4);
  pdl_enter();
  cg::cluster_group cluster = cg::this_cluster();
  const int CL = static_cast<int>(cluster.num_blocks());
  const int rank = static_cast<int>(cluster.block_rank());
  const int t = blockIdx.x / CL, b = blockIdx.y;
  const int H = p.H, G = p.G, rep = H / G, dp = p.dp, vp = p.vp;
  const RowsSmem L = rows_smem(H, dp, vp, cap);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int pos0 = window_pos0(p);
  const int i = pos0 + t;
  const long long row = static_cast<long long>(b) * p.S + t;
  const WindowKeys keys(i, p.window, p.keep);
  const int count = keys.kept + (i - keys.first + 1);
  const int chunk = (count + CL - 1) / CL;
  const int n0 = min(rank * chunk, count);
  const int nk = min(chunk, count - n0);        // keys of this block (0 possible)

  // queries, pre-scaled
  const T* qrow = static_cast<const T*>(p.q) + row * p.ldp;
  for (int c = tid; c < H * dp; c += kThreads) sm[L.q + c] = to_f32(qrow[c]) * p.scale;
  __syncthreads();

  const long long slots = p.keep + p.window;
  const T* ring_k = static_cast<const T*>(p.ring_k) + b * slots * G * dp;
  const T* ring_v = static_cast<const T*>(p.ring_v) + b * slots * G * vp;
  const T* new_k = static_cast<const T*>(p.k) + static_cast<long long>(b) * p.S * p.ldp;
  const T* new_v = static_cast<const T*>(p.v) + static_cast<long long>(b) * p.S * p.ldp;

  // scores: a thread takes one (key, key head) pair and all query heads of the group
  for (int item = tid; item < nk * G; item += kThreads) {
    const int c = item / nk, n = item - c * nk;
    const int j = keys.position(n0 + n);
    const T* kp = j >= pos0 ? new_k + (j - pos0) * p.ldp + static_cast<long long>(c) * dp
                            : ring_k + (static_cast<long long>(window_slot(j, p.window, p.keep)) * G + c) * dp;
    const float dist = static_cast<float>(i - j);
    for (int r0 = 0; r0 < rep; r0 += kRep) {
      float acc[kRep] = {};
      for (int d = 0; d < dp; d += 8) {
        float f[8];
        load8(kp + d, f);
#pragma unroll
        for (int r = 0; r < kRep; ++r) {
          if (r0 + r < rep) {
            const float4* qv = reinterpret_cast<const float4*>(sm + L.q + (c * rep + r0 + r) * dp + d);
            const float4 a = qv[0], bq = qv[1];
            acc[r] += f[0] * a.x + f[1] * a.y + f[2] * a.z + f[3] * a.w + f[4] * bq.x + f[5] * bq.y + f[6] * bq.z +
                      f[7] * bq.w;
          }
        }
      }
#pragma unroll
      for (int r = 0; r < kRep; ++r) {
        if (r0 + r < rep) {
          const int h = c * rep + r0 + r;
          const float r1 = to_f32(static_cast<const T*>(p.r1)[h]), r2 = to_f32(static_cast<const T*>(p.r2)[h]);
          sm[L.s + h * cap + n] = acc[r] - r1 * log1pf(r2 * dist);
        }
      }
    }
  }
  __syncthreads();

  // softmax statistics of this block's keys, then of the whole cluster
  for (int h = warp; h < H; h += kThreads / 32) {
    float m = -FLT_MAX, l = 0.f;
    for (int n = lane; n < nk; n += 32) m = fmaxf(m, sm[L.s + h * cap + n]);
    m = warp_max(m);
    for (int n = lane; n < nk; n += 32) l += expf(sm[L.s + h * cap + n] - m);
    l = warp_add(l);
    if (lane == 0) {
      sm[L.stat + h] = m;
      sm[L.stat + H + h] = l;
    }
  }
  if (CL > 1) cluster.sync(); else __syncthreads();
  for (int h = warp; h < H; h += kThreads / 32) {
    float m = -FLT_MAX, l = 0.f;
    for (int r = 0; r < CL; ++r) {
      const float* st = cluster.map_shared_rank(sm + L.stat, r);
      const float mr = st[h], lr = st[H + h];
      if (lr > 0.f) {
        const float mn = fmaxf(m, mr);
        l = l * expf(m - mn) + lr * expf(mr - mn);
        m = mn;
      }
    }
    const float inv = 1.0f / l;
    for (int n = lane; n < nk; n += 32) sm[L.s + h * cap + n] = expf(sm[L.s + h * cap + n] - m) * inv;
  }
  __syncthreads();

  // mixed weights
  const T* talk = static_cast<const T*>(p.talk);
  for (int item = tid; item < nk * H; item += kThreads) {
    const int h = item / nk, n = item - h * nk;
    float a = 0.f;
    for (int g = 0; g < H; ++g) a += to_f32(talk[h * H + g]) * sm[L.s + g * cap + n];
    sm[L.m + h * cap + n] = a;
  }
  __syncthreads();

  // values: a thread takes eight columns of a key head and every `groups`-th key
  const int vchunks = G * vp / 8;
  const int groups = vchunks < kThreads ? kThreads / vchunks : 1;
  const int grp = tid / vchunks;
  for (int r0 = 0; r0 < rep; r0 += kRep) {
    for (int vc0 = 0; vc0 < vchunks; vc0 += kThreads) {
      const int vc = vc0 + (groups > 1 ? tid - grp * vchunks : tid);
      const bool active = vc < vchunks && (groups == 1 || grp < groups);
      const int c = active ? vc / (vp / 8) : 0, d = active ? (vc - c * (vp / 8)) * 8 : 0;
      float acc[kRep][8] = {};
      if (active) {
        for (int n = groups > 1 ? grp : 0; n < nk; n += groups) {
          const int j = keys.position(n0 + n);
          const T* v = j >= pos0 ? new_v + (j - pos0) * p.ldp + static_cast<long long>(c) * vp + d
                                 : ring_v + (static_cast<long long>(window_slot(j, p.window, p.keep)) * G + c) * vp + d;
          float f[8];
          load8(v, f);
#pragma unroll
          for (int r = 0; r < kRep; ++r) {
            if (r0 + r < rep) {
              const float w = sm[L.m + (c * rep + r0 + r) * cap + n];
#pragma unroll
              for (int e = 0; e < 8; ++e) acc[r][e] += w * f[e];
            }
          }
        }
        float* red = sm + L.red + tid;      // [value][thread]: conflict-free
#pragma unroll
        for (int r = 0; r < kRep; ++r)
#pragma unroll
          for (int e = 0; e < 8; ++e) red[(r * 8 + e) * kThreads] = acc[r][e];
      }
      __syncthreads();
      if (vc < vchunks && (groups == 1 || grp == 0)) {
#pragma unroll
        for (int r = 0; r < kRep; ++r) {
          if (r0 + r >= rep) break;
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            float a = 0.f;
            for (int g = 0; g < groups; ++g) a += sm[L.red + (r * 8 + e) * kThreads + tid + g * vchunks];
            sm[L.o + (c * rep + r0 + r) * vp + d + e] = a;
          }
        }
      }
      __syncthreads();
    }
  }
  if (CL > 1) cluster.sync();
  T* out = static_cast<T*>(p.out) + row * p.ldo;
  for (int c = rank * kThreads + tid; c < H * vp; c += CL * kThreads) {
    float a = 0.f;
    for (int r = 0; r < CL; ++r) a += cluster.map_shared_rank(sm + L.o, r)[c];
    out[c] = from_f32<T>(a * p.out_scale);
  }
  if (CL > 1) cluster.sync();     // the other blocks read this block's shared memory until here
}

// ---------------------------------------------------------------- several queries per cluster
// The same for kTileQ queries behind one another: each key and value that a block reads serves all of them, which is what
// one query per cluster is bound by (2 x 509 tokens of 8 heads of 128 in fp32: 2 GB through L2, 263 us a layer; so 109). A thread takes
// two keys of a key head against kTileQ x 2 queries, then eight value columns of as many; the mixed weights replace the
// weights in place (a thread owns a (query, key) with all its heads: HM at most).
constexpr int kTileQ = 4, kTileRep = 2;
struct TileSmem {   // offsets in floats
  int q, s, stat, talk, o, red, total;
};
__host__ __device__ inline TileSmem tile_smem(int H, int dp, int vp, int cap) {
  TileSmem L;
  L.q = 0;                                            // [kTileQ][H][dp]
  L.o = 0;                                            // once the scores are there: [kTileQ][H][vp] this block's part of the output
  L.s = kTileQ * H * (dp > vp ? dp : vp);             // [kTileQ][H][cap] scores, weights, mixed weights
  L.stat = L.s + ((kTileQ * H * cap + 3) & ~3);       // [2][kTileQ][H] this block's maxima and sums
  L.talk = L.stat + 2 * kTileQ * H;                   // [H][H]
  L.red = L.talk + ((H * H + 3) & ~3);                // [kTileRep * 8][kThreads]
  L.total = L.red + kThreads * kTileRep * 8;
  return L;
}

template <typename T, int HM>
__global__ void __launch_bounds__(kThreads, 2)
window_tile_kernel(const WindowAttnParams p, int cap) {
  extern __shared__ float4 smem4[];
  float* sm = reinterpret_cast<float*>(smem4);
  pdl_enter();
  cg::cluster_group cluster = cg::this_cluster();
  const int CL = static_cast<int>(cluster.num_blocks());
  const int rank = static_cast<int>(cluster.block_rank());
  const int t0 = static_cast<int>(gridDim.x / CL - 1 - blockIdx.x / CL) * kTileQ, b = blockIdx.y;   // late tiles (more keys) first
  const int H = p.H, G = p.G, rep = H / G, dp = p.dp, vp = p.vp;
  const TileSmem L = tile_smem(H, dp, vp, cap);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int pos0 = window_pos0(p), i0 = pos0 + t0, nq = min(kTileQ, p.S - t0), i_last = i0 + nq - 1;
  const long long row0 = static_cast<long long>(b) * p.S;
  const WindowKeys keys(i0, p.window, p.keep);
  const int count = keys.kept + (i_last - keys.first + 1);
  const int chunk = (count + CL - 1) / CL;
  const int n0 = min(rank * chunk, count);
  const int nk = min(chunk, count - n0);        // keys of this block (0 possible)
  auto sees = [&](int qi, int j) { return j <= i0 + qi && (i0 + qi - j < p.window || j < p.keep); };

  // queries, pre-scaled (those past the end repeat the last one and are not stored), and the mixing matrix
  for (int x = tid; x < kTileQ * H * dp; x += kThreads) {
    const int qi = x / (H * dp), c = x - qi * H * dp;
    sm[L.q + x] = to_f32(static_cast<const T*>(p.q)[(row0 + t0 + min(qi, nq - 1)) * p.ldp + c]) * p.scale;
  }
  for (int x = tid; x < H * H; x += kThreads) sm[L.talk + x] = to_f32(static_cast<const T*>(p.talk)[x]);
  __syncthreads();

  const long long slots = p.keep + p.window;
  const T* ring_k = static_cast<const T*>(p.ring_k) + b * slots * G * dp;
  const T* ring_v = static_cast<const T*>(p.ring_v) + b * slots * G * vp;
  const T* new_k = static_cast<const T*>(p.k) + row0 * p.ldp;
  const T* new_v = static_cast<const T*>(p.v) + row0 * p.ldp;

  // scores
  const int pairs = (nk + 1) / 2;
  for (int item = tid; item < pairs * G; item += kThreads) {
    const int c = item / pairs, n = item - c * pairs;
    int j[2];
    const T* kp[2];
#pragma unroll
    for (int y = 0; y < 2; ++y) {
      j[y] = keys.position(n0 + min(n + y * pairs, nk - 1));
      kp[y] = j[y] >= pos0 ? new_k + (j[y] - pos0) * p.ldp + static_cast<long long>(c) * dp
                           : ring_k + (static_cast<long long>(window_slot(j[y], p.window, p.keep)) * G + c) * dp;
    }
    for (int r0 = 0; r0 < rep; r0 += kTileRep) {
      float acc[2][kTileQ][kTileRep] = {};
      float f[2][8], next[2][8];
      load8(kp[0], next[0]);
      load8(kp[1], next[1]);
      for (int d = 0; d < dp; d += 8) {
#pragma unroll
        for (int y = 0; y < 2; ++y)
#pragma unroll
          for (int e = 0; e < 8; ++e) f[y][e] = next[y][e];
        if (d + 8 < dp) {
          load8(kp[0] + d + 8, next[0]);
          load8(kp[1] + d + 8, next[1]);
        }
#pragma unroll
        for (int r = 0; r < kTileRep; ++r) {
          if (r0 + r < rep) {
#pragma unroll
            for (int qi = 0; qi < kTileQ; ++qi) {
              const float4* qv = reinterpret_cast<const float4*>(sm + L.q + (qi * H + c * rep + r0 + r) * dp + d);
              const float4 a = qv[0], e = qv[1];
#pragma unroll
              for (int y = 0; y < 2; ++y)
                acc[y][qi][r] += f[y][0] * a.x + f[y][1] * a.y + f[y][2] * a.z + f[y][3] * a.w + f[y][4] * e.x + f[y][5] * e.y +
                                 f[y][6] * e.z + f[y][7] * e.w;
            }
          }
        }
      }
#pragma unroll
      for (int r = 0; r < kTileRep; ++r) {
        if (r0 + r < rep) {
          const int h = c * rep + r0 + r;
          const float r1 = to_f32(static_cast<const T*>(p.r1)[h]), r2 = to_f32(static_cast<const T*>(p.r2)[h]);
#pragma unroll
          for (int qi = 0; qi < kTileQ; ++qi)
#pragma unroll
            for (int y = 0; y < 2; ++y)
              if (n + y * pairs < nk)
                sm[L.s + (qi * H + h) * cap + n + y * pairs] =
                    sees(qi, j[y]) ? acc[y][qi][r] - r1 * log1pf(r2 * static_cast<float>(i0 + qi - j[y])) : -FLT_MAX;
        }
      }
    }
  }
  __syncthreads();

  // softmax statistics of this block's keys, then of the whole cluster
  for (int x = warp; x < kTileQ * H; x += kThreads / 32) {
    const float* s = sm + L.s + x * cap;
    float m = -FLT_MAX, l = 0.f;
    for (int n = lane; n < nk; n += 32) m = fmaxf(m, s[n]);
    m = warp_max(m);
    for (int n = lane; n < nk; n += 32) l += s[n] != -FLT_MAX ? expf(s[n] - m) : 0.f;
    l = warp_add(l);
    if (lane == 0) {
      sm[L.stat + x] = m;
      sm[L.stat + kTileQ * H + x] = l;
    }
  }
  if (CL > 1) cluster.sync(); else __syncthreads();
  for (int x = warp; x < kTileQ * H; x += kThreads / 32) {
    float m = -FLT_MAX, l = 0.f;
    for (int y = 0; y < CL; ++y) {
      const float* st = cluster.map_shared_rank(sm + L.stat, y);
      const float mr = st[x], lr = st[kTileQ * H + x];
      if (lr > 0.f) {
        const float mn = fmaxf(m, mr);
        l = l * expf(m - mn) + lr * expf(mr - mn);
        m = mn;
      }
    }
    const float inv = 1.0f / l;
    float* s = sm + L.s + x * cap;
    for (int n = lane; n < nk; n += 32) s[n] = s[n] != -FLT_MAX ? expf(s[n] - m) * inv : 0.f;
  }
  __syncthreads();

  // A value that only some of the queries see has weight zero for the others, which keeps it out as long as it is finite: the few
  // keys at both ends of the tile's window are looked at.
  bool odd = false;
  for (int x = tid; x < 2 * (kTileQ - 1) * (G * vp / 8); x += kThreads) {
    const int y = x / (G * vp / 8), col = (x - y * (G * vp / 8)) * 8;
    const int n = (y < kTileQ - 1 ? keys.kept + y : count - 2 * (kTileQ - 1) + y) - n0;
    if (n < 0 || n >= nk) continue;
    const int j = keys.position(n0 + n);
    float f[8];
    load8(j >= pos0 ? new_v + (j - pos0) * p.ldp + col
                    : ring_v + static_cast<long long>(window_slot(j, p.window, p.keep)) * G * vp + col, f);
    float zero = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) zero = fmaf(f[e], 0.f, zero);
    odd |= zero != 0.f;                  // infinities and NaN times zero are NaN
  }

  // mixed weights
  for (int item = tid; item < nk * kTileQ; item += kThreads) {
    const int qi = item / nk, n = item - qi * nk;
    float* s = sm + L.s + qi * H * cap + n;
    float v[HM];
#pragma unroll
    for (int g = 0; g < HM; ++g) v[g] = g < H ? s[g * cap] : 0.f;
    for (int h = 0; h < H; ++h) {
      const float* talk = sm + L.talk + h * H;
      float a = 0.f;
#pragma unroll
      for (int g = 0; g < HM; ++g)
        if (g < H) a += talk[g] * v[g];
      s[h * cap] = a;
    }
  }
  const bool check_seen = __syncthreads_or(odd);

  // values: a thread takes eight columns of a key head and every `groups`-th key
  const int vchunks = G * vp / 8;
  const int groups = vchunks < kThreads ? kThreads / vchunks : 1;
  const int grp = tid / vchunks;
  for (int r0 = 0; r0 < rep; r0 += kTileRep) {
    for (int vc0 = 0; vc0 < vchunks; vc0 += kThreads) {
      const int vc = vc0 + (groups > 1 ? tid - grp * vchunks : tid);
      const bool active = vc < vchunks && (groups == 1 || grp < groups);
      const int c = active ? vc / (vp / 8) : 0, d = active ? (vc - c * (vp / 8)) * 8 : 0;
      float acc[kTileQ][kTileRep][8] = {};
      if (active) {
        float f[8], next[8];
        auto ask = [&](int n) {
          const int j = keys.position(n0 + n);
          const T* v = j >= pos0 ? new_v + (j - pos0) * p.ldp + static_cast<long long>(c) * vp + d
                                 : ring_v + (static_cast<long long>(window_slot(j, p.window, p.keep)) * G + c) * vp + d;
          load8(v, next);
        };
        auto walk = [&](auto check) {
          int n = groups > 1 ? grp : 0;
          if (n < nk) ask(n);
          for (; n < nk; n += groups) {
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = next[e];
            if (n + groups < nk) ask(n + groups);
#pragma unroll
            for (int r = 0; r < kTileRep; ++r) {
              if (r0 + r < rep) {
#pragma unroll
                for (int qi = 0; qi < kTileQ; ++qi) {
                  if (decltype(check)::value && !sees(qi, keys.position(n0 + n))) continue;
                  const float w = sm[L.s + (qi * H + c * rep + r0 + r) * cap + n];
#pragma unroll
                  for (int e = 0; e < 8; ++e) acc[qi][r][e] += w * f[e];
                }
              }
            }
          }
        };
        if (check_seen) walk(std::true_type{});
        else walk(std::false_type{});
      }
#pragma unroll
      for (int qi = 0; qi < kTileQ; ++qi) {
        if (active) {
          float* red = sm + L.red + tid;      // [value][thread]: conflict-free
#pragma unroll
          for (int r = 0; r < kTileRep; ++r)
#pragma unroll
            for (int e = 0; e < 8; ++e) red[(r * 8 + e) * kThreads] = acc[qi][r][e];
        }
        __syncthreads();
        const int cols = min(vchunks - vc0, kThreads);      // column eights of this round; every thread adds up some values
        for (int x = tid; x < cols * kTileRep * 8; x += kThreads) {
          const int val = x / cols, at = x - val * cols, r = val >> 3, cc = (vc0 + at) / (vp / 8);
          if (r0 + r >= rep) break;
          float sum = 0.f;
          for (int g = 0; g < groups; ++g) sum += sm[L.red + val * kThreads + at + g * vchunks];
          sm[L.o + (qi * H + cc * rep + r0 + r) * vp + (vc0 + at - cc * (vp / 8)) * 8 + (val & 7)] = sum;
        }
        __syncthreads();
      }
    }
  }
  if (CL > 1) cluster.sync();
  T* out = static_cast<T*>(p.out) + (row0 + t0) * p.ldo;
  for (int x = rank * kThreads + tid; x < nq * H * vp; x += CL * kThreads) {
    float a = 0.f;
    for (int y = 0; y < CL; ++y) a += cluster.map_shared_rank(sm + L.o, y)[x];
    const int qi = x / (H * vp);
    out[qi * p.ldo + x - qi * H * vp] = from_f32<T>(a * p.out_scale);
  }
  if (CL > 1) cluster.sync();     // the other blocks read this block's shared memory until here
}

constexpr int kMaxDynSmem = 227 * 1024;

template <typename T, int HM>
cudaError_t launch_tile_hm(const WindowAttnParams& p, int cl, int cap, size_t bytes, cudaStream_t st) {
  auto* kern = window_tile_kernel<T, HM>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(cl * ((p.S + kTileQ - 1) / kTileQ)), static_cast<unsigned>(p.B), 1);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = bytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cl;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kern, p, cap);
}

// Tiles of kTileQ queries, where what single queries would read is worth the longer chain of a tile (keys in pairs, values one
// by one, for four queries) and two blocks fit an SM. What the lines stand for:
//   all        what one query per cluster reads through L2. Up to 160 MB, some 20 us, a call's time is that of its blocks' chains.
//   per_query  up to 240 MB the reads only win where a query has 400 KB of them: with fewer or narrower key heads fewer threads
//              have value columns of their own, and a tile's chain over the keys is the longer for it.
//   seen       keys of a query in the middle of the prompt. With less than 128 a tile's 256 threads, two keys each, stand idle.
// us, fp32, one query per cluster / tiles: 8 heads of 128 on 4, window 512:
// 145 tokens (72 keys on average, 43 MB) 33 / 61, 300 (184 MB) 84 / 54, 800 265 / 119, 2 x 1 000 635 / 282; 145 tokens behind
// 700 107 / 87; 16 heads on 8, window 1 024: 4 x 150 (75 keys, 368 MB) 184 / 269, 300 190 / 162, 2 x 1 000 2 657 / 1 276; 6
// heads of 48 and 64 on 2, window 300: 4 x 150 behind 700 (161 MB, 270 KB a query) 74 / 77, 800 (200 MB) 64 / 66, 2 x 1 000 (250 MB)
// 147 / 115.
template <typename T>
bool launch_tiles(const WindowAttnParams& p, cudaStream_t st, cudaError_t& e) {
  const long long tiles = static_cast<long long>((p.S + kTileQ - 1) / kTileQ) * p.B;
  const int n_max = p.keep + p.window + kTileQ - 1;
  auto bytes = [&](int cl) { return static_cast<size_t>(tile_smem(p.H, p.dp, p.vp, (n_max + cl - 1) / cl).total) * sizeof(float); };
  const long long seen = min(static_cast<long long>(p.window + p.keep), p.pos_dev ? p.window : p.pos0 + (p.S + 1) / 2ll);
  const long long per_query = seen * p.G * (p.dp + p.vp) * static_cast<long long>(sizeof(T)), all = per_query * p.S * p.B;
  if (p.H > 32 || seen < 128 || all < 160000000ll || (all < 240000000ll && per_query < 400000ll)) return false;
  int cl = 1;
  while (cl < 8 && (tiles * cl < 2LL * current_sm_count() || bytes(cl) > kMaxDynSmem / 2)) cl *= 2;
  if (bytes(cl) > kMaxDynSmem / 2) return false;
  const int cap = (n_max + cl - 1) / cl;
  e = p.H <= 8 ? launch_tile_hm<T, 8>(p, cl, cap, bytes(cl), st)
               : p.H <= 16 ? launch_tile_hm<T, 16>(p, cl, cap, bytes(cl), st) : launch_tile_hm<T, 32>(p, cl, cap, bytes(cl), st);
  return true;
}

template <typename T>
cudaError_t launch_rows(const WindowAttnParams& p, cudaStream_t st) {
  cudaError_t e = cudaSuccess;
  if (launch_tiles<T>(p, st, e)) return e;
  const int n_max = p.keep + p.window;
  auto bytes = [&](int cl) {
    return static_cast<size_t>(rows_smem(p.H, p.dp, p.vp, (n_max + cl - 1) / cl).total) * sizeof(float);
  };
  // blocks per query: enough to fill the device when there are few queries, and enough for the
  // scores to fit in shared memory
  int cl = 1;
  const long long queries = static_cast<long long>(p.B) * p.S;
  while (cl < 8 && ((queries * cl < 148 && n_max / (2 * cl) >= 64) || bytes(cl) > kMaxDynSmem)) cl *= 2;
  if (bytes(cl) > kMaxDynSmem) return cudaErrorInvalidValue;
  auto kern = window_rows_kernel<T>;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(cl * p.S), static_cast<unsigned>(p.B), 1);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = bytes(cl);
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cl;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kern, p, (n_max + cl - 1) / cl);
}

}  // namespace

bool window_rows_supported(const WindowAttnParams& p) {
  return static_cast<size_t>(rows_smem(p.H, p.dp, p.vp, (p.keep + p.window + 7) / 8).total) * sizeof(float) <=
         kMaxDynSmem;
}

cudaError_t launch_head_norm(const WindowAttnParams& p, int fp32, cudaStream_t st) {
  if (p.B == 0 || p.S == 0) return cudaSuccess;
  return fp32 ? head_norm_any<float>(p, st) : head_norm_any<bf16>(p, st);
}

cudaError_t launch_window_append(const WindowAttnParams& p, int fp32, cudaStream_t st) {
  if (p.B == 0 || p.S == 0) return cudaSuccess;
  const dim3 grid(p.S, p.B);
  return fp32 ? launch_kernel(window_append_kernel<float>, grid, dim3(128), 0, st, p)
              : launch_kernel(window_append_kernel<bf16>, grid, dim3(128), 0, st, p);
}

cudaError_t launch_window_rows(const WindowAttnParams& p, int fp32, cudaStream_t st) {
  if (p.B == 0 || p.S == 0) return cudaSuccess;
  return fp32 ? launch_rows<float>(p, st) : launch_rows<bf16>(p, st);
}

}  // namespace cdeep
