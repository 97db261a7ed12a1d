// Kernels around a residual stream kept in fp32: embedding gather into the stream, RMSNorm or layer
// norm of a stream row into the operand type of the next product, and the gated unit of models that run
// entirely in fp32.
#include "elem.cuh"
#include "kernels.h"

namespace cdeep {

namespace {

struct Positions {          // learned position vectors (table nullptr: none)
  const void* table;
  int P, S, pos0;
  const int* pos_dev;
};

// x[t, :] = table[ids[t], :] (+ the vector of the row's position) in fp32; columns [W, ldx) are zero.
// Ids outside the table are clamped to it (as in the dispatch kernels), and so are positions, so a
// bad id can never read out of bounds.
template <typename T>
__global__ void __launch_bounds__(128)
embed_rows_kernel(const long long* __restrict__ ids, const T* __restrict__ table, const Positions pos,
                  float* __restrict__ x, int V, int W, int ldw, int ldx) {
  pdl_enter();
  const int t = blockIdx.x;
  long long id = ids[t];
  id = id < 0 ? 0 : (id >= V ? V - 1 : id);
  const T* src = table + id * ldw;
  const T* add = nullptr;
  if (pos.table) {
    const int p = (pos.pos_dev ? *pos.pos_dev : pos.pos0) + t % pos.S;
    add = static_cast<const T*>(pos.table) + static_cast<long long>(min(max(p, 0), pos.P - 1)) * ldw;
  }
  float* dst = x + static_cast<size_t>(t) * ldx;
  const int whole = (ldw & 7) == 0 ? (W & ~7) : 0;       // columns copied eight at a time
  for (int c = threadIdx.x * 8; c < whole; c += blockDim.x * 8) {
    float f[8];
    load8(src + c, f);
    if (add) {
      float g[8];
      load8(add + c, g);
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] += g[e];
    }
    store8(dst + c, f);
  }
  for (int c = whole + threadIdx.x; c < ldx; c += blockDim.x)
    dst[c] = c < W ? to_f32(src[c]) + (add ? to_f32(add[c]) : 0.f) : 0.f;
}

// out[t, :] = x[t, :] / sqrt(mean(x^2) + eps) * (w + offset), with kCentred of x minus its mean; the
// means run over W columns, rows are ldx apart (a multiple of 8, zero beyond W).  kWarps warps per
// row: one, or the block's four.  NV > 0: the row (at most NV * kWarps * 256 columns) stays in registers
// between the reductions and the scaling; NV = 0: it is read again for each.
template <typename T, int NV, int kWarps, bool kCentred>
__global__ void __launch_bounds__(128)
rmsnorm_f32_kernel(const float* __restrict__ x, const T* __restrict__ w, float eps, float offset,
                   T* __restrict__ out, int rows, int W, int ldx) {
  __shared__ float s_part[2][4];
  pdl_enter();
  const int row = kWarps == 1 ? blockIdx.x * 4 + (threadIdx.x >> 5) : blockIdx.x;
  if (row >= rows) return;
  constexpr int kLanes = 32 * kWarps;
  const int lane = threadIdx.x & (kLanes - 1);
  auto row_add = [&](float v, int slot) {
    v = warp_add(v);
    if constexpr (kWarps > 1) {
      if ((threadIdx.x & 31) == 0) s_part[slot][threadIdx.x >> 5] = v;
      __syncthreads();
      v = s_part[slot][0] + s_part[slot][1] + s_part[slot][2] + s_part[slot][3];
    }
    return v;
  };
  const float* xr = x + static_cast<size_t>(row) * ldx;
  T* orow = out + static_cast<size_t>(row) * ldx;
  constexpr int kBuf = NV ? NV : 1;
  float buf[kBuf][8];
  if constexpr (NV > 0) {
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int c = (v * kLanes + lane) * 8;
      if (c < ldx) load8(xr + c, buf[v]);
    }
  }
  auto each = [&](auto&& fn) {          // fn(column, eight elements) over this lane's columns
    if constexpr (NV > 0) {
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const int c = (v * kLanes + lane) * 8;
        if (c < ldx) fn(c, buf[v]);
      }
    } else {
      for (int c = lane * 8; c < ldx; c += kLanes * 8) {
        load8(xr + c, buf[0]);
        fn(c, buf[0]);
      }
    }
  };
  float mean = 0.f;
  if constexpr (kCentred) {
    float sum = 0.f;
    each([&](int, float (&f)[8]) {
#pragma unroll
      for (int e = 0; e < 8; ++e) sum += f[e];
    });
    mean = row_add(sum, 0) / static_cast<float>(W);
  }
  float ss = 0.f;
  each([&](int c, float (&f)[8]) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float d = kCentred ? (c + e < W ? f[e] - mean : 0.f) : f[e];
      ss += d * d;
    }
  });
  const float r = 1.0f / sqrtf(row_add(ss, 1) / static_cast<float>(W) + eps);
  each([&](int c, float (&f)[8]) {
    float wv[8];
    load8(w + c, wv);
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] = (f[e] - mean) * r * (wv[e] + offset);
    store8(orow + c, f);
  });
}

// h[t, j] = g * sigmoid(alpha g) * (u + offset), g = min(gu[t, j], limit), u = clamp(gu[t, I + j], +-limit)
__global__ void __launch_bounds__(256)
glu_f32_kernel(const float* __restrict__ gu, float* __restrict__ h, long long n, int I, float alpha,
               float limit, float offset) {
  pdl_enter();
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < n; i += gridDim.x * 256ll) {
    const long long t = i / I;
    const int j = static_cast<int>(i - t * I);
    const float g = fminf(gu[t * 2 * I + j], limit);
    const float u = fminf(fmaxf(gu[t * 2 * I + I + j], -limit), limit);
    h[i] = g / (1.0f + expf(-alpha * g)) * (u + offset);
  }
}

template <typename T, bool kCentred>
cudaError_t rmsnorm_any(const float* x, const void* w, float eps, float offset, void* out, int rows, int W,
                        int ldx, cudaStream_t st) {
  auto wp = static_cast<const T*>(w);
  auto op = static_cast<T*>(out);
  const dim3 grid((rows + 3) / 4), block(128);
  const int nv = (ldx + 255) / 256;
  // fewer rows than two blocks an SM, each more than two rounds of a warp wide: four warps a row. 64 rows of 2048,
  // centred: 2.7 us, with a warp a row 6.1; 32 rows of 1024 2.0 / 3.4
  if (rows <= 2 * current_sm_count() && nv > 2 && nv <= 16) {
    if (nv <= 8) return launch_kernel(rmsnorm_f32_kernel<T, 2, 4, kCentred>, dim3(rows), block, 0, st, x, wp, eps, offset, op, rows, W, ldx);
    return launch_kernel(rmsnorm_f32_kernel<T, 4, 4, kCentred>, dim3(rows), block, 0, st, x, wp, eps, offset, op, rows, W, ldx);
  }
#define CDEEP_NORM(NV) return launch_kernel(rmsnorm_f32_kernel<T, NV, 1, kCentred>, grid, block, 0, st, x, wp, eps, offset, op, rows, W, ldx)
  if (nv <= 2) CDEEP_NORM(2);
  if (nv <= 4) CDEEP_NORM(4);
  if (nv <= 8) CDEEP_NORM(8);
  CDEEP_NORM(0);
#undef CDEEP_NORM
}

}  // namespace

cudaError_t launch_embed_rows(const long long* ids, const void* table, float* x, int T, int V, int W, int ldw,
                              int ldx, int fp32, cudaStream_t st, const void* pos, int P, int S, int pos0,
                              const int* pos_dev) {
  if (T == 0) return cudaSuccess;
  const Positions ps{pos, P, S, pos0, pos_dev};
  return fp32 ? launch_kernel(embed_rows_kernel<float>, dim3(T), dim3(128), 0, st, ids,
                              static_cast<const float*>(table), ps, x, V, W, ldw, ldx)
              : launch_kernel(embed_rows_kernel<bf16>, dim3(T), dim3(128), 0, st, ids,
                              static_cast<const bf16*>(table), ps, x, V, W, ldw, ldx);
}

cudaError_t launch_rmsnorm_f32(const float* x, const void* w, float eps, float offset, void* out, int rows, int W,
                               int ldx, int fp32, cudaStream_t st, bool centred) {
  if (rows == 0) return cudaSuccess;
  if (centred)
    return fp32 ? rmsnorm_any<float, true>(x, w, eps, offset, out, rows, W, ldx, st)
                : rmsnorm_any<bf16, true>(x, w, eps, offset, out, rows, W, ldx, st);
  return fp32 ? rmsnorm_any<float, false>(x, w, eps, offset, out, rows, W, ldx, st)
              : rmsnorm_any<bf16, false>(x, w, eps, offset, out, rows, W, ldx, st);
}

cudaError_t launch_glu_f32(const float* gu, float* h, int T, int I, float alpha, float limit, float offset,
                           cudaStream_t st) {
  const long long n = static_cast<long long>(T) * I;
  if (n == 0) return cudaSuccess;
  const long long blocks = (n + 255) / 256;
  return launch_kernel(glu_f32_kernel, dim3(static_cast<unsigned>(blocks < 4096 ? blocks : 4096)), dim3(256), 0, st, gu,
                       h, n, I, alpha, limit, offset);
}

}  // namespace cdeep
