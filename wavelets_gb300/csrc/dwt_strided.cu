// Wavelet passes along an axis that is strided in memory while consecutive
// rows are neighbours on both sides (the y pass of either direction: z is
// contiguous), entirely in registers.
//
// A thread holds K consecutive elements of TWO neighbouring rows, packed as
// pairs of floats: every lifting operation is one packed instruction
// (add / fma .f32x2) for both, and every load and store moves eight bytes.
// G = L / K lanes hold a row pair; they lie C = 32 / G lanes apart, so the C
// lanes next to each other touch neighbouring memory.  All levels run on the
// K elements in place (M = K/2, K/4, .. pairs a lane), with two 64-bit
// shuffles down and two up per level for the pairs at the lane edges, and a
// finished value goes straight from its register to its place in global
// memory: no shared memory, no barriers.
//
// K = 32 for L = 32 .. 256 (five levels), 48 for L = 48, 96, 192 (four), 16
// for L = 16 (four); deeper transforms, other lengths and an odd number of
// neighbouring rows stay with the tile kernels.  With 64 to 96 values per
// thread in flight the pass is bound by HBM: the y passes of 729 cubelets of
// 128^3 (1.5 G elements) take 1.56 ms, 7.8 TB/s of their eight bytes an
// element (2.77 ms in the column-tile kernel), the inverse y passes of the
// mixed batch 0.55 ms (1.22 ms through the row kernel's tile).
//
// Each lifting step does the arithmetic of dwt.cu / dwt_cols.cu / dwt_rows.cu
// (the same operands, rounded the same), so the values are identical.
#include <cuda_runtime.h>

#include "dwt_common.cuh"
#include "wl_internal.h"

namespace wl {
namespace {
using namespace dwtc;

constexpr int kThreads = 128;
constexpr unsigned kAll = 0xffffffffu;

typedef unsigned long long f2;  // two floats: the same element of two rows

__device__ __forceinline__ f2 pack(float a) {
  f2 r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// lane position along the row: lane `seg` of G, C lanes between neighbours
template <int G> struct Along {
  static constexpr int C = 32 / G;
  int seg;
  // the value of the next / previous lane of the row, `own` at its end
  __device__ __forceinline__ f2 next(f2 v, f2 own) const {
    if (G == 1) return own;
    const f2 o = __shfl_down_sync(kAll, v, C);
    return seg == G - 1 ? own : o;
  }
  __device__ __forceinline__ f2 prev(f2 v, f2 own) const {
    if (G == 1) return own;
    const f2 o = __shfl_up_sync(kAll, v, C);
    return seg == 0 ? own : o;
  }
};

// One forward level on M pairs a lane: low-pass values in e[], details in o[]
// (dwt_rows.cu fwd_level; mirrored ends s[h] = s[h-1], d[-1] = d[0]).
template <int M, int G, bool HAAR>
__device__ __forceinline__ void fwd_level(f2 (&e)[M], f2 (&o)[M], const Along<G> &at) {
  if (HAAR) {  // dwt_cpu.cc:159-162
    const f2 c = pack(kInvSqrt2), neg = pack(-1.0f);
#pragma unroll
    for (int k = 0; k < M; k++) {
      const f2 a = e[k], b = o[k];
      o[k] = mul2(fma2(b, neg, a), c);  // a - b, rounded once
      e[k] = mul2(add2(a, b), c);
    }
    return;
  }
  const f2 ka = pack(kAlpha), kb = pack(kBeta), kg = pack(kGamma), kd = pack(kDelta);
  const f2 eN = at.next(e[0], e[M - 1]);
#pragma unroll
  for (int k = 0; k < M; k++) o[k] = fma2(ka, add2(e[k], k + 1 < M ? e[(k + 1) % M] : eN), o[k]);
  const f2 d1P = at.prev(o[M - 1], o[0]);
#pragma unroll
  for (int k = 0; k < M; k++) e[k] = fma2(kb, add2(k ? o[(k + M - 1) % M] : d1P, o[k]), e[k]);
  const f2 s1N = at.next(e[0], e[M - 1]);
#pragma unroll
  for (int k = 0; k < M; k++) o[k] = fma2(kg, add2(e[k], k + 1 < M ? e[(k + 1) % M] : s1N), o[k]);
  const f2 d2P = at.prev(o[M - 1], o[0]);
#pragma unroll
  for (int k = 0; k < M; k++) e[k] = fma2(kd, add2(k ? o[(k + M - 1) % M] : d2P, o[k]), e[k]);
}

// The inverse: low-pass e[], details o[] in, even and odd elements out
// (dwt_rows.cu inv_level).
template <int M, int G, bool HAAR>
__device__ __forceinline__ void inv_level(f2 (&e)[M], f2 (&o)[M], const Along<G> &at) {
  if (HAAR) {  // dwt_cpu.cc:193-196
    const f2 c = pack(kInvSqrt2), neg = pack(-1.0f);
#pragma unroll
    for (int k = 0; k < M; k++) {
      const f2 a = e[k], b = o[k];
      e[k] = mul2(c, add2(a, b));
      o[k] = mul2(c, fma2(b, neg, a));
    }
    return;
  }
  const f2 ka = pack(-kAlpha), kb = pack(-kBeta), kg = pack(-kGamma), kd = pack(-kDelta);
  const f2 d2P = at.prev(o[M - 1], o[0]);
#pragma unroll
  for (int k = 0; k < M; k++) e[k] = fma2(kd, add2(k ? o[(k + M - 1) % M] : d2P, o[k]), e[k]);
  const f2 s1N = at.next(e[0], e[M - 1]);
#pragma unroll
  for (int k = 0; k < M; k++) o[k] = fma2(kg, add2(e[k], k + 1 < M ? e[(k + 1) % M] : s1N), o[k]);
  const f2 d1P = at.prev(o[M - 1], o[0]);
#pragma unroll
  for (int k = 0; k < M; k++) e[k] = fma2(kb, add2(k ? o[(k + M - 1) % M] : d1P, o[k]), e[k]);
  const f2 eN = at.next(e[0], e[M - 1]);
#pragma unroll
  for (int k = 0; k < M; k++) o[k] = fma2(ka, add2(e[k], k + 1 < M ? e[(k + 1) % M] : eN), o[k]);
}

// A row pair in global memory: position q at base + q * stride floats.
struct Row {
  float *base;
  long long stride;
  bool ok;
  __device__ __forceinline__ f2 get(int q) const {
    return ok ? *reinterpret_cast<const f2 *>(base + q * stride) : 0ull;
  }
  __device__ __forceinline__ void put(int q, f2 v) const {
    if (ok) *reinterpret_cast<f2 *>(base + q * stride) = v;
  }
};

// Levels LEV .. S-1 on the 2 M values v[] of a lane, each band to its place
// with the deferred lifting scale.
template <int LEV, int M, int G, bool HAAR>
__device__ __forceinline__ void fwd_from(const f2 (&v)[2 * M], int S, const float *scale,
                                         const Along<G> &at, const Row &out) {
  constexpr int H = M * G;  // pairs of this level
  f2 e[M], o[M];
#pragma unroll
  for (int k = 0; k < M; k++) {
    e[k] = v[2 * k];
    o[k] = v[2 * k + 1];
  }
  fwd_level<M, G, HAAR>(e, o, at);
  const f2 sc = pack(scale[LEV]);
#pragma unroll
  for (int k = 0; k < M; k++) out.put(H + M * at.seg + k, mul2(o[k], sc));
  if constexpr (M % 2 == 0) {
    if (LEV + 1 < S) {
      fwd_from<LEV + 1, M / 2, G, HAAR>(e, S, scale, at, out);
      return;
    }
  }
  const f2 low = pack(scale[LEV + 1]);
#pragma unroll
  for (int k = 0; k < M; k++) out.put(M * at.seg + k, mul2(e[k], low));
}

// The 2 M values v[] of level LEV's input from the bands of levels LEV ..
// S-1 (rscale: the reciprocal of the deferred scale).
template <int LEV, int M, int G, bool HAAR>
__device__ __forceinline__ void inv_to(f2 (&v)[2 * M], int S, const float *rscale,
                                       const Along<G> &at, const Row &in) {
  constexpr int H = M * G;
  f2 e[M], o[M];
  const f2 sc = pack(rscale[LEV]);
#pragma unroll
  for (int k = 0; k < M; k++) o[k] = in.get(H + M * at.seg + k);
  bool deeper = false;
  if constexpr (M % 2 == 0) {
    if (LEV + 1 < S) {
      inv_to<LEV + 1, M / 2, G, HAAR>(e, S, rscale, at, in);
      deeper = true;
    }
  }
  if (!deeper) {
    const f2 low = pack(rscale[LEV + 1]);
#pragma unroll
    for (int k = 0; k < M; k++) e[k] = mul2(in.get(M * at.seg + k), low);
  }
#pragma unroll
  for (int k = 0; k < M; k++) o[k] = mul2(o[k], sc);
  inv_level<M, G, HAAR>(e, o, at);
#pragma unroll
  for (int k = 0; k < M; k++) {
    v[2 * k] = e[k];
    v[2 * k + 1] = o[k];
  }
}

template <int K, int G, bool HAAR, bool INV>
__device__ __forceinline__ void run_rows(const PassDesc &d, int tile, const float *scale) {
  constexpr int C = 32 / G;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Along<G> at{lane / C};
  const int row = 2 * ((tile * (kThreads / 32) + warp) * C + lane % C);
  Row in{nullptr, d.inSC, row < d.rows}, out{nullptr, d.outSC, row < d.rows};
  if (in.ok) {
    const int a = row / d.B, b = row - a * d.B;  // B even: b and b + 1 are one pair
    in.base = const_cast<float *>(static_cast<const float *>(d.in)) + (long long)a * d.inSA + b;
    out.base = static_cast<float *>(d.out) + (long long)a * d.outSA + b;
  }
  f2 v[K];
  if (INV) {
    inv_to<0, K / 2, G, HAAR>(v, d.steps, scale, at, in);
#pragma unroll
    for (int k = 0; k < K; k++) out.put(K * at.seg + k, v[k]);
  } else {
#pragma unroll
    for (int k = 0; k < K; k++) v[k] = in.get(K * at.seg + k);
    fwd_from<0, K / 2, G, HAAR>(v, d.steps, scale, at, out);
  }
}

template <int K, int G, bool INV>
__global__ void __launch_bounds__(kThreads)
dwt_strided_kernel(const PassDesc *__restrict__ passes, const int *__restrict__ tilePrefix,
                   int nPasses) {
  __shared__ float scale[16];
  const int bid = blockIdx.x;
  int lo = 0, hi = nPasses - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (tilePrefix[mid] <= bid) lo = mid; else hi = mid - 1;
  }
  const PassDesc &d = passes[lo];
  const int S = d.steps;
  const bool haar = d.wavelet == WL_HAAR;
  if ((int)threadIdx.x <= S) {
    const float s = haar ? 1.0f : lifting_scale(threadIdx.x, S);
    scale[threadIdx.x] = INV && !haar ? 1.0f / s : s;
  }
  __syncthreads();
  if (haar) run_rows<K, G, true, INV>(d, bid - tilePrefix[lo], scale);
  else run_rows<K, G, false, INV>(d, bid - tilePrefix[lo], scale);
}

// lanes per row pair and elements per lane; 0: another kernel
int strided_lanes(int L) {
  switch (L) {
    case 16: case 32: case 48: return 1;
    case 64: case 96: return 2;
    case 128: case 192: return 4;
    case 256: return 8;
    default: return 0;
  }
}

template <int K, int G>
void launch_kg(const PassDesc *p, const int *tp, int n, int blocks, bool inv, cudaStream_t s) {
  if (inv) dwt_strided_kernel<K, G, true><<<blocks, kThreads, 0, s>>>(p, tp, n);
  else dwt_strided_kernel<K, G, false><<<blocks, kThreads, 0, s>>>(p, tp, n);
}

}  // namespace

// rows per block (both rows of kThreads / 32 warps of 32 / G pairs)
int dwt_strided_rows_per_block(int L) { return 2 * (kThreads / 32) * (32 / strided_lanes(L)); }

bool dwt_strided_fits(const PassDesc &d) {
  const int g = strided_lanes(d.L);
  if (!g || d.steps < 1 || d.B % 2 || d.inSB != 1 || d.outSB != 1) return false;
  // neighbouring row pairs stay eight-byte aligned
  if ((d.inSA | d.inSC | d.outSA | d.outSC) & 1) return false;
  return d.steps <= (d.L / g == 32 ? 5 : 4);
}

void launch_dwt_strided(const PassDesc *p, const int *tp, int n, int blocks, int L, bool inverse,
                        cudaStream_t s) {
  switch (L) {
    case 16: launch_kg<16, 1>(p, tp, n, blocks, inverse, s); break;
    case 32: launch_kg<32, 1>(p, tp, n, blocks, inverse, s); break;
    case 48: launch_kg<48, 1>(p, tp, n, blocks, inverse, s); break;
    case 64: launch_kg<32, 2>(p, tp, n, blocks, inverse, s); break;
    case 96: launch_kg<48, 2>(p, tp, n, blocks, inverse, s); break;
    case 128: launch_kg<32, 4>(p, tp, n, blocks, inverse, s); break;
    case 192: launch_kg<48, 4>(p, tp, n, blocks, inverse, s); break;
    default: launch_kg<32, 8>(p, tp, n, blocks, inverse, s); break;
  }
}

}  // namespace wl
