// Wavelet passes entirely in registers, for rows whose neighbours are
// neighbours in memory: the y pass of either direction (strided rows on both
// sides, z contiguous), the forward x pass (contiguous source rows of any
// type, z contiguous in the output) and the inverse x pass (the reverse, into
// rows of any type).
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
// K = 32 for L = 32 .. 1024, 64 for 2048, 16 for 16 (every level: after one
// value is left per lane a level gathers pair j into lane j), 48 for L = 48,
// 96, 192 (four levels).  Other lengths of K = 32, 16 or 8 times at most 16
// (five, four or three levels; strided_elems) take their number of lanes from
// the pass (G = 0; the lanes of a warp that do not make a row are idle), so
// one launch holds rows of all such lengths; their source rows start at any
// address.  The x passes of 400 cubelets of odd sizes take 0.40 ms, their y
// passes 0.33 (0.55 and 0.37 in the column-tile kernel), restoring as many
// 3.4 ms a call (3.74); the x pass of a 93 x 181 x 147 16-bit volume 13 us
// (25).  Longer lengths, deeper levels and an odd number of neighbouring rows
// stay with the tile kernels.
//
// Levels below one value per lane and scales undone by division (FULL) are
// instantiations of their own: in one kernel they cost the shallow passes
// registers and branches (restoring the mixed batch 4.36 ms a call instead of
// 4.19).  A 2048^2 image's passes take 17 us each forward, 21 us inverse (42
// and 60 to 70 us in the row-cooperative kernel).
//
// With 64 to 96 values per thread in flight a large pass is bound by HBM: the
// y passes of 729 cubelets of 128^3 (1.5 G elements) take 1.56 ms, 7.8 TB/s
// of their eight bytes an element (2.77 ms in the column-tile kernel), the
// inverse y passes of the mixed batch 0.55 ms (1.22 ms through the row
// kernel's tile).
//
// The x passes read or write a lane's K elements of a source or output row
// with vectors of 32 bytes (16 where its address or K asks for it), a run cut
// by the real row length element by element; they take inputs in device memory
// and outputs whose rows start at multiples of 16 bytes.
// The inverse x passes of the mixed batch take 0.73 ms (1.47 ms through the
// row kernel's tile); forward, the half of a 2 GiB volume's cubelets that the
// kernel took first (before it accepted 16-byte starts) 0.71 ms against 0.91
// ms for the other half in the row kernel.
//
// Each lifting step does the arithmetic of dwt.cu / dwt_cols.cu / dwt_rows.cu
// (the same operands, rounded the same), so the values are identical.
#pragma once
#include <cuda_runtime.h>

#include <type_traits>

#include "dwt_common.cuh"
#include "select_common.cuh"
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
__device__ __forceinline__ f2 pack(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack(f2 v, float &a, float &b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
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

// lane position along the row: lane `seg` of `lanes` (G, or the pass's own
// number where G is 0), `c` lanes between neighbours; lanes [0, na) hold the
// level's pairs
template <int G> struct Along {
  static constexpr int C = G ? 32 / G : 0;
  int seg, lanes, c, na;
  // the value of the next / previous lane of the row, `own` at its end
  __device__ __forceinline__ f2 next(f2 v, f2 own) const {
    if (G == 1) return own;
    const f2 o = __shfl_down_sync(kAll, v, c);
    return seg == na - 1 ? own : o;
  }
  __device__ __forceinline__ f2 prev(f2 v, f2 own) const {
    if (G == 1) return own;
    const f2 o = __shfl_up_sync(kAll, v, c);
    return seg == 0 ? own : o;
  }
  // the value of lane s of the row
  __device__ __forceinline__ f2 from(f2 v, int s) const {
    return __shfl_sync(kAll, v, (s & (G - 1)) * C + (int)(threadIdx.x & (C - 1)));
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

// ---- contiguous rows (x passes: source and output; z passes) ----
// bytes per vector access of a lane's K elements
template <typename T, int K> __host__ __device__ constexpr int vec_bytes() {
  return (K * (int)sizeof(T)) % 32 == 0 ? 32 : (K * (int)sizeof(T)) % 16 == 0 ? 16 : 8;
}
template <int VB> __device__ __forceinline__ void load_vec(const void *p, unsigned *w) {
  if constexpr (VB == 32) {
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]),
                   "=r"(w[6]), "=r"(w[7])
                 : "l"(p));
  } else if constexpr (VB == 8) {
    const uint2 q = *static_cast<const uint2 *>(p);
    w[0] = q.x; w[1] = q.y;
  } else if constexpr (VB == 4) {
    w[0] = *static_cast<const unsigned *>(p);
  } else {
    const uint4 q = *static_cast<const uint4 *>(p);
    w[0] = q.x; w[1] = q.y; w[2] = q.z; w[3] = q.w;
  }
}
template <int VB> __device__ __forceinline__ void store_vec(void *p, const unsigned *w) {
  if constexpr (VB == 32) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 :: "l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]),
                    "r"(w[6]), "r"(w[7])
                 : "memory");
  } else if constexpr (VB == 8) {
    *static_cast<uint2 *>(p) = make_uint2(w[0], w[1]);
  } else if constexpr (VB == 4) {
    *static_cast<unsigned *>(p) = w[0];
  } else {
    *static_cast<uint4 *>(p) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}
// element k of a vector of 32-bit words as a float, and back
template <typename T> __device__ __forceinline__ float from_words(const unsigned *w, int k) {
  if constexpr (std::is_same<T, float>::value) return __uint_as_float(w[k]);
  else if constexpr (sizeof(T) == 4) return (float)(int)w[k];
  else if constexpr (sizeof(T) == 2) return (float)((w[k / 2] >> (16 * (k & 1))) & 0xffffu);
  else return (float)((w[k / 4] >> (8 * (k & 3))) & 0xffu);
}
template <typename T> __device__ __forceinline__ unsigned to_bits(float f) {
  T t;
  store_from_float(&t, f);
  if constexpr (std::is_same<T, float>::value) return __float_as_uint(f);
  else return (unsigned)t;
}

template <typename T, int K, int VB>
__device__ __forceinline__ void load_vecs(const T *p, float (&v)[K]) {
  constexpr int E = VB / (int)sizeof(T);
#pragma unroll
  for (int j = 0; j < K / E; j++) {
    unsigned w[VB / 4];
    load_vec<VB>(p + j * E, w);
#pragma unroll
    for (int k = 0; k < E; k++) v[j * E + k] = from_words<T>(w, k);
  }
}
template <typename T, int K, int VB>
__device__ __forceinline__ void store_vecs(T *p, const float (&v)[K]) {
  constexpr int E = VB / (int)sizeof(T), P = 4 / (int)sizeof(T);
#pragma unroll
  for (int j = 0; j < K / E; j++) {
    unsigned w[VB / 4];
#pragma unroll
    for (int i = 0; i < VB / 4; i++) {
      w[i] = 0;
#pragma unroll
      for (int k = 0; k < P; k++)
        w[i] |= to_bits<T>(v[j * E + i * P + k]) << (8 * (int)sizeof(T) * k);
    }
    store_vec<VB>(p + j * E, w);
  }
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
  template <int M> __device__ __forceinline__ void get_run(int q, f2 (&v)[M]) const {
#pragma unroll
    for (int k = 0; k < M; k++) v[k] = get(q + k);
  }
  template <int M> __device__ __forceinline__ void put_run(int q, const f2 (&v)[M]) {
#pragma unroll
    for (int k = 0; k < M; k++) put(q + k, v[k]);
  }
};

// A pair of contiguous rows (z passes); SEL: every value put also goes into
// the select statistics.
template <bool SEL> struct ZRow {
  float *base[2];  // null: no such row
  selc::SelAcc *acc;
  template <int M> __host__ __device__ static constexpr int vb() {
    return M % 8 == 0 ? 32 : M % 4 == 0 ? 16 : M % 2 == 0 ? 8 : 4;
  }
  __device__ __forceinline__ f2 get(int q) const {
    return pack(base[0] ? base[0][q] : 0.f, base[1] ? base[1][q] : 0.f);
  }
  __device__ __forceinline__ void put(int q, f2 v) {
    const f2 x[1] = {v};
    put_run<1>(q, x);
  }
  template <int M> __device__ __forceinline__ void get_run(int q, f2 (&v)[M]) const {
    float x[2][M];
#pragma unroll
    for (int r = 0; r < 2; r++) {
      if (base[r]) {
        load_vecs<float, M, vb<M>()>(base[r] + q, x[r]);
      } else {
#pragma unroll
        for (int k = 0; k < M; k++) x[r][k] = 0.f;
      }
    }
#pragma unroll
    for (int k = 0; k < M; k++) v[k] = pack(x[0][k], x[1][k]);
  }
  template <int M> __device__ __forceinline__ void put_run(int q, const f2 (&v)[M]) {
    float x[2][M];
#pragma unroll
    for (int k = 0; k < M; k++) unpack(v[k], x[0][k], x[1][k]);
#pragma unroll
    for (int r = 0; r < 2; r++) {
      if (!base[r]) continue;
      store_vecs<float, M, vb<M>()>(base[r] + q, x[r]);
      if (SEL) {
#pragma unroll
        for (int k = 0; k < M; k++) acc->visit(x[r][k]);
      }
    }
  }
};

// Levels LEV .. S-1 on the 2 M values v[] of a lane, each band to its place
// with the deferred lifting scale.
template <int LEV, int M, int G, bool HAAR, bool FULL, typename Out>
__device__ __forceinline__ void fwd_from(const f2 (&v)[2 * M], int S, const float *scale,
                                         const Along<G> &at, Out &out) {
  const int H = M * at.lanes;  // pairs of this level
  f2 e[M], o[M];
#pragma unroll
  for (int k = 0; k < M; k++) {
    e[k] = v[2 * k];
    o[k] = v[2 * k + 1];
  }
  fwd_level<M, G, HAAR>(e, o, at);
  const f2 sc = pack(scale[LEV]);
#pragma unroll
  for (int k = 0; k < M; k++) o[k] = mul2(o[k], sc);
  out.template put_run<M>(H + M * at.seg, o);
  if constexpr (M % 2 == 0) {
    if (LEV + 1 < S) {
      fwd_from<LEV + 1, M / 2, G, HAAR, FULL>(e, S, scale, at, out);
      return;
    }
  }
  if constexpr (FULL && M == 1 && G > 1) {
    if (LEV + 1 < S) {
      // one low-pass value per lane: each further level gathers pair j into
      // lane j
      f2 s = e[0];
      Along<G> in = at;
#pragma unroll 1
      for (int lev = LEV + 1; lev < S; lev++) {
        f2 ge[1] = {at.from(s, 2 * at.seg)}, go[1] = {at.from(s, 2 * at.seg + 1)};
        in.na >>= 1;
        fwd_level<1, G, HAAR>(ge, go, in);
        if (at.seg < in.na) out.put(in.na + at.seg, mul2(go[0], pack(scale[lev])));
        s = ge[0];
      }
      if (at.seg < in.na) out.put(at.seg, mul2(s, pack(scale[S])));
      return;
    }
  }
  const f2 low = pack(scale[LEV + 1]);
#pragma unroll
  for (int k = 0; k < M; k++) e[k] = mul2(e[k], low);
  out.template put_run<M>(M * at.seg, e);
}

// v / s of both, rounded correctly (rarely called: not inline)
__device__ __noinline__ f2 divide(f2 v, float s) {
  float a, b;
  unpack(v, a, b);
  return pack(__fdiv_rn(a, s), __fdiv_rn(b, s));
}

// Magnitudes of a run: the smallest but zero, the largest (NaN above all).
struct Range {
  unsigned low = ~0u;
  float high = 0.f;
  __device__ __forceinline__ void add(float v) {
    low = min(low, (__float_as_uint(v) << 1) - 1u);  // a zero becomes the largest
    asm("max.NaN.f32 %0, %0, %1;" : "+f"(high) : "f"(fabsf(v)));
  }
  // within 2^-97 .. 2^125 or zero
  __device__ __forceinline__ bool ok() const {
    return low >= ((127u - 97u) << 24) - 1u && high <= 0x1p125f;
  }
};

// The deferred lifting scale of level t undone, as the kernel that had the
// pass before did: by its reciprocal, or (divides) by a correctly rounded
// division.  That is the quotient by the reciprocal with one correction step,
// which gives it for every scale of up to kMaxLevels levels (1/K .. K^14, so
// at most 2^3) and every significand while the quotient lies in 2^-100 ..
// 2^126, where the remainder is a float (tests/test_unscale.py); a run with
// any other value but zero is divided.  The remainder's sign is chosen so that
// a zero keeps its first quotient's: the step adds minus zero.  LOW: the
// low-pass band, whose scale is positive; the details' are negative.  The
// scales of the Haar wavelet are 1.
template <bool HAAR, bool FULL> struct Unscale {
  const float *scale, *rscale;
  bool divides;
  template <bool LOW, int M> __device__ __forceinline__ void run(f2 (&v)[M], int t) const {
    if (HAAR) return;
    const f2 r = pack(rscale[t]);
    if (!FULL || !divides) {
#pragma unroll
      for (int k = 0; k < M; k++) v[k] = mul2(v[k], r);
      return;
    }
    Range range;
#pragma unroll
    for (int k = 0; k < M; k++) {
      float a, b;
      unpack(v[k], a, b);
      range.add(a);
      range.add(b);
    }
    if (!range.ok()) {
#pragma unroll
      for (int k = 0; k < M; k++) v[k] = divide(v[k], scale[t]);
      return;
    }
    // |s| q - v or (s < 0) |s| q + v, times -|1 / s|
    const f2 s = pack(LOW ? scale[t] : -scale[t]), rn = pack(LOW ? -rscale[t] : rscale[t]);
    const f2 minus = pack(-1.0f);
#pragma unroll
    for (int k = 0; k < M; k++) {
      const f2 q = mul2(v[k], r);
      v[k] = fma2(fma2(q, s, LOW ? mul2(v[k], minus) : v[k]), rn, q);
    }
  }
  template <bool LOW> __device__ __forceinline__ f2 one(f2 v, int t) const {
    f2 x[1] = {v};
    run<LOW>(x, t);
    return x[0];
  }
};

// The 2 M values v[] of level LEV's input from the bands of levels LEV ..
// S-1.
template <int LEV, int M, int G, bool HAAR, bool FULL, typename In>
__device__ __forceinline__ void inv_to(f2 (&v)[2 * M], int S, const Unscale<HAAR, FULL> &un,
                                       const Along<G> &at, const In &in) {
  const int H = M * at.lanes;
  f2 e[M], o[M];
  in.template get_run<M>(H + M * at.seg, o);
  bool deeper = false;
  if constexpr (M % 2 == 0) {
    if (LEV + 1 < S) {
      inv_to<LEV + 1, M / 2, G, HAAR, FULL>(e, S, un, at, in);
      deeper = true;
    }
  }
  if constexpr (FULL && M == 1 && G > 1) {
    if (LEV + 1 < S) {
      // the levels below one pair per lane: lane j holds pair j
      constexpr int kDeep = G == 32 ? 5 : G == 16 ? 4 : G == 8 ? 3 : G == 4 ? 2 : 1;
      f2 dg[kDeep];
#pragma unroll
      for (int k = 0; k < kDeep; k++) {
        const int n = G >> (k + 1);
        dg[k] = LEV + 1 + k < S && at.seg < n ? un.template one<false>(in.get(n + at.seg), LEV + 1 + k) : 0ull;
      }
      const int n0 = G >> (S - LEV - 1);
      f2 s = at.seg < n0 ? un.template one<true>(in.get(at.seg), S) : 0ull;
      Along<G> now = at;
#pragma unroll
      for (int k = kDeep - 1; k >= 0; k--) {
        if (LEV + 1 + k < S) {  // the same for the whole warp
          now.na = G >> (k + 1);
          f2 se[1] = {s}, so[1] = {dg[k]};
          inv_level<1, G, HAAR>(se, so, now);
          const f2 a = at.from(se[0], at.seg >> 1), b = at.from(so[0], at.seg >> 1);
          s = at.seg & 1 ? b : a;
        }
      }
      e[0] = s;
      deeper = true;
    }
  }
  if (!deeper) {
    in.template get_run<M>(M * at.seg, e);
    un.template run<true>(e, LEV + 1);  // LEV + 1 is S here
  }
  un.template run<false>(o, LEV);
  inv_level<M, G, HAAR>(e, o, at);
#pragma unroll
  for (int k = 0; k < M; k++) {
    v[2 * k] = e[k];
    v[2 * k + 1] = o[k];
  }
}

// K elements at any address: 16- and 8-bit ones from the aligned words that
// hold them
template <typename T, int K>
__device__ __forceinline__ void load_unaligned(const T *p, float (&v)[K]) {
  if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int k = 0; k < K; k++) v[k] = load_as_float(p + k);
  } else {
    constexpr int E = 4 / (int)sizeof(T), W = K / E;
    const size_t at = reinterpret_cast<size_t>(p);
    const unsigned *w = reinterpret_cast<const unsigned *>(at & ~(size_t)3);
    const int shift = 8 * (int)(at & 3);
    unsigned lo = w[0];
#pragma unroll
    for (int j = 0; j < W; j++) {
      const unsigned hi = j + 1 < W || shift ? w[j + 1] : 0u;
      const unsigned x = __funnelshift_r(lo, hi, shift);
#pragma unroll
      for (int k = 0; k < E; k++) v[j * E + k] = from_words<T>(&x, k);
      lo = hi;
    }
  }
}

// K elements [first, first + K) of a row of n real elements (REPEAT clamp);
// ANY: whatever the row's address
template <typename T, int K, bool ANY>
__device__ __forceinline__ void load_run(const T *row, int first, int n, float (&v)[K]) {
  if (first + K <= n) {
    constexpr int VB = vec_bytes<T, K>(), VS = VB < 16 ? VB : 16;
    const size_t at = reinterpret_cast<size_t>(row + first);
    if (VB == 32 && (at & 31) == 0) load_vecs<T, K, VB>(row + first, v);
    else if (ANY && (at & (VS - 1))) load_unaligned<T, K>(row + first, v);
    else load_vecs<T, K, VS>(row + first, v);
    return;
  }
#pragma unroll
  for (int k = 0; k < K; k++) v[k] = load_as_float(row + min(first + k, n - 1));
}
template <typename T, int K>
__device__ __forceinline__ void store_run(T *row, int first, int n, const float (&v)[K]) {
  if (first + K <= n) {
    constexpr int VB = vec_bytes<T, K>();
    if (VB == 32 && (reinterpret_cast<size_t>(row + first) & 31) == 0)
      store_vecs<T, K, VB>(row + first, v);
    else
      store_vecs<T, K, VB < 16 ? VB : 16>(row + first, v);
    return;
  }
#pragma unroll
  for (int k = 0; k < K; k++)
    if (first + k < n) store_from_float(row + first + k, v[k]);
}

enum Pass { kStrided, kStridedInv, kSource, kOutput };  // y forward / inverse, x forward / inverse

template <typename T, int K, int G, bool HAAR, int PASS, bool FULL>
__device__ __forceinline__ void run_rows(const PassDesc &d, int tile, const float *scale,
                                         const float *rscale) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = G ? G : d.L / K, c = G ? Along<G>::C : 32 / g;
  const Along<G> at{lane / c, g, c, g};
  const int row = 2 * ((tile * (kThreads / 32) + warp) * c + lane % c);
  const bool ok = row < d.rows && (G || at.seg < g);
  int a = 0, b = 0;
  if (ok) {
    a = row / d.B;
    b = row - a * d.B;  // B even: b and b + 1 are one pair
  }
  Row in{nullptr, d.inSC, ok}, out{nullptr, d.outSC, ok};
  if (ok && PASS != kSource)
    in.base = const_cast<float *>(static_cast<const float *>(d.in)) + (long long)a * d.inSA + b;
  if (ok && PASS != kOutput)
    out.base = static_cast<float *>(d.out) + (long long)a * d.outSA + b;
  f2 v[K];
  if constexpr (PASS == kStrided) {
#pragma unroll
    for (int k = 0; k < K; k++) v[k] = in.get(K * at.seg + k);
  }
  if constexpr (PASS == kSource) {
    float x[2][K];
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const T *src = static_cast<const T *>(d.in) + (long long)min(a, d.clampA - 1) * d.inSA +
                     (long long)min(b + r, d.clampB - 1) * d.inSB;
      if (ok) {
        load_run<T, K, G == 0>(src, K * at.seg, min(K * g, d.clampL), x[r]);
      } else {
#pragma unroll
        for (int k = 0; k < K; k++) x[r][k] = 0.f;
      }
    }
#pragma unroll
    for (int k = 0; k < K; k++) v[k] = pack(x[0][k], x[1][k]);
  }
  if constexpr (PASS == kStrided || PASS == kSource) {
    fwd_from<0, K / 2, G, HAAR, FULL>(v, d.steps, scale, at, out);
  } else {
    inv_to<0, K / 2, G, HAAR, FULL>(v, d.steps, Unscale<HAAR, FULL>{scale, rscale, d.exact != 0}, at,
                                     in);
    if constexpr (PASS == kStridedInv) {
#pragma unroll
      for (int k = 0; k < K; k++) out.put(K * at.seg + k, v[k]);
    } else {
      if (!ok || a >= d.cropA) return;
      float x[2][K];
#pragma unroll
      for (int k = 0; k < K; k++) unpack(v[k], x[0][k], x[1][k]);
#pragma unroll
      for (int r = 0; r < 2; r++)
        if (b + r < d.cropB)
          store_run<T, K>(static_cast<T *>(d.out) + (long long)a * d.outSA +
                              (long long)(b + r) * d.outSB,
                          K * at.seg, min(K * g, d.cropL), x[r]);
    }
  }
}

template <typename T, int K, int G, int PASS, bool FULL>
__global__ void __launch_bounds__(kThreads)
dwt_strided_kernel(const PassDesc *__restrict__ passes, const int *__restrict__ tilePrefix,
                   int nPasses) {
  __shared__ float scale[16], rscale[16];
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
    scale[threadIdx.x] = s;
    rscale[threadIdx.x] = 1.0f / s;
  }
  __syncthreads();
  if (haar) run_rows<T, K, G, true, PASS, FULL>(d, bid - tilePrefix[lo], scale, rscale);
  else run_rows<T, K, G, false, PASS, FULL>(d, bid - tilePrefix[lo], scale, rscale);
}

// ---- z passes: contiguous rows, in place ----
// Lengths without a row kernel (dwt_rows.cu), which went to the column tiles
// and then needed the first select pass: the z pass of a 93 x 181 x 147 16-bit
// volume takes 18 us (23), of a 200 x 176 x 208 float volume 22 (32, and its
// select 39 instead of 45); restoring 400 cubelets of odd sizes 3.0 ms a call
// (3.4).
constexpr int kZThreads = 256;

template <int K, bool HAAR, bool INV, bool SEL>
__device__ __forceinline__ void run_z(const PassDesc &d, int pair0, const float *scale,
                                      const float *rscale, selc::SelAcc &acc) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = d.L / K, c = 32 / g;
  const Along<0> at{lane / c, g, c, g};
  const int row = 2 * (pair0 + warp * c + lane % c);
  ZRow<false> in{{nullptr, nullptr}, nullptr};
  ZRow<SEL> out{{nullptr, nullptr}, &acc};
#pragma unroll
  for (int r = 0; r < 2; r++) {
    if (row + r >= d.rows || at.seg >= g) continue;
    const int a = (row + r) / d.B, b = row + r - a * d.B;
    in.base[r] = const_cast<float *>(static_cast<const float *>(d.in)) + (long long)a * d.inSA +
                 (long long)b * d.inSB;
    out.base[r] = static_cast<float *>(d.out) + (long long)a * d.outSA + (long long)b * d.outSB;
  }
  f2 v[K];
  if constexpr (!INV) {
    in.template get_run<K>(K * at.seg, v);
    __syncwarp();  // the row's lanes have read it
    fwd_from<0, K / 2, 0, HAAR, false>(v, d.steps, scale, at, out);
  } else {
    inv_to<0, K / 2, 0, HAAR, true>(v, d.steps, Unscale<HAAR, true>{scale, rscale, d.exact != 0}, at,
                                    in);
    __syncwarp();
    out.template put_run<K>(K * at.seg, v);
  }
}

template <int K, bool INV, bool SEL>
__global__ void __launch_bounds__(kZThreads)
dwt_z_kernel(const PassDesc *__restrict__ passes, const int *__restrict__ tilePrefix, int nPasses) {
  __shared__ float scale[16], rscale[16];
  __shared__ unsigned hist[SEL ? kSelectBins : 1];
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
    scale[threadIdx.x] = s;
    rscale[threadIdx.x] = 1.0f / s;
  }
  if (SEL) selc::clear_hist<kZThreads>(hist);
  selc::SelAcc acc{hist};
  __syncthreads();
  constexpr int kRounds = K < 32 ? 32 / K : 1;  // strided_z_rounds
  const int round = (kZThreads / 32) * (32 / (d.L / K));  // pairs
  for (int r = 0; r < kRounds; r++) {
    const int pair0 = ((bid - tilePrefix[lo]) * kRounds + r) * round;
    if (2 * pair0 >= d.rows) break;  // the same for every thread of the block
    if (haar) run_z<K, true, INV, SEL>(d, pair0, scale, rscale, acc);
    else run_z<K, false, INV, SEL>(d, pair0, scale, rscale, acc);
  }
  if (SEL) selc::flush<kZThreads>(acc, d.selHist, d.selState);
}

template <bool INV, bool SEL>
void launch_z(const PassDesc *p, const int *tp, int n, int blocks, int L, cudaStream_t s) {
  switch (strided_elems(L)) {
    case 8: dwt_z_kernel<8, INV, SEL><<<blocks, kZThreads, 0, s>>>(p, tp, n); break;
    case 16: dwt_z_kernel<16, INV, SEL><<<blocks, kZThreads, 0, s>>>(p, tp, n); break;
    default: dwt_z_kernel<32, INV, SEL><<<blocks, kZThreads, 0, s>>>(p, tp, n); break;
  }
}

// launch for rows of L elements
template <typename T, int PASS, int K, int G>
void launch_kg(const PassDesc *p, const int *tp, int n, int blocks, bool full, cudaStream_t s) {
  if constexpr (K * G < 512) {
    if (!full) {
      dwt_strided_kernel<T, K, G, PASS, false><<<blocks, kThreads, 0, s>>>(p, tp, n);
      return;
    }
  }
  dwt_strided_kernel<T, K, G, PASS, true><<<blocks, kThreads, 0, s>>>(p, tp, n);
}
template <typename T, int PASS, int K>
void launch_any(const PassDesc *p, const int *tp, int n, int blocks, cudaStream_t s) {
  dwt_strided_kernel<T, K, 0, PASS, PASS == kStridedInv || PASS == kOutput>
      <<<blocks, kThreads, 0, s>>>(p, tp, n);
}
// rows of any other length: strided_elems(L) elements a lane
template <typename T, int PASS>
void launch_ragged(const PassDesc *p, const int *tp, int n, int blocks, int L, cudaStream_t s) {
  switch (strided_elems(L)) {
    case 8: launch_any<T, PASS, 8>(p, tp, n, blocks, s); break;
    case 16: launch_any<T, PASS, 16>(p, tp, n, blocks, s); break;
    default: launch_any<T, PASS, 32>(p, tp, n, blocks, s); break;
  }
}
typedef void LaunchRagged(const PassDesc *p, const int *tp, int n, int blocks, int L,
                          cudaStream_t s);
template <typename T, int PASS>
void launch_len(LaunchRagged *ragged, const PassDesc *p, const int *tp, int n, int blocks, int L, bool full,
                cudaStream_t s) {
  switch (L) {
    case 16: launch_kg<T, PASS, 16, 1>(p, tp, n, blocks, full, s); break;
    case 32: launch_kg<T, PASS, 32, 1>(p, tp, n, blocks, full, s); break;
    case 48: launch_kg<T, PASS, 48, 1>(p, tp, n, blocks, full, s); break;
    case 64: launch_kg<T, PASS, 32, 2>(p, tp, n, blocks, full, s); break;
    case 96: launch_kg<T, PASS, 48, 2>(p, tp, n, blocks, full, s); break;
    case 128: launch_kg<T, PASS, 32, 4>(p, tp, n, blocks, full, s); break;
    case 192: launch_kg<T, PASS, 48, 4>(p, tp, n, blocks, full, s); break;
    case 256: launch_kg<T, PASS, 32, 8>(p, tp, n, blocks, full, s); break;
    case 512: launch_kg<T, PASS, 32, 16>(p, tp, n, blocks, full, s); break;
    case 1024: launch_kg<T, PASS, 32, 32>(p, tp, n, blocks, full, s); break;
    case 2048: launch_kg<T, PASS, 64, 32>(p, tp, n, blocks, full, s); break;
    default: ragged(p, tp, n, blocks, L, s); break;
  }
}

}  // namespace

// the instantiations of one pass and element type, each in a file of its own
// (they are many, and compile in parallel)
#define WL_STRIDED_LAUNCH(NAME, T, PASS)                                                     \
  LaunchRagged NAME##_ragged;                                                                \
  void NAME(const PassDesc *p, const int *tp, int n, int blocks, int L, bool full,           \
            cudaStream_t s) {                                                                \
    launch_len<T, PASS>(NAME##_ragged, p, tp, n, blocks, L, full, s);                        \
  }
#define WL_RAGGED_LAUNCH(NAME, T, PASS)                                                      \
  void NAME##_ragged(const PassDesc *p, const int *tp, int n, int blocks, int L,             \
                     cudaStream_t s) {                                                       \
    launch_ragged<T, PASS>(p, tp, n, blocks, L, s);                                          \
  }

}  // namespace wl
