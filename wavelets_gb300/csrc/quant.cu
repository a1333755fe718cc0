// Quantizers fused with the Huffman frequency count, plus the zero-run
// bookkeeping the Huffman coder needs.
//
// Reference: quantize (test_compress_cpu.cc:244-295) with QuantUniform
// (quant.h:189-293), QuantLog (:326-439) and QuantCodebook (:467-558);
// huffScan (test_compress_common.cc:901-921) counts every non-zero-bin value
// and splits each run of the zero bin into "dup" tokens of 2^(v+3) elements
// (v = 0..7, greedy, longest first, HuffmanDup huffman.h:13-58) plus single
// zero-bin tokens.
//
// A token chunk of 512 to 4096 consecutive coefficients (reference Z-X-Y order)
// is one warp's.  Runs wholly inside a chunk are split there, for the counts;
// runs that touch a chunk edge are joined across chunks by runs_kernel, which
// leaves every chunk the tokens that start in it of the run entering it and of
// the run leaving it (run codes), so the encoder needs no scan over chunks.
//
// Bit exactness: the uniform quantizer is evaluated with the reference's
// unfused float operations; the log quantizer compares against per-cubelet
// bin boundaries computed on the host with the host's logf (quant_host.cpp),
// because the device has no bit-identical logf; the codebook quantizer is the
// reference's lower_bound with its last-boundary special case.
#include <cfloat>

#include <algorithm>

#include "wl_internal.h"

namespace wl {
namespace {

constexpr int kThreads = kChunkThreads;
constexpr int INF = 0x7fffffff;

// ---- quantizer parameters ---------------------------------------------------
// Copies the log quantizers' tables over from the host on its way.
__global__ void quant_params_kernel(DevBatch b, Upload up) {
  stage_mark(b.head, kMarkQuant);
  const int ci = blockIdx.x * blockDim.x + threadIdx.x;
  if (up.src)
    for (int i = ci; i < up.vecs; i += gridDim.x * blockDim.x) up.dst[i] = up.src[i];
  if (ci >= b.n) return;
  const CubeletDev cd = b.cub[ci];
  CubeletState *st = b.state + ci;
  const float thr = st->threshold, maxVal = st->maxAbs;
  const int B = cd.binCount;
  if (cd.quantAlg == WL_UNIFORM) {
    // QuantUniform::init (quant.h:196-242), unfused float operations
    const int negBinCount = (B - 1) / 2, posBinCount = B / 2;
    const float range = __fsub_rn(maxVal, thr);
    st->negScale = __fdiv_rn((float)(negBinCount - 1), range);
    st->posScale = __fdiv_rn((float)(posBinCount - 1), range);
    st->negOffset = __fsub_rn(1.0f, __fmul_rn(thr, st->negScale));
    st->posOffset = __fsub_rn(1.0f, __fmul_rn(thr, st->posScale));
    st->zeroBin = (B - 1) >> 1;
  } else if (cd.quantAlg == WL_LOG) {
    st->zeroBin = (B - 1) >> 1;
    const int4 h = *up.host(b.logHdr + ci);  // computed on the host (quant_host.cpp)
    st->lowBin = h.x;
    st->highNeg = h.y;
    st->nPos = h.z;
    st->nNeg = h.w;
  }
  // Lloyd: zeroBin is set by lloyd_solve
  if (cd.quantAlg != WL_LLOYD) st->dupValue = cd.compressZeros ? st->zeroBin : -1;
}

// number of entries of the sorted table t[0..n) that are <= x / < x, by a
// fixed number of halving steps (no divergent loop exits)
__device__ __forceinline__ int count_le(const float *t, int n, float x) {
  int pos = 0;
  for (int step = n ? 1 << (31 - __clz(n)) : 0; step > 0; step >>= 1)
    if (step <= n - pos && t[pos + step - 1] <= x) pos += step;
  return pos;
}
__device__ __forceinline__ int count_lt(const float *t, int n, float x) {
  int pos = 0;
  for (int step = n ? 1 << (31 - __clz(n)) : 0; step > 0; step >>= 1)
    if (step <= n - pos && t[pos + step - 1] < x) pos += step;
  return pos;
}

// Lloyd bin lookup table.  Floats map to an order-preserving 32-bit key
// (sign flipped for positives, all bits for negatives); cell c holds the keys
// c << 20 .. (c+1) << 20, i.e. 1/8 octave of one sign.  lut[c] counts the
// boundaries below the smallest float of cell c, so for x in the cell the
// reference's lower_bound is lut[c] plus the boundaries of
// [lut[c], lut[c+1]) that are below x.
__device__ __forceinline__ unsigned order_key(float x) {
  const unsigned u = __float_as_uint(x);
  return u ^ ((unsigned)((int)u >> 31) | 0x80000000u);
}
__device__ __forceinline__ float cell_min(int c) {
  const unsigned k = (unsigned)c << 20;
  return __uint_as_float((k & 0x80000000u) ? (k ^ 0x80000000u) : ~k);
}

// ---- Lloyd on the |coefficient| histogram -----------------------------------
__device__ __forceinline__ void lloyd_range(const CubeletState *st, float &lo, float &hi) {
  lo = st->threshold;
  hi = st->maxAbs2;  // the reference skips the largest value (test_compress_cpu.cc:419-422)
  if (!(hi > lo)) hi = st->maxAbs;
}

// The Lloyd histogram counts threshold < |c| <= hi in bins of the |c| bit
// pattern, (bits - lloydBase) >> lloydShift: above the threshold bucket the
// compaction pass of the threshold select already counted them; the bucket's
// candidates are added here once the threshold is known.
__global__ void __launch_bounds__(kThreads)
lloyd_cand_kernel(DevBatch b, const unsigned *__restrict__ cand) {
  __shared__ unsigned hist[kLloydBins];
  const int ci = blockIdx.y;
  const CubeletDev cd = b.cub[ci];
  const CubeletState *st = b.state + ci;
  const unsigned n = st->candCount;
  if (cd.quantAlg != WL_LLOYD || st->lloydDeferred || (unsigned)blockIdx.x * kThreads >= n) return;
  const unsigned lo = __float_as_uint(st->threshold), hi = st->lloydHiBits, base = st->lloydBase;
  const int shift = st->lloydShift;
  for (int i = threadIdx.x; i < kLloydBins; i += kThreads) hist[i] = 0;
  __syncthreads();
  const unsigned *src = cand + cd.coefOff;
  for (unsigned i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) {
    const unsigned a = src[i];
    if (a > lo && a <= hi) atomicAdd(&hist[(a - base) >> shift], 1u);
  }
  __syncthreads();
  unsigned *g = reinterpret_cast<unsigned *>(b.lloydHist) + (size_t)ci * kLloydBins;
  for (int i = threadIdx.x; i < kLloydBins; i += kThreads)
    if (hist[i]) atomicAdd(&g[i], hist[i]);
}

// Cubelets whose Lloyd range the select passes could not settle early (the
// second largest |c| in the threshold bucket, or bucket 0): one pass over
// their coefficients with the final threshold.
__global__ void __launch_bounds__(kThreads)
lloyd_deferred_kernel(DevBatch b, const float *__restrict__ coef) {
  __shared__ unsigned hist[kLloydBins];
  const int ci = blockIdx.y;
  const CubeletDev cd = b.cub[ci];
  const CubeletState *st = b.state + ci;
  if (cd.quantAlg != WL_LLOYD || !st->lloydDeferred) return;
  const unsigned lo = st->lloydBase, hi = st->lloydHiBits;
  const int shift = st->lloydShift;
  for (int i = threadIdx.x; i < kLloydBins; i += kThreads) hist[i] = 0;
  __syncthreads();
  const float *src = coef + cd.coefOff;
  for (long long i = blockIdx.x * (long long)kThreads + threadIdx.x; i < cd.n;
       i += (long long)gridDim.x * kThreads) {
    const unsigned a = __float_as_uint(src[i]) & 0x7fffffffu;
    if (a > lo && a <= hi) atomicAdd(&hist[(a - lo) >> shift], 1u);
  }
  __syncthreads();
  unsigned *g = reinterpret_cast<unsigned *>(b.lloydHist) + (size_t)ci * kLloydBins;
  for (int i = threadIdx.x; i < kLloydBins; i += kThreads)
    if (hist[i]) atomicAdd(&g[i], hist[i]);
}

// 512 threads and shared memory sized for the batch's largest codebook:
// four CTAs per SM, so a batch of up to 4 x 152 cubelets solves in one wave.
constexpr int kSolveThreads = 512;
// prefix sums: counts (exact in 32 bits) and count * centre (double), block
// scan scratch, then two codebook buffers (cbCap each)
__host__ __device__ inline size_t lloyd_smem_bytes(int cbCap) {
  return (size_t)(kLloydBins + 1) * 8 + (size_t)(kLloydBins + 2) * 4 + 64 * 8 +
         (size_t)2 * cbCap * 4;
}

__global__ void __launch_bounds__(kSolveThreads, 4) lloyd_solve_kernel(DevBatch b, int cbCap) {
  extern __shared__ double lsm[];
  double *pwx = lsm;
  unsigned *pw = reinterpret_cast<unsigned *>(pwx + (kLloydBins + 1));
  double *scratch = reinterpret_cast<double *>(pw + (kLloydBins + 2));
  float *cb = reinterpret_cast<float *>(scratch + 64);
  float *nxt = cb + cbCap;
  const int ci = blockIdx.x;
  const CubeletDev cd = b.cub[ci];
  if (cd.quantAlg != WL_LLOYD) return;
  CubeletState *st = b.state + ci;
  const int B = cd.binCount, cbs = (B - 1) / 2;
  float lo, hi;
  lloyd_range(st, lo, hi);
  const unsigned *g = reinterpret_cast<const unsigned *>(b.lloydHist) + (size_t)ci * kLloydBins;
  const bool degenerate = !(hi > lo) || cbs < 1;
  // histogram bin i covers |c| bits [base + i 2^shift, base + (i+1) 2^shift)
  const unsigned base = st->lloydBase;
  const int shift = st->lloydShift;
  const unsigned half = (1u << shift) >> 1;
  // first bin whose centre is >= m (m > 0)
  auto first_bin = [&](float m) {
    const long long d = (long long)__float_as_uint(m) - (long long)base - (long long)half;
    const long long a = d <= 0 ? 0 : (d + (1ll << shift) - 1) >> shift;
    return (int)min(a, (long long)kLloydBins);
  };

  // prefix sums of counts and count*centre; fixed order, so the codebook is
  // deterministic: each thread sums 8 consecutive bins, then a block scan
  {
    const int per = kLloydBins / kSolveThreads;
    auto bin_at = [&](int j, double &c, double &x) {
      const int i = threadIdx.x * per + j;
      c = degenerate ? 0.0 : (double)g[i];
      x = (double)__uint_as_float(base + ((unsigned)i << shift) + half);
    };
    double sc = 0, sx = 0;
    for (int j = 0; j < per; j++) {
      double c, x;
      bin_at(j, c, x);
      sc += c;
      sx += c * x;
    }
    // inclusive warp scan of the per-thread totals
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    double ic = sc, ix = sx;
    for (int off = 1; off < 32; off <<= 1) {
      const double tc = __shfl_up_sync(0xffffffffu, ic, off);
      const double tx = __shfl_up_sync(0xffffffffu, ix, off);
      if (lane >= off) { ic += tc; ix += tx; }
    }
    double *wc = scratch;
    double *wx = wc + 32;
    if (lane == 31) { wc[wp] = ic; wx[wp] = ix; }
    __syncthreads();
    double bc = 0, bx = 0;
    for (int v = 0; v < wp; v++) { bc += wc[v]; bx += wx[v]; }
    bc += ic - sc;
    bx += ix - sx;
    if (threadIdx.x == 0) { pw[0] = 0; pwx[0] = 0; }
    // the thread's running sums again, in the same order (same values)
    double rc = 0, rx = 0;
    for (int j = 0; j < per; j++) {
      double c, x;
      bin_at(j, c, x);
      rc += c;
      rx += c * x;
      const int i = threadIdx.x * per + j;
      pw[i + 1] = (unsigned)(bc + rc);
      pwx[i + 1] = bx + rx;
    }
    __syncthreads();
  }
  // initialLloydCodebook (test_compress_common.cc:749-779)
  if (cbs >= 1) {
    const float logScale = degenerate ? 0.f : __fdiv_rn(logf(__fdiv_rn(hi, lo)), (float)cbs);
    for (int i = threadIdx.x; i < cbs; i += kSolveThreads) cb[i] = lo * expf(i * logScale);
  }
  __syncthreads();
  // one barrier per iteration: a thread forms the midpoints around its cell
  // itself, and the codebook alternates between two buffers
  float *cur = cb, *nx = nxt;
  for (int it = 0; it < cd.lloydIters && !degenerate; it++) {
    // cell i covers histogram bins [first(i), first(i+1)): first bin whose
    // centre is >= the midpoint (cb[i-1] + cb[i]) / 2
    for (int i = threadIdx.x; i < cbs; i += kSolveThreads) {
      const float c = cur[i];
      const int a = i > 0 ? first_bin(0.5f * (cur[i - 1] + c)) : 0;
      int z = i + 1 < cbs ? first_bin(0.5f * (c + cur[i + 1])) : kLloydBins;
      if (z < a) z = a;
      const double cw = (double)(pw[z] - pw[a]);
      nx[i] = cw > 0 ? (float)((pwx[z] - pwx[a]) / cw) : c;
    }
    __syncthreads();
    float *t = cur;
    cur = nx;
    nx = t;
  }
  if (cur != cb) {
    for (int i = threadIdx.x; i < cbs; i += kSolveThreads) cb[i] = cur[i];
    __syncthreads();
  }
  // setBinsFromCodebook (test_compress_common.cc:784-846), one thread, the
  // reference's float expressions
  if (threadIdx.x == 0) {
    float *bnd = b.qtable + cd.tableOff;
    float *val = b.dqtable + (size_t)ci * kMaxBins;
    const float minVal = st->minVal, maxVal = st->maxVal, thr = st->threshold;
    int nb = 0, nv = 0;
    if (cbs < 1) {
      val[nv++] = 0;
    } else {
      if ((B & 1) == 0 && fabsf(minVal) > maxVal) {
        val[nv++] = minVal;
        bnd[nb++] = __fdiv_rn(__fadd_rn(minVal, -cb[cbs - 1]), 2.0f);
      }
      val[nv++] = -cb[cbs - 1];
      for (int i = cbs - 2; i >= 0; i--) {
        bnd[nb++] = __fdiv_rn(__fadd_rn(-cb[i], -cb[i + 1]), 2.0f);
        val[nv++] = -cb[i];
      }
      bnd[nb++] = -thr;
      val[nv++] = 0;
      bnd[nb++] = thr;
      for (int i = 0; i < cbs - 1; i++) {
        val[nv++] = cb[i];
        bnd[nb++] = __fdiv_rn(__fadd_rn(cb[i], cb[i + 1]), 2.0f);
      }
      val[nv++] = cb[cbs - 1];
      if ((B & 1) == 0 && maxVal >= fabsf(minVal)) {
        val[nv++] = maxVal;
        bnd[nb++] = __fdiv_rn(__fadd_rn(maxVal, cb[cbs - 1]), 2.0f);
      }
    }
    // QuantCodebook::quant(0) (quant.h:515-526)
    int zb;
    if (nb == 0) zb = 0;
    else if (0.0f >= bnd[nb - 1]) zb = nb;
    else {
      zb = 0;
      while (zb < nb && bnd[zb] < 0.0f) zb++;
    }
    st->zeroBin = zb;
    st->dupValue = cd.compressZeros ? zb : -1;
    st->nBounds = nb;
    st->nValues = nv;
    if (nv != B) st->error = 3;
  }
  __syncthreads();
  {
    const float *bnd = b.qtable + cd.tableOff;
    const int nb = st->nBounds;
    uint16_t *lut = b.qlut + (size_t)ci * kLutStride;
    for (int c = threadIdx.x; c < kLutCells; c += kSolveThreads) {
      const float m = cell_min(c);  // NaN cells: never looked up; keep the table monotone
      lut[c] = (uint16_t)(m != m ? (c >= kLutCells / 2 ? nb : 0) : count_lt(bnd, nb, m));
    }
    if (threadIdx.x == 0) lut[kLutCells] = (uint16_t)nb;
  }
}

// ---- quantize one value ------------------------------------------------------
struct QParams {
  int alg, B, zb;
  float thr, negScale, negOffset, posScale, posOffset;
  int nb;          // codebook boundaries / log: positive table length
  int lowBin, highNeg, nPos, nNeg;
};

__device__ __forceinline__ int quant_value(float x, const QParams &q, const float *tab,
                                           const uint16_t *lut) {
  if (q.alg == WL_UNIFORM) {
    // QuantUniform::quant (quant.h:244-276)
    if (x < 0) {
      if (x >= -q.thr) return q.zb;
      const float t = __fsub_rn(__fmul_rn(x, q.negScale), q.negOffset);
      const int bin = __float2int_rz(t) + q.zb;
      return bin < 0 ? 0 : bin;
    }
    if (x <= q.thr) return q.zb;
    const float t = __fadd_rn(__fadd_rn(__fmul_rn(x, q.posScale), q.posOffset), (float)q.zb);
    if (t > (float)(q.B - 1)) return q.B - 1;
    return __float2int_rz(t);
  }
  if (q.alg == WL_LOG) {
    // tab: [P(lowBin+1 .. B-1)] then [N(0 .. highNeg-1)], nondecreasing
    if (x < 0) {
      const float y = -x;
      if (y <= q.thr) return q.zb;
      return q.highNeg - count_le(tab + q.nPos, q.nNeg, y);
    }
    if (x <= q.thr) return q.zb;
    return q.lowBin + count_le(tab, q.nPos, x);
  }
  // QuantCodebook::quant (quant.h:515-526): x >= last boundary -> nb, else
  // lower_bound (the number of boundaries below x; 0 for NaN)
  if (q.nb == 0 || x != x) return 0;
  if (x >= tab[q.nb - 1]) return q.nb;
  const int c = (int)(order_key(x) >> 20);
  const int lo = lut[c], hi = lut[c + 1];
  // a cell (1/8 octave) rarely holds more than two boundaries: compare with
  // them directly, search only when there are more
  if (hi - lo <= 2) {
    const int n = hi - lo;
    return lo + (n > 0 && tab[lo] < x ? 1 : 0) + (n > 1 && tab[lo + 1] < x ? 1 : 0);
  }
  return lo + count_lt(tab + lo, hi - lo, x);
}

__device__ __forceinline__ QParams load_qparams(const CubeletDev &cd, const CubeletState *st) {
  QParams q;
  q.alg = cd.quantAlg;
  q.B = cd.binCount;
  q.zb = st->zeroBin;
  q.thr = st->threshold;
  q.negScale = st->negScale;
  q.negOffset = st->negOffset;
  q.posScale = st->posScale;
  q.posOffset = st->posOffset;
  q.nb = 0; q.lowBin = 0; q.highNeg = 0; q.nPos = 0; q.nNeg = 0;
  if (q.alg == WL_LLOYD) q.nb = st->nBounds;
  if (q.alg == WL_LOG) {  // table layout written by the host
    q.lowBin = st->lowBin;
    q.highNeg = st->highNeg;
    q.nPos = st->nPos;
    q.nNeg = st->nNeg;
  }
  return q;
}

// ---- quantize + count + values of the chunk ----------------------------------
// Instead of storing a bin per coefficient, a chunk stores its values -- the
// elements that are not the zero bin -- in order, each with the gap to the
// value before it in the chunk (make_item).  The bit packer turns a gap into
// the zero-bin run's Huffman tokens.  Runs touching a chunk edge are left to
// runs_kernel.
//
// One warp codes one chunk from its first element to its last, so nothing but
// the tables and the histogram is shared and there is no barrier inside.  It
// reads kBlock = 512 elements at a time, 16 consecutive ones per lane (the
// next block's loads are in flight meanwhile):
//  - -thr < x < thr is the zero bin for all three quantizers (uniform and log
//    test |x| <= thr first; the codebook has the boundaries -thr and thr
//    around its zero bin and none in between), so an element costs a compare;
//    the positions of the others, the candidates, are appended in order to
//    the warp's queue (a scan over the lanes' counts places them);
//  - whenever the queue holds 32 candidates, one per lane, a round gives each
//    its exact bin (its value is read again, from L1); those that are not the
//    zero bin are values.  A value's gap to the one before it (the nearest
//    lower lane with one, else the last value of earlier rounds) gives the
//    count of its run's tokens, and its item goes out.
// Full rounds whatever the density, and no work for the zero bin beyond the
// compare.  The mixed batch (376 M coefficients, 10% kept) quantizes in 0.49
// ms, 729 cubelets of 128^3 (1.5 G, 3%) in 1.37 ms; 0.76 and 2.85 ms with
// eight warps to a chunk that met at a barrier and every token written out
// here.  Bound by its instructions: 0.87 a coefficient of the mixed batch (1.83
// with the tokens written out).
// Greedy split of a zero-bin run into dup tokens and single zero-bin tokens
// (HuffmanDup::dupCount, huffman.h:46-57) in closed form: runs of 1024, then
// one dup token per set bit of the remainder at or above 8 -- except that a
// last 8 left over is coded as 8 single tokens.
__device__ __forceinline__ void run_split_closed(int L, int &singles, int &dups) {
  const int q = L >> 10, r = L & 1023, hi = r & ~7, lo = r & 7;
  const int big = __popc(hi >> 4);
  if (hi & 8) {
    dups = q + big + (lo > 0 ? 1 : 0);
    singles = lo > 0 ? lo : 8;
  } else {
    dups = q + big;
    singles = lo;
  }
}

constexpr int kBlock = 512, kLaneRun = kBlock / 32;
constexpr int kQueue = 576;  // less than 32 left over and a block's candidates

__global__ void __launch_bounds__(32 * kQuantWarps, 4)
quantize_kernel(DevBatch b, const float *__restrict__ coef, int histOff, int lutOff, int warpOff) {
  constexpr unsigned kAll = 0xffffffffu;
  // sized by the launch: the quantizer table (Lloyd / log), the counts of the
  // batch's largest alphabet, the Lloyd cell table, then the warps' queues
  extern __shared__ __align__(16) float tab[];
  unsigned *hist = reinterpret_cast<unsigned *>(tab + histOff);
  uint16_t *lut = reinterpret_cast<uint16_t *>(tab + lutOff);
  const int ci = b.quantCub[blockIdx.x];
  const CubeletDev cd = b.cub[ci];
  const CubeletState *st = b.state + ci;
  const QParams q = load_qparams(cd, st);
  const int dupV = st->dupValue;
  const int B = cd.binCount;
  const int nTab = q.alg == WL_LLOYD ? q.nb : (q.alg == WL_LOG ? q.nPos + q.nNeg : 0);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int c = ((int)blockIdx.x - cd.quantBase) * kQuantWarps + w;  // the warp's chunk
  const unsigned ltMask = (1u << lane) - 1u;
  // zero-bin elements (-thr < x < thr) can be skipped only when they are
  // coded as runs; without runs every element is a candidate (|x| < 0 never)
  const float zthr = dupV >= 0 ? q.thr : 0.f;
  uint16_t *queue = reinterpret_cast<uint16_t *>(tab + warpOff) + w * kQueue;

  for (int i = threadIdx.x; i < B + 1; i += blockDim.x) hist[i] = 0;
  for (int i = threadIdx.x; i < nTab; i += blockDim.x) tab[i] = b.qtable[cd.tableOff + i];
  if (q.alg == WL_LLOYD) {
    const uint4 *gl = reinterpret_cast<const uint4 *>(b.qlut + (size_t)ci * kLutStride);
    uint4 *sl = reinterpret_cast<uint4 *>(lut);
    for (int i = threadIdx.x; i < kLutStride / 8; i += blockDim.x) sl[i] = gl[i];
  }
  __syncthreads();

  if (c < cd.nChunks) {
    const long long start = (long long)c << b.lgChunk;
    const int len = (int)min(1LL << b.lgChunk, cd.n - start);
    const float *src = coef + cd.coefOff + start;
    unsigned *items = b.items + cd.coefOff + start;
    int singles = 0, dups = 0;           // the lane's zero-run tokens
    int lead = -1, last = -1, nVal = 0;  // warp-uniform: first and last value, values so far

    // one round: candidates queue[at .. at + n), n <= 32
    auto round = [&](int at, int n) {
      const int pos = lane < n ? queue[at + lane] : 0;
      const int bin = quant_value(src[pos], q, tab, lut);
      const bool v = lane < n && bin != dupV;
      const unsigned m = __ballot_sync(kAll, v);
      if (m == 0) return;
      const unsigned lower = m & ltMask;
      const int pp = __shfl_sync(kAll, pos, lower ? 31 - __clz(lower) : 0);
      const int prev = lower ? pp : last;
      if (v) {
        const int gap = prev >= 0 ? pos - prev - 1 : 0;
        int sg, dp;
        run_split_closed(gap, sg, dp);  // 0, 0 for gap 0
        singles += sg;
        dups += dp;
        items[nVal + __popc(lower)] = make_item(bin, gap);
        atomicAdd(&hist[bin], 1u);
      }
      if (lead < 0) lead = __shfl_sync(kAll, pos, __ffs(m) - 1);
      last = __shfl_sync(kAll, pos, 31 - __clz(m));
      nVal += __popc(m);
    };

    float x[kLaneRun];
    auto load = [&](int base) {
      const int p0 = base + kLaneRun * lane;
      if (p0 + kLaneRun <= len) {
        const float4 *s4 = reinterpret_cast<const float4 *>(src + p0);
#pragma unroll
        for (int k = 0; k < kLaneRun / 4; k++) {
          const float4 f = s4[k];
          x[4 * k] = f.x; x[4 * k + 1] = f.y; x[4 * k + 2] = f.z; x[4 * k + 3] = f.w;
        }
      } else {
#pragma unroll
        for (int k = 0; k < kLaneRun; k++) x[k] = p0 + k < len ? src[p0 + k] : 0.f;
      }
    };
    load(0);
    int nq = 0;  // candidates in the queue
    for (int base = 0; base < len; base += kBlock) {
      unsigned mask = 0;
#pragma unroll
      for (int k = 0; k < kLaneRun; k++)
        if (!(fabsf(x[k]) < zthr)) mask |= 1u << k;  // NaN is a candidate
      const int p0 = base + kLaneRun * lane;
      if (p0 + kLaneRun > len) mask &= p0 < len ? (1u << (len - p0)) - 1u : 0u;
      if (base + kBlock < len) load(base + kBlock);
      const int cnt = __popc(mask);
      int inc = cnt;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(kAll, inc, d);
        if (lane >= d) inc += t;
      }
      int o = nq + inc - cnt;
#pragma unroll
      for (int k = 0; k < kLaneRun; k++)
        if ((mask >> k) & 1u) queue[o++] = (uint16_t)(p0 + k);
      nq += __shfl_sync(kAll, inc, 31);
      __syncwarp();
      int at = 0;
      for (; nq - at >= 32; at += 32) round(at, 32);
      if (at) {  // what is left moves to the front
        nq -= at;
        const int left = lane < nq ? queue[at + lane] : 0;
        __syncwarp();
        if (lane < nq) queue[lane] = (uint16_t)left;
        __syncwarp();
      }
    }
    if (nq) round(0, nq);

    if (lane == 0) {
      const long long chunk = cd.chunkBase + c;
      const bool any = last >= 0;
      b.chunkVal[chunk] = nVal;
      b.chunkRun[chunk] = make_int4(any ? lead : len, any ? len - 1 - last : len, any ? 0 : 1, len);
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      singles += __shfl_xor_sync(kAll, singles, d);
      dups += __shfl_xor_sync(kAll, dups, d);
    }
    if (lane == 0 && dupV >= 0) {
      if (singles) atomicAdd(&hist[dupV], (unsigned)singles);
      if (dups) atomicAdd(&hist[B], (unsigned)dups);
    }
  }
  __syncthreads();
  unsigned long long *gh = b.hist + (size_t)ci * kMaxSymbols;
  for (int i = threadIdx.x; i <= B; i += blockDim.x)
    if (hist[i]) atomicAdd(&gh[i], (unsigned long long)hist[i]);
}

// Join zero runs across chunk edges: the tokens of the runs entering and
// leaving every chunk that start in it (run codes), and their counts.  A CTA takes kRunChunks consecutive
// chunks of one cubelet (blockIdx.y), one thread each; the nearest chunks
// with a value before and after the CTA's range are searched kRunChunks at a
// time, usually found in the first step, whose loads are issued with the
// CTA's own.  Bound by the latency of a few dependent loads: one CTA of 1024 threads per cubelet left most SMs idle (59
// us for a 2048^2 image of 1024 chunks, 93 us for a 256^3 volume); spread
// over the SMs a whole call went from 523 to 468 us and from 623 to 529 us.
constexpr int kRunChunks = 256;

__global__ void __launch_bounds__(kRunChunks) runs_kernel(DevBatch b) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int kWarps = kRunChunks / 32;
  __shared__ unsigned sMask[kWarps];
  __shared__ int sPrev, sNext;
  const int ci = blockIdx.y;
  const CubeletDev cd = b.cub[ci];
  const int nc = cd.nChunks, c0 = (int)blockIdx.x * kRunChunks;
  if (c0 >= nc) return;
  const int dupV = b.state[ci].dupValue;
  if (dupV < 0) return;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int4 *cr = b.chunkRun + cd.chunkBase;
  const int c = c0 + tid;
  // chunks past the end count as all zero and are not written
  const int4 me = c < nc ? cr[c] : make_int4(0, 0, 1, 0);
  const bool val = !me.z;  // the chunk holds a value
  const int back = c0 - 1 - tid, ahead = c0 + kRunChunks + tid;
  bool hitB = back >= 0 && !cr[back].z, hitA = ahead < nc && !cr[ahead].z;
  if (tid == 0) {
    sPrev = -1;
    sNext = INF;
  }
  const unsigned m = __ballot_sync(kAll, val);
  if (lane == 0) sMask[w] = m;
  __syncthreads();
  // nearest chunks with a value before and after the CTA's range
  for (int k = 0;; k++) {
    const unsigned mb = __ballot_sync(kAll, hitB), ma = __ballot_sync(kAll, hitA);
    if (lane == 0) {
      const int o = k * kRunChunks + 32 * w;
      if (mb) atomicMax(&sPrev, c0 - 1 - (o + __ffs(mb) - 1));
      if (ma) atomicMin(&sNext, c0 + kRunChunks + o + __ffs(ma) - 1);
    }
    __syncthreads();
    const bool fb = sPrev >= 0 || c0 - (k + 1) * kRunChunks <= 0;
    const bool fa = sNext != INF || c0 + (k + 2) * kRunChunks >= nc;
    if (fb && fa) break;
    __syncthreads();  // everyone has read this step's result
    const int pb = back - (k + 1) * kRunChunks, pa = ahead + (k + 1) * kRunChunks;
    hitB = !fb && pb >= 0 && !cr[pb].z;
    hitA = !fa && pa < nc && !cr[pa].z;
  }
  // and of this chunk
  int prev = -1, next = INF;
  const unsigned lo = m & ((1u << lane) - 1u), hi = m & ~((2u << lane) - 1u);
  if (lo) {
    prev = c0 + 32 * w + 31 - __clz(lo);
  } else {
    for (int v = w - 1; v >= 0 && prev < 0; v--)
      if (sMask[v]) prev = c0 + 32 * v + 31 - __clz(sMask[v]);
    if (prev < 0) prev = sPrev;
  }
  if (hi) {
    next = c0 + 32 * w + __ffs(hi) - 1;
  } else {
    for (int v = w + 1; v < kWarps && next == INF; v++)
      if (sMask[v]) next = c0 + 32 * v + __ffs(sMask[v]) - 1;
    if (next == INF) next = sNext;
  }

  int singles = 0, dups = 0;
  if (c < nc) {
    const int n = (int)cd.n;  // positions stay below 2^31
    int runIn = 0, e = n;
    if (prev >= 0) {
      const int4 o = cr[prev];
      runIn = (prev << b.lgChunk) + o.w - o.y;
    }
    if (next != INF) e = (next << b.lgChunk) + cr[next].x;
    if (val) run_split_closed(e - ((c << b.lgChunk) + me.w - me.y), singles, dups);
    if (c == 0) {  // the run starting at element 0 belongs to no chunk's tail
      int sg, dp;
      run_split_closed(val ? me.x : e, sg, dp);
      singles += sg;
      dups += dp;
    }
    // the tokens that start in this chunk of the run entering it and of the
    // one leaving it
    const int cstart = c << b.lgChunk, cend = cstart + me.w;
    uint2 edge = make_uint2(0u, 0u);
    if (me.x > 0)
      edge.x = run_code_in(runIn, val ? cstart + me.x : e, cstart, val ? cstart + me.x : cend);
    if (val && me.y > 0) edge.y = run_code_in(cend - me.y, e, cend - me.y, cend);
    b.chunkEdge[cd.chunkBase + c] = edge;
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    singles += __shfl_xor_sync(kAll, singles, d);
    dups += __shfl_xor_sync(kAll, dups, d);
  }
  if (lane == 0) {
    unsigned long long *gh = b.hist + (size_t)ci * kMaxSymbols;
    if (singles) atomicAdd(&gh[dupV], (unsigned long long)singles);
    if (dups) atomicAdd(&gh[cd.binCount], (unsigned long long)dups);
  }
}

}  // namespace

void launch_quant_params(DevBatch &b, const Upload &up, cudaStream_t s) {
  const int copy = up.src ? std::min((up.vecs + 127) / 128, 1024) : 0;
  quant_params_kernel<<<std::max((b.n + 127) / 128, copy), 128, 0, s>>>(b, up);
}

void launch_lloyd(DevBatch &b, const float *coef, int maxBins, cudaStream_t s) {
  lloyd_cand_kernel<<<dim3(kCandSlices, b.n), kThreads, 0, s>>>(
      b, reinterpret_cast<const unsigned *>(b.coef2));
  lloyd_deferred_kernel<<<dim3(kCandSlices, b.n), kThreads, 0, s>>>(b, coef);
  const int cbCap = ((maxBins / 2 + 1) + 3) & ~3;
  const int smem = (int)lloyd_smem_bytes(cbCap);
  raise_smem_limit(lloyd_solve_kernel, smem);
  lloyd_solve_kernel<<<b.n, kSolveThreads, smem, s>>>(b, cbCap);
}

void launch_quantize(DevBatch &b, const float *coef, int maxTable, int maxSymbols, bool lloyd,
                     cudaStream_t s) {
  const int histOff = (maxTable + 3) & ~3;
  const int lutOff = (histOff + maxSymbols + 1 + 3) & ~3;
  const int warpOff = lutOff + (lloyd ? kLutStride / 2 : 0);
  const int smem = warpOff * (int)sizeof(float) + kQuantWarps * kQueue * 2;
  raise_smem_limit(quantize_kernel, smem);
  quantize_kernel<<<(unsigned)b.totalQuant, 32 * kQuantWarps, smem, s>>>(b, coef, histOff, lutOff,
                                                                          warpOff);
}

void launch_runs(DevBatch &b, cudaStream_t s) {
  runs_kernel<<<dim3((b.maxChunks + kRunChunks - 1) / kRunChunks, b.n), kRunChunks, 0, s>>>(b);
}

}  // namespace wl
