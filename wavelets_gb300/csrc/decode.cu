// Huffman decoding on the device for streams without any index (files the
// reference wrote decode too), a batch of streams at a time, straight to the
// dequantized values.
//
// Reference: HuffmanDecoder::decodeFromStream (huffman.h:96-131) walks the
// breadth-first decode table bit by bit; a zero-run key is followed by 3
// length bits and expands to 2^(v+3) copies of the zero bin.
//
// The stream is cut into subsequences of 256 bits, one thread each, and a CTA
// decodes a tile of kTileSubs consecutive ones:
//  - tile_kernel: every thread decodes speculatively from its first bit to
//    the end of its subsequence and keeps the last token boundary in each of
//    its words.  Huffman codes resynchronise after some tokens, so a thread's
//    exit (the first boundary past its end) rarely depends on where it
//    started.  Then, in rounds inside the CTA, a thread whose start differs
//    from its predecessor's exit decodes again from there until it is on the
//    speculative path at one of those words.  Thread 0 decodes the
//    subsequence before the tile only to find the tile's entry.
//  - check_kernel: a tile whose entry is not the exit of the tile before it
//    (rare: no resynchronisation within a subsequence) is decoded again from
//    that exit.  It is launched twice; the second launch changes nothing
//    unless a chain of tiles was wrong, which the host sees at the end and
//    repairs with more launches (codes that never resynchronise, e.g. all of
//    one length).
//  - scan_kernel: output offset of every tile.
//  - write_kernel: decodes each subsequence from its true start, lists the
//    tile's values in shared memory and writes the output a window at a time.
// A token costs two shared-memory reads of the stream and one of a 12-bit
// table that also expands zero-run lengths where they fit; longer codes go on
// four bits at a time.
//
// Bound by the latency of the token chain on small streams, which is why a
// thread has only 256 bits and nothing waits on the host between the passes:
// with 1024 bits a thread, tables in global memory and a host wait after
// every round, decoding a 2048^2 image (4.7 Mbit) took 830 us of a 1213 us
// call.  A wrong start is found out a word at a time: with only the first
// eight boundaries recorded a warp went through its bits five times over
// (tile_kernel 62 us, and 520 us for the mixed batch of 512, 464 Mbit);
// recorded per word it takes 34 and 345 us.
#include <cstring>

#include "wl_internal.h"

namespace wl {
namespace {

constexpr int kThreads = 256;
constexpr int kSubBits = 256, kSubWords = kSubBits / 32;
constexpr int kTileSubs = kThreads - 1;      // thread 0 warms up on the one before
constexpr int kTileBits = kTileSubs * kSubBits;
constexpr int kTileWords = kTileSubs * kSubWords;
constexpr int kLutBits = kDecodeLutBits, kLutSize = 1 << kLutBits;
constexpr int kStepBits = kDecodeStepBits, kStep = 1 << kStepBits;  // longer codes, per step
// step tables kept in shared memory: the first ones built belong to the
// shortest of the long codes (a global read of a step costs the whole warp
// several hundred cycles, and with 1024 bins most warps have one per token)
constexpr int kStageSteps = 128;
// words of a tile in shared memory: kThreads subsequences of 8 words and the
// longest token past the end; after every eighth word the next one again, so
// that words k and k + 1 are always neighbours, which also spreads the
// threads' words over the banks (stride 9)
constexpr int kStageWords = kThreads * kSubWords + 4;
constexpr int kStageSize = kStageWords + kStageWords / 8 + 1;
constexpr int kBuildNodes = 2 * kMaxSymbols;  // decode tables staged in shared memory

// Table entry.  Token: bits 0-5 bits consumed, 6-9 log2 of its elements,
// 10-22 symbol.  kSlow: kRun: the zero-run key with a code of bits 0-5 bits
// whose length bits come after it (kBad: malformed table), else bits 0-28
// the step table to go on with.
constexpr unsigned kSlow = 1u << 31, kRun = 1u << 30, kBad = 1u << 29, kSlots = kBad - 1;

struct TileAt {
  int tile;    // tile of the cubelet
  int tot;     // bits of the stream from the staged words' start (bounded)
};

// stage the words of a tile: local subsequence s (thread s) is subsequence
// kTileSubs * tile + s - 1 of the stream
__device__ __forceinline__ TileAt stage_words(const DecodeCub &c, int tile, uint32_t *sw) {
  TileAt t;
  t.tile = tile;
  const long long w0 = (long long)tile * kTileWords - kSubWords;
  for (int k = threadIdx.x; k < kStageWords; k += kThreads) {
    const long long g = w0 + k;
    const uint32_t v = g >= 0 && g < c.nWords ? c.words[g] : 0u;
    sw[k + (k >> 3)] = v;
    if ((k & 7) == 0 && k > 0) sw[k + (k >> 3) - 1] = v;
  }
  const long long bits = (c.nWords - w0) * 32;
  t.tot = (int)min(bits, (long long)2 * kTileBits);
  return t;
}
// A stream's tables for one CTA: the 12-bit table and the first `nNear` step
// tables in shared memory, the other step tables in global memory.
struct Tables {
  const unsigned *lut, *near, *steps;
  int nNear;
};
__device__ __forceinline__ void stage_lut(const DecodeCub &c, const DecodeArrays &d,
                                          unsigned *lut) {
  const uint4 *g = reinterpret_cast<const uint4 *>(d.lut + c.lutOff);
  uint4 *s = reinterpret_cast<uint4 *>(lut);
#pragma unroll
  for (int i = 0; i < kLutSize / 4 / kThreads; i++)
    s[threadIdx.x + i * kThreads] = g[threadIdx.x + i * kThreads];
}
__device__ __forceinline__ Tables stage_steps(const DecodeCub &c, const DecodeArrays &d, int ci,
                                              const unsigned *lut, unsigned *near, int room) {
  const Tables t{lut, near, d.steps + (size_t)c.stepOff * kStep, min(d.stepCount[ci], room)};
  const uint4 *g = reinterpret_cast<const uint4 *>(t.steps);
  uint4 *s = reinterpret_cast<uint4 *>(near);
  for (int i = threadIdx.x; i < t.nNear * (kStep / 4); i += kThreads) s[i] = g[i];
  return t;
}
__device__ __forceinline__ unsigned bits_at(const uint32_t *sw, int p) {
  const int k = p >> 5, a = k + (k >> 3);
  return __funnelshift_r(sw[a], sw[a + 1], p & 31);
}

// a code longer than the table, or a zero-run key whose length bits are
// outside it: the token in the table's format, 0 when malformed
__device__ __noinline__ unsigned slow_token(const uint32_t *sw, const unsigned *near,
                                            const unsigned *steps, int nNear, int p, unsigned e,
                                            int dupValue) {
  unsigned used = 0, width = kLutBits;
  while (e & kSlow) {
    if (e & kRun) {
      if (e & kBad) return 0;
      used += e & 63u;
      const unsigned lg = (bits_at(sw, p + used) & 7u) + 3;
      return (used + 3) | (lg << 6) | ((unsigned)dupValue << 10);
    }
    used += width;
    width = kStepBits;
    const int slot = (int)(e & kSlots);
    const unsigned at = slot * kStep + (bits_at(sw, p + used) & (kStep - 1));
    e = slot < nNear ? near[at] : steps[at];
  }
  return e + used;  // at most 60 bits
}

// the token at bit p of the staged words: bits consumed in bits 0-5 (0:
// malformed), log2 of its elements in 6-9, its symbol above
__device__ __forceinline__ unsigned token_at(const uint32_t *sw, const Tables &t, int p,
                                             int dupValue) {
  const unsigned e = t.lut[bits_at(sw, p) & (kLutSize - 1)];
  return e & kSlow ? slow_token(sw, t.near, t.steps, t.nNear, p, e, dupValue) : e;
}

// Elements of tokens, and above them how many are values to write (not the
// zero bin): a subsequence of 256 bits and a token has less than 2^17 and 2^9.
constexpr int kCountBits = 17, kRecShift = 26;
__device__ __forceinline__ unsigned token_count(unsigned e, int dupValue) {
  return (1u << ((e >> 6) & 15u)) + ((int)(e >> 10) != dupValue ? 1u << kCountBits : 0u);
}

struct TileSmem {
  __align__(16) unsigned lut[kLutSize];
  __align__(16) unsigned near[kStageSteps * kStep];
  uint32_t sw[kStageSize];
  // last token boundary of the speculative decode in each word: the bit in
  // bits 26-30, the counts before it below; all ones: none
  unsigned rec[kSubWords][kThreads];
  int exits[kThreads];
  unsigned sums[kThreads / 32];
};

// Decode a tile; entry: the tile's true first token boundary (bits past the
// tile's first bit), or -1 to find it speculatively.  Writes the start and
// counts of every subsequence and the tile's entry, exit and total.
__device__ void decode_tile(const DecodeCub &c, const DecodeArrays &d, int t, TileSmem &sm,
                            int entry) {
  constexpr unsigned kAll = 0xffffffffu;
  const int tile = t - c.tileBase, tid = threadIdx.x;
  const int dupValue = c.dupValue;
  const TileAt at = stage_words(c, tile, sm.sw);
  stage_lut(c, d, sm.lut);
  const Tables tab = stage_steps(c, d, d.tileCub[t], sm.lut, sm.near, kStageSteps);
  __syncthreads();
  const long long sub = (long long)tile * kTileSubs + tid - 1;  // subsequence of the stream
  const bool active = sub >= 0 && sub < c.nSub;
  const int s0 = tid * kSubBits, lim = active ? min(s0 + kSubBits, at.tot) : s0;
  bool bad = false;
  int p = s0;
  unsigned n = 0;
#pragma unroll
  for (int j = 0; j < kSubWords; j++) sm.rec[j][tid] = ~0u;
  while (p < lim) {
    sm.rec[(p - s0) >> 5][tid] = ((unsigned)(p & 31) << kRecShift) | n;
    const unsigned e = token_at(sm.sw, tab, p, dupValue);
    if ((e & 63u) == 0) { bad = true; break; }
    p += (int)(e & 63u);
    n += token_count(e, dupValue);
  }
  // A malformed token ends its subsequence: the exit is the next one's first
  // bit, never a bit before it, and nothing is counted.  (The host refuses the
  // tables that hold such tokens; whatever a table holds, a start lies in its
  // subsequence or past it and the write pass stays inside the counts.)
  if (bad) {
    p = s0 + kSubBits;
    n = 0;
  }
  const int x0 = p;           // the speculative exit and counts
  const unsigned n0 = n;
  int start = s0;
  // the first tile starts with the stream
  if (tid == 0 && tile == 0) p = kSubBits;
  if (tid == 0 && entry >= 0) p = kSubBits + entry;

  // rounds: each fixes at least the first wrong subsequence
  for (;;) {
    sm.exits[tid] = p;
    __syncthreads();
    const int ns = tid > 0 ? sm.exits[tid - 1] : start;
    bool changed = false;
    if (active && tid > 0 && ns != start && !bad) {
      bad = ns < s0;
      start = bad ? s0 : ns;
      int q = start;
      unsigned m = 0;
      while (q < lim && !bad) {
        const unsigned r = sm.rec[(q - s0) >> 5][tid];
        if (r >> kRecShift == (unsigned)(q & 31)) {  // on the speculative path from here
          m += n0 - (r & ((1u << kRecShift) - 1));
          q = x0;
          break;
        }
        const unsigned e = token_at(sm.sw, tab, q, dupValue);
        if ((e & 63u) == 0) { bad = true; break; }
        q += (int)(e & 63u);
        m += token_count(e, dupValue);
      }
      if (bad) {
        q = s0 + kSubBits;
        m = 0;
      }
      changed = q != p;
      p = q;
      n = m;
    }
    if (!__syncthreads_or(changed)) break;
  }
  const bool out = active && tid > 0;
  if (out) {
    d.subStart[c.subBase + sub] = (uint8_t)(start - s0);
    d.subCount[c.subBase + sub] = n;
  }
  unsigned sum = out ? n & ((1u << kCountBits) - 1) : 0u;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(kAll, sum, o);
  if ((tid & 31) == 0) sm.sums[tid >> 5] = sum;
  if (tid == 1) d.tileEntry[t] = start - s0;
  if (tid == kThreads - 1) d.tileExit[t] = p - (s0 + kSubBits);
  if (bad) atomicAdd(&d.flags[kDecodeBad], 1);
  __syncthreads();
  if (tid == 0) {
    unsigned all = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; w++) all += sm.sums[w];
    d.tileCount[t] = all;
  }
}

__global__ void __launch_bounds__(kThreads) tile_kernel(const DecodeCub *__restrict__ cubs,
                                                        DecodeArrays d) {
  extern __shared__ __align__(16) unsigned char dsm[];
  const DecodeCub c = cubs[d.tileCub[blockIdx.x]];
  decode_tile(c, d, blockIdx.x, *reinterpret_cast<TileSmem *>(dsm), -1);
}

// flag: counter of tiles decoded again
__global__ void __launch_bounds__(kThreads) check_kernel(const DecodeCub *__restrict__ cubs,
                                                         DecodeArrays d, int flag) {
  extern __shared__ __align__(16) unsigned char dsm[];
  __shared__ int entry;
  const int t = blockIdx.x;
  const DecodeCub c = cubs[d.tileCub[t]];
  if (t == c.tileBase) return;
  // read once for the CTA: the tile before may be decoded again meanwhile
  // (the next launch then sees its new exit)
  if (threadIdx.x == 0) {
    const int e = d.tileExit[t - 1];
    entry = e == d.tileEntry[t] ? -1 : e;
  }
  __syncthreads();
  const int e = entry;
  if (e < 0) return;
  if (threadIdx.x == 0) atomicAdd(&d.flags[flag], 1);
  decode_tile(c, d, t, *reinterpret_cast<TileSmem *>(dsm), e);
}

// per cubelet: exclusive scan of its tiles' element counts
__global__ void __launch_bounds__(kThreads) scan_kernel(const DecodeCub *__restrict__ cubs,
                                                        DecodeArrays d) {
  __shared__ long long sh[kThreads / 32];
  const DecodeCub c = cubs[blockIdx.x];
  long long carry = 0;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int seg = 0; seg < c.nTiles; seg += kThreads) {
    const int j = seg + threadIdx.x;
    const long long v = j < c.nTiles ? d.tileCount[c.tileBase + j] : 0;
    long long inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long x = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += x;
    }
    if (lane == 31) sh[w] = inc;
    __syncthreads();
    long long before = 0, all = 0;
#pragma unroll
    for (int k = 0; k < kThreads / 32; k++) {
      if (k < w) before += sh[k];
      all += sh[k];
    }
    if (j < c.nTiles) d.tileOff[c.tileBase + j] = carry + before + inc - v;
    carry += all;
    __syncthreads();
  }
  // fewer values than the cubelet holds
  if (threadIdx.x == 0 && carry < c.n) atomicAdd(&d.flags[kDecodeShort], 1);
}

// Shared memory of write_kernel: with kPool words four CTAs fit on an SM.  The
// pool holds the list of the tile's values and, before them, the step tables
// that fit (kMinNear at least, else the values are written one by one).
constexpr int kPool = 7600, kMinNear = 16, kWindow = 6400;
constexpr int kPosBits = 19;  // elements of a listed tile, a bin above them
struct WriteSmem {
  union {
    struct {
      __align__(16) unsigned lut[kLutSize];
      uint32_t sw[kStageSize];
    };
    float4 window[kWindow / 4];  // once the tile is decoded
  };
  __align__(16) unsigned pool[kPool];
  uint2 sums[kThreads / 32];
};

// The values, from each subsequence's true start.
//
// With zero runs (dupValue >= 0) a tile's output is mostly the zero bin's
// value.  All threads decode their subsequences at once into a list of the
// tile's values, then the output goes by in windows: a window of the zero
// bin's value in shared memory, the list's next values into it, and out with
// 16-byte stores, every output line written once.  Writing the values one by
// one over a filled output cost the mixed batch 0.90 ms (the lines of all
// resident tiles, some 200 MB, do not stay in L2 between fill and value; every
// value is a partial sector); this way 0.55 ms
// (volume 256^3: 52 -> 51 us, one tile per SM).  Step tables beyond the pool
// are read from memory: with 64 of them the volume's 1024 bins took 57 us.
//
// Tiles with more values than the pool holds are filled and written one by
// one; so are sparse cubelets, whose tiles cover so much output that one CTA
// would be long at it (filled beforehand by launch_fill_batch,
// DecodeCub::fill 0), and streams without zero runs, which have no fill.
__global__ void __launch_bounds__(kThreads) write_kernel(const DecodeCub *__restrict__ cubs,
                                                         DecodeArrays d) {
  constexpr unsigned kAll = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char dsm[];
  WriteSmem &sm = *reinterpret_cast<WriteSmem *>(dsm);
  const int t = blockIdx.x, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const DecodeCub c = cubs[d.tileCub[t]];
  const long long tileOff = d.tileOff[t];
  // the launches before settled the flags; the host looks at them before it
  // lets anything reach the outputs
  const int refused = d.flags[kDecodeBad];
  if (t == 0 && tid < kDecodeFlags) d.hostFlags[tid] = d.flags[tid];
  if (refused || tileOff >= c.n) return;  // padding bits after the last value
  const int tile = t - c.tileBase, dupValue = c.dupValue, bins = c.binCount;
  const TileAt at = stage_words(c, tile, sm.sw);
  stage_lut(c, d, sm.lut);
  const long long sub = (long long)tile * kTileSubs + tid - 1;
  const bool active = tid > 0 && sub < c.nSub;
  const unsigned cnt = active ? d.subCount[c.subBase + sub] : 0u;
  int p = tid * kSubBits + (active ? (int)d.subStart[c.subBase + sub] : 0);
  // elements and values before the subsequence
  const unsigned n = cnt & ((1u << kCountBits) - 1), nv = cnt >> kCountBits;
  uint2 inc = make_uint2(n, nv);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned x = __shfl_up_sync(kAll, inc.x, o), y = __shfl_up_sync(kAll, inc.y, o);
    if (lane >= o) {
      inc.x += x;
      inc.y += y;
    }
  }
  if (lane == 31) sm.sums[w] = inc;
  __syncthreads();
  unsigned o = inc.x - n, v = inc.y - nv, values = 0;
#pragma unroll
  for (int k = 0; k < kThreads / 32; k++) {
    const uint2 x = sm.sums[k];
    if (k < w) {
      o += x.x;
      v += x.y;
    }
    values += x.y;
  }
  const unsigned vEnd = v + nv;
  const long long room = c.n - tileOff;  // elements from the tile's first on
  const unsigned end = (unsigned)min(room, (long long)0xffffffffu);
  const int lim = active ? min(tid * kSubBits + kSubBits, at.tot) : p;
  float *F = c.out + tileOff;
  const unsigned tileEnd = (unsigned)min((long long)end, (long long)d.tileCount[t]);
  const bool listed = c.fill && tileEnd < (1u << kPosBits) &&
                      values <= kPool - kMinNear * kStep;
  // the pool: step tables, then the list (element from the tile's first on,
  // ascending, and bin)
  const int listAt = listed ? (int)(kPool - values) : kPool;
  unsigned *list = sm.pool + listAt;
  const Tables tab = stage_steps(c, d, d.tileCub[t], sm.lut, sm.pool, listAt / kStep);
  const float zero = dupValue >= 0 ? c.dq[min(dupValue, bins - 1)] : 0.f;
  if (c.fill && !listed) {
    const int total = (int)tileEnd;
    const int head = min((int)((16 - (reinterpret_cast<size_t>(F) & 15)) & 15) / 4, total);
    const int quads = (total - head) / 4, tail = head + 4 * quads;
    if (tid < head) F[tid] = zero;
    float4 *g4 = reinterpret_cast<float4 *>(F + head);
    for (int i = tid; i < quads; i += kThreads) g4[i] = make_float4(zero, zero, zero, zero);
    if (tid < total - tail) F[tail + tid] = zero;
  }
  __syncthreads();  // the tables are there, and the fill comes before the values
  while (p < lim && o < end) {
    const unsigned e = token_at(sm.sw, tab, p, dupValue);
    if ((e & 63u) == 0) break;
    p += (int)(e & 63u);
    const int sym = (int)(e >> 10);
    if (sym != dupValue) {
      if (listed) {
        if (v < vEnd) list[v++] = o | ((unsigned)min(sym, bins - 1) << kPosBits);
      } else {
        F[o] = __ldg(c.dq + min(sym, bins - 1));
      }
    }
    o += 1u << ((e >> 6) & 15u);
  }
  if (!listed) return;
  // values counted in the padding bits past the cubelet's end
  for (; v < vEnd; v++) list[v] = ~0u;

  // ---- the tile's output, window by window: windows start at multiples of
  // 16 bytes, the first up to three floats before the tile
  if (tileEnd == 0) return;
  const unsigned shift = (unsigned)((reinterpret_cast<size_t>(F) & 15) / 4);
  const unsigned span = tileEnd + shift;
  float4 *G = reinterpret_cast<float4 *>(F - shift);
  float *win = reinterpret_cast<float *>(sm.window);
  const float4 zero4 = make_float4(zero, zero, zero, zero);
  __syncthreads();  // the list is complete, the tables are done with
  const float *dq = c.dq;
  if (bins <= listAt) {  // in the place of the step tables
    float *near = reinterpret_cast<float *>(sm.pool);
    for (int i = tid; i < bins; i += kThreads) near[i] = c.dq[i];
    dq = near;
  }
  for (int i = tid; i < kWindow / 4; i += kThreads) sm.window[i] = zero4;
  __syncthreads();
  unsigned i = tid;  // the thread's next value of the list
  for (unsigned w0 = 0; w0 < span; w0 += kWindow) {
    const unsigned w1 = min(w0 + kWindow, span);
    for (; i < values; i += kThreads) {
      const unsigned x = list[i], at = (x & ((1u << kPosBits) - 1)) + shift;
      if (at >= w1) break;
      win[at - w0] = dq[x >> kPosBits];
    }
    __syncthreads();
    for (unsigned k = tid; k < kWindow / 4; k += kThreads) {
      const unsigned q = w0 + 4 * k;
      if (q >= span) break;
      const float4 x = sm.window[k];
      if (q >= shift && q + 4 <= span) {
        G[q / 4] = x;
      } else {
        const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int j = 0; j < 4; j++)
          if (q + j >= shift && q + j < span) F[q + j - shift] = xs[j];
      }
      sm.window[k] = zero4;
    }
    __syncthreads();
  }
}

// 12-bit table and step tables of every stream's decode table
__global__ void __launch_bounds__(1024) build_lut_kernel(const DecodeCub *__restrict__ cubs,
                                                         DecodeArrays d) {
  extern __shared__ ushort2 nodes[];  // the decode table, when it fits
  __shared__ int nSlots;
  const DecodeCub c = cubs[blockIdx.x];
  const int nNodes = c.nTable / 2;
  const bool staged = nNodes <= kBuildNodes && c.dupKey < 0x10000;  // 16 bits an entry
  const int2 *tab = reinterpret_cast<const int2 *>(c.table);
  if (staged)
    for (int i = threadIdx.x; i < nNodes; i += blockDim.x) {
      const int2 v = tab[i];
      nodes[i] = make_ushort2((unsigned short)v.x, (unsigned short)v.y);
    }
  if (threadIdx.x == 0) nSlots = 0;
  __syncthreads();
  auto node = [&](int k) {
    if (!staged) return tab[k];
    const ushort2 v = nodes[k];
    return make_int2(v.x, v.y);
  };
  unsigned *L = d.lut + c.lutOff, *T = d.steps + (size_t)c.stepOff * kStep;
  // the entry reached from node `k` with `width` bits `p`, `above` bits
  // already consumed
  auto entry = [&](int k, unsigned p, int width, int above) {
    int dep = 0;
    int2 v = node(k);
    while (v.x != 0 && dep < width) {  // x == 0: a leaf, y its symbol
      k = (p >> dep) & 1u ? v.y : v.x;
      dep++;
      if (k < 0 || k >= nNodes) return kSlow | kRun | kBad;
      v = node(k);
    }
    if (v.x != 0) {  // goes on: a step table of its own
      if (above + dep + kStepBits > kMaxDecodeCode) return kSlow | kRun | kBad;
      const int slot = atomicAdd(&nSlots, 1);
      if (slot >= c.nSteps) return kSlow | kRun | kBad;
      T[slot * kStep] = (unsigned)k;  // until it is filled
      return kSlow | (unsigned)slot;
    }
    if (v.y == c.dupKey && c.dupKey >= 0) {
      if (above > 0 || dep + 3 > width) return kSlow | kRun | (unsigned)dep;
      const unsigned run = ((p >> dep) & 7u) + 3;
      return (unsigned)(dep + 3) | (run << 6) | ((unsigned)c.dupValue << 10);
    }
    if (above + dep == 0) return kSlow | kRun | kBad;  // a zero-length code
    return (unsigned)dep | ((unsigned)v.y << 10);
  };
  for (int p = threadIdx.x; p < kLutSize; p += blockDim.x) L[p] = entry(0, (unsigned)p, kLutBits, 0);
  __syncthreads();
  int head = 0, above = kLutBits;
  for (;;) {
    const int tail = min(nSlots, c.nSteps);
    __syncthreads();  // everyone has read the count
    if (head >= tail) break;
    // whole warps, kStep lanes per table
    const int lo = head * kStep, hi = tail * kStep;
    for (int i = (lo & ~31) + threadIdx.x; i < ((hi + 31) & ~31); i += blockDim.x) {
      const bool ok = i >= lo && i < hi;
      const int k = ok ? (int)T[i & ~(kStep - 1)] : 0;
      __syncwarp();
      if (ok) T[i] = entry(k, (unsigned)(i & (kStep - 1)), kStepBits, above);
    }
    __syncthreads();
    head = tail;
    above += kStepBits;
  }
  if (threadIdx.x == 0) d.stepCount[blockIdx.x] = min(nSlots, c.nSteps);
}

__global__ void __launch_bounds__(256) fill_batch_kernel(const FillItem *__restrict__ items,
                                                         int nItems) {
  int lo = 0, hi = nItems - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (items[mid].blockBase <= (long long)blockIdx.x) lo = mid; else hi = mid - 1;
  }
  const FillItem it = items[lo];
  const long long b0 = ((long long)blockIdx.x - it.blockBase) * kFillBlock;
  const long long e = min(b0 + kFillBlock, it.n);
  const float4 v4 = make_float4(it.v, it.v, it.v, it.v);
  // b0 is a multiple of kFillBlock, so whole float4 words up to the end
  for (long long i = b0 + 4 * threadIdx.x; i + 4 <= e; i += 4 * 256)
    *reinterpret_cast<float4 *>(it.out + i) = v4;
  const long long tail = b0 + ((e - b0) & ~3LL);
  if (threadIdx.x < e - tail) it.out[tail + threadIdx.x] = it.v;
}

}  // namespace

void launch_fill_batch(const FillItem *items, int nItems, long long totalBlocks, cudaStream_t s) {
  if (nItems > 0 && totalBlocks > 0)
    fill_batch_kernel<<<(unsigned)totalBlocks, 256, 0, s>>>(items, nItems);
}

long long decode_subs(long long nWords) {
  const long long k = (nWords * 32 + kSubBits - 1) / kSubBits;
  return k > 0 ? k : 1;
}
int decode_tiles(long long nWords) {
  return (int)((decode_subs(nWords) + kTileSubs - 1) / kTileSubs);
}
int decode_lut_size() { return kLutSize; }
size_t decode_step_bytes(long long steps) { return (size_t)steps * kStep * sizeof(unsigned); }

int launch_decode(const DecodeCub *cubs, const DecodeBatch &b, const DecodeArrays &d,
                  cudaStream_t s) {
  const int build = (b.maxTable / 2 <= kBuildNodes ? b.maxTable / 2 : kBuildNodes) * 4 + 16;
  if (build > 48 * 1024) raise_smem_limit(build_lut_kernel, build);
  build_lut_kernel<<<b.n, 1024, build, s>>>(cubs, d);
  tile_kernel<<<b.tiles, kThreads, sizeof(TileSmem), s>>>(cubs, d);
  check_kernel<<<b.tiles, kThreads, sizeof(TileSmem), s>>>(cubs, d, kDecodeFirst);
  check_kernel<<<b.tiles, kThreads, sizeof(TileSmem), s>>>(cubs, d, kDecodeAgain);
  return 4 + launch_decode_write(cubs, b, d, s);
}
void launch_decode_check(const DecodeCub *cubs, const DecodeBatch &b, const DecodeArrays &d,
                         cudaStream_t s) {
  check_kernel<<<b.tiles, kThreads, sizeof(TileSmem), s>>>(cubs, d, kDecodeAgain);
}
int launch_decode_write(const DecodeCub *cubs, const DecodeBatch &b, const DecodeArrays &d,
                        cudaStream_t s) {
  scan_kernel<<<b.n, kThreads, 0, s>>>(cubs, d);
  const int smem = (int)sizeof(WriteSmem);
  if (smem > 48 * 1024) raise_smem_limit(write_kernel, smem);
  write_kernel<<<b.tiles, kThreads, smem, s>>>(cubs, d);
  return 2;
}

}  // namespace wl
