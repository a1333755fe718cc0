// Huffman coding on the device: exact tree construction, code assignment and
// decode table per cubelet, then a parallel bit packer.
//
// Tree (Huffman::computeHuffmanCoding, huffman.cc:42-97): the reference pops
// the two nodes of smallest count from a priority queue ordered by
// (count, node address) with ties going to the LARGER node index
// (CompareHuffmanNode, huffman.cc:9-18); the first popped becomes the 0
// branch.  Leaves are symbol indices 0..S-1 (S = bins, +1 for the zero-run
// key), merged nodes are numbered from S upward.  Here the leaves are sorted
// by (count asc, index desc), the order they are popped in, and merged in
// rounds of independent pairs (huffman_build_kernel).
// Codes are root-first, bit d of the code word = branch taken at depth d
// (computeEncodedBits :147-174), the decode table lists nodes breadth first
// as (left id, right id) or (0, symbol) (computeDecodeTable :177-228).
//
// Packing (Huffman::encodeToStream, huffman.h:242-296; BitStreamWriter
// bit_stream.h:60-162): every coefficient yields zero or one token -- its own
// code, a single zero-bin code, or at the first element of a dup chunk the
// zero-run key code followed by 3 length bits.  Token lengths are summed per
// token chunk, chunk offsets are scanned per cubelet, and lanes pack slices of
// a chunk's values in registers (the bit packer below).
#include "wl_internal.h"

namespace wl {
namespace {

constexpr int kMaxCodeBits = 58;  // + 3 dup bits fits 61 bits -> at most 3 words

// ---- tree -------------------------------------------------------------------
// Shared memory of one tree build for up to S symbols (P = S rounded up to a
// power of two).  The sort keys are dead once the leaf list is taken from
// them and the lists are dead after the last round, so their space is reused.
struct BuildSmem {
  unsigned long long *keys;        // P sort keys
  unsigned *cntA, *cntB;           // S each: counts of the active list (two buffers)
  uint16_t *idA, *idB;             // S each: its node ids
  unsigned *sum;                   // S / 2 + 1: counts of the round's new nodes
  uint16_t *lch, *rch;             // S each: children of merged node (id - S)
  uint16_t *par;                   // 2 S: parent's (id - S) * 2 + branch
  uint16_t *bfs;                   // 2 S: nodes in breadth-first order
};

__host__ __device__ inline int build_pow2(int S) {
  int P = 32;
  while (P < S) P <<= 1;
  return P;
}
// keys (aliased by cntB, idB) | cntA (aliased by bfs) | sum | idA |
// lch | rch | par
__host__ __device__ inline size_t build_smem_bytes(int S) {
  const size_t s = (size_t)((S + 3) & ~3);
  return (size_t)build_pow2(S) * 8 + s * 4 + (s / 2 + 4) * 4 + s * 2 * 3 + s * 2 * 2;
}

// number of entries of the ascending list v[0..n) below x, by a whole warp:
// 32 probes at a time
__device__ __forceinline__ int list_rank_warp(const unsigned *v, int n, unsigned x, int lane) {
  int lo = 0, len = n;
  while (len > 0) {
    const int step = (len + 31) >> 5;
    const int p = lo + (lane + 1) * step - 1;
    const int c = __popc(__ballot_sync(0xffffffffu, p < lo + len && v[p] < x));
    lo += c * step;
    len = min(step - 1, len - c * step);
  }
  return lo;
}

// One CTA builds one cubelet's tree, codes and decode table; nothing in it is
// a serial chain over the symbols.  A one-thread merge, depth pass and
// breadth-first walk took 120 and 578 us for 257 and 1025 symbols.  It is bound
// by the latency of its dependent steps in shared memory and, with many warps,
// by the instructions they all issue between two barriers; so the searches of
// a round run side by side, the last rounds and the breadth-first numbering,
// whose lists are short, belong to one warp without barriers, and the other
// warps walk the codes meanwhile: 42 K cycles instead of 55 K for 257 symbols
// and 82 K instead of 118 K for 1025 (a 256^3 volume's call 380 -> 363 us), of
// which the rounds take 27 and 46 K, the numbering 9 and 20 K.  (Ranks by
// ballots over a warp's registers in the last rounds were no faster.)
//
// Merging in rounds.  The active list holds the parentless nodes in the order
// the reference pops them (count ascending, on equal counts the larger index
// first).  With s the sum of its two smallest counts, every node created from
// now on counts at least s, so the entries below s are popped in list order:
// they pair off two by two at once (an odd last one stays for the next
// round), and the new nodes -- counts ascending, equal counts in reverse
// order, before old nodes of equal count since their indices are larger --
// are merged into the rest of the list by rank.  Two rounds at least double
// the smallest count, so there are at most about 62 of them (25 in practice),
// each a handful of shared-memory searches.
//
// Codes: a thread per symbol walks up the parents (at most 58 steps).  The
// decode table's breadth-first numbering is a scan of the inner nodes, level
// by level.
template <int T>
__global__ void __launch_bounds__(T) huffman_build_kernel(DevBatch b) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int kTail = 64;  // lists that one warp merges
  extern __shared__ __align__(16) unsigned char hsm[];
  __shared__ int nLeaves;
  __shared__ bool overflow;
  stage_mark(b.head, kMarkBuild);
  const int ci = blockIdx.x;
  const CubeletDev cd = b.cub[ci];
  CubeletState *st = b.state + ci;
  const int dupV = st->dupValue;
  const int S = cd.binCount + (dupV >= 0 ? 1 : 0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  BuildSmem m;
  {
    const int s4 = (S + 3) & ~3;
    unsigned char *p = hsm;
    m.keys = reinterpret_cast<unsigned long long *>(p);
    m.cntB = reinterpret_cast<unsigned *>(p);
    m.idB = reinterpret_cast<uint16_t *>(p + 4 * s4);
    p += (size_t)build_pow2(S) * 8;
    m.cntA = reinterpret_cast<unsigned *>(p);
    m.bfs = reinterpret_cast<uint16_t *>(p); p += 4 * s4;
    m.sum = reinterpret_cast<unsigned *>(p); p += (s4 / 2 + 4) * 4;
    m.idA = reinterpret_cast<uint16_t *>(p); p += 2 * s4;
    m.lch = reinterpret_cast<uint16_t *>(p); p += 2 * s4;
    m.rch = reinterpret_cast<uint16_t *>(p); p += 2 * s4;
    m.par = reinterpret_cast<uint16_t *>(p);
  }

  // ---- leaves with a nonzero count, key = count:51 | (8191 - symbol):13
  const unsigned long long *cnt = b.hist + (size_t)ci * kMaxSymbols;
  if (tid == 0) nLeaves = 0;
  __syncthreads();
  for (int i = tid; i < S; i += T) {
    const unsigned long long c = cnt[i];
    if (c > 0) {
      const int slot = atomicAdd(&nLeaves, 1);
      m.keys[slot] = (c << 13) | (unsigned long long)(8191 - i);
    }
  }
  __syncthreads();
  const int nL = nLeaves;
  const int P = build_pow2(nL);
  for (int i = nL + tid; i < P; i += T) m.keys[i] = ~0ull;
  __syncthreads();
  // ---- bitonic sort, ascending: distances below 32 inside a warp
  auto warp_stages = [&](unsigned long long v, int i, int k, int j0) {
    for (int j = j0; j > 0; j >>= 1) {
      const unsigned long long o = __shfl_xor_sync(kAll, v, j);
      const bool keepMin = ((i & k) == 0) == ((i & j) == 0);
      v = keepMin == (v < o) ? v : o;
    }
    return v;
  };
  for (int i = tid; i < P; i += T) {  // P is a multiple of 32: whole warps
    unsigned long long v = m.keys[i];
    for (int k = 2; k <= 32; k <<= 1) v = warp_stages(v, i, k, k >> 1);
    m.keys[i] = v;
  }
  __syncthreads();
  for (int k = 64; k <= P; k <<= 1) {
    for (int j = k >> 1; j >= 32; j >>= 1) {
      for (int p = tid; p < P / 2; p += T) {
        const int i = 2 * p - (p & (j - 1)), l = i + j;
        const unsigned long long a = m.keys[i], c = m.keys[l];
        if ((a > c) == ((i & k) == 0)) { m.keys[i] = c; m.keys[l] = a; }
      }
      __syncthreads();
    }
    for (int i = tid; i < P; i += T) m.keys[i] = warp_stages(m.keys[i], i, k, 16);
    __syncthreads();
  }
  // the counts of a cubelet's tokens sum to at most its element count (below
  // 2^31), so 32 bits hold every node's count
  for (int i = tid; i < nL; i += T) {
    const unsigned long long key = m.keys[i];
    m.cntA[i] = (unsigned)(key >> 13);
    m.idA[i] = (uint16_t)(8191 - (int)(key & 8191ull));
  }
  __syncthreads();

  // ---- merge rounds
  unsigned *cc = m.cntA, *cn = m.cntB;
  uint16_t *ic = m.idA, *in = m.idB;
  int len = nL, next = S;
  // one round by threads t0, t0 + step, .. (sync: a barrier among them); false
  // when the counts overflow 32 bits: not from a token count
  auto merge_round = [&](int t0, int step, auto sync) {
    const unsigned s = cc[0] + cc[1];
    const int kp = list_rank_warp(cc, len, s, lane) & ~1;  // entries paired off
    if (kp < 2) return false;
    const int q = kp >> 1, r = len - kp;
    for (int j = t0; j < q; j += step) {
      const int a = ic[2 * j], c = ic[2 * j + 1], node = next - S + j;
      m.sum[j] = cc[2 * j] + cc[2 * j + 1];
      m.lch[node] = (uint16_t)a;
      m.rch[node] = (uint16_t)c;
      m.par[a] = (uint16_t)(2 * node);
      m.par[c] = (uint16_t)(2 * node + 1);
    }
    sync();
    const unsigned *rest = cc + kp;
    const int top = 1 << (31 - __clz(max(q, r)));
    // new nodes go before, old ones after entries of equal count in the other
    // list; a run of equal counts among the new nodes is reversed
    for (int t = t0; t < len - q; t += step) {
      const bool isNew = t < q;
      const unsigned c = isNew ? m.sum[t] : rest[t - q];
      const unsigned *v = isNew ? rest : m.sum;
      const int n = isNew ? r : q;
      const bool run = isNew && ((t > 0 && m.sum[max(t - 1, 0)] == c) |
                                 (t + 1 < q && m.sum[min(t + 1, q - 1)] == c));
      // three searches side by side, without branches: in the other list, and
      // for a run's ends (an index at or past the end reads some entry of ours)
      int at = 0, lo = 0, hi = 0;
      for (int d = top; d > 0; d >>= 1) {
        const unsigned x = v[min(at + d, n) - (n > 0)], y = m.sum[min(lo + d, q) - 1],
                       z = m.sum[min(hi + d, q) - 1];
        at += (d <= n - at) & ((x < c) | (!isNew & (x == c))) ? d : 0;
        lo += (d <= q - lo) & (y < c) ? d : 0;
        hi += (d <= q - hi) & (z <= c) ? d : 0;
      }
      at += !isNew ? t - q : run ? lo + hi - 1 - t : t;
      cn[at] = c;
      in[at] = isNew ? (uint16_t)(next + t) : ic[kp + t - q];
    }
    next += q;
    len -= q;
    unsigned *tc = cc;
    cc = cn;
    cn = tc;
    uint16_t *ti = ic;
    ic = in;
    in = ti;
    sync();
    return true;
  };
  bool bad = false;
  while (len > kTail && !bad) bad = !merge_round(tid, T, [] { __syncthreads(); });
  if (warp == 0) {
    while (len > 1 && !bad) bad = !merge_round(lane, 32, [] { __syncwarp(); });
    if (lane == 0) overflow = bad;
  }
  __syncthreads();
  bad = overflow;
  const int root = S + nL - 2;  // with two or more leaves

  // ---- codes: up from each leaf (root-first bits, bit d = branch at depth d)
  if (warp > 0) {
    unsigned long long *gcode = b.codes + (size_t)ci * kMaxSymbols;
    uint8_t *glen = b.codeLen + (size_t)ci * kMaxSymbols;
    for (int i = tid - 32; i < S; i += T - 32) {
      unsigned long long code = 0;
      int d = 0;
      if (nL > 1 && cnt[i] > 0 && !bad) {
        int nd = i;
        while (nd != root && d < 64) {
          const int pb = m.par[nd];
          code = (code << 1) | (unsigned)(pb & 1);
          d++;
          nd = S + (pb >> 1);
        }
      }
      gcode[i] = code;
      glen[i] = (uint8_t)d;
    }
    return;
  }

  // ---- decode table, breadth first: (left id, right id) or (0, symbol);
  // kWide nodes a lane and step
  constexpr int kWide = 2;
  int2 *dec = reinterpret_cast<int2 *>(b.decode + (size_t)ci * 4 * kMaxSymbols);
  int base = 0, width = nL > 0 && !bad ? 1 : 0, levels = 0;
  if (nL > 0 && lane == 0)
    m.bfs[0] = (uint16_t)(nL > 1 ? root : 8191 - (int)(m.keys[0] & 8191ull));
  __syncwarp();
  while (width > 0) {
    int child = base + width;  // the next level's first node
    for (int t0 = 0; t0 < width; t0 += 32 * kWide) {
      int nd[kWide], left[kWide], right[kWide];
#pragma unroll
      for (int k = 0; k < kWide; k++) {
        const int t = t0 + 32 * k + lane;
        const int x = m.bfs[base + min(t, width - 1)];
        nd[k] = t < width ? x : -1;
      }
#pragma unroll
      for (int k = 0; k < kWide; k++) {
        left[k] = m.lch[max(nd[k] - S, 0)];
        right[k] = m.rch[max(nd[k] - S, 0)];
      }
#pragma unroll
      for (int k = 0; k < kWide; k++) {
        const unsigned bal = __ballot_sync(kAll, nd[k] >= S);
        const int at = base + t0 + 32 * k + lane;
        const int c = child + 2 * __popc(bal & ((1u << lane) - 1u));
        if (nd[k] >= S) {
          m.bfs[c] = (uint16_t)left[k];
          m.bfs[c + 1] = (uint16_t)right[k];
          dec[at] = make_int2(c, c + 1);
        } else if (nd[k] >= 0) {
          dec[at] = make_int2(0, nd[k]);
        }
        child += 2 * __popc(bal);
      }
    }
    __syncwarp();
    base += width;
    width = child - base;
    levels++;
  }
  if (lane == 0) {
    const int longest = levels > 0 ? levels - 1 : 0;
    st->nDecode = 2 * base;
    st->longest = longest;
    st->nLeaves = nL;
    if (longest > kMaxCodeBits || bad) st->error = 2;
  }
}

// ---- bit packer -------------------------------------------------------------
// A chunk's stream is the tokens of the zero run entering it that start in it,
// then for each of its values the tokens of the zero run before it and the
// value's own, then the tokens of the run leaving it that start in it
// (quantize_kernel stores the values, runs_kernel the edge runs).
//
// A chunk's values are cut into F slices of ceil(n / F) (F from enc_slices,
// per launch); lane s of the chunk's F lanes packs slice s, the first lane the
// entering run and the last the leaving run besides, and a CTA of kEncThreads
// lanes takes kEncThreads / F consecutive chunks of one cubelet.  The bit
// counter sums each slice's code lengths and places the slices inside their
// chunk with an F-lane exclusive scan; the packer starts each slice at its
// chunk's offset (from the per-cubelet scan) plus that place.  A lane keeps
// its bits in a 64-bit register and stores whole words: words wholly inside
// its slice are stored directly, its first and last word (which it may share
// with neighbouring slices) are OR-ed in.  A word shared by slices of one
// chunk is zeroed by the lane whose slice starts in it, before any lane of the
// chunk ORs (the chunk's lanes are one warp); the chunk's first and last
// words, shared with neighbouring chunks, were zeroed by encode_zero_kernel.
//
// The run before a value costs no loop over its tokens, which would run as
// long as the longest in the warp: the tokens of its multiple of 16 below 1024
// (powers of two) and of what is below 16 (an eight and singles) are two
// ready-made bit strings, joined with the value's code and appended at once.
// Only runs of 1024 and more, and alphabets whose codes make such strings
// longer than 64 bits, take the loops.  Values are read one at a time, the
// next one ahead (for_entries).
//
// The encode stage (bit counts, scans, packer) of the mixed batch takes 0.42
// ms, of 729 cubelets of 128^3 0.51 ms; 0.49 and 0.79 ms when it read every
// token as a 16-bit word.

// code bits (below kMaxCodeBits) and length (above) of one symbol
constexpr unsigned long long kCodeMask = (1ull << kMaxCodeBits) - 1;

// Slice geometry shared by the bit counter and the packer: chunk `cl` of the
// cubelet (within its CTA's run), slice `sub` of it, values [t0, t1) of the
// chunk's.
struct SliceAt {
  int cl, sub, n, t0, t1;  // n: values of the chunk
  bool ok;                 // the chunk exists
  long long chunk;
  uint2 edge;              // run codes at the chunk's edges
};
__device__ __forceinline__ SliceAt slice_at(const DevBatch &b, const CubeletDev &cd, int lgF) {
  SliceAt r;
  const int lane = threadIdx.x;
  r.cl = (((int)blockIdx.x - cd.encBase) << (7 - lgF)) + (lane >> lgF);
  r.sub = lane & ((1 << lgF) - 1);
  r.ok = r.cl < cd.nChunks;
  r.chunk = cd.chunkBase + r.cl;
  const int n = r.ok ? b.chunkVal[r.chunk] : 0;
  const int m = (n + (1 << lgF) - 1) >> lgF;
  r.n = n;
  r.t0 = min(n, r.sub * m);
  r.t1 = min(n, r.t0 + m);
  // the chunk's entering run comes before its first value, the leaving run
  // after its last
  r.edge = make_uint2(0u, 0u);
  if (r.ok && b.state[(int)b.encCub[blockIdx.x]].dupValue >= 0) {
    r.edge = b.chunkEdge[r.chunk];
    if (r.sub == 0) r.t0 = -1;
    if (r.sub == (1 << lgF) - 1) r.t1 = n + 1;
  }
  return r;
}
// f(bin or -1, run code) for the entries [t0, t1) of the slice, in order: the
// entering run (-1), the values with the run before each, the leaving run (n).
// One entry per step and the next value's load in flight: one copy of f keeps
// the packer's code inside the instruction cache (with four values unrolled
// and an append for every kind of token, its warps waited for instructions
// most of the time: 1.46 ms for 729 cubelets against 0.43).
template <class Fn>
__device__ __forceinline__ void for_entries(const unsigned *items, const SliceAt &sl, Fn &&f) {
  auto load = [&](int j) { return (unsigned)j < (unsigned)sl.n ? items[j] : 0u; };
  unsigned nx = load(sl.t0);
#pragma unroll 1
  for (int j = sl.t0; j < sl.t1; j++) {
    const unsigned it = nx;
    nx = load(j + 1);
    if ((unsigned)j < (unsigned)sl.n) f((int)(it >> 16), run_code((int)(it & 0xffff)));
    else f(-1, j < 0 ? sl.edge.x : sl.edge.y);
  }
}
// Bits of every slice: lane s of a chunk's F lanes sums its values' code
// lengths and their runs' (a run's length from its token counts), an F-lane
// exclusive scan places the slice inside the chunk (sliceOff), and the chunk's
// last lane writes the chunk's bit count.
__global__ void __launch_bounds__(kEncThreads) encode_count_kernel(DevBatch b) {
  extern __shared__ uint8_t sLen[];
  stage_mark(b.head, kMarkEncode);
  const int ci = b.encCub[blockIdx.x];
  const CubeletDev cd = b.cub[ci];
  const int lgF = __ffs(b.encF) - 1, F = 1 << lgF;
  const int dupV = b.state[ci].dupValue, dupKey = cd.binCount, S = cd.binCount + 1;
  for (int i = threadIdx.x; i < S; i += kEncThreads) sLen[i] = b.codeLen[(size_t)ci * kMaxSymbols + i];
  __syncthreads();
  const SliceAt sl = slice_at(b, cd, lgF);
  unsigned mine = 0;  // at most 4096 tokens of at most 61 bits
  if (sl.ok) {
    const unsigned one = dupV >= 0 ? sLen[dupV] : 0u, dup = sLen[dupKey] + 3u;
    for_entries(b.items + cd.coefOff + ((long long)sl.cl << b.lgChunk), sl,
                [&](int bin, unsigned run) {
      if (bin >= 0) mine += sLen[bin];
      const int lo = run & 255;
      const int keys = (int)(run >> 16) + __popc(run & 0x3f00) + (lo > 8);
      mine += dup * keys + one * (lo > 8 ? (lo & 15) - (lo < kEightAlone ? 8 : 0) : lo);
    });
  }
  unsigned inc = mine;
  for (int d = 1; d < F; d <<= 1) {
    const unsigned x = __shfl_up_sync(0xffffffffu, inc, d, F);
    if (sl.sub >= d) inc += x;
  }
  if (sl.ok) {
    b.sliceOff[sl.chunk * 32 + sl.sub] = inc - mine;
    if (sl.sub == F - 1) b.chunkLen[sl.chunk] = inc;
  }
}

// Per cubelet: exclusive scan of the chunk bit counts, kScanRun consecutive
// chunks per thread, so that one round covers 8192 chunks (the most a call
// that fills no more than the GPU has: a round is all latency).  A round's
// bits fit 32 bits (4096 elements of at most 61 each per chunk).
constexpr int kScanRun = 8;
__global__ void __launch_bounds__(1024) encode_scan_kernel(DevBatch b) {
  __shared__ unsigned sh[32];
  __shared__ unsigned v[1024 * (kScanRun + 1)];  // a thread's run at stride 9
  const int ci = blockIdx.x, tid = threadIdx.x;
  const CubeletDev cd = b.cub[ci];
  CubeletState *st = b.state + ci;
  unsigned long long carry = 0;
  const int lane = tid & 31, w = tid >> 5;
  const unsigned *len = b.chunkLen + cd.chunkBase;
  unsigned long long *bits = b.chunkBits + cd.chunkBase;
  for (int seg = 0; seg < cd.nChunks; seg += 1024 * kScanRun) {
    const int n = min(1024 * kScanRun, cd.nChunks - seg);
#pragma unroll
    for (int k = 0; k < kScanRun; k++) {
      const int i = k * 1024 + tid;
      v[i + i / kScanRun] = i < n ? len[seg + i] : 0u;
    }
    __syncthreads();
    unsigned mine = 0;
#pragma unroll
    for (int k = 0; k < kScanRun; k++) {  // exclusive inside the run
      const unsigned t = v[tid * (kScanRun + 1) + k];
      v[tid * (kScanRun + 1) + k] = mine;
      mine += t;
    }
    unsigned inc = mine;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned t = __shfl_up_sync(0xffffffffu, inc, off);
      if (lane >= off) inc += t;
    }
    if (lane == 31) sh[w] = inc;
    __syncthreads();
    unsigned before = sh[lane];  // inclusive over the warps
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned t = __shfl_up_sync(0xffffffffu, before, off);
      if (lane >= off) before += t;
    }
    const unsigned all = __shfl_sync(0xffffffffu, before, 31);
    const unsigned upTo = __shfl_sync(0xffffffffu, before, w > 0 ? w - 1 : 0);
    const unsigned at = (w > 0 ? upTo : 0u) + inc - mine;
#pragma unroll
    for (int k = 0; k < kScanRun; k++) v[tid * (kScanRun + 1) + k] += at;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kScanRun; k++) {
      const int i = k * 1024 + tid;
      if (i < n) bits[seg + i] = carry + v[i + i / kScanRun];
    }
    carry += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    st->totalBits = carry;
    const unsigned long long words = (carry + 31) / 32;
    st->nWords = (int)words;
    if ((long long)words > cd.wordsCap) st->error = 4;
  }
}

// packed word and metadata offsets of every cubelet: exclusive scans over
// the cubelets, 1024 at a time
__global__ void __launch_bounds__(1024) cubelet_offsets_kernel(DevBatch b) {
  __shared__ long long sw[32], sm[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  long long carryW = 0, carryM = 0;
  for (int base = 0; base < b.n; base += 1024) {
    const int i = base + threadIdx.x;
    long long vw = 0, vm = 0;
    if (i < b.n) {
      const CubeletState *st = b.state + i;
      vw = st->error ? 0 : st->nWords;
      vm = st->nDecode + (b.cub[i].quantAlg == WL_LLOYD ? st->nBounds + st->nValues : 0);
    }
    long long iw = vw, im = vm;
    for (int off = 1; off < 32; off <<= 1) {
      const long long tw = __shfl_up_sync(0xffffffffu, iw, off);
      const long long tm = __shfl_up_sync(0xffffffffu, im, off);
      if (lane >= off) { iw += tw; im += tm; }
    }
    if (lane == 31) { sw[w] = iw; sm[w] = im; }
    __syncthreads();
    long long bw = 0, bm = 0, tw = 0, tm = 0;
    for (int v = 0; v < 32; v++) {
      if (v < w) { bw += sw[v]; bm += sm[v]; }
      tw += sw[v];
      tm += sm[v];
    }
    if (i < b.n) {
      CubeletState *st = b.state + i;
      st->wordsBase = carryW + bw + iw - vw;
      st->metaBase = carryM + bm + im - vm;
    }
    carryW += tw;
    carryM += tm;
    __syncthreads();
  }
  if (b.head && threadIdx.x == 0) {
    b.head[kHeadWords] = carryW;
    b.head[kHeadMeta] = carryM;
  }
}

// decode table and Lloyd codebook of every cubelet into one buffer
__device__ __forceinline__ void pack_meta(const DevBatch &b, int ci, int *m) {
  const CubeletState *st = b.state + ci;
  const CubeletDev cd = b.cub[ci];
  const int *dec = b.decode + (size_t)ci * 4 * kMaxSymbols;
  const int nDecode = st->nDecode;
  for (int i = threadIdx.x; i < nDecode; i += blockDim.x) m[i] = dec[i];
  if (cd.quantAlg == WL_LLOYD) {
    const float *bnd = b.qtable + cd.tableOff;
    const float *val = b.dqtable + (size_t)ci * kMaxBins;
    const int nBounds = st->nBounds, nValues = st->nValues;
    for (int i = threadIdx.x; i < nBounds; i += blockDim.x)
      m[nDecode + i] = __float_as_int(bnd[i]);
    for (int i = threadIdx.x; i < nValues; i += blockDim.x)
      m[nDecode + nBounds + i] = __float_as_int(val[i]);
  }
}
__global__ void pack_meta_kernel(DevBatch b) {
  if (b.hostState == nullptr) stage_mark(b.head, kMarkEnd);
  pack_meta(b, blockIdx.x, b.meta + b.state[blockIdx.x].metaBase);
}

// The results of a small call straight to page-locked host memory: words and
// metadata when they fit in the slab the host set aside, states and head
// always.  The host then waits once, instead of waiting for the sizes and
// again for the copies; with the one-launch set-up and the clock marks in
// place of event nodes a 2048^2 image went from 425 to 366 us a call, a 64^2
// tile from 282 to 223 us.
constexpr int kDeliverThreads = 256, kDeliverBlocks = 64;
__global__ void __launch_bounds__(kDeliverThreads) deliver_kernel(DevBatch b) {
  stage_mark(b.head, kMarkEnd);
  const OutSlab o = *b.outSlab;
  const long long words = b.head[kHeadWords], meta = b.head[kHeadMeta];
  const long long wordsBytes = (words * 4 + 15) & ~15LL;
  const bool fits = wordsBytes + meta * 4 <= o.cap && wordsBytes + meta * 4 > o.above;
  const int t0 = blockIdx.x * kDeliverThreads + threadIdx.x, step = kDeliverBlocks * kDeliverThreads;
  if (fits) {
    const uint4 *src = reinterpret_cast<const uint4 *>(b.words);
    uint4 *dst = reinterpret_cast<uint4 *>(o.base);
    const long long quads = words / 4;
    for (long long i = t0; i < quads; i += step) dst[i] = src[i];
    if (t0 < words - quads * 4)
      reinterpret_cast<uint32_t *>(o.base)[quads * 4 + t0] = b.words[quads * 4 + t0];
  }
  for (int ci = blockIdx.x; ci < b.n; ci += kDeliverBlocks) {
    const CubeletState *st = b.state + ci;
    const unsigned *w = reinterpret_cast<const unsigned *>(st);
    unsigned *hw = reinterpret_cast<unsigned *>(b.hostState + ci);
    for (int i = threadIdx.x; i < (int)(sizeof(CubeletState) / 4); i += kDeliverThreads) hw[i] = w[i];
    if (fits) pack_meta(b, ci, reinterpret_cast<int *>(o.base + wordsBytes) + st->metaBase);
  }
  if (blockIdx.x == 0 && threadIdx.x < kHeadCount) {
    // this block's own mark comes from thread 0, of the same warp
    __syncwarp((1u << kHeadCount) - 1u);
    b.hostHead[threadIdx.x] = threadIdx.x == kHeadDelivered ? (fits ? 1 : 0) : b.head[threadIdx.x];
  }
}

// zero the first and last word of every chunk (the words chunks share)
__global__ void encode_zero_kernel(DevBatch b) {
  const long long chunk = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (chunk >= b.totalChunks) return;
  const int ci = b.chunkCub[chunk];
  const CubeletState *st = b.state + ci;
  if (st->error) return;
  const unsigned long long off = b.chunkBits[chunk];
  const unsigned long long end = (chunk + 1 < b.cub[ci].chunkBase + b.cub[ci].nChunks)
                                     ? b.chunkBits[chunk + 1] : st->totalBits;
  if (end == off) return;
  uint32_t *w = b.words + st->wordsBase;
  w[off >> 5] = 0;
  w[(end - 1) >> 5] = 0;
}

// ready-made strings: runs below 16 elements, multiples of 16 below 1024 (in
// 16s), zero-run keys with their length bits
constexpr int kLowRuns = 17, kHighRuns = 64, kDupRuns = 8;

__global__ void __launch_bounds__(kEncThreads, 8) encode_write_kernel(DevBatch b) {
  extern __shared__ unsigned long long sTab[];  // code | length << kMaxCodeBits
  __shared__ unsigned long long sLow[kLowRuns], sHigh[kHighRuns], sDup[kDupRuns];
  __shared__ unsigned char sLowLen[kLowRuns], sHighLen[kHighRuns];
  const int ci = b.encCub[blockIdx.x];
  const CubeletDev cd = b.cub[ci];
  const CubeletState *st = b.state + ci;
  if (st->error) return;
  const int lane = threadIdx.x;
  const int lgF = __ffs(b.encF) - 1, F = 1 << lgF;
  const int dupV = st->dupValue, dupKey = cd.binCount, S = cd.binCount + 1;
  const unsigned long long *gc = b.codes + (size_t)ci * kMaxSymbols;
  const uint8_t *gl = b.codeLen + (size_t)ci * kMaxSymbols;
  for (int i = lane; i < S; i += kEncThreads)
    sTab[i] = (gc[i] & kCodeMask) | ((unsigned long long)gl[i] << kMaxCodeBits);
  const bool runs = dupV >= 0;
  const int oneLen = runs ? gl[dupV] : 0, dupLen = runs ? gl[dupKey] + 3 : 0;
  const unsigned long long one = runs ? gc[dupV] : 0, dup = runs ? gc[dupKey] : 0;
  // an eight and eight singles, and six powers of two, in 64 bits each: any
  // but extreme code lengths
  const bool ready = dupLen + 8 * oneLen <= 64 && 6 * dupLen <= 64;
  if (ready && lane < kLowRuns) {
    unsigned long long v = lane > 8 ? dup : 0;
    int l = lane > 8 ? dupLen : 0;
    for (int k = lane == kEightAlone ? 0 : lane > 8 ? lane - 8 : lane; k > 0; k--) {
      if (l < 64) v |= one << l;
      l += oneLen;
    }
    sLow[lane] = v;
    sLowLen[lane] = (unsigned char)l;
  } else if (ready && lane >= 32 && lane < 32 + kHighRuns) {
    unsigned long long v = 0;
    int l = 0;
    for (int lg = 5; lg >= 0; lg--)  // 2^(lg + 4) elements, length bits lg + 1
      if (((lane - 32) >> lg) & 1) {
        v |= (dup | ((unsigned long long)(lg + 1) << (dupLen - 3))) << l;
        l += dupLen;
      }
    sHigh[lane - 32] = v;
    sHighLen[lane - 32] = (unsigned char)l;
  }
  if (lane < kDupRuns && runs) sDup[lane] = dup | ((unsigned long long)lane << (dupLen - 3));
  __syncthreads();
  const SliceAt sl = slice_at(b, cd, lgF);
  unsigned long long off = 0, end = 0;
  if (sl.ok) {
    off = b.chunkBits[sl.chunk];
    end = sl.cl + 1 < cd.nChunks ? b.chunkBits[sl.chunk + 1] : st->totalBits;
  }
  // the slice's first bit and bit count
  const unsigned rel = sl.ok ? b.sliceOff[sl.chunk * 32 + sl.sub] : 0u;
  unsigned nxt = __shfl_down_sync(0xffffffffu, rel, 1, F);
  if (sl.sub == F - 1) nxt = (unsigned)(end - off);
  const unsigned long long sb = nxt - rel, pos = off + rel;
  uint32_t *gw = b.words + st->wordsBase;
  const bool any = sl.ok && sb > 0;
  if (any && F > 1) {
    const unsigned long long fw = pos >> 5;
    if (fw > (off >> 5) && fw < ((end - 1) >> 5)) gw[fw] = 0;
  }
  __syncwarp();
  if (!any) return;
  unsigned long long w = pos >> 5;
  const unsigned long long wFirst = w;
  unsigned long long acc = 0;  // bit 0 = bit 0 of word w
  int bits = (int)(pos & 31);
  for_entries(b.items + cd.coefOff + ((long long)sl.cl << b.lgChunk), sl,
              [&](int bin, unsigned run) {
    const unsigned long long e = bin >= 0 ? sTab[bin] : 0ull;
    const unsigned long long code = e & kCodeMask;
    const int codeLen = (int)(e >> kMaxCodeBits);
    // usually one step: the run's two strings and the code together; else as
    // many as it takes, the code in the last
    bool more = true;
#pragma unroll 1
    while (more) {
      const int hi = (run >> 8) & 63, lo = run & 255;
      unsigned long long v;
      int l;
      if (run >> 16) {
        v = sDup[7];
        l = dupLen;
        run -= 1u << 16;
      } else if (ready) {
        v = sHigh[hi];
        l = sHighLen[hi];
        const int ll = sLowLen[lo];
        run = (unsigned)lo;
        if (l + ll <= 64) {
          v |= l < 64 ? sLow[lo] << l : 0ull;
          l += ll;
          run = 0;
          if (l + codeLen <= 64) {
            v |= l < 64 ? code << l : 0ull;
            l += codeLen;
            more = false;
          }
        }
      } else if (hi) {
        const int lg = 31 - __clz(hi);
        v = sDup[lg + 1];
        l = dupLen;
        run ^= 256u << lg;
      } else if (lo > 8) {
        v = sDup[0];
        l = dupLen;
        run = lo == kEightAlone ? 0u : (unsigned)(lo - 8);
      } else if (lo) {
        v = one;
        l = oneLen;
        run--;
      } else {
        v = code;
        l = codeLen;
        more = false;
      }
      // l <= 64 bits of v, none above them; bits < 32 before and after
      unsigned long long over = bits ? v >> (64 - bits) : 0;  // above the accumulator
      acc |= v << bits;
      bits += l;
#pragma unroll 1
      while (bits >= 32) {
        if (w == wFirst) atomicOr(&gw[w], (unsigned)acc);
        else gw[w] = (unsigned)acc;
        w++;
        acc = (acc >> 32) | (over << 32);
        over >>= 32;
        bits -= 32;
      }
    }
  });
  if (bits > 0) atomicOr(&gw[w], (unsigned)acc);
}

}  // namespace

void launch_huffman_build(DevBatch &b, int maxSymbols, cudaStream_t s) {
  const int smem = (int)build_smem_bytes(maxSymbols);
  // wide CTAs for a large alphabet (the sort and the list moves are as long as
  // it is); a batch of more than two cubelets per SM keeps 256 threads, eight
  // CTAs to an SM, so that all of them build in one wave
  if (maxSymbols > 600 && b.n <= 2 * 152) {
    raise_smem_limit(huffman_build_kernel<1024>, smem);
    huffman_build_kernel<1024><<<b.n, 1024, smem, s>>>(b);
  } else {
    raise_smem_limit(huffman_build_kernel<256>, smem);
    huffman_build_kernel<256><<<b.n, 256, smem, s>>>(b);
  }
}

void launch_pack_meta(DevBatch &b, cudaStream_t s) { pack_meta_kernel<<<b.n, 256, 0, s>>>(b); }

void launch_deliver(DevBatch &b, cudaStream_t s) {
  deliver_kernel<<<kDeliverBlocks, kDeliverThreads, 0, s>>>(b);
}

void launch_encode(DevBatch &b, int maxSymbols, cudaStream_t s) {
  const unsigned chunks = (unsigned)b.totalChunks;
  encode_count_kernel<<<(unsigned)b.totalEnc, kEncThreads, (maxSymbols + 15) & ~15, s>>>(b);
  encode_scan_kernel<<<b.n, 1024, 0, s>>>(b);
  cubelet_offsets_kernel<<<1, 1024, 0, s>>>(b);
  encode_zero_kernel<<<(chunks + 255) / 256, 256, 0, s>>>(b);
  const int smem = maxSymbols * (int)sizeof(unsigned long long);
  raise_smem_limit(encode_write_kernel, smem);
  encode_write_kernel<<<(unsigned)b.totalEnc, kEncThreads, smem, s>>>(b);
}

}  // namespace wl
