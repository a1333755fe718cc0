// Internal declarations shared by the libwlgpu translation units.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <vector>

#include "wlgpu.h"

namespace wl {

#ifdef __CUDACC__
// a stage mark of the call (DevBatch::head)
__device__ __forceinline__ void stage_mark(long long *head, int i) {
  if (head && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    head[i] = (long long)t;
  }
}
#endif

__host__ __device__ inline int clz32(unsigned x) {
#ifdef __CUDA_ARCH__
  return __clz(x);
#else
  return __builtin_clz(x);
#endif
}

constexpr int kMaxBins = 4096;          // bins per cubelet (kernel tables)
constexpr int kMaxSymbols = kMaxBins + 1;
constexpr int kChunk = 4096;            // elements per select chunk
// Token chunks: the elements one warp quantizes and a group of bit-packer
// lanes packs, 1 << lg (DevBatch::lgChunk).  4096 for large batches (little
// per-chunk work), down to 512 -- a block of the quantizer -- where a call of
// n elements would otherwise run on fewer than 32 warps per SM of a 152-SM
// GB300: a warp codes its chunk from end to end (with 4096 always, a 64^2
// tile took 260 us a call, 180 us with 512; a 2048^2 image 342 and 323 us).
constexpr int kMinLgChunk = 9, kMaxLgChunk = 12;
inline int token_chunk_lg(long long n) {
  int lg = kMinLgChunk;
  while (lg < kMaxLgChunk && (n >> (lg + 1)) >= 152 * 32) lg++;
  return lg;
}
constexpr int kQuantWarps = 8;  // token chunks per quantize CTA, a warp each
constexpr int kChunkThreads = 256;
constexpr int kSelectBins = 4096;       // radix-select digit histogram
constexpr int kLloydBins = 4096;        // |coefficient| histogram for Lloyd
constexpr int kCandSlices = 64;        // CTAs per cubelet over its threshold candidates
constexpr int kLutCells = 4096;         // Lloyd bin lookup: cells of the float order key
constexpr int kLutStride = kLutCells + 8;  // per-cubelet table stride (16-byte rows)
// Chunks per select CTA: up to eight for large batches (few histogram
// flushes), fewer where eight would leave CTA slots empty (four CTAs of 256
// threads on each of a GB300's 152 SMs).
constexpr int kMaxSelGroup = 8;
inline int sel_group(long long chunks) {
  const long long slots = 152 * 4, g = (chunks + slots - 1) / slots;
  return (int)(g < 1 ? 1 : g > kMaxSelGroup ? kMaxSelGroup : g);
}
// Bit packer: a token chunk's values are split into F slices (F a power of
// two, 1..32), one lane each; a CTA of kEncThreads lanes packs kEncThreads / F
// consecutive chunks of one cubelet (four warps: few CTAs, so kernels of
// another stream still find CTA slots on the SMs).  Short slices keep many
// warps in flight (a lane's values are a serial chain), long ones share fewer
// words with their neighbours: 16 lanes per 4096 elements for large batches
// (encode stage of the mixed batch 0.53, 0.42 and 0.39 ms with 8, 16 and 32,
// of 729 sparser cubelets of 128^3 0.52, 0.51 and 0.64 ms); a call with fewer
// than kEncLanes lanes that way takes as many more as bring it there, at most
// 32 a chunk (packer of a 256^3 volume: 39, 21 and 14 us with 2^16, 2^17 and
// 2^18 lanes).
constexpr int kEncThreads = 128;
constexpr long long kEncLanes = 1 << 18;
inline int enc_slices(long long chunks, int lgChunk) {
  int f = 16 >> (kMaxLgChunk - lgChunk);
  while (f < 32 && chunks * f < kEncLanes) f *= 2;
  return f;
}
constexpr int kTileBudget = 16384;      // floats of shared memory per DWT tile
constexpr int kMaxAxis = 16384;         // longest padded axis (one row per tile)

// A value of a token chunk: its bin in bits 16 and up, the zero-bin elements
// between it and the chunk's value before it (0 for the first) below.
__host__ __device__ inline unsigned make_item(int bin, int gap) {
  return ((unsigned)bin << 16) | (unsigned)gap;
}

// Tokens of a zero-bin run, or of the part of one that starts in a chunk:
// 1024s from bit 16 on, powers of two 512 .. 16 as bits 5 .. 0 of bits 8 .. 13,
// below that 0 .. 8 singles, 8 + k for an eight and k = 1 .. 7 singles, or
// kEightAlone.  A whole run of L: see run_code.
constexpr int kEightAlone = 16;
__host__ __device__ inline unsigned run_code(int L) {
  return ((unsigned)(L >> 10) << 16) | ((unsigned)((L >> 4) & 63) << 8) | (unsigned)(L & 15);
}

// Tokens of a zero-bin run [s, e) that start inside [w0, w1) as a run code
// (HuffmanDup::dupCount / Huffman::dupEncodeString, huffman.h:31-57, 278-296:
// greedy runs of 1024, then the largest power of two >= 8 while more than 8
// remain, then single zero-bin tokens).
__host__ __device__ inline unsigned run_code_in(int s, int e, int w0, int w1) {
  const int q = (e - s) >> 10;
  int j0 = w0 > s ? (int)(((unsigned)(w0 - s) + 1023u) >> 10) : 0;
  int j1 = w1 > s ? (int)(((unsigned)(w1 - s) + 1023u) >> 10) : 0;
  if (j0 > q) j0 = q;
  if (j1 > q) j1 = q;
  unsigned code = (unsigned)(j1 - j0) << 16;
  int pos = s + (q << 10), r = e - pos;
  bool eight = false;
  while (r > 8) {
    const int lg = 31 - clz32(r);
    if (pos >= w0 && pos < w1) {
      if (lg == 3) eight = true;
      else code |= 1u << (8 + lg - 4);
    }
    pos += 1 << lg;
    r -= 1 << lg;
  }
  const int a = pos > w0 ? pos : w0, z = pos + r < w1 ? pos + r : w1;
  const int singles = z > a ? z - a : 0;
  return code | (unsigned)(eight ? (singles ? 8 + singles : kEightAlone) : singles);
}

struct CubeletState;

// One pass of the separable transform over one cubelet, as seen by the
// row kernel.  Rows are flattened r = b + B*a; row (a,b) of the input starts
// at in + a*inSA + b*inSB (contiguous along c); element (a,b,c) of the
// output goes to out + a*outSA + b*outSB + c*outSC.
struct PassDesc {
  const void *in;
  void *out;
  long long inSA, inSB;
  long long inSC;                   // input element stride (column-tile kernel)
  long long outSA, outSB, outSC;
  int L;          // row length (padded)
  int B;          // rows per 'a'
  int rows;       // total rows (A*B)
  int T;          // rows per tile (power of two)
  int tiles;
  int steps;
  int wavelet;    // WL_HAAR / WL_CDF97
  int exact;      // reference float order (filter bank) instead of lifting; inverse passes of
                  // the register kernels: the deferred scale undone by division
  int clampL, clampB, clampA;  // forward load: source sizes (REPEAT padding)
  int cropL, cropB, cropA;     // inverse store: destination sizes (crop)
  int vecLoad;                 // source is page-locked host memory: 16-byte row loads
  // last forward pass of a compression (row-register z pass): also gather the
  // first radix-select digit histogram and the extremes of the values it
  // writes into these (null: no statistics)
  unsigned *selHist;
  CubeletState *selState;
};

// Per-cubelet state written by the kernels and read back by the host.
struct CubeletState {
  // select
  unsigned minOrd, maxOrd;       // order-preserving encodings of min/max
  unsigned absMax, absMax2;      // bits of the two largest |c|
  unsigned prefix;               // radix-select prefix of the threshold bits
  unsigned long long rank;       // remaining rank inside the prefix bucket
  float threshold;
  float minVal, maxVal, maxAbs, maxAbs2;
  // quantizer
  int zeroBin;
  int dupValue;                  // -1 when zero runs are off
  float negScale, negOffset, posScale, posOffset;  // uniform
  // quantizer tables: Lloyd boundary/value counts; log table layout
  int nBounds, nValues;
  int lowBin, highNeg, nPos, nNeg;
  // Huffman
  unsigned long long totalBits;
  long long wordsBase;           // word offset of this cubelet in the packed output
  long long metaBase;            // int offset of its decode table (+ codebook) in the packed metadata
  int nWords;
  int longest;
  int nDecode;
  int nLeaves;
  int error;                     // nonzero: kernel-side failure code
  int pad_;
  // threshold bucket candidates, compacted into the cubelet's own region of
  // the second coefficient buffer (free once the transform is done)
  unsigned candCount;
  // Lloyd histogram bins: bin = (bits(|c|) - lloydBase) >> lloydShift for
  // threshold < |c| <= the Lloyd range top (bits lloydHiBits)
  unsigned lloydBase, lloydHiBits;
  int lloydShift;
  int lloydDeferred;             // 1: the compaction pass cannot tell; separate pass
  int pad2_;
};

// Everything a kernel needs about one cubelet of a batch.
struct CubeletDev {
  long long n;            // padded element count
  long long coefOff;      // float offset of the coefficients
  long long chunkBase;    // first token chunk
  long long wordsOff;     // word offset of the Huffman output
  long long wordsCap;     // capacity in words
  int nChunks;            // token chunks
  int selChunks;          // chunks of kChunk elements (select)
  int quantBase;          // first quantize CTA (kQuantWarps token chunks per CTA)
  int binCount;
  int quantAlg;
  int compressZeros;
  float frac;
  int lloydIters;
  int tableOff;           // offset into per-cubelet quantizer tables (floats)
  int nTable;             // entries in the table (log: boundaries; lloyd: boundaries)
  int groupBase;          // first select group (DevBatch::group chunks of kChunk)
  int encBase;            // first bit-packer CTA (kEncThreads / F chunks per CTA)
  int selFused;           // 1: the last transform pass gathered the first select
                          // digit and the extremes (no stand-alone first pass)
};

// Page-locked result storage of a call: words from `base` on, then (at the
// next multiple of 16 bytes) each cubelet's decode table and codebook; used
// when they take more than `above` and at most `cap` bytes.
struct OutSlab {
  char *base;
  long long cap, above;
};

// Device workspace for one batch.
struct DevBatch {
  int n;                          // cubelets
  CubeletDev *cub;                // [n]
  CubeletState *state;            // [n]
  float *coef;                    // coefficients (ping)
  float *coef2;                   // second buffer (pong)
  unsigned *items;                // values (make_item): a token chunk's from its first element's
                                  // place on (the second coefficient buffer, free by then)
  int lgChunk;                    // log2 of the elements per token chunk
  int *chunkVal;                  // values per token chunk
  uint2 *chunkEdge;               // per chunk: tokens (run_code) that start in it of the zero run
                                  // entering it and of the one leaving it
  unsigned *selHist;              // [n][kSelectBins]
  float *lloydHist;               // [n][kLloydBins][2] (count, sum)
  float *qtable;                  // quantizer tables
  uint16_t *qlut;                 // [n][kLutStride] Lloyd boundaries below each key cell
  float *dqtable;                 // dequant values [n][binCount]
  unsigned long long *hist;       // [n][kMaxSymbols] Huffman counts
  int4 *chunkRun;                 // per chunk: lead, trail, allZero, len
  unsigned *chunkLen;             // per chunk bit count
  unsigned long long *chunkBits;  // per chunk bit offset in its cubelet's stream
  unsigned long long *codes;      // [n][kMaxSymbols] code bits
  uint8_t *codeLen;               // [n][kMaxSymbols]
  int *decode;                    // [n][4*kMaxSymbols]
  uint32_t *words;                // Huffman output
  int *chunkCub;                  // [totalChunks] cubelet of every chunk
  int *groupCub;                  // [totalGroups] cubelet of every select group
  int *quantCub;                  // [totalQuant] cubelet of every quantize CTA
  long long totalQuant;
  long long totalGroups;
  int group;                      // chunks per select group
  int *encCub;                    // [totalEnc] cubelet of every bit-packer CTA
  long long totalEnc;
  int encF;                       // bit-packer slices per chunk
  unsigned *sliceOff;             // [totalChunks][32] bit offset of each slice in its chunk
  int4 *logHdr;                   // [n] log table layout from the host
  int *meta;                      // packed decode tables and Lloyd codebooks
  long long totalChunks;
  int maxChunks;                  // most chunks of one cubelet
  // Stage marks and output sizes of the call (null for a second half): the
  // marks are nanosecond clock readings taken by the first thread of the
  // kernel that starts a stage (event nodes between the kernels of a graph
  // cost 5 to 8 us each)
  long long *head;
  float2 *hostSel;                // page-locked: threshold, largest |c| of every cubelet
  const OutSlab *outSlab;         // in the upload block: where deliver_kernel puts the results
  CubeletState *hostState;        // page-locked copy of the states, deliver_kernel's
  long long *hostHead;            // and of head
};
enum { kMarkStart, kMarkSelect, kMarkQuant, kMarkBuild, kMarkEncode, kMarkEnd, kHeadWords,
       kHeadMeta, kHeadDelivered, kHeadCount };

// launchers (dwt.cu)
// Raise a kernel's dynamic shared-memory limit to at least `bytes`.  The
// limit is per kernel and process-wide; it only ever grows here, so a launch
// on one host thread cannot be undercut by a smaller setting from another.
void raise_smem_limit(const void *func, int bytes);
template <class F> inline void raise_smem_limit(F *func, int bytes) {
  raise_smem_limit(reinterpret_cast<const void *>(func), bytes);
}

void launch_dwt_pass(const PassDesc *d_passes, const int *d_tilePrefix,
                     int nPasses, int totalTiles, int smemBytes, int inType,
                     int outType, bool inverse, cudaStream_t s);
int dwt_tile_rows(int L, bool exact);
int dwt_smem_bytes(int L, int T, bool exact);
// column-tile passes (dwt_cols.cu): lifting / Haar, rows up to kColsMaxL
constexpr int kColsMaxL = 512;
void launch_dwt_cols(const PassDesc *d_passes, const int *d_tilePrefix, int nPasses, int tiles,
                     int smem, int rows, int warps, int inType, int outType, bool inverse,
                     bool vecLoad,
                     cudaStream_t s);
int dwt_cols_tile_rows(int L);               // default tile height for rows of L
int dwt_cols_smem_bytes(int L, int rows);
bool dwt_cols_rows_fit(int L, int rows);      // rows in {32, 64, 128} and smem fits
// row-register forward passes (dwt_rows.cu): float rows contiguous on both
// sides, L a power of two in 16 .. 256, 1 <= steps <= log2 L
bool dwt_rowreg_fits(int L, int steps);
// rows per block; sel: the last pass, which also gathers the select
// statistics of the values it writes (PassDesc::selHist), several row rounds
// per block
int dwt_rowreg_rows_per_block(int L, bool sel = false);
void launch_dwt_rowreg(const PassDesc *d_passes, const int *d_tilePrefix, int nPasses, int blocks,
                       int L, bool sel, cudaStream_t s);
// the inverse of the in-place pass (the first inverse pass, z)
void launch_dwt_rowreg_inv(const PassDesc *d_passes, const int *d_tilePrefix, int nPasses,
                           int blocks, int L, cudaStream_t s);
int dwt_rowreg_t_rows_per_block(int L);
// inverse y and x passes (rows strided in the input, neighbouring rows
// neighbours in memory): rows through a shared-memory tile of
// dwt_rowreg_t_rows_per_block(L) rows, out to outType (the x pass: rows
// contiguous in the output, cropped) or back through the tile (the y pass)
void launch_dwt_rowreg_inv_t(const PassDesc *d_passes, const int *d_tilePrefix, int nPasses,
                             int blocks, int L, int outType, cudaStream_t s);
// the same with the rows read from any element type (REPEAT clamp) and
// stored through a shared-memory tile to an output where consecutive rows
// are neighbours (forward x and y passes)
void launch_dwt_rowreg_t(const PassDesc *d_passes, const int *d_tilePrefix, int nPasses,
                         int blocks, int L, int inType, cudaStream_t s);

// passes in registers whose neighbouring rows are neighbours in memory
// (dwt_strided.cu): the y passes; the forward x pass of source rows of es-byte
// elements in device memory; the inverse x pass into such rows
bool dwt_strided_fits(const PassDesc &d);
bool dwt_strided_source_fits(const PassDesc &d, int es);
bool dwt_strided_output_fits(const PassDesc &d, int es);
// full: the kernel with levels across lanes and division (all passes of a
// launch, or none, need it)
bool dwt_strided_full(const PassDesc &d, bool inverse);
void launch_dwt_strided_x(const PassDesc *d_passes, const int *d_tilePrefix, int nPasses,
                          int blocks, int L, int dtype, bool inverse, bool full, cudaStream_t s);
int dwt_strided_rows_per_block(int L);
// a length with a kernel of its own (else: all of strided_elems(L) in one launch)
bool dwt_strided_own(int L);
// elements a lane holds of rows whose length has no kernel of its own, 0: not
// taken.  They halve five, four or three times; at most 16 lanes a row, so
// that neighbouring lanes still share sectors.  (With 48, 40 and 24 besides, a
// batch of 40 odd sizes had a third more launches and took as long, and the y
// passes of 400 of them took 0.38 ms instead of 0.34.)
constexpr int strided_elems(int L) {
  for (int k : {32, 16, 8})
    if (L % k == 0 && L / k <= 16) return k;
  return 0;
}
// z passes of the same kernels: contiguous rows, in place, as many levels as a
// lane's elements halve; the forward pass may gather the select statistics.
// One launch for all lengths of the same strided_elems.
bool dwt_z_fits(const PassDesc &d);
int dwt_z_rows_per_block(int L);
void launch_dwt_z(const PassDesc *d_passes, const int *d_tilePrefix, int nPasses, int blocks,
                  int L, bool inverse, bool sel, cudaStream_t s);
// rounds of a block over rows of k elements a lane: some 16 K values
constexpr int strided_z_rounds(int k) { return k < 32 ? 32 / k : 1; }
void launch_dwt_strided(const PassDesc *d_passes, const int *d_tilePrefix, int nPasses, int blocks,
                        int L, bool inverse, bool full, cudaStream_t s);

// ---- column-tile heights per size class (tune.cpp) ----
enum TuneKind { kTuneFwdX, kTuneFwdY, kTuneFwdZ, kTuneInvZ, kTuneInvY, kTuneInvX, kTuneKinds };
int tune_type_index(int dtype, bool vec);
// tile shape (rows, warps) for rows of up to L elements: the tuned entry,
// else the default
struct TileShape {
  int rows, warps;
};
constexpr int kTileShapes = 6;  // candidates: rows 32/64/128 x warps 4/8
constexpr TileShape kTileShape[kTileShapes] = {{32, 4}, {64, 4}, {128, 4},
                                               {32, 8}, {64, 8}, {128, 8}};
TileShape tuned_cols_shape(int kind, int typeIdx, int L);
void set_tuned_cols_shape(int kind, int typeIdx, int cls, TileShape t,
                          const float us[kTileShapes]);
unsigned tune_version();  // changes whenever the table does

// A block of page-locked host memory that a kernel copies to the device on its
// way.  A copy node in front of a graph's kernels is handed to the copy engine
// apart from them; with a
// copy node each graph of a 64^3 call and of a 2048^2 image took some 3 us more
// (calls: 160 -> 155 us, 250 -> 244 us, mixed batch of 40: 797 -> 761 us).
struct Upload {
  const uint4 *src;  // null: already there
  uint4 *dst;
  int vecs;          // of 16 bytes
  // the host's copy of something at a device address inside the block
  template <typename T> __device__ const T *host(const T *p) const {
    return src ? reinterpret_cast<const T *>(
                     reinterpret_cast<const char *>(src) +
                     (reinterpret_cast<const char *>(p) - reinterpret_cast<const char *>(dst)))
               : p;
  }
};
// launchers (select.cu)
// everything a call's kernels expect set: histograms and states zeroed, the
// select state (extremes from FLT_MAX / FLT_MIN), cubelet of every chunk;
// runs before the transform, whose last pass may gather the first digit
void launch_init(DevBatch &b, bool lloyd, const Upload &up, cudaStream_t s);
// pass0: run the stand-alone first digit pass for the cubelets whose last
// transform pass did not gather it (CubeletDev::selFused == 0)
void launch_select(DevBatch &b, const float *coef, bool pass0, cudaStream_t s);

// launchers (quant.cu)
void launch_quant_params(DevBatch &b, const Upload &up, cudaStream_t s);
void launch_lloyd(DevBatch &b, const float *coef, int maxBins, cudaStream_t s);
// sum of squared differences of two u8 arrays into *out (opt.cu)
void launch_sq_err_u8(const uint8_t *a, const uint8_t *b, long long n, unsigned long long *out,
                      cudaStream_t s);
void launch_quantize(DevBatch &b, const float *coef, int maxTable, int maxSymbols, bool lloyd,
                     cudaStream_t s);
void launch_runs(DevBatch &b, cudaStream_t s);

// error metrics (errors.cu): per-CTA double sums {a, a*a, |d|, d*d} of the
// original (dtype) against the restored floats, blocks = err_sums_blocks(n)
int err_sums_blocks(long long n);
void launch_err_sums(const void *orig, int dtype, const float *rest, long long n, double *part,
                     int blocks, cudaStream_t s);

// launchers (huffman.cu)
void launch_huffman_build(DevBatch &b, int maxSymbols, cudaStream_t s);
void launch_encode(DevBatch &b, int maxSymbols, cudaStream_t s);
void launch_pack_meta(DevBatch &b, cudaStream_t s);
// states, head and (when they fit in the slab) words, decode tables and
// codebooks straight to page-locked host memory
void launch_deliver(DevBatch &b, cudaStream_t s);

// batched Huffman decoding (decode.cu): the streams of n cubelets to their
// dequantized values
struct DecodeCub {
  const uint32_t *words;  // device
  long long nWords;
  const int *table;       // device
  int nTable;
  int dupKey, dupValue, binCount;
  long long n;            // elements
  float *out;             // values
  int fill;               // dupValue >= 0: 1: the decoder sets dq[dupValue] everywhere
                          // first, 0: the output holds it already
  const float *dq;        // dequantized value of every bin
  long long subBase, nSub;   // subsequences (decode_subs)
  int tileBase, nTiles;      // tiles (decode_tiles)
  long long lutOff;          // decode_lut_size() entries
  long long stepOff;         // step tables (decode_table_steps)
  int nSteps;
};
// elements of a tile's output up to which the decoder fills it itself
constexpr long long kDecodeFillTile = 1 << 20;
struct DecodeArrays {
  unsigned *lut, *steps;
  int *stepCount;         // step tables of every stream
  uint8_t *subStart;      // first token boundary of every subsequence
  unsigned *subCount;     // elements and values of every subsequence
  const int *tileCub;     // cubelet of every tile
  int *tileEntry, *tileExit;
  unsigned *tileCount;
  long long *tileOff;
  int *flags;             // kDecodeFlags counters, zero before the first launch
  int *hostFlags;         // page-locked copy of them, the write pass's
};
enum {
  kDecodeFirst, kDecodeAgain,  // tiles decoded again by the first / second check
  kDecodeBad,                  // malformed streams
  kDecodeShort,                // streams with fewer values than their cubelet
  kDecodeFlags
};
struct DecodeBatch {
  int n, tiles;           // streams, tiles in all
  int maxTable;
};
constexpr int kMaxDecodeCode = 60;  // longest code decoded (with its length bits 63)
constexpr int kDecodeLutBits = 12, kDecodeStepBits = 4;  // of a code, per table
// step tables of a decode table, -1: not one that the decoder takes
// (decode_table.cpp)
int decode_table_steps(const int *t, int n, int binCount, int dupKey);
long long decode_subs(long long nWords);
int decode_tiles(long long nWords);
int decode_lut_size();
size_t decode_step_bytes(long long steps);
// the whole decode (returns the kernels launched); if flags[kDecodeAgain] is
// not zero afterwards: zero it and launch_decode_check until it stays zero,
// then fill the outputs and launch_decode_write again
int launch_decode(const DecodeCub *cubs, const DecodeBatch &b, const DecodeArrays &d,
                  cudaStream_t s);
void launch_decode_check(const DecodeCub *cubs, const DecodeBatch &b, const DecodeArrays &d,
                         cudaStream_t s);
int launch_decode_write(const DecodeCub *cubs, const DecodeBatch &b, const DecodeArrays &d,
                        cudaStream_t s);
// n floats at out set to v, for many ranges in one launch (blocks of
// kFillBlock elements; blockBase = the range's first block)
constexpr int kFillBlock = 4096;
struct FillItem {
  float *out;  // 16-byte aligned
  long long n;
  float v;
  long long blockBase;
};
void launch_fill_batch(const FillItem *items, int nItems, long long totalBlocks, cudaStream_t s);

// host-side exact log-quantizer tables (quant_host.cpp)
struct LogTable {
  std::vector<float> bounds;   // see quant_host.cpp for the layout
  int lowBin, highNeg, nPos, nNeg;
  float negScale, negOffset, posScale, posOffset;
};
void log_quant_table(int binCount, float threshold, float maxVal, LogTable &t);
void dequant_values(int quantAlg, int binCount, float threshold, float maxVal,
                    const float *codebookValues, float *out);

}  // namespace wl
