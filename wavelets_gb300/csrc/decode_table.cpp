// What a Huffman decode table has to be before a stream is decoded with it.
#include <cstdlib>
#include <memory>

#include "wl_internal.h"

namespace wl {

// A table of n ints describes n / 2 nodes: (0, symbol) for a leaf, the two
// children for an inner node.  Accepted are trees: every inner node's children
// come after it, every node but the root is the child of exactly one, no code
// is longer than kMaxDecodeCode bits, and symbols are bins or the zero-run key.
// A table that loops, shares a node or ends nowhere would give the decoder
// tokens without an end or a length.
//
// The reference lists the nodes breadth first, the two children of a node next
// to each other (Huffman::computeDecodeTable, huffman.cc:177-228); that layout
// is checked in one pass without a branch per node, anything else with a depth
// per node.
//
// Returns the step tables that the decoder builds for it, -1 when it is not
// accepted.  A step table belongs to an inner node at the depth where the
// lookup table or another step table ends.
int decode_table_steps(const int *t, int n, int binCount, int dupKey) {
  if (n < 2 || n % 2) return -1;
  const int nodes = n / 2;
  const unsigned bins = (unsigned)binCount;
  const int key = dupKey < 0 ? 0 : dupKey;
  const auto symbol = [&](int s) { return ((unsigned)s < bins) | (s == key); };
  const auto stepDepth = [](int d) {
    return d >= kDecodeLutBits && (d - kDecodeLutBits) % kDecodeStepBits == 0;
  };
  if (t[0] == 0) return nodes == 1 && symbol(t[1]) ? 0 : -1;
  int next = 1, levelEnd = 1, depth = 0, steps = 0;
  unsigned off = 0;  // anything but the reference's layout
  for (int i = 0; i < nodes; i++) {
    if (i == levelEnd) {  // the next level: two nodes for every inner one of this
      if (stepDepth(depth)) steps += (next - i) / 2;
      levelEnd = next;
      depth++;
    }
    const int a = t[2 * i], b = t[2 * i + 1];
    // all ones for an inner node (a branch would be mispredicted every few nodes)
    const unsigned ua = (unsigned)a, inner = 0u - ((ua | (0u - ua)) >> 31);
    off |= (unsigned)(i >= next) | (~inner & (unsigned)!symbol(b)) |
           (inner & ((unsigned)(a ^ next) | (unsigned)(b ^ (next + 1))));
    next += (int)(inner & 2u);
  }
  if (off == 0 && next == nodes) return depth <= kMaxDecodeCode ? steps : -1;
  steps = 0;
  // depth of every node, 0: no parent yet
  const std::unique_ptr<unsigned char, void (*)(void *)> depths(
      static_cast<unsigned char *>(calloc(nodes, 1)), free);
  unsigned char *at = depths.get();
  if (!at) return -1;
  for (int i = 0; i < nodes; i++) {
    const int a = t[2 * i], b = t[2 * i + 1];
    if (i > 0 && at[i] == 0) return -1;
    if (a == 0) {
      if (!symbol(b)) return -1;
      continue;
    }
    if (a <= i || a >= nodes || b <= i || b >= nodes || a == b || at[a] || at[b] ||
        at[i] >= kMaxDecodeCode)
      return -1;
    steps += stepDepth(at[i]);
    at[a] = at[b] = (unsigned char)(at[i] + 1);
  }
  return steps;
}

}  // namespace wl

// for callers without a GPU
extern "C" int wl_internal_decode_table_steps(const int *t, int n, int binCount, int dupKey) {
  return wl::decode_table_steps(t, n, binCount, dupKey);
}
