// Register passes (dwt_strided.cuh): which passes they take, and their launch.
#include "wl_internal.h"

namespace wl {

// one per pass and element type (dwt_strided_*.cu)
#define WL_STRIDED_DECLARE(NAME) \
  void NAME(const PassDesc *p, const int *tp, int n, int blocks, int L, bool full,  \
            cudaStream_t s);
WL_STRIDED_DECLARE(strided_y)
WL_STRIDED_DECLARE(strided_y_inv)
WL_STRIDED_DECLARE(strided_x_u8)
WL_STRIDED_DECLARE(strided_x_u16)
WL_STRIDED_DECLARE(strided_x_i32)
WL_STRIDED_DECLARE(strided_x_f32)
WL_STRIDED_DECLARE(strided_x_inv_u8)
WL_STRIDED_DECLARE(strided_x_inv_u16)
WL_STRIDED_DECLARE(strided_x_inv_i32)
WL_STRIDED_DECLARE(strided_x_inv_f32)
void strided_z(const PassDesc *p, const int *tp, int n, int blocks, int L, cudaStream_t s);
void strided_z_sel(const PassDesc *p, const int *tp, int n, int blocks, int L, cudaStream_t s);
void strided_z_inv(const PassDesc *p, const int *tp, int n, int blocks, int L, cudaStream_t s);

bool dwt_strided_own(int L) {
  return (L >= 16 && (L & (L - 1)) == 0) || L == 48 || L == 96 || L == 192;
}

namespace {

constexpr int kWarps = 4;  // per block (dwt_strided.cuh kThreads)

// lanes per row pair (0: another kernel), elements per lane and the most levels
int strided_lanes(int L) {
  switch (L) {
    case 16: case 32: case 48: return 1;
    case 64: case 96: return 2;
    case 128: case 192: return 4;
    case 256: return 8;
    case 512: return 16;
    case 1024: case 2048: return 32;
    default: return strided_elems(L) ? L / strided_elems(L) : 0;
  }
}
int strided_levels(int L) {
  if (!dwt_strided_own(L) || L % 48 == 0) {  // as often as a lane's elements halve
    int n = 0;
    for (int k = dwt_strided_own(L) ? 48 : strided_elems(L); k % 2 == 0; k /= 2) n++;
    return n;
  }
  int n = 0;
  while ((2 << n) <= L) n++;
  return n;
}

// length, levels and paired rows as the kernels take them
bool shape_fits(const PassDesc &d) {
  return strided_lanes(d.L) && d.steps >= 1 && d.B % 2 == 0 && d.steps <= strided_levels(d.L);
}
// rows at base with these strides (elements of es bytes) start at multiples
// of 16 bytes, so that every lane's K elements start at their vectors' size
bool rows_aligned(const void *base, long long sa, long long sb, int es) {
  return reinterpret_cast<size_t>(base) % 16 == 0 && sa * es % 16 == 0 && sb * es % 16 == 0;
}

}  // namespace

// rows per block (both rows of kWarps warps of 32 / G pairs)
int dwt_strided_rows_per_block(int L) { return 2 * kWarps * (32 / strided_lanes(L)); }

bool dwt_strided_fits(const PassDesc &d) {
  // neighbouring row pairs stay eight-byte aligned
  return shape_fits(d) && d.inSB == 1 && d.outSB == 1 &&
         ((d.inSA | d.inSC | d.outSA | d.outSC) & 1) == 0;
}
bool dwt_strided_source_fits(const PassDesc &d, int es) {
  return shape_fits(d) && d.inSC == 1 && d.outSB == 1 && ((d.outSA | d.outSC) & 1) == 0 &&
         (!dwt_strided_own(d.L) || rows_aligned(d.in, d.inSA, d.inSB, es));
}
bool dwt_strided_output_fits(const PassDesc &d, int es) {
  return shape_fits(d) && d.outSC == 1 && d.inSB == 1 && ((d.inSA | d.inSC) & 1) == 0 &&
         rows_aligned(d.out, d.outSA, d.outSB, es);
}

bool dwt_z_fits(const PassDesc &d) {
  // lengths of the row kernel stay with it, which is faster there: the z pass
  // of the mixed batch takes 0.67 ms there and 0.89 here, with whole sectors
  // a lane but a quarter of the warps
  const int k = strided_elems(d.L);
  if (!k || (dwt_strided_own(d.L) && d.L <= 256) || d.steps < 1 || d.inSC != 1 || d.outSC != 1)
    return false;
  int own = 0;
  for (int e = k; e % 2 == 0; e /= 2) own++;
  const auto at32 = [](const void *p, long long a, long long b) {
    return reinterpret_cast<size_t>(p) % 32 == 0 && a % 8 == 0 && b % 8 == 0;
  };
  return d.steps <= own && at32(d.in, d.inSA, d.inSB) && at32(d.out, d.outSA, d.outSB);
}
int dwt_z_rows_per_block(int L) {
  const int k = strided_elems(L);
  return 2 * 8 * (32 / (L / k)) * strided_z_rounds(k);
}
void launch_dwt_z(const PassDesc *p, const int *tp, int n, int blocks, int L, bool inverse,
                  bool sel, cudaStream_t s) {
  (inverse ? strided_z_inv : sel ? strided_z_sel : strided_z)(p, tp, n, blocks, L, s);
}

bool dwt_strided_full(const PassDesc &d, bool inverse) {
  int own = 0;  // levels on a lane's own elements
  for (int k = d.L / strided_lanes(d.L); k % 2 == 0; k /= 2) own++;
  return d.steps > own || (inverse && d.exact);
}

void launch_dwt_strided(const PassDesc *p, const int *tp, int n, int blocks, int L, bool inverse,
                        bool full, cudaStream_t s) {
  (inverse ? strided_y_inv : strided_y)(p, tp, n, blocks, L, full, s);
}
void launch_dwt_strided_x(const PassDesc *p, const int *tp, int n, int blocks, int L, int dtype,
                          bool inverse, bool full, cudaStream_t s) {
  switch (dtype) {
    case WL_U8: (inverse ? strided_x_inv_u8 : strided_x_u8)(p, tp, n, blocks, L, full, s); break;
    case WL_U16: (inverse ? strided_x_inv_u16 : strided_x_u16)(p, tp, n, blocks, L, full, s); break;
    case WL_I32: (inverse ? strided_x_inv_i32 : strided_x_i32)(p, tp, n, blocks, L, full, s); break;
    default: (inverse ? strided_x_inv_f32 : strided_x_f32)(p, tp, n, blocks, L, full, s); break;
  }
}

}  // namespace wl
