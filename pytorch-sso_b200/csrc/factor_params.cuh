// Launch parameters shared by the factor-construction kernels.
#pragma once
#include <stdint.h>

namespace sso {

struct FactorParams {
  const void* x;
  const float* weight;  // per-sample, nullable
  float* out;
  float* partial;  // workspace [tile][split][128*128]
  int64_t sn, sc, sh, sw;
  int64_t ldo;
  int64_t rows;  // n*ho*wo
  int n, c, h, w, ho, wo;
  int kh, kw, stride_h, stride_w, pad_h, pad_w, dil_h, dil_w;
  int d;        // columns incl. the ones column
  int dcols;    // c*kh*kw
  int splits;
  int rows_per_split;
  float alpha, beta;
  // tensor-core path only
  int* status;      // device word: 0 ok, else the code of the wait that gave up
  int perm_c;       // > 0: kernel columns are ordered (kh, kw, c) with c < perm_c; 0: natural order
  int perm_kk;      // kh*kw
  int perm_pub;     // > 0: public channel count (a group's columns past it are padding); 0: perm_c
  int perm_fold;    // > 0: the columns of a group are kx*perm_pub + c with kx < perm_fold (kernel width), groups are ky
  int accumulate;   // the partial tiles already hold the sums of earlier launches of this factor
  // finishing inside the producing kernel (factor_finish.cuh); tickets == nullptr: separate kernel
  int* tickets;     // [ticket_tiles] per-tile counters, then [ticket_tiles][16] per-group counters
  int ticket_tiles;
};

// Element (r, c) of a 128x128 partial tile of the tensor-core kernels: groups of four columns, rows inside a group.  An
// accumulate warp holds one row per lane, so its 16-byte stores are 512 contiguous bytes per instruction (row by row
// every store touched 32 lines: 6 us for the two tiles of a CTA).
__host__ __device__ __forceinline__ int part_at(int r, int c) { return ((c >> 2) * 128 + r) * 4 + (c & 3); }

// Public column of internal column j (the finishing kernels), -1 for padding.
__device__ __forceinline__ int public_column(const FactorParams& p, int j) {
  if (p.perm_c <= 0) return j;
  const int pub = p.perm_pub > 0 ? p.perm_pub : p.perm_c;
  if (j >= p.dcols) return pub * p.perm_kk;      // the ones column
  const int grp = j / p.perm_c, r = j - grp * p.perm_c;
  if (p.perm_fold > 0) {
    const int kx = r / pub;
    return kx < p.perm_fold ? (r - kx * pub) * p.perm_kk + grp * p.perm_fold + kx : -1;
  }
  return r < pub ? r * p.perm_kk + grp : -1;
}

// Scratch layout of the tensor-core factor kernels: [status word, 256 bytes][ticket counters]
// [partial tiles].  The header is cleared on the stream by every launch.
inline size_t factor_header_bytes(int tiles) {
  return 256 + (((size_t)tiles * 17 * sizeof(int) + 255) / 256) * 256;
}

struct RowInfo {   // one im2col row (n, ho, wo)
  int64_t base;    // n*sn
  int ih0, iw0;    // top-left input coordinate of the patch
  float wgt;       // sample weight (A operand only)
  int valid;
};
struct ColInfo {   // one im2col column (c, kh, kw) or the ones column
  int64_t off;     // c*sc
  int dh, dw;      // kh*dil_h, kw*dil_w
  int kind;        // 0 data, 1 ones, 2 out of range
  int pad;
};

}  // namespace sso
