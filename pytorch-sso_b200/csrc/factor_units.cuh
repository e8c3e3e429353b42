// Finishing of a factor whose partial tiles lie in the scratch: splits summed, alpha / beta, the column permutation of
// k x k windows and the mirror.
//
// Internal columns are (k, c) - kernel position, channel - and public ones (c, k).  A unit is a pair of channel blocks
// (I, J), I >= J, of B channels each, at ALL kernel positions: the public rows and columns of such a block are
// contiguous (B * kk of them), and every element of the lower triangle that the unit's output and its mirror need
// belongs to no other unit.  So the partial tiles are read once, as 16 bytes per thread with eight rows of a column
// group next to each other (part_at), turned in shared memory, and written as contiguous runs of B * kk in both
// directions.  Without a permutation kk is 1 and B up to 64.
//
// Bound: the partial tiles (read once) and the result (written once, read once more if beta != 0).  The kernels before
// this one went by output rows and read each element of the lower triangle again for its mirror, four bytes at a time,
// or scattered four-byte stores.  Whole factors, us: fp32 512 channels 3x3 on 4x4 (d 4609, 128 images) 375 -> 323, adding
// to a running average 443 -> 356; bf16 512 channels 3x3 on 7x7 (d 4608, 32 images) 170 -> 123 and 234 -> 152.
// Items taken apart by shifts and results written 16 bytes at a time: the finishing of VGG-16's factors (four samples)
// 1508 -> 1238, of ResNet-50's 504 -> 427.
#pragma once
#include "common.cuh"
#include "factor_params.cuh"

namespace sso {
namespace units {

constexpr int SMEM_MAX = 200 * 1024;

struct Problem {
  const float* partial;    // [tile][split][128*128], part_at
  float* out;
  int64_t ldo;
  int c, kk, pub;          // pitch of a kernel position's columns, positions, channels that are public
  int dcols, d, splits;
  int block;               // channels of a unit's side: 4, or a multiple of 8 that divides 128
  int lanes;               // log2 of the lanes that share a sum
  int units;
  float alpha, beta;
};

// The column permutation (if any) is one that units cover, and a unit fits shared memory.
inline bool supported(const FactorParams& p) {
  if (p.perm_c <= 0) return true;
  return p.perm_fold == 0 && p.perm_c % 8 == 0 && (int64_t)(4 * p.perm_kk) * ((4 * p.perm_kk) | 1) * 4 <= SMEM_MAX;
}

inline int side(const Problem& u) { return u.block * u.kk; }
inline size_t smem_bytes(const Problem& u) { return (size_t)side(u) * (side(u) | 1) * sizeof(float); }

// `fill`: CTAs that would fill the GPU if this problem were alone (0: it is one of many).
inline Problem plan(const FactorParams& p, int fill) {
  Problem u;
  u.partial = p.partial; u.out = p.out; u.ldo = p.ldo;
  u.dcols = p.dcols; u.d = p.d; u.splits = p.splits;
  u.alpha = p.alpha; u.beta = p.beta;
  auto count = [&](int b) { const int n = ceil_div(u.pub, b); return n * (n + 1) / 2; };
  if (p.perm_c > 0) {
    u.c = p.perm_c; u.kk = p.perm_kk; u.pub = p.perm_pub > 0 ? p.perm_pub : p.perm_c;
    // eight channels read whole 128-byte lines and write longer runs; four where eight would leave SMs without a unit,
    // or a unit's square is more than a third of shared memory
    u.block = count(8) >= fill && 8 * u.kk <= 136 ? 8 : 4;
  } else {
    u.c = p.d; u.kk = 1; u.pub = p.d; u.dcols = p.d;
    u.block = 64;
    while (u.block > 16 && count(u.block) < 2 * fill) u.block >>= 1;
  }
  u.units = count(u.block);
  // lanes per sum: chains of at most eight partial tiles, where there are threads for it
  u.lanes = 0;
  while (u.lanes < 4 && u.splits >= (8 << u.lanes)) ++u.lanes;
  return u;
}

// Threads of a unit's CTA: more where units are few.
inline int threads(const Problem& u) {
  int64_t items = (int64_t)side(u) * side(u) / 4 << u.lanes;
  int t = 256;
  while (t < 1024 && (int64_t)u.units * t < 148 * 1024 && items > t) t *= 2;
  return t;
}

__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// The splits sub, sub + step, ... of four elements: two chains, in a fixed order.
__device__ __forceinline__ float4 sum_splits(const float* __restrict__ src, int sub, int step, int splits) {
  constexpr int64_t S = 128 * 128;
  float4 a = __ldcs(reinterpret_cast<const float4*>(src + sub * S));
  if (sub + step >= splits) return a;
  float4 b = __ldcs(reinterpret_cast<const float4*>(src + (sub + step) * S));
  int sp = sub + 2 * step;
#pragma unroll 2
  for (; sp + step < splits; sp += 2 * step) {
    const float4 v = __ldcs(reinterpret_cast<const float4*>(src + sp * S)), w = __ldcs(reinterpret_cast<const float4*>(src + (sp + step) * S));
    a = add4(a, v);
    b = add4(b, w);
  }
  if (sp < splits) a = add4(a, __ldcs(reinterpret_cast<const float4*>(src + sp * S)));
  return add4(a, b);
}

// One direction of a unit: rows x cols of the result from (row0, col0) on; an element's sum is s[r][c], or s[c][r] in the other
// direction.  Four columns at a time where the result allows 16-byte accesses.
template <bool TURNED>
__device__ __forceinline__ void write_block(const Problem& u, int row0, int col0, int rows, int cols, float alpha, const float* __restrict__ s, int pitch) {
  auto at = [&](int r, int c) { return TURNED ? s[c * pitch + r] : s[r * pitch + c]; };
  float* base = u.out + (int64_t)row0 * u.ldo + col0;
  if (cols % 4 == 0 && u.ldo % 4 == 0 && (reinterpret_cast<uintptr_t>(base) & 15) == 0) {
    const int quads = cols >> 2, dr = (int)blockDim.x / quads, dq = (int)blockDim.x - dr * quads;
    int r = (int)threadIdx.x / quads, q = (int)threadIdx.x - r * quads;
    while (r < rows) {
      float4 old[4];
      int rr[4], c[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {        // old values before the first store, so that the four are in flight together
        rr[j] = r;
        c[j] = 4 * q;
        if (u.beta != 0.f && r < rows) old[j] = *reinterpret_cast<const float4*>(base + (int64_t)r * u.ldo + c[j]);
        r += dr;
        q += dq;
        if (q >= quads) { q -= quads; ++r; }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (rr[j] >= rows) break;
        float4 v = make_float4(alpha * at(rr[j], c[j]), alpha * at(rr[j], c[j] + 1), alpha * at(rr[j], c[j] + 2), alpha * at(rr[j], c[j] + 3));
        if (u.beta != 0.f) v = make_float4(fmaf(u.beta, old[j].x, v.x), fmaf(u.beta, old[j].y, v.y), fmaf(u.beta, old[j].z, v.z), fmaf(u.beta, old[j].w, v.w));
        *reinterpret_cast<float4*>(base + (int64_t)rr[j] * u.ldo + c[j]) = v;
      }
    }
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int r0 = warp; r0 < rows; r0 += 4 * nw) {
    for (int c = lane; c < cols; c += 32) {
      float old[4];
      if (u.beta != 0.f) {
#pragma unroll
        for (int j = 0; j < 4; ++j) old[j] = r0 + j * nw < rows ? base[(int64_t)(r0 + j * nw) * u.ldo + c] : 0.f;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int r = r0 + j * nw;
        if (r >= rows) break;
        const float v = alpha * at(r, c);
        base[(int64_t)r * u.ldo + c] = u.beta == 0.f ? v : fmaf(u.beta, old[j], v);
      }
    }
  }
}

__device__ __forceinline__ void finish(const Problem& u, int unit, float* __restrict__ s, const int* status) {
  const int tid = threadIdx.x, nt = blockDim.x;
  const int B = u.block, kk = u.kk, E = B * kk, pitch = E | 1;
  int I, J;
  tri_decode(unit, I, J);
  const bool diag = I == J;
  const int64_t tile_floats = (int64_t)u.splits * (128 * 128);
  auto at = [&](int r, int c) {      // element (r, c), r >= c or in its tile, of the first split
    const int bi = r >> 7, bj = c >> 7;
    return u.partial + (int64_t)(bi * (bi + 1) / 2 + bj) * tile_floats + part_at(r & 127, c & 127);
  };
  // lanes: rows (up to eight), then the lanes of a sum, then column groups, then the rest of the rows
  const int rbits = min(B < 8 ? 2 : 3, 5 - u.lanes), rsub = 1 << rbits, sub_n = 1 << u.lanes;
  // a unit's side is a power of two, so that an item is taken apart by shifts; the pair of kernel positions (below 56 * 56)
  // by a multiplication.  With divisions the kernel was bound by its instructions (69 % of the issue slots)
  const int quad_bits = __ffs(B) - 3, pair_bits = quad_bits + __ffs(B) - 1 - rbits, pairs = kk * kk;
  const uint32_t inv_kk = (1u << 20) / (uint32_t)kk + 1u;
  const int n = pairs << (pair_bits + rbits + u.lanes);
  const int r_lo = tid & (rsub - 1), sub = (tid >> rbits) & (sub_n - 1);
#pragma unroll 2
  for (int t0 = tid & ~31; t0 < n; t0 += nt) {
    const int w = (t0 + (tid & 31)) >> (rbits + u.lanes);
    const int pair = w >> pair_bits, e = w & ((1 << pair_bits) - 1);
    const int q = e & ((1 << quad_bits) - 1), r = (e >> quad_bits) << rbits | r_lo;
    const int k1 = (int)(((uint32_t)pair * inv_kk) >> 20), k2 = pair - k1 * kk;
    bool valid = pair < pairs && sub < u.splits && !(diag && k1 < k2);
    const bool below = k1 >= k2;
    const int ri = below ? k1 * u.c + I * B + r : k2 * u.c + J * B + r;
    const int cj = below ? k2 * u.c + J * B + 4 * q : k1 * u.c + I * B + 4 * q;
    const bool on_diag = diag && k1 == k2;
    if (on_diag && 4 * q > r) valid = false;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (valid) v = sum_splits(at(ri, cj), sub, sub_n, u.splits);
    for (int o = rsub; o < rsub << u.lanes; o <<= 1) {
      v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
      v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
      v.z += __shfl_xor_sync(0xffffffffu, v.z, o);
      v.w += __shfl_xor_sync(0xffffffffu, v.w, o);
    }
    if (!valid || sub != 0) continue;
    const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = 4 * q + i;
      if (below) {
        if (on_diag && c > r) break;
        s[(r * kk + k1) * pitch + c * kk + k2] = x[i];
        if (diag) s[(c * kk + k2) * pitch + r * kk + k1] = x[i];
      } else {
        s[(c * kk + k1) * pitch + r * kk + k2] = x[i];
      }
    }
  }
  __syncthreads();
  const bool bad = status && *status != 0;
  const float alpha = bad ? __int_as_float(0x7fc00000) : u.alpha;      // NaN in place of a result whose kernel gave up
  const int row0 = I * E, col0 = J * E, rows = min(E, u.pub * kk - row0), cols = min(E, u.pub * kk - col0);
  write_block<false>(u, row0, col0, rows, cols, alpha, s, pitch);
  if (!diag) {
    write_block<true>(u, col0, row0, cols, rows, alpha, s, pitch);
    return;
  }
  // the ones column of a k x k window: its row and column next to this block, and the corner
  if (u.d == u.dcols) return;
  const int last = u.pub * kk;
  for (int b = tid; b < rows + (unit == 0 ? 1 : 0); b += nt) {
    const bool corner = b == rows;
    const int c = corner ? u.dcols : (b % kk) * u.c + J * B + b / kk, col = corner ? last : row0 + b;
    const float* src = at(u.dcols, c);
    float v = 0.f;
    for (int sp = 0; sp < u.splits; ++sp) v += src[(int64_t)sp * (128 * 128)];
    v *= alpha;
    float* o1 = u.out + (int64_t)last * u.ldo + col;
    float* o2 = u.out + (int64_t)col * u.ldo + last;
    const float v1 = u.beta != 0.f ? fmaf(u.beta, *o1, v) : v, v2 = u.beta != 0.f ? fmaf(u.beta, *o2, v) : v;
    *o1 = v1;
    if (!corner) *o2 = v2;
  }
}

}  // namespace units
}  // namespace sso
