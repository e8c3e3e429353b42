// Diagonal block of a 128-column Cholesky panel, done by eight warps: L = chol(D) and L^-1 for a
// (<=128)x(<=128) SPD block D, all in fp32 FMA arithmetic, in shared memory (pitch 132: the 16-byte loads of
// eight consecutive rows meet no bank conflict).
//
// The block is eight panels of 16 columns.  What bounds it is the chain of 128 pivots, so warp 0 does nothing but
// that chain: of panel k it takes the 16x16 diagonal block, subtracts the panel before, eliminates, and next solves
// the one 16x16 block that its next diagonal block needs.  The other warps follow half a step behind: trailing update
// by panel k - 1 and, in the idle half of the matrix, the sums G(k, c) = sum_j L(k, j) Inv(j, c) of row k of the
// inverse (20 to 28 block products a step, spread over seven warps by a table).  Two barriers a step:
//   X : panel k's block and its inverse are there, panel k - 1 has been subtracted everywhere
//       then, one 16x16 product per warp: L(i, k) = A(i, k) Inv_kk^T below, Inv(k, c) = -Inv_kk G(k, c) to the left
//   Y : those are there (warp 0 only announces its own and goes on)
// The elimination: lane l of warp 0 holds row l of the block, lane l + 16 row l of an identity that goes through the
// same steps, which leaves the inverse's column l in it for no further instruction; per pivot one round of shuffles
// (the raw column, and the next diagonal element so that the next pivot's rsqrt starts early).
// Rows and columns past the block's size behave as an identity block.  A pivot that is not a positive normal number
// (non-positive, denormal or NaN) is recorded once per matrix (LAPACK numbering) and replaced by 1, like the 64-wide
// kernel does for non-positive ones.
// Measured: 17 us for 128 rows (clocks: 1600 to 3100 per elimination, 750 per round of products, which are bound by
// the 512 bytes per 16-byte load and warp that shared memory returns); a chain of four barriers per panel with all
// warps in step and the inverse by three levels of doubling afterwards took 23.  Inside the dataflow kernel, with the
// inverse of the block announced before the other results are written: 1000 402 -> 307 us, 577+64 264 -> 203, the six
// factors of 784-1000-1000-10 433 -> 339, 4608+512 2208 -> 1715.
#pragma once
#include "common.cuh"

namespace sso {
namespace dpanel {

constexpr int PN = 128;        // rows / columns handled by one CTA
constexpr int PP = 132;        // pitch of the shared-memory matrices (floats)
constexpr int PK = 16;         // panel width inside the block
constexpr int THREADS = 256;
constexpr size_t SMEM_BYTES = (size_t)(2 * PN * PP) * sizeof(float);

// MUFU.RSQ alone (2 ulp); the argument is a positive normal number wherever this is called
__device__ __forceinline__ float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float x, float y, float z, float w) {
  *reinterpret_cast<float4*>(p) = make_float4(x, y, z, w);
}

// Barriers 1 and 2 of the eight warps that factorise a block, which may be part of a larger CTA.
__device__ __forceinline__ void sync_x() { asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory"); }
__device__ __forceinline__ void sync_y() { asm volatile("bar.sync 2, %0;" ::"n"(THREADS) : "memory"); }
__device__ __forceinline__ void arrive_y() { asm volatile("bar.arrive 2, %0;" ::"n"(THREADS) : "memory"); }

// A warp's 16x16x16 product: lane (rg, cg) holds rows rg, rg + 8; columns cg + 4 v of A B^T, 4 cg + v of A B.
struct Acc {
  float v[2][4];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) v[i][j] = 0.f;
  }
  __device__ __forceinline__ void add(int i, float4 a, const float4 (&b)[4]) {      // along q
#pragma unroll
    for (int j = 0; j < 4; ++j) v[i][j] = fmaf(a.x, b[j].x, v[i][j]);
#pragma unroll
    for (int j = 0; j < 4; ++j) v[i][j] = fmaf(a.y, b[j].y, v[i][j]);
#pragma unroll
    for (int j = 0; j < 4; ++j) v[i][j] = fmaf(a.z, b[j].z, v[i][j]);
#pragma unroll
    for (int j = 0; j < 4; ++j) v[i][j] = fmaf(a.w, b[j].w, v[i][j]);
  }
  __device__ __forceinline__ void nt(const float* __restrict__ A, const float* __restrict__ B, int rg, int cg) {
#pragma unroll
    for (int q = 0; q < PK; q += 4) {
      const float4 a0 = ld4(A + rg * PP + q), a1 = ld4(A + (rg + 8) * PP + q);
      float4 b[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = ld4(B + (cg + 4 * j) * PP + q);
      add(0, a0, b);
      add(1, a1, b);
    }
  }
  __device__ __forceinline__ void nn(const float* __restrict__ A, const float* __restrict__ B, int rg, int cg) {
#pragma unroll
    for (int q = 0; q < PK; q += 4) {
      const float4 a[2] = {ld4(A + rg * PP + q), ld4(A + (rg + 8) * PP + q)};
      float4 b[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = ld4(B + (q + j) * PP + 4 * cg);
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float x = j == 0 ? a[i].x : j == 1 ? a[i].y : j == 2 ? a[i].z : a[i].w;
          v[i][0] = fmaf(x, b[j].x, v[i][0]);
          v[i][1] = fmaf(x, b[j].y, v[i][1]);
          v[i][2] = fmaf(x, b[j].z, v[i][2]);
          v[i][3] = fmaf(x, b[j].w, v[i][3]);
        }
    }
  }
};

// What warps 1 to 7 do while warp 0 eliminates panel k >= 1: trailing blocks (i, j) and sums G(k, c), longest first to
// the warp with the least so far.
struct Schedule {
  unsigned char task[8][7][8];      // 0xFF: none; 0x80 | c: G(k, c); else i << 3 | j
};
constexpr Schedule make_schedule() {
  Schedule s{};
  for (int k = 0; k < 8; ++k) {
    int load[7] = {}, count[7] = {};
    for (int w = 0; w < 7; ++w)
      for (int t = 0; t < 8; ++t) s.task[k][w][t] = 0xFF;
    if (k == 0) continue;
    auto give = [&](int code, int cost) {
      int best = -1;
      for (int w = 0; w < 7; ++w)
        if (count[w] < 8 && (best < 0 || load[w] < load[best])) best = w;
      s.task[k][best][count[best]++] = (unsigned char)code;
      load[best] += cost;
    };
    for (int c = 0; c < k; ++c)
      if (k - c > 1) give(0x80 | c, 8 * (k - c) + 2);
    for (int i = k; i < 8; ++i)
      for (int j = k; j <= i; ++j)
        if (i != k) give(i << 3 | j, 10);
    give(0x80 | (k - 1), 10);
  }
  return s;
}
static __constant__ Schedule c_schedule = make_schedule();

// The elimination of panel k's diagonal block by one warp, after the subtraction of panel k - 1.
__device__ __forceinline__ void eliminate(float* __restrict__ S, float* __restrict__ V, int k, int n, int* __restrict__ info, int row0, int lane) {
  const int l = lane & 15, h = lane >> 4, c0 = PK * k;
  float* D = S + c0 * PP + c0;
  // row l of the block, columns 8 h ..: both halves of the warp subtract, the lower one collects
  float d[8];
  {
    const float4 u = ld4(D + l * PP + 8 * h), w = ld4(D + l * PP + 8 * h + 4);
    d[0] = u.x; d[1] = u.y; d[2] = u.z; d[3] = u.w; d[4] = w.x; d[5] = w.y; d[6] = w.z; d[7] = w.w;
  }
  if (k > 0) {
    const float* P = D - PK;
#pragma unroll
    for (int q = 0; q < PK; q += 4) {
      const float4 a = ld4(P + l * PP + q);
      float4 b[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) b[c] = ld4(P + (8 * h + c) * PP + q);
#pragma unroll
      for (int c = 0; c < 8; ++c) d[c] = fmaf(-a.x, b[c].x, d[c]);
#pragma unroll
      for (int c = 0; c < 8; ++c) d[c] = fmaf(-a.y, b[c].y, d[c]);
#pragma unroll
      for (int c = 0; c < 8; ++c) d[c] = fmaf(-a.z, b[c].z, d[c]);
#pragma unroll
      for (int c = 0; c < 8; ++c) d[c] = fmaf(-a.w, b[c].w, d[c]);
    }
  }
  float v[PK];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const float up = __shfl_down_sync(0xffffffffu, d[c], 16);
    v[c] = h ? (c == l ? 1.f : 0.f) : (c <= l ? d[c] : 0.f);
    v[c + 8] = h ? (c + 8 == l ? 1.f : 0.f) : (c + 8 <= l ? up : 0.f);
  }
  float pv = __shfl_sync(0xffffffffu, v[0], 0);
  int first_bad = -1;
#pragma unroll
  for (int j = 0; j < PK; ++j) {
    float t[PK];
#pragma unroll
    for (int c = j + 1; c < PK; ++c) t[c] = __shfl_sync(0xffffffffu, v[j], c);      // a[c][j]
    float d1 = 0.f;
    if (j + 1 < PK) d1 = __shfl_sync(0xffffffffu, v[j + 1], j + 1);                 // a[j+1][j+1] before this step
    const bool bad = !(pv >= 1.17549435e-38f);
    if (bad && first_bad < 0) first_bad = j;
    const float rs = bad ? 1.f : rsqrt_approx(pv);
    const float w = v[j] * (rs * rs);
#pragma unroll
    for (int c = j + 1; c < PK; ++c) v[c] = fmaf(-w, t[c], v[c]);
    v[j] = lane == j ? (bad ? 1.f : pv) * rs : v[j] * rs;
    if (j + 1 < PK) {
      const float x = t[j + 1] * rs;
      pv = fmaf(-x, x, d1);
    }
  }
  if (first_bad >= 0 && lane == 0 && info && c0 + first_bad < n) atomicCAS(info, 0, row0 + c0 + first_bad + 1);
  if (h == 0) {
#pragma unroll
    for (int q = 0; q < PK; q += 4)
      st4(D + l * PP + q, q <= l ? v[q] : 0.f, q + 1 <= l ? v[q + 1] : 0.f, q + 2 <= l ? v[q + 2] : 0.f, q + 3 <= l ? v[q + 3] : 0.f);
  } else {
#pragma unroll
    for (int r = 0; r < PK; ++r) V[(c0 + r) * PP + c0 + l] = v[r];
  }
}

// The factorisation itself, by 256 threads (barriers 1 and 2).  S holds the lower triangle on entry, visible to all of
// them, with an identity past the first n rows and columns; on return (behind a barrier) L in its lower triangle and
// L^-1, with zeros above the diagonal and the identity past n, in V.  `info` (nullable) receives the 1-based number
// row0 + pivot + 1 of the first bad pivot.
__device__ __forceinline__ void factor_block(float* __restrict__ S, float* __restrict__ V, int n, int* __restrict__ info, int row0, int tid) {
  const int lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int rg = lane >> 2, cg = lane & 3;
  const int np = (n + PK - 1) / PK;     // panels that hold columns of the matrix
  auto at = [](float* m, int i, int j) { return m + (PK * i) * PP + PK * j; };
  for (int k = 0; k < np; ++k) {
    if (warp == 0) {
      eliminate(S, V, k, n, info, row0, lane);
    } else if (k == 0) {
      // the inverse's upper half, and its identity past the matrix
      for (int e = tid - 32; e < PN * PN / 4; e += THREADS - 32) {
        const int r = e / (PN / 4), c = e % (PN / 4) * 4;
        if (c / PK > r / PK || r >= PK * np) st4(V + r * PP + c, c == r ? 1.f : 0.f, c + 1 == r ? 1.f : 0.f, c + 2 == r ? 1.f : 0.f, c + 3 == r ? 1.f : 0.f);
      }
    } else {
#pragma unroll 1
      for (int slot = 0; slot < 8; ++slot) {
        const int code = c_schedule.task[k][warp - 1][slot];
        if (code == 0xFF) break;
        Acc acc;
        acc.zero();
        if (code & 0x80) {
          const int c = code & 7;
#pragma unroll 1
          for (int j = c; j < k; ++j) acc.nn(at(S, k, j), at(V, j, c), rg, cg);
          float* G = at(S, c, k);
#pragma unroll
          for (int i = 0; i < 2; ++i) st4(G + (rg + 8 * i) * PP + 4 * cg, acc.v[i][0], acc.v[i][1], acc.v[i][2], acc.v[i][3]);
        } else {
          const int i0 = code >> 3, j0 = code & 7;
          if (i0 >= np) continue;
          acc.nt(at(S, i0, k - 1), at(S, j0, k - 1), rg, cg);
          float* C = at(S, i0, j0) + rg * PP + cg;
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) C[8 * i * PP + 4 * j] -= acc.v[i][j];
        }
      }
    }
    sync_x();
    // warp 0: the block below the diagonal one; the others: k blocks of the inverse's row, then the blocks further below
    const int m = warp - 1;
    const bool left = warp != 0 && m < k;
    const int i = warp == 0 ? k + 1 : k + 2 + (m - k);
    Acc acc;
    acc.zero();
    if (left) {
      acc.nn(at(V, k, k), at(S, m, k), rg, cg);
      float* O = at(V, k, m);
#pragma unroll
      for (int r = 0; r < 2; ++r) st4(O + (rg + 8 * r) * PP + 4 * cg, -acc.v[r][0], -acc.v[r][1], -acc.v[r][2], -acc.v[r][3]);
    } else if (i < np) {
      acc.nt(at(S, i, k), at(V, k, k), rg, cg);
      __syncwarp();
      float* O = at(S, i, k) + rg * PP + cg;
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int j = 0; j < 4; ++j) O[8 * r * PP + 4 * j] = acc.v[r][j];
    }
    if (warp == 0) {
      __syncwarp();
      if (k + 1 < np) arrive_y();
      else sync_y();
    } else {
      sync_y();
    }
  }
}

static __global__ void __launch_bounds__(THREADS, 1) diag_panel_kernel(const sso_diag_rec* __restrict__ recs,
                                                               int* __restrict__ info) {
  extern __shared__ __align__(16) float psm[];
  float* S = psm;               // the block, then L (lower triangle)
  float* V = psm + PN * PP;     // L^-1
  const sso_diag_rec rec = recs[blockIdx.x];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = rec.size;
  for (int r = warp; r < PN; r += THREADS / 32)
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int c = lane + 32 * u;
      if (c <= r) S[r * PP + c] = r < n ? rec.L[(int64_t)r * rec.ld_l + c] : (r == c ? 1.f : 0.f);
    }
  __syncthreads();
  factor_block(S, V, n, info ? info + 2 * rec.mat + rec.info_slot : nullptr, rec.row0, tid);
  // ---- results: the lower triangle of L, L^-1 with zeros above its diagonal, and optionally the upper
  // triangle of the transpose of L^-1.  Nothing reads L above the diagonal, and the buffer of the transpose
  // is zeroed before the factorisation starts.
  for (int r = warp; r < n; r += THREADS / 32) {
    float* lrow = rec.L + (int64_t)r * rec.ld_l;
    float* vrow = rec.Linv + (int64_t)r * rec.ld_inv;
    float* trow = rec.LinvT ? rec.LinvT + (int64_t)r * rec.ld_invt : nullptr;
    float lv[4], vv[4], tv[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {           // all loads of the row first, then all stores
      const int c = lane + 32 * u;
      lv[u] = S[r * PP + c];
      vv[u] = V[r * PP + c];
      tv[u] = V[c * PP + r];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int c = lane + 32 * u;
      if (c < n) {
        if (c <= r) lrow[c] = lv[u];
        vrow[c] = (c <= r) ? vv[u] : 0.f;     // read in full (K = 128) by the tasks of the rows below
        if (trow && c >= r) trow[c] = tv[u];
      }
    }
  }
}

}  // namespace dpanel
}  // namespace sso
