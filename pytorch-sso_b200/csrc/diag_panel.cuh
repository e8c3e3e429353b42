// Diagonal block of a 128-column Cholesky panel, done by eight warps: L = chol(D) and L^-1 for a
// (<=128)x(<=128) SPD block D, in shared memory (pitch 132: the 16-byte loads of
// eight consecutive rows meet no bank conflict).
//
// The block is eight panels of 16 columns.  What bounds it is the chain of 128 pivots, so warp 0 does nothing but
// that chain: of panel k it takes the 16x16 diagonal block, subtracts the panel before, eliminates, and next solves
// the one 16x16 block that its next diagonal block needs.  The other warps follow half a step behind with two things
// that are one and the same update: the trailing matrix (lower blocks), and the rows of an identity that go through
// the elimination with it and become L^-T (kept in the idle upper blocks).  Two barriers a step:
//   X : panel k's block and its inverse are there, panel k - 1 has been subtracted everywhere
//       then, one 16x16 product per warp: row block b of the panel, X(b, k) Inv_kk^T
//   Y : those are there (warp 0 only announces its own and goes on)
// The products are mma.sync on three bf16 parts of the fp32 operands, six products each as in factor_f32.cu (fp32
// grade); the parts of a panel are made once, when its row blocks are finished.  In fp32 FMA, with 2x4 outputs per
// lane, they were bound by the 512 bytes that shared memory returns per 16-byte load and warp, and took the
// elimination's shuffles along (17 us for 128 rows).
// The elimination: lane l of warp 0 holds row l of the block, lane l + 16 row l of an identity that goes through the
// same steps, which leaves the inverse's column l in it for no further instruction; per pivot one round of shuffles
// (the raw column, and the next diagonal element so that the next pivot's reciprocal starts early).
// Rows and columns past the block's size behave as an identity block.  A pivot that is not a positive normal number
// (non-positive, denormal or NaN) is recorded once per matrix (LAPACK numbering) and replaced by 1, like the 64-wide
// kernel does for non-positive ones.
// Measured: a 16x16 block in 1500 clocks (2280 with a reciprocal square root, a select and the scaling of the column on the
// chain between two pivots, and with the entries above the diagonal cleared), 128 rows in 22610 clocks (26270).  Before
// the elimination went in two steps of eight and took the next block from registers 14.4 us; a chain of four barriers per
// panel with all warps in step and the inverse by three levels of doubling afterwards took 23.  Elimination and products
// are straight-line code that issues an instruction in three to four clocks.
#pragma once
#include "common.cuh"

namespace sso {
namespace dpanel {

constexpr int PN = 128;        // rows / columns handled by one CTA
constexpr int PP = 132;        // pitch of the shared-memory matrices (floats)
constexpr int PK = 16;         // panel width inside the block
constexpr int THREADS = 256;
constexpr size_t SMEM_BYTES = (size_t)(2 * PN * PP) * sizeof(float) + 3 * PN * 48;      // two matrices, parts of a panel

// MUFU.RSQ alone (2 ulp); the argument is a positive normal number wherever this is called
__device__ __forceinline__ float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// MUFU.RCP alone (1 ulp); the same, but that it gives 0 above 2^126 (eliminate_large)
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
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

// The bf16 parts of the current panel: [part][row 0..127][16 columns], rows 48 bytes apart (eight consecutive ones on
// different banks).  Row block b > k holds L(b, k), b <= k column block k of L^-T.
constexpr uint32_t PL_ROW = 48, PL_PART = PN * PL_ROW;

__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t saddr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(saddr));
}
__device__ __forceinline__ void mma16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// A warp's 16x16x16 product A B^T of operands in three parts (six products; what is dropped is below 2^-24): lane
// (g, t) gets rows g, g + 8, columns 8 h + 2 t, + 1 of half h.  b[..][2 h], b[..][2 h + 1]: half h of B's rows.
__device__ __forceinline__ void product(float (&out)[2][4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][4]) {
  float small[2][4];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int i = 0; i < 4; ++i) out[h][i] = small[h][i] = 0.f;
#pragma unroll
  for (int h = 0; h < 2; ++h) { mma16(small[h], a[2], b[0][2 * h], b[0][2 * h + 1]); mma16(out[h], a[1], b[0][2 * h], b[0][2 * h + 1]); }
#pragma unroll
  for (int h = 0; h < 2; ++h) { mma16(small[h], a[0], b[2][2 * h], b[2][2 * h + 1]); mma16(out[h], a[0], b[1][2 * h], b[1][2 * h + 1]); }
#pragma unroll
  for (int h = 0; h < 2; ++h) { mma16(small[h], a[1], b[1][2 * h], b[1][2 * h + 1]); mma16(out[h], a[0], b[0][2 * h], b[0][2 * h + 1]); }
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int i = 0; i < 4; ++i) out[h][i] += small[h][i];
}
// C(i, j) -= P_i P_j^T (C = -P_i P_j^T if `fresh`), C a 16x16 block of S.
__device__ __forceinline__ void subtract(float* __restrict__ C, uint32_t planes, int i, int j, bool fresh, int lane) {
  uint32_t a[3][4], b[3][4];
  const uint32_t ra = planes + (16 * i + (lane & 15)) * PL_ROW + (lane >> 4) * 16;
  const uint32_t rb = planes + (16 * j + (lane & 7) + (lane >> 4) * 8) * PL_ROW + ((lane >> 3) & 1) * 16;
#pragma unroll
  for (int q = 0; q < 3; ++q) { ldmatrix4(a[q], ra + q * PL_PART); ldmatrix4(b[q], rb + q * PL_PART); }
  float2* c = reinterpret_cast<float2*>(C + (lane >> 2) * PP + 2 * (lane & 3));
  float2 v[2][2];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int r = 0; r < 2; ++r) v[h][r] = fresh ? make_float2(0.f, 0.f) : c[(8 * r * PP + 8 * h) / 2];
  float o[2][4];
  product(o, a, b);
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int r = 0; r < 2; ++r) c[(8 * r * PP + 8 * h) / 2] = make_float2(v[h][r].x - o[h][2 * r], v[h][r].y - o[h][2 * r + 1]);
}
// Three parts of the values at a lane's places (rows g, g + 8; columns 2 t, + 1 and 2 t + 8, + 9) of row block b: into
// `q` as the registers of an A operand, and to shared memory.
__device__ __forceinline__ void put_parts(uint32_t planes, int b, const float (&o)[2][4], uint32_t (&q)[3][4], int lane) {
  const uint32_t at = planes + (16 * b + (lane >> 2)) * PL_ROW + 4 * (lane & 3);
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      split2(o[h][2 * r], o[h][2 * r + 1], q[0][2 * h + r], q[1][2 * h + r], q[2][2 * h + r]);
#pragma unroll
      for (int i = 0; i < 3; ++i)
        asm volatile("st.shared.b32 [%0], %1;" ::"r"(at + i * PL_PART + 8 * r * PL_ROW + 16 * h), "r"(q[i][2 * h + r]) : "memory");
    }
}

// What warps 1 to 7 do while warp 0 eliminates panel k >= 1, one after the other: the blocks (i, j), j >= k, that panel
// k - 1 reaches - of the trailing matrix (i >= j, all but (k, k)) and of L^-T (i < k) - with those of column k first.
struct Schedule {
  unsigned char count[8], task[8][36];      // i << 3 | j
};
constexpr Schedule make_schedule() {
  Schedule s{};
  for (int k = 1; k < 8; ++k)
    for (int j = k; j < 8; ++j)
      for (int i = 0; i < 8; ++i)
        if ((i < k || i >= j) && !(i == k && j == k)) s.task[k][s.count[k]++] = (unsigned char)(i << 3 | j);
  return s;
}
static __constant__ Schedule c_schedule = make_schedule();

// A 16x16 block with an element above 2^125 on its diagonal, whose reciprocal may be no normal number: columns are scaled by
// reciprocal square roots before they are subtracted.  In shared memory and slow, for matrices near the largest float only.  D: the
// block, then L; V: L^-1.  Returns the bad pivots, a bit each.
__device__ __forceinline__ uint32_t eliminate_large(float* __restrict__ D, float* __restrict__ V, int lane) {
  const int l = lane & 15, h = lane >> 4;
  float* const row = h ? V + l : D + l * PP;      // as in eliminate: a row of the block, or a column of the inverse
  const int step = h ? PP : 1;
#pragma unroll 1
  for (int c = 0; h && c < PK; ++c) row[c * step] = c == l ? 1.f : 0.f;
  uint32_t bad_pivots = 0;
#pragma unroll 1
  for (int j = 0; j < PK; ++j) {
    __syncwarp();
    const float pv = D[j * PP + j];
    const bool bad = !(pv >= 1.17549435e-38f);
    if (bad) bad_pivots |= 1u << j;
    const float pivot = bad ? 1.f : pv, x = (lane == j ? pivot : row[j * step]) * rsqrt_approx(pivot);
    __syncwarp();
    row[j * step] = x;
    __syncwarp();
#pragma unroll 1
    for (int c = j + 1; c < PK; ++c) row[c * step] = fmaf(-x, D[c * PP + j], row[c * step]);
  }
  return bad_pivots;
}

// The elimination of panel k's diagonal block by one warp.  The block's entries above the diagonal are not looked at.
__device__ __forceinline__ void eliminate(float* __restrict__ S, float* __restrict__ V, int k, int n, int* __restrict__ info, int first, int dir, int lane) {
  const int l = lane & 15, h = lane >> 4, c0 = PK * k;
  float* D = S + c0 * PP + c0;
  float v[PK];
#pragma unroll
  for (int q = 0; q < PK; q += 4) {
    const float4 u = ld4(D + l * PP + q);
    const float d[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) v[q + i] = h ? (q + i == l ? 1.f : 0.f) : d[i];
  }
  auto report = [&](uint32_t bad_pivots) {
    if (!bad_pivots || lane != 0 || !info) return;
    const int bad = __ffs(bad_pivots) - 1;
    if (c0 + bad < n) atomicCAS(info, 0, first + dir * (c0 + bad));
  };
  const bool large = __any_sync(0xffffffffu, D[l * PP + l] > 0x1p125f);      // no pivot is larger than what it began as
  uint32_t bad_pivots = 0;
#pragma unroll
  for (int j0 = 0; j0 < PK; j0 += 8) {
    if (j0 > 0) {
      if (large) {      // asked here, when the answer has long been there; nothing has been stored yet
        report(eliminate_large(D, V + c0 * PP + c0, lane));
        return;
      }
      // the first eight columns from the other eight, all at once: rows 8 to 15 of them by way of shared memory (a
      // shuffle costs more than four cycles, 64 of them more than the sixteen loads)
      if (lane >= 8 && lane < 16) {
        st4(D + l * PP, v[0], v[1], v[2], v[3]);
        st4(D + l * PP + 4, v[4], v[5], v[6], v[7]);
      }
      __syncwarp();
#pragma unroll
      for (int c = 8; c < PK; ++c) {
        const float4 x = ld4(D + c * PP), y = ld4(D + c * PP + 4);
        float s0 = v[0] * x.x, s1 = v[4] * y.x;
        s0 = fmaf(v[1], x.y, s0); s1 = fmaf(v[5], y.y, s1);
        s0 = fmaf(v[2], x.z, s0); s1 = fmaf(v[6], y.z, s1);
        s0 = fmaf(v[3], x.w, s0); s1 = fmaf(v[7], y.w, s1);
        v[c] -= s0 + s1;
      }
    }
    // Columns stay unscaled (w = a[.][j] / pivot) until all eight are done: on the chain from one pivot to the next are a
    // reciprocal, a product and a sum, and the two shuffles it waits for go first.
    float scale[8], pv = __shfl_sync(0xffffffffu, v[j0], j0);
#pragma unroll
    for (int j = j0; j < j0 + 8; ++j) {
      float t[PK], d1 = 0.f;
      if (j + 1 < j0 + 8) {
        t[j + 1] = __shfl_sync(0xffffffffu, v[j], j + 1);          // a[j+1][j]
        d1 = __shfl_sync(0xffffffffu, v[j + 1], j + 1);            // a[j+1][j+1] before this step
      }
#pragma unroll
      for (int c = j + 2; c < j0 + 8; ++c) t[c] = __shfl_sync(0xffffffffu, v[j], c);
      const bool bad = !(pv >= 1.17549435e-38f);
      if (bad) bad_pivots |= 1u << j;
      const float pivot = bad ? 1.f : pv;
      const float inv = rcp_approx(pivot), w = v[j] * inv;
#pragma unroll
      for (int c = j + 1; c < j0 + 8; ++c) v[c] = fmaf(-w, t[c], v[c]);
      scale[j - j0] = rsqrt_approx(pivot);
      if (lane == j) v[j] = pivot;
      if (j + 1 < j0 + 8) pv = fmaf(-(t[j + 1] * inv), t[j + 1], d1);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j0 + j] *= scale[j];
  }
  if (h) {
#pragma unroll
    for (int r = 0; r < PK; ++r) V[(c0 + r) * PP + c0 + l] = v[r];
  } else {
#pragma unroll
    for (int q = 0; q < PK; q += 4) st4(D + l * PP + q, v[q], v[q + 1], v[q + 2], v[q + 3]);
  }
  report(bad_pivots);
}

// The factorisation itself, by 256 threads (barriers 1 and 2).  S holds the lower triangle on entry, visible to all of
// them, with an identity past the first n rows and columns; on return (behind a barrier) L in its lower triangle and
// L^-1, with zeros above the diagonal and the identity past n, in V.  `info` (nullable) receives the 1-based number
// of the first bad pivot, which is first + dir * pivot.
__device__ __forceinline__ void factor_block(float* __restrict__ S, float* __restrict__ V, int n, int* __restrict__ info, int first, int dir, int tid) {
  const int lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int g = lane >> 2, t = lane & 3;
  const int np = (n + PK - 1) / PK;     // panels that hold columns of the matrix
  const uint32_t planes = (uint32_t)__cvta_generic_to_shared(V + PN * PP);
  auto at = [](float* m, int i, int j) { return m + (PK * i) * PP + PK * j; };
  for (int k = 0; k < np; ++k) {
    if (warp == 0) {
      eliminate(S, V, k, n, info, first, dir, lane);
    } else if (k == 0) {
      // the inverse's upper half, and its identity past the matrix
      for (int e = tid - 32; e < PN * PN / 4; e += THREADS - 32) {
        const int r = e / (PN / 4), c = e % (PN / 4) * 4;
        if (c / PK > r / PK || r >= PK * np) st4(V + r * PP + c, c == r ? 1.f : 0.f, c + 1 == r ? 1.f : 0.f, c + 2 == r ? 1.f : 0.f, c + 3 == r ? 1.f : 0.f);
      }
    } else {
      const int count = c_schedule.count[k];
#pragma unroll 1
      for (int s = warp - 1; s < count; s += THREADS / 32 - 1) {
        const int code = c_schedule.task[k][s], i = code >> 3, j = code & 7;
        if (i < np && j < np) subtract(at(S, i, j), planes, i, j, i == k - 1, lane);
      }
    }
    sync_x();
    // row block b of the panel: warp 0 the one below the diagonal block, the others the rest
    const int b = warp == 0 ? k + 1 : warp - 1 <= k ? warp - 1 : warp;
    const bool more = k + 1 < np;       // a panel follows that needs this one's parts
    if (b == k) {
      if (more) {                       // L^-T's own block: the transposed inverse of the diagonal block
        const float* I = at(V, k, k);
        float o[2][4];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int i = 0; i < 4; ++i) o[h][i] = I[(8 * h + 2 * t + (i & 1)) * PP + g + 8 * (i >> 1)];
        uint32_t q[3][4];
        put_parts(planes, k, o, q, lane);
      }
    } else if (b < np) {                // X Inv_kk^T, X = S(b, k): below the diagonal a block of L, above one of L^-T
      float2* X = reinterpret_cast<float2*>(at(S, b, k) + g * PP + 2 * t);
      const float* I = at(V, k, k) + g * PP + 2 * t;
      uint32_t xa[3][4], xb[3][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {     // operand registers: row + 8 (i & 1), column + 8 (i >> 1); of B the other way round
        const float2 x = X[(8 * (i & 1) * PP + 8 * (i >> 1)) / 2];
        split2(x.x, x.y, xa[0][i], xa[1][i], xa[2][i]);
        const float2 y = *reinterpret_cast<const float2*>(I + 8 * (i >> 1) * PP + 8 * (i & 1));
        split2(y.x, y.y, xb[0][i], xb[1][i], xb[2][i]);
      }
      float o[2][4];
      product(o, xa, xb);
      if (b > k) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int r = 0; r < 2; ++r) X[(8 * r * PP + 8 * h) / 2] = make_float2(o[h][2 * r], o[h][2 * r + 1]);
      } else {
        float* O = at(V, k, b) + 2 * t * PP + g;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int i = 0; i < 4; ++i) O[(8 * h + (i & 1)) * PP + 8 * (i >> 1)] = o[h][i];
      }
      if (more) put_parts(planes, b, o, xa, lane);
      if (warp == 0) {
        __syncwarp();
        arrive_y();
        // the next diagonal block minus this panel: both operands are the block just finished, still in registers
#pragma unroll
        for (int i = 0; i < 3; ++i) { xb[i][0] = xa[i][0]; xb[i][1] = xa[i][2]; xb[i][2] = xa[i][1]; xb[i][3] = xa[i][3]; }
        float2* D = reinterpret_cast<float2*>(at(S, b, b) + g * PP + 2 * t);
        product(o, xa, xb);
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            float2& c = D[(8 * r * PP + 8 * h) / 2];
            c = make_float2(c.x - o[h][2 * r], c.y - o[h][2 * r + 1]);
          }
        __syncwarp();
      }
    }
    if (warp == 0) {
      if (!more) sync_y();
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
  factor_block(S, V, n, info ? info + 2 * rec.mat + rec.info_slot : nullptr, rec.row0 + 1, 1, tid);
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
