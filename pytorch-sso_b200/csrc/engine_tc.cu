// Tile tasks on the tensor cores:  C[m x n] <- alpha * op(A)[m x k] * op(B)[k x n] + beta * C  with
// m, n <= 128, fp32 in / fp32 out, computed as 3xTF32 on tcgen05 (x = hi + lo, hi = rna_tf32(x);
// lo*hi + hi*lo + hi*hi into one TMEM accumulator that is drained into fp32 registers every two
// stages, because the tensor core's own accumulation truncates).
//
// One CTA per task, 17 warps: 8 accumulate warps, 1 MMA warp, 8 load warps.  Both operands end up
// K-major in shared memory in the canonical SWIZZLE_128B layout: one operand row = 32 k = 128
// bytes, eight rows = one 1024-byte atom, the 16-byte chunk index XOR-ed with (row & 7).  Core
// matrices are then aligned to 128-byte lines, which the tensor core needs to read shared memory
// at full rate (padded no-swizzle layouts halve it), and the swizzle keeps the stores free of
// bank conflicts:
//   * operand contiguous along k in global memory (A not transposed, B transposed): a thread loads
//     16 bytes = 4 consecutive k of one row and stores them as one chunk; 8 lanes = one row;
//   * operand contiguous along its row/column index (A transposed, B not transposed): a thread loads
//     4 consecutive indices of one k and scatters them with scalar stores; a warp covers 16 k x 8
//     indices so that its 32 stores fall into 32 different banks.
// Unaligned bases / leading dimensions (odd matrix sizes) fall back to element loads.
// Every wait is bounded; a timeout sets *status and the task writes nothing.
#include "common.cuh"
#include "tc_common.cuh"
#include "tc_pair.cuh"

namespace sso {
namespace etc {

using namespace tc;

constexpr int TILE = 128, KS = 32, STAGES = 3;
constexpr int EPI_WARPS = 8, MMA_WARP = 8, LOAD_WARPS = 8;
constexpr int THREADS = 32 * (EPI_WARPS + 1 + LOAD_WARPS);
constexpr uint32_t OPB = TILE * 128;                // bytes of one operand part (hi or lo) of one stage
constexpr uint32_t STAGE_BYTES = 4 * OPB;           // A_hi A_lo B_hi B_lo
constexpr uint32_t TMEM_COLS = 256;
constexpr int FLUSH = 2;
constexpr int CT_LD = TILE + 1;           // row pitch of the output tile staged in shared memory

__device__ __forceinline__ uint64_t smem_desc_sw128_kmajor(uint32_t saddr) {
  // start address, LBO unused for a K-major operand one swizzle atom wide, SBO = 1024 (eight
  // rows), descriptor version 1, layout type 2 = SWIZZLE_128B
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(1024u >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// byte offset of element (row r, k) inside one operand part
__device__ __forceinline__ uint32_t sw_off(int r, int k) {
  return (uint32_t)(r >> 3) * 1024u + (uint32_t)(r & 7) * 128u + (uint32_t)(((k >> 2) ^ (r & 7)) << 4) + (uint32_t)(k & 3) * 4u;
}

__device__ __forceinline__ void split_store4(uint32_t addr, float4 v) {
  const uint32_t h0 = rna_tf32(v.x), h1 = rna_tf32(v.y), h2 = rna_tf32(v.z), h3 = rna_tf32(v.w);
  const uint32_t l0 = __float_as_uint(v.x - __uint_as_float(h0)), l1 = __float_as_uint(v.y - __uint_as_float(h1));
  const uint32_t l2 = __float_as_uint(v.z - __uint_as_float(h2)), l3 = __float_as_uint(v.w - __uint_as_float(h3));
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(h0), "r"(h1), "r"(h2), "r"(h3) : "memory");
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr + OPB), "r"(l0), "r"(l1), "r"(l2), "r"(l3) : "memory");
}
__device__ __forceinline__ void split_store1(uint32_t addr, float x) {
  const uint32_t h = rna_tf32(x);
  const uint32_t l = __float_as_uint(x - __uint_as_float(h));
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(h) : "memory");
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr + OPB), "r"(l) : "memory");
}

// 4 consecutive elements along the contiguous direction starting at (fixed, first); elements whose
// contiguous index is >= lim_c or whose other index is out of range read as zero.
__device__ __forceinline__ float4 load4(const float* __restrict__ P, int64_t ld, int fixed, int first, bool fixed_ok,
                                        int lim_c, bool vec_ok) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (!fixed_ok || first >= lim_c) return v;
  const float* q = P + (int64_t)fixed * ld + first;
  if (vec_ok && first + 3 < lim_c) return __ldg(reinterpret_cast<const float4*>(q));
  v.x = __ldg(q);
  if (first + 1 < lim_c) v.y = __ldg(q + 1);
  if (first + 2 < lim_c) v.z = __ldg(q + 2);
  if (first + 3 < lim_c) v.w = __ldg(q + 3);
  return v;
}

// Stage-invariant addressing of one operand for one load thread (lt = 0..255).
//   k-contiguous operand: chunk j is row (lt>>3) + 32j, k = (lt&7)*4 .. +3;
//   other operand: with w = lt>>5, kq = lt&15, rc = (lt>>4)&1, chunk j is k = (j&1)*16 + kq and the
//   four indices 4c .. 4c+3, c = 4w + 2(j>>1) + rc.
struct OpLoad {
  const float* p0;      // chunk j of stage s is at p0 + joff(j) + s*step
  int64_t ja, step;     // k-contiguous: joff = j*ja;  other: joff = (j&1)*ja + (j>>1)*8
  uint32_t so0;         // k-contiguous: chunk j is stored at so0 + j*4096
  uint32_t okmask;
  bool fast;
};
__device__ __forceinline__ OpLoad make_op(const float* P, int ld, bool kc, int lim, int lt, bool vec) {
  OpLoad o;
  o.okmask = 0u;
  o.fast = vec;
  o.step = kc ? (int64_t)KS : (int64_t)KS * ld;
  if (kc) {
    const int q = lt >> 3, l8 = lt & 7;
    o.p0 = P + (int64_t)q * ld + l8 * 4;
    o.ja = (int64_t)32 * ld;
    o.so0 = sw_off(q, l8 * 4);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (q + 32 * j < lim) o.okmask |= 1u << j;
  } else {
    const int w = lt >> 5, kq = lt & 15, rc = (lt >> 4) & 1;
    o.p0 = P + (int64_t)kq * ld + (4 * w + rc) * 4;
    o.ja = (int64_t)16 * ld;
    o.so0 = 0u;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int idx = (4 * w + 2 * (j >> 1) + rc) * 4;
      if (idx + 3 < lim) o.okmask |= 1u << j;
      else if (idx < lim) o.fast = false;    // a chunk straddling the edge needs the checked loads
    }
  }
  return o;
}

// Role of the 8 accumulate warps: drain the TMEM accumulator chunk by chunk into fp32 registers,
// then write the tile.  accfull0 / accempty0 are the shared addresses of barrier pairs (b = 0, 1
// at +8 bytes).  `ct` is shared memory that is free once the last commit has fired.
__device__ __forceinline__ void accumulate_and_store(const sso_tile_task& t, uint32_t tmem_base, uint32_t accfull0,
                                                     uint32_t accempty0, int nchunks, int* status, float* ct,
                                                     int warp, int lane) {
  auto accfull_bar = [&](int b) { return accfull0 + 8u * b; };
  auto accempty_bar = [&](int b) { return accempty0 + 8u * b; };
  const int q = warp & 3, half = warp >> 2;
  float acc[64];
#pragma unroll
  for (int i = 0; i < 64; ++i) acc[i] = 0.f;
  bool ok = true;
  for (int c = 0; c < nchunks; ++c) {
    const int b = c & 1;
    if (!mbar_wait(accfull_bar(b), (c >> 1) & 1, status, 13)) { ok = false; break; }
    tc_fence_after();
    const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * TILE + half * 64);
    uint32_t v0[32], v1[32];
    tmem_ld32(taddr, v0);
    tmem_ld32(taddr + 32, v1);
    tmem_ld_wait();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(accempty_bar(b));
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      acc[i] += __uint_as_float(v0[i]);
      acc[32 + i] += __uint_as_float(v1[i]);
    }
  }
  // The operand buffers are free now (the last commit has fired, so every MMA has read them):
  // stage the tile there, row r at r*129 floats, and write C (and its mirror) with whole
  // warps per row so that global accesses are coalesced.
  // A wait that gave up leaves the accumulator incomplete: the tile is written all the same, as NaN, so
  // that nothing downstream can mistake a stale or partial result for a valid one.
  const int r = q * 32 + lane;
  if (!ok) {
#pragma unroll
    for (int i = 0; i < 64; ++i) acc[i] = __int_as_float(0x7fc00000);
  }
#pragma unroll
  for (int i = 0; i < 64; ++i) ct[r * CT_LD + half * 64 + i] = t.alpha * acc[i];
  asm volatile("bar.sync 1, %0;" ::"n"(32 * EPI_WARPS) : "memory");
  {
    const bool sym = (t.flags & 4u) != 0;
    if (t.beta != 0.f) {
      // an updated tile: the old values of four rows (16 loads per lane) are fetched before anything is
      // stored; one row at a time, every load would wait behind the previous row's stores to the same
      // array, i.e. 64 round trips to L2 in a row per warp (measured: 29 us against 13 us for the same
      // task with beta = 0)
      for (int r0 = warp; r0 < t.m; r0 += 4 * EPI_WARPS) {
        float old[4][TILE / 32];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int rr = r0 + j * EPI_WARPS;
#pragma unroll
          for (int u = 0; u < TILE / 32; ++u) {
            const int c = lane + 32 * u;
            old[j][u] = (rr < t.m && c < t.n) ? t.C[(int64_t)rr * t.ldc + c] : 0.f;
          }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int rr = r0 + j * EPI_WARPS;
#pragma unroll
          for (int u = 0; u < TILE / 32; ++u) {
            const int c = lane + 32 * u;
            if (rr < t.m && c < t.n) {
              const float v = (sym && c > rr) ? ct[c * CT_LD + rr] : ct[rr * CT_LD + c];
              t.C[(int64_t)rr * t.ldc + c] = fmaf(t.beta, old[j][u], v);
            }
          }
        }
      }
    } else {
      for (int rr = warp; rr < t.m; rr += EPI_WARPS) {
        float* crow = t.C + (int64_t)rr * t.ldc;
        for (int c = lane; c < t.n; c += 32)
          // symmetric tile: only the lower half was computed to be used; mirror it
          crow[c] = (sym && c > rr) ? ct[c * CT_LD + rr] : ct[rr * CT_LD + c];
      }
    }
  }
  // the mirror of an updated tile (beta != 0) reads back what other warps have just written
  if (t.C2 && t.beta != 0.f) asm volatile("bar.sync 1, %0;" ::"n"(32 * EPI_WARPS) : "memory");
  if (t.C2) {
    for (int c = warp; c < t.n; c += EPI_WARPS) {
      float* orow = t.C2 + (int64_t)c * t.ldc2;
      for (int rr = lane; rr < t.m; rr += 32)
        orow[rr] = (t.beta != 0.f) ? t.C[(int64_t)rr * t.ldc + c] : ct[rr * CT_LD + c];
    }
  }
}

__global__ void __launch_bounds__(THREADS, 1) tile_task_tc_kernel(const sso_tile_task* __restrict__ tasks, int* status) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bars[2 * STAGES + 4];
  __shared__ uint32_t tmem_base_slot;
  const sso_tile_task t = tasks[blockIdx.x];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool ta = t.flags & 1u, tb = t.flags & 2u;
  const bool a_kc = !ta, b_kc = tb;
  const int nstages = ceil_div(t.k, KS);
  const int nchunks = ceil_div(nstages, FLUSH);

  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (STAGES + s); };
  auto accfull_bar = [&](int b) { return bar0 + 8u * (2 * STAGES + b); };
  auto accempty_bar = [&](int b) { return bar0 + 8u * (2 * STAGES + 2 + b); };
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), LOAD_WARPS);
      mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(accfull_bar(b), 1);
      mbar_init(accempty_bar(b), EPI_WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) tmem_alloc(smem_u32(&tmem_base_slot), TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;

  if (warp < EPI_WARPS) {
    // ------------------------------------------------------------------ accumulate + epilogue
    float* ct = reinterpret_cast<float*>(smem_raw + (smem0 - smem_u32(smem_raw)));
    accumulate_and_store(t, tmem_base, accfull_bar(0), accempty_bar(0), nchunks, status, ct, warp, lane);
  } else if (warp == MMA_WARP) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      const uint32_t idesc = instr_desc(2u, 0u);   // tf32, K-major
      bool ok = true;
      int s = 0;
      for (; s < nstages && ok; ++s) {
        const int slot = s % STAGES, c = s / FLUSH, b = c & 1;
        const bool first_of_chunk = (s % FLUSH) == 0;
        if (first_of_chunk && c >= 2) ok = mbar_wait(accempty_bar(b), ((c >> 1) - 1) & 1, status, 12);
        if (!ok) break;
        ok = mbar_wait(full_bar(slot), (s / STAGES) & 1, status, 11);
        if (!ok) break;
        tc_fence_after();
        const uint32_t sb = smem0 + slot * STAGE_BYTES;
        const uint32_t ah = sb, al = sb + OPB, bh = sb + 2 * OPB, bl = sb + 3 * OPB;
        const uint32_t d_tmem = tmem_base + (uint32_t)(b * TILE);
#pragma unroll
        for (int ks = 0; ks < KS / 8; ++ks) {
          // one k-slice = 8 tf32 = 32 bytes further along the 128-byte rows
          const uint64_t adh = smem_desc_sw128_kmajor(ah + ks * 32u), adl = smem_desc_sw128_kmajor(al + ks * 32u);
          const uint64_t bdh = smem_desc_sw128_kmajor(bh + ks * 32u), bdl = smem_desc_sw128_kmajor(bl + ks * 32u);
          umma<true>(d_tmem, adl, bdh, idesc, (first_of_chunk && ks == 0) ? 0u : 1u);
          umma<true>(d_tmem, adh, bdl, idesc, 1u);
          umma<true>(d_tmem, adh, bdh, idesc, 1u);
        }
        umma_commit(empty_bar(slot));
        if ((s % FLUSH) == FLUSH - 1 || s == nstages - 1) umma_commit(accfull_bar(b));
      }
      mmas_done<STAGES>(s, empty_bar, status, 18);
    }
  } else {
    // ------------------------------------------------------------------ load warps
    const int lt = tid - 32 * (MMA_WARP + 1);
    const int l8 = lt & 7, q = lt >> 3;               // k-contiguous mapping
    const int w = lt >> 5, kq = lt & 15, rc = (lt >> 4) & 1;   // mapping of the other kind
    const bool a_vec = ((reinterpret_cast<uintptr_t>(t.A) & 15) == 0) && (t.lda % 4 == 0);
    const bool b_vec = ((reinterpret_cast<uintptr_t>(t.B) & 15) == 0) && (t.ldb % 4 == 0);
    // Addresses that do not change from stage to stage are computed once.  Interior stages of
    // aligned operands then cost one 16-byte load per chunk; edges and unaligned operands take
    // the checked element loads.
    const OpLoad oa = make_op(t.A, t.lda, a_kc, t.m, lt, a_vec);
    const OpLoad ob = make_op(t.B, t.ldb, b_kc, t.n, lt, b_vec);
    auto load_op = [&](const OpLoad& o, const float* P, int ld, bool kc, int lim, bool vec, int s, float4 (&v)[4]) {
      const int k0 = s * KS;
      if (k0 + KS <= t.k && o.fast) {
        const float* base = o.p0 + (int64_t)s * o.step;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int64_t joff = kc ? j * o.ja : (j & 1) * o.ja + (j >> 1) * 8;
          v[j] = ((o.okmask >> j) & 1u) ? __ldg(reinterpret_cast<const float4*>(base + joff))
                                        : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (kc) {          // P[i*ld + k]
            const int i = q + 32 * j;
            v[j] = load4(P, ld, i, k0 + l8 * 4, i < lim, t.k, vec);
          } else {           // P[k*ld + index]
            const int k = k0 + (j & 1) * 16 + kq;
            v[j] = load4(P, ld, k, (4 * w + 2 * (j >> 1) + rc) * 4, k < t.k, lim, vec);
          }
        }
      }
    };
    auto store_op = [&](const OpLoad& o, bool kc, uint32_t base, const float4 (&v)[4]) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (kc) {
          split_store4(base + o.so0 + j * 4096u, v[j]);
        } else {
          const int k = (j & 1) * 16 + kq, r0 = (4 * w + 2 * (j >> 1) + rc) * 4;
          split_store1(base + sw_off(r0, k), v[j].x);
          split_store1(base + sw_off(r0 + 1, k), v[j].y);
          split_store1(base + sw_off(r0 + 2, k), v[j].z);
          split_store1(base + sw_off(r0 + 3, k), v[j].w);
        }
      }
    };
    auto load_stage = [&](int s, float4 (&va)[4], float4 (&vb)[4]) {
      load_op(oa, t.A, t.lda, a_kc, t.m, a_vec, s, va);
      load_op(ob, t.B, t.ldb, b_kc, t.n, b_vec, s, vb);
    };
    auto store_stage = [&](int s, const float4 (&va)[4], const float4 (&vb)[4]) -> bool {
      const int slot = s % STAGES;
      if (s >= STAGES && !mbar_wait(empty_bar(slot), ((s / STAGES) - 1) & 1, status, 14)) return false;
      const uint32_t sa = smem0 + slot * STAGE_BYTES;
      store_op(oa, a_kc, sa, va);
      store_op(ob, b_kc, sa + 2 * OPB, vb);
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(full_bar(slot));
      return true;
    };
    // the global loads of stage s+1 are in flight while stage s is split and stored
    float4 a0[4], b0[4], a1[4], b1[4];
    if (nstages > 0) load_stage(0, a0, b0);
    for (int s = 0; s < nstages; s += 2) {
      if (s + 1 < nstages) load_stage(s + 1, a1, b1);
      if (!store_stage(s, a0, b0) || s + 1 >= nstages) break;
      if (s + 2 < nstages) load_stage(s + 2, a0, b0);
      if (!store_stage(s + 1, a1, b1)) break;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------------------
// Fast variant for tasks whose operands are both contiguous along k (A not transposed, B
// transposed) with 16-byte aligned rows: the fp32 tiles travel global -> shared with cp.async
// into a ring of RAW_SLOTS raw stages, so several stages of loads are in flight without holding
// registers; the load warps then split each of their own chunks in place (hi overwrites the raw
// value, lo goes to a ring of LO_SLOTS stages) and hand the stage to the MMA warp.
// ------------------------------------------------------------------------------------------
constexpr uint32_t PART = 2 * OPB;                       // A and B of one stage, one flavour (raw/hi or lo)
constexpr uint32_t TS_COLS = 512;                        // two accumulators and the A operands of up to four stages
constexpr uint32_t KC_SMEM = 7 * PART;                   // RAW_SLOTS + LO_SLOTS = 7 in every variant

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}

template <int RAW_SLOTS, int LO_SLOTS, int PREFETCH>
__global__ void __launch_bounds__(THREADS, 1) tile_task_kc_kernel(const sso_tile_task* __restrict__ tasks, int* status) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bars[RAW_SLOTS + 2 * LO_SLOTS + 4];
  __shared__ uint32_t tmem_base_slot;
  const sso_tile_task t = tasks[blockIdx.x];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nstages = ceil_div(t.k, KS);
  const int nchunks = ceil_div(nstages, FLUSH);

  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t lo0 = smem0 + RAW_SLOTS * PART;
  const uint32_t bar0 = smem_u32(bars);
  auto rawfree_bar = [&](int s) { return bar0 + 8u * s; };
  auto full_bar = [&](int s) { return bar0 + 8u * (RAW_SLOTS + s); };
  auto lofree_bar = [&](int s) { return bar0 + 8u * (RAW_SLOTS + LO_SLOTS + s); };
  const uint32_t accfull0 = bar0 + 8u * (RAW_SLOTS + 2 * LO_SLOTS), accempty0 = accfull0 + 16u;
  if (tid == 0) {
    for (int s = 0; s < RAW_SLOTS; ++s) mbar_init(rawfree_bar(s), 1);
    for (int s = 0; s < LO_SLOTS; ++s) {
      mbar_init(full_bar(s), LOAD_WARPS);
      mbar_init(lofree_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(accfull0 + 8u * b, 1);
      mbar_init(accempty0 + 8u * b, EPI_WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) tmem_alloc(smem_u32(&tmem_base_slot), TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;

  if (warp < EPI_WARPS) {
    float* ct = reinterpret_cast<float*>(smem_raw + (smem0 - smem_u32(smem_raw)));
    accumulate_and_store(t, tmem_base, accfull0, accempty0, nchunks, status, ct, warp, lane);
  } else if (warp == MMA_WARP) {
    if (lane == 0) {
      const uint32_t idesc = instr_desc(2u, 0u);   // tf32, K-major
      bool ok = true;
      int s = 0;
      for (; s < nstages && ok; ++s) {
        const int rs = s % RAW_SLOTS, ls = s % LO_SLOTS, c = s / FLUSH, b = c & 1;
        const bool first_of_chunk = (s % FLUSH) == 0;
        if (first_of_chunk && c >= 2) ok = mbar_wait(accempty0 + 8u * b, ((c >> 1) - 1) & 1, status, 22);
        if (!ok) break;
        ok = mbar_wait(full_bar(ls), (s / LO_SLOTS) & 1, status, 21);
        if (!ok) break;
        tc_fence_after();
        const uint32_t ah = smem0 + rs * PART, bh = ah + OPB, al = lo0 + ls * PART, bl = al + OPB;
        const uint32_t d_tmem = tmem_base + (uint32_t)(b * TILE);
#pragma unroll
        for (int ks = 0; ks < KS / 8; ++ks) {
          const uint64_t adh = smem_desc_sw128_kmajor(ah + ks * 32u), adl = smem_desc_sw128_kmajor(al + ks * 32u);
          const uint64_t bdh = smem_desc_sw128_kmajor(bh + ks * 32u), bdl = smem_desc_sw128_kmajor(bl + ks * 32u);
          umma<true>(d_tmem, adl, bdh, idesc, (first_of_chunk && ks == 0) ? 0u : 1u);
          umma<true>(d_tmem, adh, bdl, idesc, 1u);
          umma<true>(d_tmem, adh, bdh, idesc, 1u);
        }
        umma_commit(rawfree_bar(rs));
        umma_commit(lofree_bar(ls));
        if ((s % FLUSH) == FLUSH - 1 || s == nstages - 1) umma_commit(accfull0 + 8u * b);
      }
      mmas_done<LO_SLOTS>(s, lofree_bar, status, 28);
    }
  } else {
    // ------------------------------------------------------------------ load + split warps
    const int lt = tid - 32 * (MMA_WARP + 1);
    const int q = lt >> 3, l8 = lt & 7;
    const uint32_t so0 = sw_off(q, l8 * 4);
    const float* pa = t.A + (int64_t)q * t.lda + l8 * 4;
    const float* pb = t.B + (int64_t)q * t.ldb + l8 * 4;
    const int64_t ja = (int64_t)32 * t.lda, jb = (int64_t)32 * t.ldb;
    uint32_t oka = 0u, okb = 0u;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (q + 32 * j < t.m) oka |= 1u << j;
      if (q + 32 * j < t.n) okb |= 1u << j;
    }
    bool ok = true;
    auto issue = [&](int s) {       // cp.async of this thread's 8 chunks of stage s (zero fill past the edges)
      const int rs = s % RAW_SLOTS;
      if (s >= RAW_SLOTS && !mbar_wait(rawfree_bar(rs), ((s / RAW_SLOTS) - 1) & 1, status, 24)) { ok = false; return; }
      const int kk = s * KS + l8 * 4;
      const uint32_t nb = (uint32_t)min(16, max(0, (t.k - kk) * 4));
      const uint32_t dst = smem0 + rs * PART + so0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        cp_async16(dst + j * 4096u, pa + j * ja + s * KS, ((oka >> j) & 1u) ? nb : 0u);
        cp_async16(dst + OPB + j * 4096u, pb + j * jb + s * KS, ((okb >> j) & 1u) ? nb : 0u);
      }
    };
    for (int s = 0; s < PREFETCH; ++s) {     // always PREFETCH groups, so that wait_group counts stages
      if (s < nstages) issue(s);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int s = 0; s < nstages && ok; ++s) {
      if (s + PREFETCH < nstages) issue(s + PREFETCH);
      asm volatile("cp.async.commit_group;" ::: "memory");
      if (!ok) break;
      asm volatile("cp.async.wait_group %0;" ::"n"(PREFETCH) : "memory");
      const int rs = s % RAW_SLOTS, ls = s % LO_SLOTS;
      if (s >= LO_SLOTS && !mbar_wait(lofree_bar(ls), ((s / LO_SLOTS) - 1) & 1, status, 25)) break;
      const uint32_t hi = smem0 + rs * PART + so0, lo = lo0 + ls * PART + so0;
      // all loads before the first store: one chunk at a time, each would wait for the one before
      float4 v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t off = (uint32_t)(j & 3) * 4096u + (uint32_t)(j >> 2) * OPB;
        asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v[j].x), "=f"(v[j].y), "=f"(v[j].z), "=f"(v[j].w) : "r"(hi + off));
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t off = (uint32_t)(j & 3) * 4096u + (uint32_t)(j >> 2) * OPB;
        // hi is rounded to nearest and written back in place.  Leaving the raw word as hi (the MMA
        // reads only its top 19 bits) saves this store and 10-15 % of the kernel, but a truncated hi
        // doubles |lo| and makes the dropped lo*lo term one-signed: on ill-conditioned factors the
        // preconditioned gradient then misses the 1e-4 bound (3.7e-4 measured against 2e-4).
        const uint32_t h0 = rna_tf32(v[j].x), h1 = rna_tf32(v[j].y), h2 = rna_tf32(v[j].z), h3 = rna_tf32(v[j].w);
        const uint32_t l0 = __float_as_uint(v[j].x - __uint_as_float(h0)), l1 = __float_as_uint(v[j].y - __uint_as_float(h1));
        const uint32_t l2 = __float_as_uint(v[j].z - __uint_as_float(h2)), l3 = __float_as_uint(v[j].w - __uint_as_float(h3));
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(hi + off), "r"(h0), "r"(h1), "r"(h2), "r"(h3) : "memory");
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(lo + off), "r"(l0), "r"(l1), "r"(l2), "r"(l3) : "memory");
      }
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(full_bar(ls));
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------------------
// TMA-fed variant of the k-contiguous kernel: the two operand boxes of a stage (128 rows x 32 k,
// fp32) are fetched by one thread with cp.async.bulk.tensor into the raw ring (tensor maps made
// on the host when the plan is built, two per task), so the loads no longer pass through the
// load/store units.  The load warps only split: A into tensor memory (hi and lo, a row per lane, which
// takes its part of the operand traffic off shared memory), B's hi in place and lo into a second ring.
// Bound: the feed of the operands for large tasks (4608 x 512 preconditioned in 152 us, 159 TFLOP/s), set-up, pipeline fill
// and store of a task (about 10 us) for small ones.  us, with A in shared memory and chunks split one by one / in
// shared memory / in tensor memory: that layer 175 / 161 / 152, ResNet-50's preconditioning 1122 / 1037 / 1005.
// ------------------------------------------------------------------------------------------
struct alignas(128) TaskMaps {
  unsigned char a[128];
  unsigned char b[128];
};

template <int RAW_SLOTS, int LO_SLOTS, int PREFETCH>
__global__ void __launch_bounds__(THREADS, 1) tile_task_tma_kernel(const sso_tile_task* tasks,      // written by the launches before: no non-coherent loads
                                                                    const TaskMaps* __restrict__ maps, int* status) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bars[2 * RAW_SLOTS + 2 * LO_SLOTS + 4];
  __shared__ uint32_t tmem_base_slot;
  // the descriptors of this task's two operands: fetched while barriers and TMEM are set up
  if (threadIdx.x == 32 * (MMA_WARP + 1)) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(maps[blockIdx.x].a)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(maps[blockIdx.x].b)) : "memory");
  }
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");      // launched beside the phase before: its results, and a scale in the tasks, are there
  const sso_tile_task t = tasks[blockIdx.x];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nstages = ceil_div(t.k, KS);
  const int nchunks = ceil_div(nstages, FLUSH);

  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t lo0 = smem0 + RAW_SLOTS * PART;
  const uint32_t bar0 = smem_u32(bars);
  auto rawfree_bar = [&](int s) { return bar0 + 8u * s; };
  auto rawfull_bar = [&](int s) { return bar0 + 8u * (RAW_SLOTS + s); };
  auto full_bar = [&](int s) { return bar0 + 8u * (2 * RAW_SLOTS + s); };
  auto lofree_bar = [&](int s) { return bar0 + 8u * (2 * RAW_SLOTS + LO_SLOTS + s); };
  const uint32_t accfull0 = bar0 + 8u * (2 * RAW_SLOTS + 2 * LO_SLOTS), accempty0 = accfull0 + 16u;
  if (tid == 0) {
    for (int s = 0; s < RAW_SLOTS; ++s) {
      mbar_init(rawfree_bar(s), 1);
      mbar_init(rawfull_bar(s), 1);
    }
    for (int s = 0; s < LO_SLOTS; ++s) {
      mbar_init(full_bar(s), LOAD_WARPS);
      mbar_init(lofree_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(accfull0 + 8u * b, 1);
      mbar_init(accempty0 + 8u * b, EPI_WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) tmem_alloc(smem_u32(&tmem_base_slot), TS_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;

  if (warp < EPI_WARPS) {
    float* ct = reinterpret_cast<float*>(smem_raw + (smem0 - smem_u32(smem_raw)));
    accumulate_and_store(t, tmem_base, accfull0, accempty0, nchunks, status, ct, warp, lane);
  } else if (warp == MMA_WARP) {
    if (lane == 0) {
      const uint32_t idesc = instr_desc(2u, 0u);   // tf32, K-major
      bool ok = true;
      int s = 0;
      for (; s < nstages && ok; ++s) {
        const int rs = s % RAW_SLOTS, ls = s % LO_SLOTS, c = s / FLUSH, b = c & 1;
        const bool first_of_chunk = (s % FLUSH) == 0;
        if (first_of_chunk && c >= 2) ok = mbar_wait(accempty0 + 8u * b, ((c >> 1) - 1) & 1, status, 42);
        if (!ok) break;
        ok = mbar_wait(full_bar(ls), (s / LO_SLOTS) & 1, status, 41);
        if (!ok) break;
        tc_fence_after();
        const uint32_t bh = smem0 + rs * PART + OPB, bl = lo0 + ls * OPB;
        const uint32_t ah = tmem_base + TMEM_COLS + ls * 2 * KS, al = ah + KS;
        const uint32_t d_tmem = tmem_base + (uint32_t)(b * TILE);
#pragma unroll
        for (int ks = 0; ks < KS / 8; ++ks) {
          const uint64_t bdh = smem_desc_sw128_kmajor(bh + ks * 32u), bdl = smem_desc_sw128_kmajor(bl + ks * 32u);
          umma_tf32_ts(d_tmem, al + ks * 8, bdh, idesc, (first_of_chunk && ks == 0) ? 0u : 1u);
          umma_tf32_ts(d_tmem, ah + ks * 8, bdl, idesc, 1u);
          umma_tf32_ts(d_tmem, ah + ks * 8, bdh, idesc, 1u);
        }
        umma_commit(rawfree_bar(rs));
        umma_commit(lofree_bar(ls));
        if ((s % FLUSH) == FLUSH - 1 || s == nstages - 1) umma_commit(accfull0 + 8u * b);
      }
      mmas_done<LO_SLOTS>(s, lofree_bar, status, 48);
    }
  } else {
    // ------------------------------------------------------------------ producer thread + split warps
    const int lt = tid - 32 * (MMA_WARP + 1);
    const int q = lt >> 3, l8 = lt & 7;
    const uint32_t so0 = sw_off(q, l8 * 4);
    const int a_row = 32 * (warp & 3) + lane, a_col = ((lt >> 5) >> 2) * (KS / 2);      // a warp reaches the lanes of its quarter
    const uint64_t map_a = reinterpret_cast<uint64_t>(maps[blockIdx.x].a), map_b = reinterpret_cast<uint64_t>(maps[blockIdx.x].b);
    bool ok = true;
    int issued = 0;
    auto issue = [&](int s) {       // one thread: both boxes of stage s
      const int rs = s % RAW_SLOTS;
      ok = ok && (s < RAW_SLOTS || mbar_wait(rawfree_bar(rs), ((s / RAW_SLOTS) - 1) & 1, status, 44));
      if (!ok) return;
      issued = s + 1;
      const uint32_t fb = rawfull_bar(rs), dst = smem0 + rs * PART;
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fb), "r"(PART) : "memory");
      asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                   ::"r"(dst), "l"(map_a), "r"(s * KS), "r"(0), "r"(fb) : "memory");
      asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                   ::"r"(dst + OPB), "l"(map_b), "r"(s * KS), "r"(0), "r"(fb) : "memory");
    };
    const bool producer = (lt == 0) && !g_inject_stall;     // stalled: nothing is ever loaded
    if (producer)
      for (int s = 0; s < PREFETCH && s < nstages; ++s) issue(s);
    for (int s = 0; s < nstages; ++s) {
      if (producer && s + PREFETCH < nstages) issue(s + PREFETCH);
      const int rs = s % RAW_SLOTS, ls = s % LO_SLOTS;
      if (!mbar_wait(rawfull_bar(rs), (s / RAW_SLOTS) & 1, status, 46)) break;
      if (s >= LO_SLOTS && !mbar_wait(lofree_bar(ls), ((s / LO_SLOTS) - 1) & 1, status, 45)) break;
      tc_fence_after();                          // the MMAs that read this slot of tensor memory are done
      // A: a row per lane, half of the stage's columns per warp, into tensor memory; B: hi in place, lo into its ring.
      // hi is rounded to nearest.  Leaving the raw word as hi (the MMA reads only its top 19 bits) was faster, but a
      // truncated hi doubles |lo| and makes the dropped lo*lo term one-signed: on ill-conditioned factors the
      // preconditioned gradient then misses the 1e-4 bound (3.7e-4 measured against 2e-4).
      // All loads before the first store: one chunk at a time, each would wait for the one before.
      const uint32_t ra = smem0 + rs * PART, hi = ra + OPB + so0, lo = lo0 + ls * OPB + so0;
      float4 v[4], u[4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v[j].x), "=f"(v[j].y), "=f"(v[j].z), "=f"(v[j].w) : "r"(ra + sw_off(a_row, a_col + 4 * j)));
#pragma unroll
      for (int j = 0; j < 4; ++j)
        asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(u[j].x), "=f"(u[j].y), "=f"(u[j].z), "=f"(u[j].w) : "r"(hi + j * 4096u));
      {
        uint32_t h[16], l[16];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float x[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            h[4 * j + i] = rna_tf32(x[i]);
            l[4 * j + i] = __float_as_uint(x[i] - __uint_as_float(h[4 * j + i]));
          }
        }
        const uint32_t ta = tmem_base + ((uint32_t)(a_row & ~31) << 16) + TMEM_COLS + ls * 2 * KS + a_col;
        tmem_st16(ta, h);
        tmem_st16(ta + KS, l);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t h0 = rna_tf32(u[j].x), h1 = rna_tf32(u[j].y), h2 = rna_tf32(u[j].z), h3 = rna_tf32(u[j].w);
        const uint32_t l0 = __float_as_uint(u[j].x - __uint_as_float(h0)), l1 = __float_as_uint(u[j].y - __uint_as_float(h1));
        const uint32_t l2 = __float_as_uint(u[j].z - __uint_as_float(h2)), l3 = __float_as_uint(u[j].w - __uint_as_float(h3));
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(hi + j * 4096u), "r"(h0), "r"(h1), "r"(h2), "r"(h3) : "memory");
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(lo + j * 4096u), "r"(l0), "r"(l1), "r"(l2), "r"(l3) : "memory");
      }
      tmem_st_wait();
      tc_fence_before();
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(full_bar(ls));
    }
    if (producer) ring_landed<RAW_SLOTS>(issued, rawfull_bar, status, 47);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, TS_COLS);
  }
}

// ------------------------------------------------------------------------------------------
// Blocks of 256x256: a cluster of two CTAs computes one with tcgen05.mma.cta_group::2.  A CTA fetches and splits 128 rows of
// either operand and its tensor core reads them for 256 columns, so that a stage brings in half the bytes per
// multiplication of the 128x128 tasks, which are bound by that (32 KB per SM and 0.91 us, 5.2 TB/s over the chip).  Eight
// accumulate warps (128 sums per thread), one that issues the MMAs (the leader's), one that issues the boxes, eight that
// split in two groups of every other stage.  Bound: the MMAs.  A stage of a long block takes 1.16 us, its twelve MMAs 1.13 at half
// the measured bf16 rate (of the SMs that have a block the tensor pipe is busy 79 % of the time, the shared-memory pipe 58 %); then
// the last round of blocks, of which 74 run at a time (108 blocks of 4608 x 512: 0.73 of the chip).  us, tiles of 128 / blocks of 256 and what tiles are left: preconditioning of ResNet-50's layers 1010 / 750, of VGG-16's 882 / 673, a
// posterior draw of VGG-16's 555 / 482.
// ------------------------------------------------------------------------------------------
namespace pair {
constexpr int RAW = 4, LO = 3, BLOCK = 256;
// five warpgroups: 0-1 accumulate, 2 issues, 3-4 split; they share the block's 640 x 96 registers as 168 + 168 + 32 + 56 + 56
constexpr int THREADS = 640, PROD_WARP = 9, SPLIT_WARP0 = 12, SPLIT_WARPS = 8;
constexpr size_t SMEM = (RAW + LO) * PART + 1024;

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
tile_pair_kernel(const sso_tile_task* tasks, const TaskMaps* __restrict__ maps, int* status) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bars[2 * RAW + 2 * LO + 4];
  __shared__ uint32_t tmem_base_slot;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;      // uniform, for setmaxnreg
  const uint32_t rank = cluster_ctarank();
  const int task = blockIdx.x >> 1;
  if (tid == 32 * PROD_WARP) {      // fetched while barriers and TMEM are set up
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(maps[task].a)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(maps[task].b)) : "memory");
  }
  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t lo0 = smem0 + RAW * PART;
  const uint32_t bar0 = smem_u32(bars);
  auto rawfull = [&](int s) { return bar0 + 8u * s; };
  auto rawfree = [&](int s) { return bar0 + 8u * (RAW + s); };
  auto full = [&](int s) { return bar0 + 8u * (2 * RAW + s); };
  auto lofree = [&](int s) { return bar0 + 8u * (2 * RAW + LO + s); };
  const uint32_t accfull0 = bar0 + 8u * (2 * RAW + 2 * LO), accempty0 = accfull0 + 16u;
  if (tid == 0) {
    for (int s = 0; s < RAW; ++s) { mbar_init(rawfull(s), 1); mbar_init(rawfree(s), 1); }
    for (int s = 0; s < LO; ++s) { mbar_init(full(s), SPLIT_WARPS); mbar_init(lofree(s), 1); }      // four warps of either CTA
    for (int b = 0; b < 2; ++b) { mbar_init(accfull0 + 8u * b, 1); mbar_init(accempty0 + 8u * b, 2 * EPI_WARPS); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) tmem_alloc2(smem_u32(&tmem_base_slot), TMEM_COLS2);
  tc_fence_before();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");      // as in tile_task_tma_kernel
  const sso_tile_task t = tasks[task];
  const int nstages = ceil_div(t.k, KS), nchunks = ceil_div(nstages, FLUSH);

  if (warp < EPI_WARPS) {
    // ------------------------------------------------------------------ accumulate and store
    asm volatile("setmaxnreg.inc.sync.aligned.u32 168;");
    const int q = warp & 3, half = warp >> 2;
    const uint32_t leader_accempty0 = map_to_cta(accempty0, 0u);
    float acc[128];
#pragma unroll
    for (int i = 0; i < 128; ++i) acc[i] = 0.f;
    bool ok = true;
    for (int c = 0; c < nchunks; ++c) {
      const int b = c & 1;
      if (!mbar_wait(accfull0 + 8u * b, (c >> 1) & 1, status, 53)) { ok = false; break; }
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * BLOCK + half * 128);
#pragma unroll
      for (int part = 0; part < 8; ++part) {
        uint32_t v[16];
        tmem_ld16(taddr + part * 16, v);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[part * 16 + i] += __uint_as_float(v[i]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(leader_accempty0 + 8u * b);
    }
    // A wait that gave up leaves the sums incomplete: the block is written all the same, as NaN.  The ring is free: every
    // MMA has read its operands before the last accumulator was published.
    const float nan = __int_as_float(0x7fc00000);
    float* stg = reinterpret_cast<float*>(smem_raw + (smem0 - smem_u32(smem_raw))) + warp * 1024;
    const int row0 = (int)rank * TILE + q * 32, rows = min(32, t.m - row0);
#pragma unroll
    for (int part = 0; part < 4; ++part) {
      const int col0 = half * 128 + part * 32;
      if (col0 >= t.n || !ok) break;
#pragma unroll
      for (int i = 0; i < 32; ++i) stg[lane * 32 + (i ^ lane)] = t.alpha * acc[part * 32 + i];
      __syncwarp();
      const int c = col0 + lane;
      float* o = t.C + (int64_t)row0 * t.ldc + c;
      if (c < t.n) {
        for (int r0 = 0; r0 < rows; r0 += 8) {
          float old[8];
          if (t.beta != 0.f) {        // eight rows in flight before the first store
#pragma unroll
            for (int j = 0; j < 8; ++j) old[j] = r0 + j < rows ? o[(int64_t)(r0 + j) * t.ldc] : 0.f;
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int r = r0 + j;
            if (r >= rows) break;
            const float v = stg[r * 32 + (lane ^ r)];
            o[(int64_t)r * t.ldc] = t.beta != 0.f ? fmaf(t.beta, old[j], v) : v;
          }
        }
      }
      __syncwarp();
    }
    if (!ok)
      for (int r = 0; r < rows; ++r)
        for (int c = half * 128 + lane; c < min(half * 128 + 128, t.n); c += 32) t.C[(int64_t)(row0 + r) * t.ldc + c] = nan;
  } else if (warp < SPLIT_WARP0) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");      // one instruction for the whole warpgroup
    if (warp == MMA_WARP && lane == 0 && rank == 0) {
      const uint32_t idesc = instr_desc_pair(2u, 0u);   // tf32, K-major
      bool ok = true;
      int s = 0;
      for (; s < nstages; ++s) {
        const int rs = s % RAW, ls = s % LO, c = s / FLUSH, b = c & 1;
        const bool first_of_chunk = (s % FLUSH) == 0;
        if (first_of_chunk && c >= 2) ok = mbar_wait(accempty0 + 8u * b, ((c >> 1) - 1) & 1, status, 52);
        if (ok) ok = mbar_wait(full(ls), (s / LO) & 1, status, 51);
        if (!ok) break;
        tc_fence_after();
        const uint32_t ah = smem0 + rs * PART, bh = ah + OPB, al = lo0 + ls * PART, bl = al + OPB;
        const uint32_t d_tmem = tmem_base + (uint32_t)(b * BLOCK);
#pragma unroll
        for (int ks = 0; ks < KS / 8; ++ks) {
          const uint64_t adh = smem_desc_sw128_kmajor(ah + ks * 32u), adl = smem_desc_sw128_kmajor(al + ks * 32u);
          const uint64_t bdh = smem_desc_sw128_kmajor(bh + ks * 32u), bdl = smem_desc_sw128_kmajor(bl + ks * 32u);
          umma2<true>(d_tmem, adl, bdh, idesc, (first_of_chunk && ks == 0) ? 0u : 1u);
          umma2<true>(d_tmem, adh, bdl, idesc, 1u);
          umma2<true>(d_tmem, adh, bdh, idesc, 1u);
        }
        umma2_commit_both(rawfree(rs));
        umma2_commit_both(lofree(ls));
        if ((s % FLUSH) == FLUSH - 1 || s == nstages - 1) umma2_commit_both(accfull0 + 8u * b);
      }
      mmas_done<LO>(s, lofree, status, 58);
    } else if (warp == PROD_WARP && lane == 0 && !g_inject_stall) {      // stalled: nothing is ever loaded
      const uint64_t map_a = reinterpret_cast<uint64_t>(maps[task].a), map_b = reinterpret_cast<uint64_t>(maps[task].b);
      const int row = (int)rank * TILE;
      int s = 0;
      for (; s < nstages; ++s) {
        const int rs = s % RAW;
        if (s >= RAW && !mbar_wait(rawfree(rs), ((s / RAW) - 1) & 1, status, 54)) break;
        const uint32_t fb = rawfull(rs), dst = smem0 + rs * PART;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fb), "r"(PART) : "memory");
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                     ::"r"(dst), "l"(map_a), "r"(s * KS), "r"(row), "r"(fb) : "memory");
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                     ::"r"(dst + OPB), "l"(map_b), "r"(s * KS), "r"(row), "r"(fb) : "memory");
      }
      ring_landed<RAW>(s, rawfull, status, 57);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ split warps
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    const int group = (warp - SPLIT_WARP0) >> 2;
    const uint32_t at0 = sw_off(32 * (warp & 3) + lane, 0);      // a thread has this row of both operands; chunk j: bits 4 to 6 xor j
    const uint32_t leader_full0 = map_to_cta(full(0), 0u);
    for (int s = group; s < nstages; s += 2) {
      const int rs = s % RAW, ls = s % LO;
      if (!mbar_wait(rawfull(rs), (s / RAW) & 1, status, 56)) break;
      if (s >= LO && !mbar_wait(lofree(ls), ((s / LO) - 1) & 1, status, 55)) break;
#pragma unroll 1
      for (int side = 0; side < 2; ++side) {
        const uint32_t hi = smem0 + rs * PART + side * OPB + at0, lo = lo0 + ls * PART + side * OPB + at0;
        // all loads before the first store: one chunk at a time, each would wait for the one before.  hi is rounded to
        // nearest (see tile_task_tma_kernel)
        float4 v[KS / 4];
#pragma unroll
        for (int j = 0; j < KS / 4; ++j)
          asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v[j].x), "=f"(v[j].y), "=f"(v[j].z), "=f"(v[j].w) : "r"(hi ^ (j << 4)));
#pragma unroll
        for (int j = 0; j < KS / 4; ++j) {
          const uint32_t h0 = rna_tf32(v[j].x), h1 = rna_tf32(v[j].y), h2 = rna_tf32(v[j].z), h3 = rna_tf32(v[j].w);
          const uint32_t l0 = __float_as_uint(v[j].x - __uint_as_float(h0)), l1 = __float_as_uint(v[j].y - __uint_as_float(h1));
          const uint32_t l2 = __float_as_uint(v[j].z - __uint_as_float(h2)), l3 = __float_as_uint(v[j].w - __uint_as_float(h3));
          asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(hi ^ (j << 4)), "r"(h0), "r"(h1), "r"(h2), "r"(h3) : "memory");
          asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(lo ^ (j << 4)), "r"(l0), "r"(l1), "r"(l2), "r"(l3) : "memory");
        }
      }
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(leader_full0 + 8u * ls);
    }
  }
  tc_fence_before();
  cluster_sync_all();          // neither CTA leaves while its peer's MMAs may still read its shared memory
  if (warp == MMA_WARP) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc2(tmem_base, TMEM_COLS2);
  }
}
}  // namespace pair

}  // namespace etc

int launch_tile_pairs(const sso_tile_task* tasks_dev, const void* maps_dev, int count, int* status_dev, cudaStream_t st) {
  SSO_ENSURE_SMEM(etc::pair::tile_pair_kernel, etc::pair::SMEM);
  launch_early(etc::pair::tile_pair_kernel, dim3(2 * count), etc::pair::THREADS, etc::pair::SMEM, st, tasks_dev, reinterpret_cast<const etc::TaskMaps*>(maps_dev), status_dev);
  SSO_LAUNCH_OK("tile_pair_kernel");
  return 0;
}

int engine_tc_set_wait_controls(long long cycles, int stall) { return tc::set_wait_controls(cycles, stall); }

int launch_tile_tasks_tma(const sso_tile_task* tasks_dev, const void* maps_dev, int count, int* status_dev, cudaStream_t st) {
  constexpr int RAW = 5, LO = 3;
  const size_t smem = (size_t)RAW * etc::PART + (size_t)LO * etc::OPB + 1024;
  SSO_ENSURE_SMEM((etc::tile_task_tma_kernel<RAW, LO, 3>), smem);
  launch_early(etc::tile_task_tma_kernel<RAW, LO, 3>, dim3(count), etc::THREADS, smem, st, tasks_dev, reinterpret_cast<const etc::TaskMaps*>(maps_dev), status_dev);
  SSO_LAUNCH_OK("tile_task_tma_kernel");
  return 0;
}

int launch_tile_tasks_kc(const sso_tile_task* tasks_dev, int count, int* status_dev, cudaStream_t st) {
  const size_t smem = (size_t)etc::KC_SMEM + 1024;
  SSO_ENSURE_SMEM((etc::tile_task_kc_kernel<5, 2, 3>), smem);
  etc::tile_task_kc_kernel<5, 2, 3><<<count, etc::THREADS, smem, st>>>(tasks_dev, status_dev);
  SSO_LAUNCH_OK("tile_task_kc_kernel");
  return 0;
}

int launch_tile_tasks_tc(const sso_tile_task* tasks_dev, int count, int* status_dev, cudaStream_t st) {
  const size_t smem = (size_t)etc::STAGES * etc::STAGE_BYTES + 1024;
  SSO_ENSURE_SMEM(etc::tile_task_tc_kernel, (int)smem);
  etc::tile_task_tc_kernel<<<count, etc::THREADS, smem, st>>>(tasks_dev, status_dev);
  SSO_LAUNCH_OK("tile_task_tc_kernel");
  return 0;
}

}  // namespace sso
