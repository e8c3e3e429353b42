// Blocked Cholesky factorisation and SPD inverse of many matrices as ONE persistent kernel.
//
// The work is tile tasks (128x128, flow.cuh) in one list that is topologically sorted and ordered by when a task can
// start (engine.cu simulates the schedule); one CTA per SM takes the next task from a counter, so a task only ever
// waits for tasks that running CTAs have taken before it.  A tile is announced by a flag in global memory, and a task
// waits for its operands block by block along K: all but the last 128 columns of a panel update run before the
// previous panel is done.  The chain from one panel to the next is then one diagonal block (its inverse is announced
// before its other results are written), one multiplication by that inverse and the last 128 columns of one update,
// without a kernel boundary in it; as phases of launches every one of these was a kernel of at least 11 us (4608: 36
// panels of three launches, 20 more for the inverse).
//
// Inside a CTA (16 warps): 0-7 accumulate, store and factor diagonal blocks; 8 issues MMAs; 9 takes tasks, waits for flags
// and issues TMA loads; 12-15 split the landed fp32 stages into tf32 hi (in place) and lo.  Products are 3xTF32
// with both operands along k (every matrix is kept in the orientation in which it is read), drained into fp32 registers
// every two stages.  The pipeline runs on across tasks: loads of the next task start while this one is stored.
// The multiplication by Linv^T that ends a PANEL or INVT task takes its A operand from the accumulator: the accumulate
// warps write it into the raw slots of four more stages.
//
// Bound: for one large matrix the chain of diagonal blocks, for many the shared-memory traffic of the 3xTF32 stages
// (as tile_task_tma_kernel).  Against one launch per phase (us): 577+64 508 -> 180, 1000 637 -> 265, six factors of a
// 784-1000-1000-10 network 1196 -> 296, 4608+512 3363 -> 1424, the 106 factors of ResNet-50 8970 -> 3600, those of VGG-16
// with sampling factors 19416 -> 6440, and 4290 with these out of the same factorisation.
// Sampling factors: with J the reversal of rows and columns and J M J = L L^T, the lower Cholesky factor of M^-1 is J L^-T J.  A
// matrix whose factor is wanted is therefore read, and its results are written, in reverse; in between nothing differs.
// Every wait is bounded; a CTA whose wait gives up sets the status word and writes NaN for this and all further tasks.
#include "common.cuh"
#include "diag_panel.cuh"
#include "flow.cuh"
#include "tc_common.cuh"

namespace sso {
namespace flow {

using namespace tc;

constexpr int TILE = 128, KS = 32, RAW = 4, LO = 2, FLUSH = 2, QUEUE = 4;
constexpr int ACC_WARPS = 8, MMA_WARP = 8, PROD_WARP = 9, SPLIT_WARP0 = 12, SPLIT_WARPS = 4;
constexpr int THREADS = 512;
constexpr uint32_t OPB = TILE * 128;           // one operand of one stage: 128 rows of 32 fp32
constexpr uint32_t PART = 2 * OPB;             // A and B
constexpr uint32_t STAGING = 32 * 128;         // a warp's 32x32 staging tile
constexpr uint32_t RING_BYTES = (RAW + LO) * PART;
constexpr size_t SMEM = RING_BYTES + ACC_WARPS * STAGING + 1024;
static_assert(dpanel::SMEM_BYTES <= RING_BYTES, "a diagonal block is factored in the operand ring");

__device__ __forceinline__ uint64_t desc_k(uint32_t saddr) {      // K-major SWIZZLE_128B
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(1024u >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ uint32_t sw_off(int r, int chunk) {    // 16-byte chunk of row r
  return (uint32_t)(r >> 3) * 1024u + (uint32_t)(r & 7) * 128u + (uint32_t)((chunk ^ (r & 7)) << 4);
}
__device__ __forceinline__ int load_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void store_release(int* p, int v) { asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
__device__ __forceinline__ bool flag_wait(const int* f, int epoch, int* status, int code) {
  if (load_acquire(f) == epoch) return true;
  const long long t0 = clock64(), limit = g_wait_cycles;
  while (load_acquire(f) != epoch)
    if (clock64() - t0 > limit) {
      atomicCAS(status, 0, code);
      return false;
    }
  return true;
}

// What a task multiplies: K blocks [kb0, kb1), the rows of its two operands, whether a multiplication by Linv follows.
struct Shape {
  int kb0, kb1, n1, n2;          // stages of the sum, of the multiplication
  int row_a, row_b;              // block rows of the operands
  bool share;                    // both operands are the same tile
};
__device__ __forceinline__ Shape shape_of(const Task& t, int d) {
  Shape s;
  s.n2 = 0; s.share = false;
  switch (t.kind) {
    case DIAG: s.kb0 = 0; s.kb1 = t.a; s.row_a = s.row_b = t.a; s.share = true; break;
    case PANEL: s.kb0 = 0; s.kb1 = t.b; s.row_a = t.a; s.row_b = t.b; s.n2 = TILE / KS; break;
    case INVT: s.kb0 = t.a; s.kb1 = t.b; s.row_a = t.a; s.row_b = t.b; s.n2 = TILE / KS; break;
    default: s.kb0 = t.a; s.kb1 = (d + TILE - 1) / TILE; s.row_a = t.a; s.row_b = t.b; s.share = t.a == t.b; break;
  }
  s.n1 = s.kb1 > s.kb0 ? (min(s.kb1 * TILE, d) - s.kb0 * TILE + KS - 1) / KS : 0;
  return s;
}

// Before a run: next epoch, traces of the matrices, info cleared.
__global__ void __launch_bounds__(256) begin_kernel(const Mat* __restrict__ mats, int n_mats, int* sync, float* __restrict__ traces, int* info,
                                                    int clear_info, int with_traces, const float* src, int ld_src) {
  __shared__ float red[256];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");      // the next kernel sets itself up meanwhile
  const int tid = threadIdx.x;
  if (blockIdx.x == 0 && tid == 0) { sync[1] += 1; sync[2] = sync[0]; }
  if (info && clear_info && tid < 2) info[2 * mats[blockIdx.x].mat + tid] = 0;
  if (!with_traces) return;
  const Mat& m = mats[blockIdx.x];
  if (!src) { src = m.src; ld_src = m.ld_src; }
  float s = 0.f;
  for (int i = tid; i < m.pub; i += 256) s += src[(int64_t)i * ld_src + i];
  red[tid] = s;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (tid < o) red[tid] += red[tid + o];
    __syncthreads();
  }
  if (tid == 0) traces[m.mat] = red[0];
}

// v of M + v I: r*pi for the first of a pair, r/pi for the second, pi = sqrt(mean diagonal of one / of the other)
__device__ __forceinline__ float shift_of(const Mat& m, const float* traces, const float* damp_r) {
  if (!m.shifted) return 0.f;
  const float r = damp_r[m.mat];
  if (m.partner < 0) return r;
  const float mine = traces[m.mat] / (float)m.pub, other = traces[m.partner] / (float)m.d_partner;
  const float pi = m.role == 0 ? sqrtf(mine / other) : sqrtf(other / mine);
  return m.role == 0 ? r * pi : r / pi;
}

// REV: every matrix of the run is taken in reverse (a variant of its own: the addresses of the results cost 2 % of a run otherwise)
template <bool REV>
__global__ void __launch_bounds__(THREADS, 1) flow_kernel(const Args g) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bars[2 * RAW + 2 * LO + 4 + 2 + 2 * QUEUE];
  __shared__ uint32_t tmem_base_slot;
  __shared__ Task queue[QUEUE];
  __shared__ volatile int dead;          // a wait of this CTA gave up
  // for that case: queue entries pushed, the first one not finished, stages loaded; the task that the accumulate warps
  // left (they release its entry when they take it, so that another may lie there by now), one taken but not pushed
  __shared__ volatile uint32_t pushed, acc_at, issued;
  __shared__ volatile uint32_t gave_up;  // first queue entry at which one of the accumulate warps gave up
  __shared__ Task left, lost;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t lo0 = smem0 + RAW * PART;
  const uint32_t bar0 = smem_u32(bars);
  auto rawfull = [&](uint32_t s) { return bar0 + 8u * s; };
  auto rawfree = [&](uint32_t s) { return bar0 + 8u * (RAW + s); };
  auto full = [&](uint32_t s) { return bar0 + 8u * (2 * RAW + s); };
  auto lofree = [&](uint32_t s) { return bar0 + 8u * (2 * RAW + LO + s); };
  const uint32_t accfull0 = bar0 + 8u * (2 * RAW + 2 * LO), accempty0 = accfull0 + 16u;
  const uint32_t afull = accempty0 + 16u, ddone = afull + 8u, qfull0 = ddone + 8u, qempty0 = qfull0 + 8u * QUEUE;
  if (tid == 0) {
    for (int s = 0; s < RAW; ++s) { mbar_init(rawfull(s), 1); mbar_init(rawfree(s), 1); }
    for (int s = 0; s < LO; ++s) { mbar_init(full(s), SPLIT_WARPS); mbar_init(lofree(s), 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(accfull0 + 8u * b, 1); mbar_init(accempty0 + 8u * b, ACC_WARPS); }
    mbar_init(afull, ACC_WARPS);
    mbar_init(ddone, ACC_WARPS);
    for (int s = 0; s < QUEUE; ++s) { mbar_init(qfull0 + 8u * s, 1); mbar_init(qempty0 + 8u * s, ACC_WARPS + 1 + SPLIT_WARPS); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    dead = 0;
    pushed = acc_at = issued = 0;
    gave_up = 0xffffffffu;
    left.kind = lost.kind = -1;
  }
  if (warp == MMA_WARP) tmem_alloc(smem_u32(&tmem_base_slot), 256);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  int* status = g.status;
  asm volatile("griddepcontrol.wait;" ::: "memory");      // begin_kernel, and all before it, are done
  const int epoch = g.sync[1];
  // next entry of the task queue; every consumer warp reads it and arrives on its "empty" barrier
  auto take = [&](uint32_t n, Task& t) -> bool {
    const uint32_t s = n % QUEUE;
    if (!mbar_wait(qfull0 + 8u * s, (n / QUEUE) & 1, status, 81)) return false;
    t = queue[s];
    __syncwarp();
    if (lane == 0) mbar_arrive(qempty0 + 8u * s);
    return true;
  };

  if (warp >= ACC_WARPS && warp < SPLIT_WARP0) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");      // one instruction for the whole warpgroup
    if (warp == PROD_WARP && lane == 0) {
      // ---------------------------------------------------------------- task queue, flags, TMA loads (one thread)
      uint32_t stage = 0, n = 0, n_diag = 0;
      const unsigned base = (unsigned)g.sync[2];
      bool ok = true;
      for (; ok; ++n) {
        const unsigned idx = (unsigned)atomicAdd(&g.sync[0], 1) - base;
        Task t;
        t.kind = -1; t.mat = 0; t.a = 0; t.b = 0;
        if (idx < (unsigned)g.n_tasks) t = g.tasks[idx];
        const uint32_t qs = n % QUEUE;
        if (n >= QUEUE && !mbar_wait(qempty0 + 8u * qs, ((n / QUEUE) - 1) & 1, status, 82)) { lost = t; ok = false; break; }
        queue[qs] = t;
        mbar_arrive(qfull0 + 8u * qs);
        pushed = n + 1;
        if (t.kind < 0) break;
        const Mat& m = g.mats[t.mat];
        const Shape sh = shape_of(t, m.d);
        const bool over_x = t.kind == INVT || t.kind == PROD;      // A operand of the sum: X (else L); B: L, X for PROD
        const uint64_t map_w = reinterpret_cast<uint64_t>(m.map_w);
        auto x_flag = [&](int j, int k) { return g.flags + m.flag_x + j * m.np + k; };
        auto w_flag = [&](int i, int k) { return g.flags + m.flag_w + i * m.np + k; };
        auto issue = [&](uint64_t ma, int row_a, int ka, uint64_t mb, int row_b, int kb, bool a_on, bool b_on) {
          const uint32_t s = stage % RAW;
          if (stage >= RAW && !mbar_wait(rawfree(s), ((stage / RAW) - 1) & 1, status, 84)) return false;
          const uint32_t dst = smem0 + s * PART, fb = rawfull(s);
          if (g_inject_stall) { ++stage; return true; }      // stalled: nothing is ever loaded
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(fb), "r"((a_on ? OPB : 0u) + (b_on ? OPB : 0u)) : "memory");
          if (a_on)
            asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                         ::"r"(dst), "l"(ma), "r"(ka), "r"(row_a), "r"(fb) : "memory");
          if (b_on)
            asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                         ::"r"(dst + OPB), "l"(mb), "r"(kb), "r"(row_b), "r"(fb) : "memory");
          ++stage;
          return true;
        };
        for (int st = 0; ok && st < sh.n1; ++st) {
          const int kb = sh.kb0 + st * KS / TILE;
          if (st % (TILE / KS) == 0) {           // a new block of K: both tiles must have been announced
            const int* fa = over_x ? x_flag(sh.row_a, kb) : w_flag(sh.row_a, kb);
            const int* fb = t.kind == PROD ? x_flag(sh.row_b, kb) : w_flag(sh.row_b, kb);
            ok = flag_wait(fa, epoch, status, 83) && (sh.share || flag_wait(fb, epoch, status, 83));
            if (!ok) break;
            asm volatile("fence.proxy.async;" ::: "memory");      // written by other SMs' stores, read by TMA
          }
          const int k = sh.kb0 * TILE + st * KS;
          ok = issue(map_w, sh.row_a * TILE, k, map_w, sh.row_b * TILE, k, true, !sh.share);
        }
        if (ok && sh.n2) {
          const int p = t.b;                     // panel whose Linv the sum is multiplied by
          ok = flag_wait(g.flags + m.flag_d + p, epoch, status, 85);
          asm volatile("fence.proxy.async;" ::: "memory");
          for (int st = 0; ok && st < sh.n2; ++st) ok = issue(0, 0, 0, reinterpret_cast<uint64_t>(m.map_li), p * TILE, st * KS, false, true);
        }
        if (ok && t.kind == DIAG) {              // the block is factored in the ring: no load may land meanwhile
          ok = mbar_wait(ddone, n_diag & 1, status, 86);
          ++n_diag;
        }
      }
      issued = stage;
      if (!ok) dead = 1;
    }
    // ------------------------------------------------------------------ MMA issuer
    const uint32_t idesc = instr_desc(2u, 0u);   // tf32, K-major
    uint32_t stage = 0, chunk = 0;
    for (uint32_t n = 0; warp == MMA_WARP; ++n) {
      Task t;
      if (!take(n, t)) { dead = 1; break; }
      if (t.kind < 0) break;
      const Shape sh = shape_of(t, g.mats[t.mat].d);
      bool ok = true;
      if (lane == 0) {
        for (int phase = 0; phase < 2 && ok; ++phase) {
          const int ns = phase == 0 ? sh.n1 : sh.n2;
          const bool share = phase == 0 && sh.share;
          for (int s = 0; s < ns; ++s, ++stage) {
            const uint32_t rs = stage % RAW, ls = stage % LO, b = chunk & 1;
            const bool first = (s % FLUSH) == 0;
            if (first && chunk >= 2) ok = mbar_wait(accempty0 + 8u * b, ((chunk >> 1) - 1) & 1, status, 88);
            if (ok) ok = mbar_wait(full(ls), (stage / LO) & 1, status, 87);
            if (!ok) break;
            tc_fence_after();
            const uint32_t ah = smem0 + rs * PART, bh = share ? ah : ah + OPB, al = lo0 + ls * PART, bl = share ? al : al + OPB;
            const uint32_t d_tmem = tmem_base + b * TILE;
#pragma unroll
            for (int ks = 0; ks < KS / 8; ++ks) {
              const uint64_t adh = desc_k(ah + ks * 32u), adl = desc_k(al + ks * 32u), bdh = desc_k(bh + ks * 32u), bdl = desc_k(bl + ks * 32u);
              umma<true>(d_tmem, adl, bdh, idesc, (first && ks == 0) ? 0u : 1u);
              umma<true>(d_tmem, adh, bdl, idesc, 1u);
              umma<true>(d_tmem, adh, bdh, idesc, 1u);
            }
            umma_commit(rawfree(rs));
            umma_commit(lofree(ls));
            if ((s % FLUSH) == FLUSH - 1 || s == ns - 1) {
              umma_commit(accfull0 + 8u * b);
              ++chunk;
            }
          }
        }
      }
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) { dead = 1; break; }
    }
    if (warp == MMA_WARP && lane == 0) mmas_done<LO>((int)stage, lofree, status, 98);
  } else if (warp >= SPLIT_WARP0) {
    // ------------------------------------------------------------------ split warps
    asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
    const int lt = tid - 32 * SPLIT_WARP0;       // 0 .. 127: 16-byte chunk lt & 7 of rows lt >> 3, + 16, ..
    const uint32_t so0 = sw_off(lt >> 3, lt & 7);
    uint32_t stage = 0, n_mult = 0;
    bool ok = true;
    for (uint32_t n = 0; ok; ++n) {
      Task t;
      if (!take(n, t)) { ok = false; break; }
      if (t.kind < 0) break;
      const Shape sh = shape_of(t, g.mats[t.mat].d);
      for (int s = 0; s < sh.n1 + sh.n2; ++s, ++stage) {
        const uint32_t rs = stage % RAW, ls = stage % LO;
        const bool mult = s >= sh.n1, share = sh.share && !mult;
        if (s == sh.n1) ok = mbar_wait(afull, n_mult & 1, status, 91);      // the sum has been written into the raw slots
        if (ok && !mult) ok = mbar_wait(rawfull(rs), (stage / RAW) & 1, status, 92);
        if (ok && stage >= LO) ok = mbar_wait(lofree(ls), ((stage / LO) - 1) & 1, status, 93);
        if (!ok) break;
        const uint32_t hi = smem0 + rs * PART + so0, lo = lo0 + ls * PART + so0;
        // all loads of a side before the first store: one chunk at a time, each would wait for the one before
        auto split = [&](uint32_t side) {
          float4 v[8];
#pragma unroll
          for (int j = 0; j < 8; ++j)            // sixteen rows further = 2048 bytes
            asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v[j].x), "=f"(v[j].y), "=f"(v[j].z), "=f"(v[j].w) : "r"(hi + side + j * 2048u));
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            // hi rounded to nearest, written back in place (see tile_task_tma_kernel)
            const uint32_t h0 = rna_tf32(v[j].x), h1 = rna_tf32(v[j].y), h2 = rna_tf32(v[j].z), h3 = rna_tf32(v[j].w);
            const uint32_t l0 = __float_as_uint(v[j].x - __uint_as_float(h0)), l1 = __float_as_uint(v[j].y - __uint_as_float(h1));
            const uint32_t l2 = __float_as_uint(v[j].z - __uint_as_float(h2)), l3 = __float_as_uint(v[j].w - __uint_as_float(h3));
            asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(hi + side + j * 2048u), "r"(h0), "r"(h1), "r"(h2), "r"(h3) : "memory");
            asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(lo + side + j * 2048u), "r"(l0), "r"(l1), "r"(l2), "r"(l3) : "memory");
          }
        };
        split(0);
        if (mult) ok = mbar_wait(rawfull(rs), (stage / RAW) & 1, status, 92);      // the sum is split while the inverse is awaited
        if (!ok) break;
        if (!share) split(OPB);
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(full(ls));
      }
      if (sh.n2) ++n_mult;
    }
    if (!ok) dead = 1;
  } else {
    // ------------------------------------------------------------------ accumulate, store, diagonal blocks
    asm volatile("setmaxnreg.inc.sync.aligned.u32 192;");
    const int q = warp & 3, half = warp >> 2;
    const int row = q * 32 + lane, col0 = half * 64;         // this thread's row of the tile and first of its 64 columns
    float* ring = reinterpret_cast<float*>(smem_raw + (smem0 - smem_u32(smem_raw)));
    float* stg = ring + (RING_BYTES + warp * STAGING) / 4;
    const uint32_t stg0 = smem0 + RING_BYTES + warp * STAGING;
    uint32_t stage = 0, chunk = 0;
    uint32_t n = 0;
    bool ok = true;
    for (;; ++n) {
      // Barriers have no limit, so the eight warps leave a task together: a wait may run out for one of them and just not
      // for another.  Each passes all_well once per task, whatever happens, and reads the same answer behind it (a warp
      // that is already at the next task may have given up there).
      auto all_well = [&]() {
        dpanel::sync_x();
        return gave_up > n;
      };
      auto fail = [&]() {
        gave_up = n;
        all_well();
        ok = false;
      };
      Task t;
      if (!take(n, t)) { fail(); break; }
      if (t.kind < 0) { ok = all_well(); break; }
      const Mat& m = g.mats[t.mat];
      const int d = m.d;
      const Shape sh = shape_of(t, d);
      float acc[64];
      // rows and columns of the matrix that the tile covers
      const int r0 = t.a * TILE;
      const int c0 = (t.kind == DIAG ? t.a : t.b) * TILE;
#pragma unroll
      for (int i = 0; i < 64; ++i) acc[i] = 0.f;
      if (t.kind == DIAG || t.kind == PANEL) {
        const int gr = r0 + row, gc = c0 + col0;
        const float* const src = g.src ? g.src : m.src;
        const int ld_src = g.src ? g.ld_src : m.ld_src;
        if (REV) {
          // element (d - 1 - gc - i, d - 1 - gr), which lies in the lower triangle as (gr, gc + i) does: a row of it for the lanes
          // of a warp; the padding rows come first and are those of an identity
          const int col_p = d - 1 - gr;
          if (col_p >= m.pub) {
#pragma unroll
            for (int i = 0; i < 64; ++i) acc[i] = gc + i == gr ? 1.f : 0.f;
          } else if (col_p >= 0) {
            const float* p = src + (int64_t)(d - 1 - gc) * ld_src + col_p;
#pragma unroll
            for (int i = 0; i < 64; ++i, p -= ld_src)
              if (gc + i < d && d - 1 - gc - i < m.pub) acc[i] = __ldcg(p);
          }
        } else if (gr < d) {
          const float* p = src + (int64_t)gr * ld_src + gc;
          if (ld_src % 4 == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0 && gc + 64 <= d) {
#pragma unroll
            for (int i = 0; i < 64; i += 4) {
              const float4 v = __ldcg(reinterpret_cast<const float4*>(p + i));
              acc[i] = v.x; acc[i + 1] = v.y; acc[i + 2] = v.z; acc[i + 3] = v.w;
            }
          } else {
#pragma unroll
            for (int i = 0; i < 64; ++i)
              if (gc + i < d) acc[i] = __ldcg(p + i);
          }
        }
        if (t.kind == DIAG) {
          const float v = shift_of(m, g.traces, g.damp_r);
#pragma unroll
          for (int i = 0; i < 64; ++i)
            if (gc + i == gr && (!REV || gr >= d - m.pub)) acc[i] += v;
        }
      }
      auto drain = [&](int chunks, float sign) {
        for (int c = 0; c < chunks; ++c, ++chunk) {
          const uint32_t b = chunk & 1;
          if (!mbar_wait(accfull0 + 8u * b, (chunk >> 1) & 1, status, 95)) return false;
          tc_fence_after();
          const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + b * TILE + (uint32_t)col0;
#pragma unroll
          for (int part = 0; part < 2; ++part) {
            uint32_t v[32];
            tmem_ld32(taddr + part * 32, v);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) acc[part * 32 + i] = fmaf(sign, __uint_as_float(v[i]), acc[part * 32 + i]);
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(accempty0 + 8u * b);
        }
        return true;
      };
      auto leave = [&]() {
        if (lane == 0) left = t;
        ok = false;
      };
      if (!drain(ceil_div(sh.n1, FLUSH), t.kind == PROD ? 1.f : -1.f)) { fail(); leave(); break; }
      stage += sh.n1;
      if (sh.n2) {
        // the sum becomes the A operand of four more stages: 64 columns = two of them (every MMA that read these
        // slots has completed: its accumulator has been drained)
#pragma unroll
        for (int i = 0; i < 64; i += 4) {
          const uint32_t s = (stage + half * 2 + i / 32) % RAW;
          asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(smem0 + s * PART + sw_off(row, (i % 32) / 4)), "f"(acc[i]), "f"(acc[i + 1]),
                       "f"(acc[i + 2]), "f"(acc[i + 3]) : "memory");
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(afull);
        stage += sh.n2;
#pragma unroll
        for (int i = 0; i < 64; ++i) acc[i] = 0.f;
        if (!drain(ceil_div(sh.n2, FLUSH), 1.f)) { fail(); leave(); break; }
      }
      const int nr = min(TILE, d - r0), nc = min(TILE, d - c0);
      // Results in the order of M: element (r, c) of the tile at o + r * sr + c * sc, of which the padding is left out.
      float* const T = g.out ? g.out : m.T;
      float* const U = m.U && g.out ? g.out : m.U;
      const int ldt = g.out ? g.ld_out : m.ldt, ldu = g.out ? g.ld_out : m.ldu;
      const int pad = REV ? d - m.pub : 0;
      constexpr int dir = REV ? -1 : 1;
      auto place = [&](float* base, int ld, int r, int c) {
        return REV ? base + (int64_t)(d - 1 - r) * ld + (d - 1 - c) : base + (int64_t)r * ld + c;
      };
      // rows along lanes, through 32 columns of this warp's staging tile at a time
      auto store_rows = [&](float* o, int ld, bool lower) {
#pragma unroll
        for (int part = 0; part < 2; ++part) {
#pragma unroll
          for (int i = 0; i < 32; ++i) stg[lane * 32 + (i ^ lane)] = acc[part * 32 + i];
          __syncwarp();
          const int c = col0 + part * 32 + lane;
          for (int rr = 0; rr < 32; ++rr) {
            const int r = q * 32 + rr;
            if (r < nr && c < nc && r0 + r >= pad && c0 + c >= pad && !(lower && c > r))
              o[(int64_t)r * (dir * ld) + dir * c] = stg[rr * 32 + (lane ^ rr)];
          }
          __syncwarp();
        }
      };
      // the tile as the scratch matrix' block (r0, c0), a box of 32x32 per warp and copy: TMA clips it at the matrix edge.  (Through
      // store_rows a panel tile took 4.1 us from its sum to its flag.)
      auto store_boxes = [&]() {
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          const int gr = r0 + q * 32, gc = c0 + col0 + part * 32;
          if (part) {
            if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            __syncwarp();
          }
#pragma unroll
          for (int i = 0; i < 32; i += 4)
            asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(stg0 + sw_off(lane, i / 4)), "f"(acc[part * 32 + i]), "f"(acc[part * 32 + i + 1]),
                         "f"(acc[part * 32 + i + 2]), "f"(acc[part * 32 + i + 3]) : "memory");
          fence_async_smem();
          __syncwarp();
          if (lane == 0 && gr < d && gc < d) {
            asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(reinterpret_cast<uint64_t>(m.map_box)),
                         "r"(gc), "r"(gr), "r"(stg0) : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        }
        if (lane == 0) {
          asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
          asm volatile("fence.proxy.async;" ::: "memory");
        }
        __syncwarp();
      };
      auto store_columns = [&](float* o, int ld, bool lower) {      // the transposed tile: a column per instruction
        o += (int64_t)col0 * (dir * ld) + dir * row;
#pragma unroll
        for (int i = 0; i < 64; ++i, o += dir * ld) {
          const int c = col0 + i;
          if (row < nr && c < nc && r0 + row >= pad && c0 + c >= pad && !(lower && c >= row)) *o = acc[i];
        }
      };
      // the tile, transposed, as a block of U, and zeros across the diagonal
      auto store_u = [&]() {
        store_columns(place(U, ldu, c0, r0), ldu, false);
        float* z = place(U, ldu, r0, c0);
        for (int rr = warp; rr < nr; rr += ACC_WARPS)
          for (int c = lane; c < nc; c += 32)
            if (r0 + rr >= pad && c0 + c >= pad) z[(int64_t)rr * (dir * ldu) + dir * c] = 0.f;
      };
      const bool with_u = U && g.with_u;
      int* flag = nullptr;
      if (t.kind != DIAG) {
        if (t.kind == PANEL) {
          store_boxes();
          flag = g.flags + m.flag_w + t.a * m.np + t.b;
        } else if (t.kind == INVT) {
          store_boxes();
          flag = g.flags + m.flag_x + t.a * m.np + t.b;
        } else {
          store_rows(place(T, ldt, r0, c0), ldt, t.a == t.b);
          store_columns(place(T, ldt, c0, r0), ldt, t.a == t.b);
        }
        if (!all_well()) { leave(); break; }      // and the tile is stored by all eight warps
      } else {
        // ---------------------------------------------------------------- diagonal block, in the operand ring
        float* S = ring;
        float* V = S + dpanel::PN * dpanel::PP;
        if (row < nr) {
#pragma unroll
          for (int i = 0; i < 64; i += 4) dpanel::st4(S + row * dpanel::PP + col0 + i, acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
        } else {
#pragma unroll
          for (int i = 0; i < 64; ++i) S[row * dpanel::PP + col0 + i] = col0 + i == row ? 1.f : 0.f;
        }
        if (!all_well()) { leave(); break; }
        dpanel::factor_block(S, V, nr, g.info ? g.info + 2 * m.mat + m.info_slot : nullptr, REV ? d - r0 : r0 + 1, dir, tid);
        float* li = m.Li + (int64_t)t.a * (TILE * TILE);
        for (int e = tid; e < TILE * TILE / 4; e += 256) {
          const int r = e / (TILE / 4), c = e % (TILE / 4) * 4;
          reinterpret_cast<float4*>(li)[e] = dpanel::ld4(V + r * dpanel::PP + c);
        }
        dpanel::sync_x();                        // the next panel waits for this alone: announced before the other results
        if (tid == 0) {
          __threadfence();
          store_release(g.flags + m.flag_d + t.a, epoch);
        }
        for (int r = warp; r < nr; r += ACC_WARPS) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int c = lane + 32 * u;
            if (c >= nr) continue;
            if (m.X) m.X[(int64_t)(r0 + r) * m.ldw + r0 + c] = V[c * dpanel::PP + r];
            if (with_u && !m.X) U[(int64_t)(r0 + r) * ldu + r0 + c] = c >= r ? S[c * dpanel::PP + r] : 0.f;
            if (with_u && m.X && r0 + r >= pad && r0 + c >= pad) *place(U, ldu, r0 + r, r0 + c) = c <= r ? V[r * dpanel::PP + c] : 0.f;
          }
        }
        if (m.X) flag = g.flags + m.flag_x + t.a * m.np + t.a;
        fence_async_smem();                      // the ring goes back to TMA
        __syncwarp();
        if (lane == 0) mbar_arrive(ddone);
        if (flag) dpanel::sync_x();
      }
      if (flag && tid == 0) {
        __threadfence();
        store_release(flag, epoch);
      }
      if (with_u && t.kind == (m.X ? INVT : PANEL)) store_u();      // nobody waits for U
    }
    if (!ok) dead = 1;
    if (tid == 0) acc_at = n;
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 256);
  }
  if (!dead) return;
  // A wait of this CTA gave up.  Its copies in flight must have landed before it leaves; then the tasks that it holds
  // and all that it can still take are answered with NaN, so that nothing stale passes for a result and nobody waits
  // for them.
  if (tid == 0 && !g_inject_stall)
    for (uint32_t s = issued > RAW ? issued - RAW : 0; s < issued; ++s) mbar_wait(rawfull(s % RAW), (s / RAW) & 1, status, 97);
  const float nan = __int_as_float(0x7fc00000);
  auto poison = [&](const Task& t) {
    const Mat& m = g.mats[t.mat];
    const int r0 = t.a * TILE, c0 = (t.kind == DIAG ? t.a : t.b) * TILE, nr = min(TILE, m.d - r0), nc = min(TILE, m.d - c0);
    auto fill = [&](float* o, int ld, int rows, int cols) {
      for (int e = tid; e < rows * cols; e += THREADS) o[(int64_t)(e / cols) * ld + e % cols] = nan;
    };
    auto fill_result = [&](float* base, int ld, int row, int col, int rows, int cols) {      // a block in the order of M
      for (int e = tid; e < rows * cols; e += THREADS) {
        const int r = row + e / cols, c = col + e % cols, pad = m.d - m.pub;
        if (r >= pad && c >= pad) base[REV ? (int64_t)(m.d - 1 - r) * ld + (m.d - 1 - c) : (int64_t)r * ld + c] = nan;
      }
    };
    if (t.kind == DIAG) {
      fill(m.Li + (int64_t)t.a * (TILE * TILE), TILE, TILE, TILE);
      if (m.X) fill(m.X + (int64_t)r0 * m.ldw + r0, m.ldw, nr, nr);
    }
    if (t.kind == PANEL) fill(m.W + (int64_t)r0 * m.ldw + c0, m.ldw, nr, nc);
    if (t.kind == INVT) fill(m.X + (int64_t)r0 * m.ldw + c0, m.ldw, nr, nc);
    float* const T = g.out ? g.out : m.T;
    float* const U = m.U && g.out ? g.out : m.U;
    const int ldt = g.out ? g.ld_out : m.ldt, ldu = g.out ? g.ld_out : m.ldu;
    if (t.kind == PROD) { fill_result(T, ldt, r0, c0, nr, nc); fill_result(T, ldt, c0, r0, nc, nr); }
    if (m.U && g.with_u && (t.kind == DIAG || t.kind == (m.X ? INVT : PANEL))) fill_result(U, ldu, c0, r0, nc, nr);
    __syncthreads();
    if (tid == 0 && t.kind != PROD) {
      __threadfence();
      if (t.kind == DIAG) store_release(g.flags + m.flag_d + t.a, epoch);
      if (t.kind == PANEL) store_release(g.flags + m.flag_w + t.a * m.np + t.b, epoch);
      else if (m.X) store_release(g.flags + m.flag_x + t.a * m.np + (t.kind == DIAG ? t.a : t.b), epoch);
    }
  };
  if (left.kind >= 0) poison(left);
  for (uint32_t n = acc_at + (left.kind >= 0 ? 1 : 0); n < pushed; ++n)
    if (queue[n % QUEUE].kind >= 0) poison(queue[n % QUEUE]);
  if (lost.kind >= 0) poison(lost);
  for (;;) {
    __syncthreads();
    if (tid == 0) {
      const unsigned idx = (unsigned)atomicAdd(&g.sync[0], 1) - (unsigned)g.sync[2];
      lost.kind = -1;
      if (idx < (unsigned)g.n_tasks) lost = g.tasks[idx];
    }
    __syncthreads();
    if (lost.kind < 0) break;
    poison(lost);
  }
  if (tid == 0 && g.info) g.info[0] = -(1000 + *reinterpret_cast<volatile int*>(status));
}

}  // namespace flow

int flow_set_wait_controls(long long cycles, int stall) { return tc::set_wait_controls(cycles, stall); }

int flow_launch(const flow::Args& a, int n_mats, int clear_info, int with_traces, cudaStream_t st) {
  SSO_ENSURE_SMEM(flow::flow_kernel<false>, flow::SMEM);
  SSO_ENSURE_SMEM(flow::flow_kernel<true>, flow::SMEM);
  flow::begin_kernel<<<n_mats, 256, 0, st>>>(a.mats, n_mats, a.sync, const_cast<float*>(a.traces), a.info, clear_info, with_traces, a.src, a.ld_src);
  SSO_LAUNCH_OK("flow begin");
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(a.n_tasks < 148 ? a.n_tasks : 148);
  cfg.blockDim = dim3(flow::THREADS);
  cfg.dynamicSmemBytes = flow::SMEM;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // set-up beside begin_kernel
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, a.rev ? flow::flow_kernel<true> : flow::flow_kernel<false>, a);
  SSO_LAUNCH_OK("flow_kernel");
  return 0;
}

}  // namespace sso
