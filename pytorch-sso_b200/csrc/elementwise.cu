// HBM-streaming kernels of the K-FAC path: EMA / scaled accumulation over flat factor pools,
// BatchNorm diagonal curvature, diagonal inverse + precondition, triangular pack / unpack.
// All are bandwidth bound: 16-byte vector accesses where alignment allows, grids sized as a
// multiple of the 148 SMs with a grid-stride loop.
#include <algorithm>

#include "common.cuh"

namespace sso {

constexpr int kSMs = 148;

__device__ __forceinline__ float ema_op(float data, float ema, float beta, float omb) {
  return fmaf(beta, data, omb * ema);
}

// dst <- a*src + b*dst, rounded once where one of the factors is 1: a scaled sum has the same bits whichever of the two holds
// the terms before (with a multiplication of its own, three closures' factors were 3.6e-8 off instead of 3.3e-8).
__device__ __forceinline__ float axpby_op(float a, float s, float b, float d) {
  return a == 1.f ? fmaf(b, d, s) : fmaf(a, s, b * d);
}

// dst <- a*src + b*dst  (b == 0: dst is not read)
__global__ void __launch_bounds__(256) axpby_kernel(const float* __restrict__ src, float* __restrict__ dst,
                                                    int64_t count, float a, float b) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool vec = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0;
  if (vec) {
    const int64_t n4 = count >> 2;
    const float4* s4 = reinterpret_cast<const float4*>(src);
    float4* d4 = reinterpret_cast<float4*>(dst);
    for (int64_t i = tid; i < n4; i += stride) {
      const float4 s = __ldg(s4 + i);
      float4 o;
      if (b == 0.f) {
        o = make_float4(a * s.x, a * s.y, a * s.z, a * s.w);
      } else {
        const float4 d = d4[i];
        o = make_float4(axpby_op(a, s.x, b, d.x), axpby_op(a, s.y, b, d.y), axpby_op(a, s.z, b, d.z), axpby_op(a, s.w, b, d.w));
      }
      d4[i] = o;
    }
    for (int64_t i = (n4 << 2) + tid; i < count; i += stride)
      dst[i] = (b == 0.f) ? a * src[i] : axpby_op(a, src[i], b, dst[i]);
  } else {
    for (int64_t i = tid; i < count; i += stride)
      dst[i] = (b == 0.f) ? a * src[i] : axpby_op(a, src[i], b, dst[i]);
  }
}

static int grid_for(int64_t count, int per_thread) {
  const int64_t want = ceil_div64(count, (int64_t)256 * per_thread);
  const int64_t cap = (int64_t)kSMs * 8;
  return (int)std::max<int64_t>(1, std::min(want, cap));
}

// ------------------------------------------------------------------------------------------
// BatchNorm diagonal curvature
// ------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) bn_plane_sums_pcontig(const T* __restrict__ y, const T* __restrict__ g,
                                                             int n, int c, int hw, int64_t syn, int64_t syc, int64_t syp,
                                                             int64_t sgn, int64_t sgc, int64_t sgp,
                                                             const float* __restrict__ scale,
                                                             const float* __restrict__ shift,
                                                             float* __restrict__ sx, float* __restrict__ sg) {
  // one warp per (n, c) plane
  const int warp = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (warp >= n * c) return;
  const int in = warp / c, ic = warp % c;
  const float inv_scale = scale ? 1.f / scale[ic] : 1.f, sh = shift ? shift[ic] : 0.f;
  const T* py = y + (int64_t)in * syn + (int64_t)ic * syc;
  const T* pg = g + (int64_t)in * sgn + (int64_t)ic * sgc;
  float ax = 0.f, ag = 0.f;
  for (int p = lane; p < hw; p += 32) {
    if (y) {
      const float xv = (to_f32<T>(py[(int64_t)p * syp]) - sh) * inv_scale;
      ax = fmaf(xv, xv, ax);
    }
    if (g) {
      const float gv = to_f32<T>(pg[(int64_t)p * sgp]);
      ag = fmaf(gv, gv, ag);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ax += __shfl_xor_sync(0xffffffffu, ax, o);
    ag += __shfl_xor_sync(0xffffffffu, ag, o);
  }
  if (lane == 0) {
    if (y) sx[warp] = ax;
    if (g) sg[warp] = ag;
  }
}

template <typename T>
__global__ void __launch_bounds__(256) bn_plane_sums_ccontig(const T* __restrict__ y, const T* __restrict__ g,
                                                             int n, int c, int hw, int64_t syn, int64_t syc, int64_t syp,
                                                             int64_t sgn, int64_t sgc, int64_t sgp,
                                                             const float* __restrict__ scale,
                                                             const float* __restrict__ shift,
                                                             float* __restrict__ sx, float* __restrict__ sg) {
  // block = 32 channels x 8 pixel lanes; grid = (ceil(c/32), n)
  __shared__ float rx[8][33], rg[8][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int ic = blockIdx.x * 32 + tx, in = blockIdx.y;
  float ax = 0.f, ag = 0.f;
  if (ic < c) {
    const float inv_scale = scale ? 1.f / scale[ic] : 1.f, sh = shift ? shift[ic] : 0.f;
    const T* py = y + (int64_t)in * syn + (int64_t)ic * syc;
    const T* pg = g + (int64_t)in * sgn + (int64_t)ic * sgc;
    for (int p = ty; p < hw; p += 8) {
      if (y) {
        const float xv = (to_f32<T>(py[(int64_t)p * syp]) - sh) * inv_scale;
        ax = fmaf(xv, xv, ax);
      }
      if (g) {
        const float gv = to_f32<T>(pg[(int64_t)p * sgp]);
        ag = fmaf(gv, gv, ag);
      }
    }
  }
  rx[ty][tx] = ax;
  rg[ty][tx] = ag;
  __syncthreads();
  if (ty == 0 && ic < c) {
    float tx_sum = 0.f, tg_sum = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      tx_sum += rx[i][tx];
      tg_sum += rg[i][tx];
    }
    if (y) sx[(int64_t)in * c + ic] = tx_sum;
    if (g) sg[(int64_t)in * c + ic] = tg_sum;
  }
}

// Channels-contiguous planes, vectorised: a thread owns V = 16 bytes / sizeof(T) consecutive channels
// and walks pixels; LP lanes cover one pixel's channels (LP*V >= c), 256/LP pixels are processed in
// parallel per block, and the pixel range of one image is cut into `splits` blocks.  Partial sums go
// to out[(n*splits + split)*c + channel]; the finishing kernel adds the splits.
template <typename T, bool IS_Y>
__device__ __forceinline__ void bn_plane_sums_block(const T* __restrict__ t, int c, int hw, int64_t sn, int64_t sp, int lp,
                                                    int splits, const float* __restrict__ scale,
                                                    const float* __restrict__ shift, float* __restrict__ out, int in,
                                                    int split, float* __restrict__ red_) {
  constexpr int V = 16 / sizeof(T);
  float (*red)[V + 1] = reinterpret_cast<float (*)[V + 1]>(red_);
  const int cv = threadIdx.x % lp, pp = threadIdx.x / lp, npp = 256 / lp;
  const int per = (hw + splits - 1) / splits;
  const int p0 = split * per, p1 = min(hw, p0 + per);
  const int c0 = cv * V;
  float acc[V];
#pragma unroll
  for (int i = 0; i < V; ++i) acc[i] = 0.f;
  if (c0 < c) {
    float isc[V], sh[V];
#pragma unroll
    for (int i = 0; i < V; ++i) {
      isc[i] = (IS_Y && scale) ? 1.f / scale[c0 + i] : 1.f;
      sh[i] = (IS_Y && shift) ? shift[c0 + i] : 0.f;
    }
    const T* base = t + (int64_t)in * sn + c0;
    auto add = [&](const uint4& raw) {
      const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const float v = (to_f32<T>(e[i]) - sh[i]) * isc[i];
        acc[i] = fmaf(v, v, acc[i]);
      }
    };
    int p = p0 + pp;
    for (; p + 3 * npp < p1; p += 4 * npp) {      // four independent 16-byte loads in flight per thread
      const uint4 r0 = __ldg(reinterpret_cast<const uint4*>(base + (int64_t)p * sp));
      const uint4 r1 = __ldg(reinterpret_cast<const uint4*>(base + (int64_t)(p + npp) * sp));
      const uint4 r2 = __ldg(reinterpret_cast<const uint4*>(base + (int64_t)(p + 2 * npp) * sp));
      const uint4 r3 = __ldg(reinterpret_cast<const uint4*>(base + (int64_t)(p + 3 * npp) * sp));
      add(r0); add(r1); add(r2); add(r3);
    }
    for (; p < p1; p += npp) add(__ldg(reinterpret_cast<const uint4*>(base + (int64_t)p * sp)));
  }
#pragma unroll
  for (int i = 0; i < V; ++i) red[threadIdx.x][i] = acc[i];
  __syncthreads();
  const int channels = lp * V;
  if (channels < 256) {
    // few channels are many pixel lanes: neighbouring threads share those of a channel (by the first lane alone this was
    // a chain of npp loads: 16 channels of 8 images 9.7 -> 4.4 us, 64 of 32 56x56 images 7.0 -> 6.0)
    const int share = min(32, 256 / channels), part = threadIdx.x % share;
    for (int k = threadIdx.x / share; k < channels; k += 256 / share) {
      float sum = 0.f;
      for (int q = part; q < npp; q += share) sum += red[q * lp + k / V][k % V];
      for (int o = 1; o < share; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (part == 0 && k < c) out[((int64_t)in * splits + split) * c + k] = sum;
    }
  } else if (pp == 0 && c0 < c) {
    float* o = out + ((int64_t)in * splits + split) * c + c0;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      float sum = 0.f;
      for (int q = 0; q < npp; ++q) sum += red[q * lp + cv][i];
      o[i] = sum;
    }
  }
}

template <typename T, bool IS_Y>
__global__ void __launch_bounds__(256) bn_plane_sums_vec(const T* __restrict__ t, int c, int hw, int64_t sn, int64_t sp, int lp,
                                                         int splits, const float* __restrict__ scale,
                                                         const float* __restrict__ shift, float* __restrict__ out) {
  __shared__ float red[256 * (16 / sizeof(T) + 1)];
  bn_plane_sums_block<T, IS_Y>(t, c, hw, sn, sp, lp, splits, scale, shift, out, blockIdx.y, blockIdx.x, red);
}

// block = 8 channels x 32 image lanes: with the usual 32..256 images a thread owns one to eight
// images, issues the loads of all their split partials back to back, and the 32 lanes are combined
// in shared memory (fixed order: deterministic).  Many small blocks keep this latency-bound step short.
__device__ __forceinline__ void bn_finish_block(const float* __restrict__ sx, const float* __restrict__ sg,
                                                const float* __restrict__ weight, int n, int c, int splits_x, int splits_g,
                                                float alpha, float beta, float* __restrict__ w_out,
                                                float* __restrict__ b_out, int block) {
  __shared__ float rw[32][9], rb[32][9];
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
  const int ic = block * 8 + tx;
  float aw = 0.f, ab = 0.f;
  if (ic < c) {
    for (int in = ty; in < n; in += 32) {
      const float* px = sx + (int64_t)in * splits_x * c + ic;
      const float* pg = sg + (int64_t)in * splits_g * c + ic;
      float x0 = 0.f, x1 = 0.f, g0 = 0.f, g1 = 0.f;
      int q = 0;
      for (; q + 1 < splits_x; q += 2) { x0 += px[(int64_t)q * c]; x1 += px[(int64_t)(q + 1) * c]; }
      if (q < splits_x) x0 += px[(int64_t)q * c];
      for (q = 0; q + 1 < splits_g; q += 2) { g0 += pg[(int64_t)q * c]; g1 += pg[(int64_t)(q + 1) * c]; }
      if (q < splits_g) g0 += pg[(int64_t)q * c];
      const float gsum = (weight ? weight[in] : 1.f) * (g0 + g1);
      aw = fmaf(x0 + x1, gsum, aw);
      ab += gsum;
    }
  }
  rw[ty][tx] = aw;
  rb[ty][tx] = ab;
  __syncthreads();
  if (ty == 0 && ic < c) {
    float tw = 0.f, tb = 0.f;
#pragma unroll
    for (int i = 0; i < 32; ++i) { tw += rw[i][tx]; tb += rb[i][tx]; }
    const float s = alpha / (float)n;
    w_out[ic] = (beta == 0.f) ? s * tw : fmaf(beta, w_out[ic], s * tw);
    if (b_out) b_out[ic] = (beta == 0.f) ? s * tb : fmaf(beta, b_out[ic], s * tb);
  }
}

__global__ void __launch_bounds__(256) bn_finish_kernel(const float* __restrict__ sx, const float* __restrict__ sg,
                                                        const float* __restrict__ weight, int n, int c,
                                                        int splits_x, int splits_g, float alpha, float beta,
                                                        float* __restrict__ w_out, float* __restrict__ b_out) {
  bn_finish_block(sx, sg, weight, n, c, splits_x, splits_g, alpha, beta, w_out, b_out, blockIdx.x);
}

// The gradient sums of many layers in one launch and their results in a second: a ResNet has a layer of a few
// microseconds' work per convolution, and launches of one layer each filled the chip for a fraction of their time (the 53
// layers of ResNet-50 at 32 images in bf16: 800 us layer by layer, 239 us in two launches, 711 MB read).  The records
// travel in the kernel's parameter space.
constexpr int BN_BATCH = 64;
struct BnRec {
  sso_bn_desc d;
  int lp, sum0, fin0;      // lanes of a pixel; first block of this layer in either launch
};
struct BnBatch {
  int n;
  BnRec rec[BN_BATCH];
};

template <bool FINISH>
__device__ __forceinline__ int bn_find(const BnBatch& b) {
  int lo = 0, hi = b.n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if ((FINISH ? b.rec[mid].fin0 : b.rec[mid].sum0) <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
  }
  return lo;
}

__global__ void __launch_bounds__(256) bn_batch_sums_kernel(const __grid_constant__ BnBatch b) {
  __shared__ float red[256 * 9];
  const BnRec& r = b.rec[bn_find<false>(b)];
  const int j = (int)blockIdx.x - r.sum0, in = j / r.d.splits_g, split = j - in * r.d.splits_g;
  const int c = (int)r.d.c, hw = (int)r.d.hw;
  if (r.d.dtype == SSO_F32)
    bn_plane_sums_block<float, false>(reinterpret_cast<const float*>(r.d.g), c, hw, r.d.sn, r.d.sp, r.lp, r.d.splits_g, nullptr,
                                      nullptr, r.d.sg, in, split, red);
  else if (r.d.dtype == SSO_BF16)
    bn_plane_sums_block<__nv_bfloat16, false>(reinterpret_cast<const __nv_bfloat16*>(r.d.g), c, hw, r.d.sn, r.d.sp, r.lp,
                                              r.d.splits_g, nullptr, nullptr, r.d.sg, in, split, red);
  else
    bn_plane_sums_block<__half, false>(reinterpret_cast<const __half*>(r.d.g), c, hw, r.d.sn, r.d.sp, r.lp, r.d.splits_g,
                                       nullptr, nullptr, r.d.sg, in, split, red);
}

__global__ void __launch_bounds__(256) bn_batch_finish_kernel(const __grid_constant__ BnBatch b) {
  const BnRec& r = b.rec[bn_find<true>(b)];
  bn_finish_block(r.d.sx, r.d.sg, r.d.sample_weight, (int)r.d.n, (int)r.d.c, r.d.splits_x, r.d.splits_g, r.d.alpha, r.d.beta,
                  r.d.w_out, r.d.b_out, (int)blockIdx.x - r.fin0);
}

// pixel-range splits of the vectorised kernel for a [n, c, hw] tensor (1 when it is not used)
static int bn_vec_lanes(int64_t c, int vec) {
  if (c % vec != 0 || c / vec > 256) return 0;
  int lp = 1;
  while (lp < c / vec) lp <<= 1;
  return lp;
}
static int bn_vec_splits(int64_t n, int64_t c, int64_t hw, int vec) {
  const int lp = bn_vec_lanes(c, vec);
  if (lp == 0 || hw <= 1) return 1;
  const int npp = 256 / lp;
  int64_t s = ceil_div64(4 * kSMs, n);                       // about four blocks per SM
  const int64_t most = std::max<int64_t>(1, hw / (8 * npp)); // at least eight pixels per lane
  if (s > most) s = most;
  return (int)std::max<int64_t>(1, s);
}

template <typename T>
static int bn_sums_typed(const void* y, const void* g, int64_t n, int64_t c, int64_t hw, int64_t syn,
                         int64_t syc, int64_t syp, int64_t sgn, int64_t sgc, int64_t sgp,
                         const float* scale, const float* shift, float* sx, float* sg, int splits,
                         cudaStream_t st) {
  const T* ty = reinterpret_cast<const T*>(y);
  const T* tg = reinterpret_cast<const T*>(g);
  constexpr int V = 16 / sizeof(T);
  const int lp = bn_vec_lanes(c, V);
  auto vec_ok = [&](const T* p, int64_t sc_, int64_t sn_, int64_t sp_) {
    return p != nullptr && sc_ == 1 && lp > 0 && hw > 1 && (reinterpret_cast<uintptr_t>(p) & 15) == 0 &&
           (sn_ * sizeof(T)) % 16 == 0 && (sp_ * sizeof(T)) % 16 == 0;
  };
  if (splits > 1 || (vec_ok(ty, syc, syn, syp) || !y) && (vec_ok(tg, sgc, sgn, sgp) || !g) && hw > 1 && lp > 0) {
    SSO_CHECK_ARG((!y || vec_ok(ty, syc, syn, syp)) && (!g || vec_ok(tg, sgc, sgn, sgp)),
                  "bn_plane_sums: splits > 1 needs channels-contiguous, 16-byte aligned planes");
    dim3 grid((unsigned)splits, (unsigned)n);
    if (y) {
      bn_plane_sums_vec<T, true><<<grid, 256, 0, st>>>(ty, (int)c, (int)hw, syn, syp, lp, splits, scale, shift, sx);
      SSO_LAUNCH_OK("bn_plane_sums_vec");
    }
    if (g) {
      bn_plane_sums_vec<T, false><<<grid, 256, 0, st>>>(tg, (int)c, (int)hw, sgn, sgp, lp, splits, nullptr, nullptr, sg);
      SSO_LAUNCH_OK("bn_plane_sums_vec");
    }
    return 0;
  }
  if (syc == 1 && sgc == 1 && hw > 1) {
    dim3 grid((unsigned)ceil_div64(c, 32), (unsigned)n);
    bn_plane_sums_ccontig<T><<<grid, 256, 0, st>>>(ty, tg, (int)n, (int)c, (int)hw, syn, syc, syp, sgn, sgc,
                                                    sgp, scale, shift, sx, sg);
  } else {
    const int64_t warps = n * c;
    bn_plane_sums_pcontig<T><<<(unsigned)ceil_div64(warps * 32, 256), 256, 0, st>>>(
        ty, tg, (int)n, (int)c, (int)hw, syn, syc, syp, sgn, sgc, sgp, scale, shift, sx, sg);
  }
  SSO_LAUNCH_OK("bn_plane_sums");
  return 0;
}

// ------------------------------------------------------------------------------------------
// diagonal inverse / precondition
// ------------------------------------------------------------------------------------------
__global__ void diag_inv_precond_kernel(const float* __restrict__ ema, float* __restrict__ inv,
                                        float* __restrict__ grad, int64_t count, float damping,
                                        int use_sqrt, int update_inv) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += stride) {
    float v;
    if (update_inv) {
      float x = ema[i];
      if (use_sqrt) x = sqrtf(x);
      v = 1.f / (x + damping);
      inv[i] = v;
    } else {
      v = inv[i];
    }
    if (grad) grad[i] *= v;
  }
}

// ------------------------------------------------------------------------------------------
// triangular pack / unpack over a table of row runs
// ------------------------------------------------------------------------------------------
// Both kernels read through the read-only path in batches of four loads per thread: the source and the
// destination come out of one record, so with plain loads every load would wait for the previous store.
__global__ void __launch_bounds__(256) tri_pack_kernel(const sso_tri_rec* __restrict__ recs, float scale) {
  const sso_tri_rec r = recs[blockIdx.x];
  for (int row = r.row0; row < r.row0 + r.nrows; ++row) {
    const int64_t base = (int64_t)r.n * row - (int64_t)row * (row + 1) / 2;
    const float* src = r.m + (int64_t)row * r.ld;
    float* dst = r.packed + base;
    for (int x0 = row + threadIdx.x; x0 < r.n; x0 += 4 * 256) {
      float v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = (x0 + 256 * u < r.n) ? __ldg(src + x0 + 256 * u) : 0.f;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (x0 + 256 * u < r.n) dst[x0 + 256 * u] = scale * v[u];
    }
  }
}
// A record of at most 32 rows: the part on and above the diagonal is copied row by row (contiguous in the
// packed form); the part below it is the transpose of packed rows, moved in 32 x 32 tiles through shared
// memory so that the packed rows are read and the matrix rows written in whole 128-byte lines.  Longer
// records take the element-wise path (strided reads below the diagonal).
__global__ void __launch_bounds__(256) tri_unpack_kernel(const sso_tri_rec* __restrict__ recs, float scale,
                                                         int symmetric) {
  __shared__ float tile[2][32][33];
  const sso_tri_rec r = recs[blockIdx.x];
  const int n = r.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float* pk = r.packed;
  auto base = [n](int row) { return (int64_t)n * row - (int64_t)row * (row + 1) / 2; };
  if (r.nrows > 32) {
    if (blockIdx.y != 0) return;
    for (int row = r.row0; row < r.row0 + r.nrows; ++row) {
      float* dst = r.m + (int64_t)row * r.ld;
      for (int x = tid; x < n; x += 256) {
        const int lo = min(row, x), hi = max(row, x);
        const float v = scale * __ldg(pk + base(lo) + hi);
        dst[x] = (symmetric || x >= row) ? v : 0.f;
      }
    }
    return;
  }
  // gridDim.y CTAs share a record: rows of the upper part and tiles of the lower part are dealt round robin
  const int part = blockIdx.y, parts = gridDim.y;
  for (int rr = part; rr < r.nrows; rr += parts) {
    const int row = r.row0 + rr;
    const float* src = pk + base(row);
    float* dst = r.m + (int64_t)row * r.ld;
    for (int x0 = row + tid; x0 < n; x0 += 4 * 256) {
      float v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = (x0 + 256 * u < n) ? __ldg(src + x0 + 256 * u) : 0.f;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (x0 + 256 * u < n) dst[x0 + 256 * u] = scale * v[u];
    }
  }
  const int xend = r.row0 + r.nrows - 1;        // columns x < xend have elements below the diagonal in this band
  int buf = 0;
  for (int x0 = 32 * part; x0 < xend; x0 += 32 * parts, buf ^= 1) {
    float v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int x = x0 + warp + 8 * k, row = r.row0 + lane;
      v[k] = (symmetric && lane < r.nrows && x < row) ? __ldg(pk + base(x) + row) : 0.f;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) tile[buf][warp + 8 * k][lane] = v[k];
    __syncthreads();          // (two buffers: the next tile's stores cannot overtake this tile's reads)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int rr = warp + 8 * k, row = r.row0 + rr, x = x0 + lane;
      if (rr < r.nrows && x < row) r.m[(int64_t)row * r.ld + x] = scale * tile[buf][lane][rr];
    }
  }
}

// scaled copies of many flat segments in one launch (one CTA per record)
__global__ void __launch_bounds__(256) copy_segments_kernel(const sso_seg_rec* __restrict__ recs, float scale) {
  const sso_seg_rec r = recs[blockIdx.x];
  const bool vec = ((reinterpret_cast<uintptr_t>(r.src) | reinterpret_cast<uintptr_t>(r.dst)) & 15) == 0;
  if (vec) {
    const int64_t n4 = r.count >> 2;
    // four 16-byte loads in flight per thread: one at a time leaves an SM with ~10 KB on its way to it
    for (int64_t i0 = threadIdx.x; i0 < n4; i0 += 4 * 256) {
      float4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i0 + 256 * u < n4) v[u] = __ldg(reinterpret_cast<const float4*>(r.src) + i0 + 256 * u);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i0 + 256 * u < n4)
          reinterpret_cast<float4*>(r.dst)[i0 + 256 * u] = make_float4(scale * v[u].x, scale * v[u].y, scale * v[u].z, scale * v[u].w);
    }
    for (int64_t i = (n4 << 2) + threadIdx.x; i < r.count; i += 256) r.dst[i] = scale * r.src[i];
  } else {
    for (int64_t i = threadIdx.x; i < r.count; i += 256) r.dst[i] = scale * r.src[i];
  }
}

// One warp per row; the comparison is on the quotients, ties go to the lower class.  Launch bound.
__global__ void __launch_bounds__(256) sample_classes_kernel(const float* __restrict__ prob, const float* __restrict__ q, int64_t rows,
                                                             int64_t classes, int64_t* __restrict__ out) {
  const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const float* p = prob + row * classes;
  const float* e = q + row * classes;
  auto clean = [](float v) { return (v > 0.f && v <= 3.402823466e38f) ? v : 0.f; };
  float best = -1.f, flat = -1.f, sum = 0.f;     // the race over the probabilities, and over a uniform row
  int64_t best_c = 0, flat_c = 0;
  for (int64_t c = lane; c < classes; c += 32) {
    const float v = clean(p[c]), r = v / e[c], u = 1.f / e[c];
    sum += v;
    if (r > best) { best = r; best_c = c; }
    if (u > flat) { flat = u; flat_c = c; }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float b = __shfl_xor_sync(0xffffffffu, best, o), f = __shfl_xor_sync(0xffffffffu, flat, o);
    const int64_t bc = __shfl_xor_sync(0xffffffffu, best_c, o), fc = __shfl_xor_sync(0xffffffffu, flat_c, o);
    if (b > best || (b == best && bc < best_c)) { best = b; best_c = bc; }
    if (f > flat || (f == flat && fc < flat_c)) { flat = f; flat_c = fc; }
  }
  if (lane == 0) out[row] = sum > 0.f ? best_c : flat_c;
}

// Bound: HBM (up to seven streams of 4 bytes per element), at small sizes the launch.  One CTA per record of
// at most 4096 elements, so that a network of two million parameters already gives every SM several CTAs
// (with 32768-element records it was 55 CTAs of one scalar load chain each: 65 us for 1.8 M parameters,
// 8 us now).  Where a record's arrays start on 16 bytes a thread moves float4s, the loads of two of them
// issued before the first store (source and destination come out of one record, so the compiler must
// assume that they alias); the scalars travel in kernel parameters, one set per distinct combination, so
// that a schedule that changes them does not rebuild the table.
struct TailSets { sso_tail_set s[SSO_TAIL_MAX_SETS]; };

__device__ __forceinline__ void tail_element(const sso_tail_set& q, bool has_m, bool has_e, float& p, float& g, float& m, float& e) {
  float v = fmaf(q.add, p, g);
  if (has_m) { v = fmaf(q.momentum, m, v); m = v; }
  if (has_e) { v = fmaf(q.ema, v, (1.f - q.ema) * e); e = v; }
  v *= q.scale;
  g = v;
  p = fmaf(-q.lr, v, p);
}

template <bool OWN>
__global__ void __launch_bounds__(256) optimizer_tail_kernel(const sso_tail_rec* __restrict__ recs,
                                                             const __grid_constant__ TailSets sets) {
  const sso_tail_rec r = recs[blockIdx.x];
  sso_tail_set q;
  if (OWN) { q.add = r.add; q.momentum = r.momentum; q.ema = r.ema; q.scale = r.scale; q.lr = r.lr; }
  else q = sets.s[r.set];
  const bool has_m = r.mbuf != nullptr, has_e = r.ebuf != nullptr, upd = q.lr != 0.f;
  const int64_t n = r.count;
  int64_t done = 0;
  if (((reinterpret_cast<uintptr_t>(r.p) | reinterpret_cast<uintptr_t>(r.g) | reinterpret_cast<uintptr_t>(r.mbuf) |
        reinterpret_cast<uintptr_t>(r.ebuf)) & 15) == 0) {
    const int64_t n4 = n >> 2;
    done = n4 << 2;
    auto at = [](float* base, int64_t i) { return reinterpret_cast<float4*>(base) + i; };
    for (int64_t i0 = threadIdx.x; i0 < n4; i0 += 2 * 256) {
      float4 p[2], g[2], m[2], e[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int64_t i = i0 + 256 * u;
        const bool in = i < n4;
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        p[u] = in ? *at(r.p, i) : z;
        g[u] = in ? *at(r.g, i) : z;
        m[u] = in && has_m ? *at(r.mbuf, i) : z;
        e[u] = in && has_e ? *at(r.ebuf, i) : z;
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int64_t i = i0 + 256 * u;
        if (i >= n4) break;
        tail_element(q, has_m, has_e, p[u].x, g[u].x, m[u].x, e[u].x);
        tail_element(q, has_m, has_e, p[u].y, g[u].y, m[u].y, e[u].y);
        tail_element(q, has_m, has_e, p[u].z, g[u].z, m[u].z, e[u].z);
        tail_element(q, has_m, has_e, p[u].w, g[u].w, m[u].w, e[u].w);
        *at(r.g, i) = g[u];
        if (upd) *at(r.p, i) = p[u];
        if (has_m) *at(r.mbuf, i) = m[u];
        if (has_e) *at(r.ebuf, i) = e[u];
      }
    }
  }
  for (int64_t i = done + threadIdx.x; i < n; i += 256) {
    float p = r.p[i], g = r.g[i], m = has_m ? r.mbuf[i] : 0.f, e = has_e ? r.ebuf[i] : 0.f;
    tail_element(q, has_m, has_e, p, g, m, e);
    r.g[i] = g;
    if (upd) r.p[i] = p;
    if (has_m) r.mbuf[i] = m;
    if (has_e) r.ebuf[i] = e;
  }
}

}  // namespace sso

using namespace sso;

// ---- 16-bit wire format of the exchange ---------------------------------------------------------
// A packed fp32 buffer is a sequence of arrays; a chunk record names a run of elements of one array.
// absmax: maxima[array] = max |x| (non-negative floats order like their bit patterns, so an integer
// atomicMax gives a deterministic result).  encode: out16 = cast(x * 65000 / sums[array]).
// decode: out32 = float(x16) * sums[array] / 65000.  `sums` holds the per-array maxima summed over
// the ranks, so that the sum of the scaled values of all ranks stays inside the fp16 range.
__global__ void __launch_bounds__(256) wire_absmax_kernel(const float* __restrict__ buf, const sso_wire_rec* __restrict__ recs,
                                                          float* __restrict__ maxima) {
  const sso_wire_rec r = recs[blockIdx.x];
  const float* src = buf + r.offset;
  float m = 0.f;
  for (int64_t i = threadIdx.x; i < r.count; i += 256) m = fmaxf(m, fabsf(src[i]));
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  __shared__ float sm[8];
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) m = fmaxf(m, sm[w]);
    if (!(m == m)) m = __int_as_float(0x7f800000);     // a NaN in the array: scale by infinity's reciprocal
    atomicMax(reinterpret_cast<int*>(maxima + r.array), __float_as_int(m));
  }
}

template <typename T>
__device__ __forceinline__ T wire_cast(float v);
template <>
__device__ __forceinline__ __nv_bfloat16 wire_cast<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <>
__device__ __forceinline__ __half wire_cast<__half>(float v) { return __float2half_rn(v); }

template <typename T>
__global__ void __launch_bounds__(256) wire_encode_kernel(const float* __restrict__ buf, const sso_wire_rec* __restrict__ recs,
                                                          const float* __restrict__ sums, T* __restrict__ out) {
  const sso_wire_rec r = recs[blockIdx.x];
  const float s = sums[r.array];
  const float scale = (s > 0.f && s < __int_as_float(0x7f800000)) ? 65000.f / s : 1.f;
  const float* src = buf + r.offset;
  T* dst = out + r.offset;
  for (int64_t i = threadIdx.x; i < r.count; i += 256) dst[i] = wire_cast<T>(src[i] * scale);
}

template <typename T>
__global__ void __launch_bounds__(256) wire_decode_kernel(const T* __restrict__ in, const sso_wire_rec* __restrict__ recs,
                                                          const float* __restrict__ sums, float* __restrict__ out) {
  const sso_wire_rec r = recs[blockIdx.x];
  const float s = sums[r.array];
  const float scale = (s > 0.f && s < __int_as_float(0x7f800000)) ? s / 65000.f : 1.f;
  const T* src = in + r.offset;
  float* dst = out + r.offset;
  for (int64_t i = threadIdx.x; i < r.count; i += 256) dst[i] = to_f32<T>(src[i]) * scale;
}

extern "C" {

int sso_optimizer_tail(const sso_tail_rec* recs_dev, int n_recs, void* stream) {
  SSO_CHECK_ARG(recs_dev != nullptr && n_recs >= 0, "optimizer_tail: bad argument");
  if (n_recs == 0) return 0;
  optimizer_tail_kernel<true><<<n_recs, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(recs_dev, TailSets{});
  SSO_LAUNCH_OK("optimizer_tail_kernel");
  return 0;
}

int sso_sample_classes(const float* prob, const float* q, int64_t rows, int64_t classes, int64_t* out, void* stream) {
  SSO_CHECK_ARG(prob && q && out && rows > 0 && classes > 0, "sample_classes: bad argument");
  sample_classes_kernel<<<(unsigned)ceil_div64(rows, 8), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(prob, q, rows, classes, out);
  SSO_LAUNCH_OK("sample_classes_kernel");
  return 0;
}

int sso_optimizer_tail_sets(const sso_tail_rec* recs_dev, int n_recs, const sso_tail_set* sets, int n_sets, void* stream) {
  SSO_CHECK_ARG(recs_dev != nullptr && n_recs >= 0, "optimizer_tail: bad argument");
  SSO_CHECK_ARG(sets != nullptr && n_sets > 0 && n_sets <= SSO_TAIL_MAX_SETS, "optimizer_tail: %d sets of scalars, at most %d", n_sets,
                SSO_TAIL_MAX_SETS);
  if (n_recs == 0) return 0;
  TailSets all{};
  for (int i = 0; i < n_sets; ++i) all.s[i] = sets[i];
  optimizer_tail_kernel<false><<<n_recs, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(recs_dev, all);
  SSO_LAUNCH_OK("optimizer_tail_kernel");
  return 0;
}

int sso_axpby(const float* src, float* dst, int64_t count, float a, float b, void* stream) {
  SSO_CHECK_ARG(src && dst && count >= 0, "axpby: bad argument");
  if (count == 0) return 0;
  axpby_kernel<<<grid_for(count, 16), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(src, dst, count, a, b);
  SSO_LAUNCH_OK("axpby_kernel");
  return 0;
}

int sso_ema_update(const float* data, float* ema, int64_t count, float beta, int first, void* stream) {
  // first (or beta == 1): ema <- data; else ema <- beta*data + (1-beta)*ema
  if (first || beta == 1.f) return sso_axpby(data, ema, count, 1.f, 0.f, stream);
  return sso_axpby(data, ema, count, beta, 1.f - beta, stream);
}

int sso_bn_plane_splits(int dtype, int64_t n, int64_t c, int64_t hw, int64_t stride_c) {
  if (stride_c != 1) return 1;
  return bn_vec_splits(n, c, hw, dtype == SSO_F32 ? 4 : 8);
}

int sso_bn_plane_sums(const void* y, const void* g, int dtype, int64_t n, int64_t c, int64_t hw,
                      int64_t syn, int64_t syc, int64_t syp, int64_t sgn, int64_t sgc, int64_t sgp,
                      const float* scale, const float* shift, float* sx, float* sg, int splits, void* stream) {
  SSO_CHECK_ARG((y && sx) || (g && sg), "bn_plane_sums: nothing to do");
  SSO_CHECK_ARG(!y || sx, "bn_plane_sums: y without sx");
  SSO_CHECK_ARG(!g || sg, "bn_plane_sums: g without sg");
  SSO_CHECK_ARG(n > 0 && c > 0 && hw > 0 && n * c < (int64_t)1 << 26 && splits >= 1, "bn_plane_sums: bad shape");
  if (!y) { syn = sgn; syc = sgc; syp = sgp; }
  if (!g) { sgn = syn; sgc = syc; sgp = syp; }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  switch (dtype) {
    case SSO_F32:
      return bn_sums_typed<float>(y, g, n, c, hw, syn, syc, syp, sgn, sgc, sgp, scale, shift, sx, sg, splits, st);
    case SSO_BF16:
      return bn_sums_typed<__nv_bfloat16>(y, g, n, c, hw, syn, syc, syp, sgn, sgc, sgp, scale, shift, sx, sg, splits, st);
    case SSO_F16:
      return bn_sums_typed<__half>(y, g, n, c, hw, syn, syc, syp, sgn, sgc, sgp, scale, shift, sx, sg, splits, st);
  }
  return fail(-1, "bn_plane_sums: unknown dtype %d", dtype);
}

int sso_bn_diag_finish(const float* sx, const float* sg, const float* sample_weight, int64_t n, int64_t c,
                       int splits_x, int splits_g, float alpha, float beta, float* w_out, float* b_out,
                       void* stream) {
  SSO_CHECK_ARG(sx && sg && w_out && n > 0 && c > 0 && splits_x >= 1 && splits_g >= 1, "bn_diag_finish: bad argument");
  bn_finish_kernel<<<(unsigned)ceil_div64(c, 8), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      sx, sg, sample_weight, (int)n, (int)c, splits_x, splits_g, alpha, beta, w_out, b_out);
  SSO_LAUNCH_OK("bn_finish_kernel");
  return 0;
}

int sso_bn_batch(int n, const sso_bn_desc* descs, void* stream) {
  SSO_CHECK_ARG(n >= 0 && (n == 0 || descs != nullptr), "bn_batch: bad argument");
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  static thread_local BnBatch b;
  int sums = 0, blocks = 0;
  b.n = 0;
  auto flush = [&]() -> int {
    if (b.n == 0) return 0;
    bn_batch_sums_kernel<<<sums, 256, 0, st>>>(b);
    SSO_LAUNCH_OK("bn_batch_sums_kernel");
    bn_batch_finish_kernel<<<blocks, 256, 0, st>>>(b);
    SSO_LAUNCH_OK("bn_batch_finish_kernel");
    b.n = sums = blocks = 0;
    return 0;
  };
  for (int i = 0; i < n; ++i) {
    const sso_bn_desc& d = descs[i];
    SSO_CHECK_ARG(d.g && d.sg && d.sx && d.w_out, "bn_batch: null pointer");
    SSO_CHECK_ARG(d.n > 0 && d.c > 0 && d.hw > 0 && d.n * d.c < (int64_t)1 << 26 && d.splits_g >= 1 && d.splits_x >= 1,
                  "bn_batch: bad shape");
    const int size = d.dtype == SSO_F32 ? 4 : 2, lp = bn_vec_lanes(d.c, 16 / size);
    if (lp > 0 && d.hw > 1 && d.sc == 1 && (reinterpret_cast<uintptr_t>(d.g) & 15) == 0 && d.sn * size % 16 == 0 && d.sp * size % 16 == 0) {
      b.rec[b.n] = {d, lp, sums, blocks};
      ++b.n;
      sums += (int)(d.n * d.splits_g);
      blocks += (int)ceil_div64(d.c, 8);
      if (b.n == BN_BATCH) {
        const int rc = flush();
        if (rc) return rc;
      }
      continue;
    }
    int rc = sso_bn_plane_sums(nullptr, d.g, d.dtype, d.n, d.c, d.hw, 0, 0, 0, d.sn, d.sc, d.sp, nullptr, nullptr, nullptr, d.sg, d.splits_g, stream);
    if (!rc) rc = sso_bn_diag_finish(d.sx, d.sg, d.sample_weight, d.n, d.c, d.splits_x, d.splits_g, d.alpha, d.beta, d.w_out, d.b_out, stream);
    if (rc) return rc;
  }
  return flush();
}

int sso_diag_inv_precondition(const float* ema, float* inv, float* grad, int64_t count, float damping,
                              int use_sqrt, int update_inv, void* stream) {
  SSO_CHECK_ARG(inv && count >= 0 && (ema || !update_inv), "diag_inv_precondition: bad argument");
  if (count == 0) return 0;
  diag_inv_precond_kernel<<<grid_for(count, 4), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      ema, inv, grad, count, damping, use_sqrt, update_inv);
  SSO_LAUNCH_OK("diag_inv_precond_kernel");
  return 0;
}

int sso_tri_pack(const sso_tri_rec* recs_dev, int n_recs, float scale, void* stream) {
  SSO_CHECK_ARG(recs_dev && n_recs >= 0, "tri_pack: bad argument");
  if (n_recs == 0) return 0;
  tri_pack_kernel<<<n_recs, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(recs_dev, scale);
  SSO_LAUNCH_OK("tri_pack_kernel");
  return 0;
}

int sso_tri_unpack(const sso_tri_rec* recs_dev, int n_recs, float scale, int symmetric, void* stream) {
  SSO_CHECK_ARG(recs_dev && n_recs >= 0, "tri_unpack: bad argument");
  if (n_recs == 0) return 0;
  tri_unpack_kernel<<<dim3((unsigned)n_recs, 8), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(recs_dev, scale, symmetric);
  SSO_LAUNCH_OK("tri_unpack_kernel");
  return 0;
}

int sso_copy_segments(const sso_seg_rec* recs_dev, int n_recs, float scale, void* stream) {
  SSO_CHECK_ARG(recs_dev && n_recs >= 0, "copy_segments: bad argument");
  if (n_recs == 0) return 0;
  copy_segments_kernel<<<n_recs, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(recs_dev, scale);
  SSO_LAUNCH_OK("copy_segments_kernel");
  return 0;
}

int sso_wire_absmax(const float* buf, const sso_wire_rec* recs_dev, int n_recs, float* maxima, void* stream) {
  SSO_CHECK_ARG(buf && recs_dev && maxima && n_recs >= 0, "wire_absmax: bad argument");
  if (n_recs == 0) return 0;
  wire_absmax_kernel<<<n_recs, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(buf, recs_dev, maxima);
  SSO_LAUNCH_OK("wire_absmax_kernel");
  return 0;
}

int sso_wire_encode(const float* buf, const sso_wire_rec* recs_dev, int n_recs, const float* sums, void* out16,
                    int dtype, void* stream) {
  SSO_CHECK_ARG(buf && recs_dev && sums && out16 && n_recs >= 0, "wire_encode: bad argument");
  SSO_CHECK_ARG(dtype == SSO_BF16 || dtype == SSO_F16, "wire_encode: the wire type must be bf16 or fp16");
  if (n_recs == 0) return 0;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (dtype == SSO_BF16)
    wire_encode_kernel<__nv_bfloat16><<<n_recs, 256, 0, st>>>(buf, recs_dev, sums, static_cast<__nv_bfloat16*>(out16));
  else
    wire_encode_kernel<__half><<<n_recs, 256, 0, st>>>(buf, recs_dev, sums, static_cast<__half*>(out16));
  SSO_LAUNCH_OK("wire_encode_kernel");
  return 0;
}

int sso_wire_decode(const void* in16, const sso_wire_rec* recs_dev, int n_recs, const float* sums, float* out32,
                    int dtype, void* stream) {
  SSO_CHECK_ARG(in16 && recs_dev && sums && out32 && n_recs >= 0, "wire_decode: bad argument");
  SSO_CHECK_ARG(dtype == SSO_BF16 || dtype == SSO_F16, "wire_decode: the wire type must be bf16 or fp16");
  if (n_recs == 0) return 0;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (dtype == SSO_BF16)
    wire_decode_kernel<__nv_bfloat16><<<n_recs, 256, 0, st>>>(static_cast<const __nv_bfloat16*>(in16), recs_dev, sums, out32);
  else
    wire_decode_kernel<__half><<<n_recs, 256, 0, st>>>(static_cast<const __half*>(in16), recs_dev, sums, out32);
  SSO_LAUNCH_OK("wire_decode_kernel");
  return 0;
}

}  // extern "C"
