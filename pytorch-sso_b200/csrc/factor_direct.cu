// Small factors in one launch: out <- alpha * U^T U + beta * out for few rows (a Linear layer's batch, a small output
// plane), exact fp32 FFMA, no scratch, no second kernel.
//
// One CTA owns a lower-triangle TxT tile (64, or 32 where that leaves most SMs without one) and walks all rows, 32 per
// stage; the loads of the next stage are in registers while this one is multiplied.  G groups of (T/4)^2 threads, 4x4
// elements each, take every G-th stage and their sums are added in order, so that an SM with one CTA has enough
// warps to hide the latency of its shared-memory loads.  Bound: FFMA (about 0.6 of its rate), a launch, a round trip.  The tensor-core path has three launches (split, multiply,
// finish) and fills a pipeline first: 24 us for 128 x 1000 where this takes 10.5, 14.5 for 16 x 20 where this takes 3.5;
// the line between the two is drawn on this kernel's own estimate (factor_direct_supported).
#include <algorithm>

#include "common.cuh"
#include "factor_params.cuh"

namespace sso {
namespace direct {

template <typename E>
__device__ __forceinline__ float4 load4(const E* p);
template <>
__device__ __forceinline__ float4 load4<float>(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
template <>
__device__ __forceinline__ float4 load4<__nv_bfloat16>(const __nv_bfloat16* p) {
  const uint2 v = __ldg(reinterpret_cast<const uint2*>(p));
  return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xFFFF0000u), __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xFFFF0000u));
}
template <>
__device__ __forceinline__ float4 load4<__half>(const __half* p) {
  const uint2 v = __ldg(reinterpret_cast<const uint2*>(p));
  const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&v.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
  return make_float4(a.x, a.y, b.x, b.y);
}

// MODE 0: columns contiguous, 4-element aligned; 1: columns contiguous; 2: rows contiguous (or any strides)
template <typename E, int MODE, int T, int G>
__global__ void __launch_bounds__((T / 4) * (T / 4) * G) factor_direct_kernel(const FactorParams p, int64_t plane_stride) {
  constexpr int NT = (T / 4) * (T / 4), NV = KT / (T / 4), PER = 2 * KT * T;      // threads, float4s per thread, floats of a group
  extern __shared__ __align__(16) float smem[];      // per group: 32 rows of the two column ranges, later its TxT sums
  const int tid = threadIdx.x % NT, group = threadIdx.x / NT;
  float* As = smem + group * PER;
  float* Bs = As + KT * T;
  int bi, bj;
  tri_decode(blockIdx.x, bi, bj);
  const bool diag = bi == bj;
  const E* x = reinterpret_cast<const E*>(p.x);
  const int hw = p.ho * p.wo, rows = (int)p.rows;
  auto row_at = [&](int r) { return x + ((int64_t)(r / hw) * p.sn + (int64_t)(r % hw) * plane_stride); };
  // MODE 0, 1: four columns of rows tid / (T/4), + T/4, ..; MODE 2: one row, every (NT/32)-th column
  float4 ra[NV], rb[NV];
  auto load = [&](int c0, int r0, float4 (&v)[NV]) {
    if (MODE == 2) {
      const int r = r0 + (tid & 31);
      const E* row = row_at(min(r, rows - 1));
      auto at = [&](int i) {
        const int c = c0 + (tid >> 5) + (NT / 32) * i;
        return (r < rows && c < p.dcols) ? to_f32<E>(__ldg(row + c * p.sc)) : (r < rows && c == p.dcols && c < p.d ? 1.f : 0.f);
      };
#pragma unroll
      for (int j = 0; j < NV; ++j) v[j] = make_float4(at(4 * j), at(4 * j + 1), at(4 * j + 2), at(4 * j + 3));
      return;
    }
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int r = r0 + tid / (T / 4) + (T / 4) * j, c = c0 + (tid % (T / 4)) * 4;
      v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r < rows) {
        const E* row = row_at(r);
        if (MODE == 0 && c + 3 < p.dcols) {
          v[j] = load4<E>(row + c);
        } else {
          auto at = [&](int cc) { return cc < p.dcols ? to_f32<E>(__ldg(row + cc)) : (cc == p.dcols && cc < p.d ? 1.f : 0.f); };
          v[j] = make_float4(at(c), at(c + 1), at(c + 2), at(c + 3));
        }
      }
    }
  };
  auto store = [&](float* S, const float4 (&v)[NV]) {
    if (MODE == 2) {
      const int k = tid & 31;
      auto put = [&](int i, float x) { S[k * T + swz(k, (tid >> 5) + (NT / 32) * i)] = x; };
#pragma unroll
      for (int j = 0; j < NV; ++j) { put(4 * j, v[j].x); put(4 * j + 1, v[j].y); put(4 * j + 2, v[j].z); put(4 * j + 3, v[j].w); }
      return;
    }
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int k = tid / (T / 4) + (T / 4) * j;
      *reinterpret_cast<float4*>(S + k * T + swz(k, (tid % (T / 4)) * 4)) = v[j];
    }
  };
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  const int ty = tid / (T / 4), tx = tid % (T / 4);
  const int stages = ceil_div(rows, KT);
  if (group < stages) {
    load(bi * T, group * KT, ra);
    if (!diag) load(bj * T, group * KT, rb);
  }
  for (int s0 = 0; s0 < stages; s0 += G) {
    const int s = s0 + group;
    if (s < stages) {
      store(As, ra);
      if (!diag) store(Bs, rb);
    }
    __syncthreads();
    if (s + G < stages) {
      load(bi * T, (s + G) * KT, ra);
      if (!diag) load(bj * T, (s + G) * KT, rb);
    }
    if (s < stages) {
      const float* B = diag ? As : Bs;
#pragma unroll 8
      for (int k = 0; k < KT; ++k) {
        const float4 va = *reinterpret_cast<const float4*>(As + k * T + swz(k, ty * 4)), vb = *reinterpret_cast<const float4*>(B + k * T + swz(k, tx * 4));
        const float a[4] = {va.x, va.y, va.z, va.w}, b[4] = {vb.x, vb.y, vb.z, vb.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
      }
    }
    __syncthreads();
  }
  // the groups' tiles go to shared memory, columns rotated by the row so that rows and columns of it are read without
  // bank conflicts; the tile and its mirror are then written along rows of the output
  auto at = [](int r, int c) { return r * T + (c ^ (r & 31)); };
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) As[at(ty * 4 + i, tx * 4 + j)] = acc[i][j];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // pass 0: the tile, pass 1: its mirror; the lower triangle serves both, bit for bit.  With beta the old values of a
  // warp's rows are fetched before anything is stored (a load would wait behind the stores to the same array).
  constexpr int RW = T / (NT * G / 32);      // rows per warp
  for (int pass = 0; pass < (diag ? 1 : 2); ++pass) {
    const int row0 = (pass == 0 ? bi : bj) * T, col0 = (pass == 0 ? bj : bi) * T;
    float old[RW][T / 32];
    if (p.beta != 0.f) {
#pragma unroll
      for (int i = 0; i < RW; ++i)
#pragma unroll
        for (int u = 0; u < T / 32; ++u) {
          const int gr = row0 + warp * RW + i, gc = col0 + lane + 32 * u;
          old[i][u] = (gr < p.d && gc < p.d) ? p.out[(int64_t)gr * p.ldo + gc] : 0.f;
        }
    }
#pragma unroll
    for (int i = 0; i < RW; ++i)
#pragma unroll
      for (int u = 0; u < T / 32; ++u) {
        const int r = warp * RW + i, c = lane + 32 * u, gr = row0 + r, gc = col0 + c;
        if (gr >= p.d || gc >= p.d) continue;
        const bool flip = pass == 1 || (diag && c > r);
        const int e = flip ? at(c, r) : at(r, c);
        float v = smem[e];
#pragma unroll
        for (int g = 1; g < G; ++g) v += smem[g * PER + e];
        v *= p.alpha;
        p.out[(int64_t)gr * p.ldo + gc] = (p.beta == 0.f) ? v : fmaf(p.beta, old[i][u], v);
      }
  }
}

static int tiles_of(int d, int t) {
  const int nb = ceil_div(d, t);
  return nb * (nb + 1) / 2;
}

template <typename E, int MODE, int T, int G>
static int launch_one(const FactorParams& p, int64_t plane_stride, cudaStream_t st) {
  constexpr int BYTES = G * 2 * KT * T * (int)sizeof(float);
  SSO_ENSURE_SMEM((factor_direct_kernel<E, MODE, T, G>), BYTES);
  factor_direct_kernel<E, MODE, T, G><<<tiles_of(p.d, T), (T / 4) * (T / 4) * G, BYTES, st>>>(p, plane_stride);
  SSO_LAUNCH_OK("factor_direct_kernel");
  return 0;
}

template <typename E, int MODE>
static int launch_mode(const FactorParams& p, int64_t plane_stride, cudaStream_t st) {
  if (tiles_of(p.d, 64) <= 74) return p.rows > 4 * KT ? launch_one<E, MODE, 32, 8>(p, plane_stride, st) : launch_one<E, MODE, 32, 4>(p, plane_stride, st);
  return p.rows > 2 * KT ? launch_one<E, MODE, 64, 4>(p, plane_stride, st) : launch_one<E, MODE, 64, 2>(p, plane_stride, st);
}

template <typename E>
static int launch(const FactorParams& p, int64_t plane_stride, cudaStream_t st) {
  const size_t esz = sizeof(E);
  auto even = [&](int64_t s) { return s * esz % (4 * esz) == 0; };
  if (p.sc == 1 || p.c == 1) {
    const bool vec = reinterpret_cast<uintptr_t>(p.x) % (4 * esz) == 0 && even(p.sn) && even(plane_stride);
    return vec ? launch_mode<E, 0>(p, plane_stride, st) : launch_mode<E, 1>(p, plane_stride, st);
  }
  return launch_mode<E, 2>(p, plane_stride, st);
}

}  // namespace direct

static int64_t plane_stride_of(const FactorParams& p) { return p.w > 1 ? p.sw : p.h > 1 ? p.sh : 0; }

// 1x1 windows over evenly spaced pixels, unweighted, whose estimated time (multiply-adds of the fullest SM at 0.6 of the
// FFMA rate) stays below what the launches of the tensor-core path take by themselves.
bool factor_direct_supported(const FactorParams& p, int dtype) {
  if (p.kh != 1 || p.kw != 1 || p.pad_h || p.pad_w || p.stride_h != 1 || p.stride_w != 1 || p.weight) return false;
  if (p.w > 1 && p.h > 1 && p.sh != p.w * p.sw) return false;
  const int t64 = direct::tiles_of(p.d, 64);
  const double tiles = t64 <= 74 ? std::max(1.0, direct::tiles_of(p.d, 32) / 148.0) : 4.0 * std::max(1.0, t64 / 148.0);      // of 32x32, per SM
  const double us = tiles * (double)p.rows * (1024.0 / 128 / 0.6) / 1850.0;
  return us <= (dtype == SSO_F32 ? 12.0 : 5.0);
}

int factor_direct_launch(const FactorParams& p, int dtype, cudaStream_t st) {
  switch (dtype) {
    case SSO_F32: return direct::launch<float>(p, plane_stride_of(p), st);
    case SSO_BF16: return direct::launch<__nv_bfloat16>(p, plane_stride_of(p), st);
    case SSO_F16: return direct::launch<__half>(p, plane_stride_of(p), st);
  }
  return fail(-1, "unknown dtype %d", dtype);
}

}  // namespace sso
