// Kronecker-factor construction from fp32 inputs on the tensor cores (three-way bf16 split, fused im2col gather).
//
//   partial[tile][split] = sum over this split's rows r of  w_r u_r[I] u_r[J]^T
//
// x = hi + mid + lo in bf16, exact to fp32's 24 bits; the six products down to 2^-16 (lo*hi, hi*lo, mid*mid, mid*hi,
// hi*mid, hi*hi; what is dropped is below 2^-24) go into one TMEM accumulator that is drained into fp32 registers
// every FLUSH stages (the tensor core's own running sum truncates).  Two kernels:
//
// split_kernel writes the three parts of the input once, as pixel rows [part][pixel][C8] of 16-bit values with the
// channels padded to a multiple of eight (the ones column of a 1x1 window without padding is one of them).  Every activation is converted
// once instead of once per kernel position and tile, and whatever layout the input has (NCHW, odd channel counts,
// unaligned rows) the gather sees 16-byte chunks of channels.  Bound: memory, 4 bytes in and 6 out per element.
//
// factor_f32_kernel brings im2col rows of the parts straight into the operand layout (MN-major SWIZZLE_128B: 64 columns =
// 128 bytes of one row, zero-filled outside the image), in one of three shapes:
//   PAIR, BOX  a cluster of two CTAs computes a 256x256 block with tcgen05.mma.cta_group::2; a stage is a box of 32 whole
//              pixels, fetched by one thread with TMA, the three parts of 64 columns in one piece;
//   PAIR       the same where no box covers the output exactly: eight warps gather with cp.async;
//   single     one CTA, one 128x128 tile (narrow factors, where a pair would compute padding), gathered.
// Bound: with boxes the MMAs, twelve per stage of 32 rows and pair (1536 cycles per SM, 0.98 us as measured without any
// loads; 1.1 with them); gathered, the copies: 48 KB of parts per stage come in at 1.4 us whatever the number of stages
// in flight, MMAs or not (5 TB/s over the chip: what the load/store path of an SM keeps outstanding).  us, 3xTF32 on
// 128x128 tiles / gathered / boxes / with narrow last block rows: 5x5 over 64 channels, d = 1601 from 65536 rows 1810 /
// 1127 / 896 / 840; 3x3 over 64, d = 577 from 131072 rows 495 gathered, 391 / 363; d = 4608 from 8192 rows 1710 / 1016 / 876.  Measured alternatives:
// splitting in the gather warps is bound by their instructions (650 per warp and stage, 2.3 us per stage, in bf16 as in
// 3xTF32), and 32-bit MN-major operands are read at half the rate.
// The input is processed in runs of whole images whose parts fit the scratch; each run adds to the partial tiles of
// the one before.
// Partial tiles, tickets and the finishing kernels are those of the other factor kernels.
#include <cuda.h>

#include <algorithm>
#include <numeric>

#include "common.cuh"
#include "factor_finish.cuh"
#include "factor_params.cuh"
#include "tc_pair.cuh"

namespace sso {

int factor_tc_run_reduce(const FactorParams& p, int tiles, cudaStream_t st);
decltype(&cuTensorMapEncodeTiled) tensor_map_encoder();      // factor_tma.cu; null if the driver has none

namespace f32 {

using namespace tc;

constexpr int TILE = 128, KS = 32, STAGES = 4, LAG = 2, FLUSH = 2;
// five warpgroups: 0-1 accumulate (128 sums per thread of a pair), 2 issues the MMAs (one thread), 3-4 gather; they
// share the block's 640 x 96 registers as 168 + 168 + 24 + 56 + 56 per thread
constexpr int EPI_WARPS = 8, MMA_WARP = 8, LOAD_WARP0 = 12, LOAD_WARPS = 8;
constexpr int THREADS = 640;
constexpr uint32_t BLK = KS * 128u;              // 64 columns of one stage, one part
constexpr uint32_t OPB = 2 * BLK;                // 128 columns
constexpr uint32_t SIDE = 3 * OPB;               // hi mid lo
constexpr uint32_t SLOT_BYTES = 2 * SIDE;        // both sides
constexpr size_t SMEM = STAGES * SLOT_BYTES + 1024;

struct Parts {
  const __nv_bfloat16* a;      // hi part of the (weighted) row side, the other two `stride` elements apart
  const __nv_bfloat16* b;      // of the column side; equal to a without weights
  int64_t stride;
  int c8;                      // channels per pixel, a multiple of eight
};

// Stages as boxes of whole pixels (32 = bw * bh * bn), fetched by TMA: a view {c8, width, h, n, part} of the parts.
struct alignas(64) Boxes {
  CUtensorMap map;
  int bw, bh, bn, across, down;      // a box; boxes per image in either direction
  int narrow;                        // N of the last block row's MMAs (narrow_columns), 0: an ordinary row
};

// First kernel of a factor: let the next one set itself up meanwhile (it waits for this one's end before it touches
// memory), clear the status word and the tickets that it will use.
__device__ __forceinline__ void begin_factor(const FactorParams& p, int header_words) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (blockIdx.x == 0 && blockIdx.y == 0)
    for (int i = threadIdx.x; i < header_words; i += blockDim.x) p.status[i] = 0;
}

// A CTA turns 32 pixels x 64 channels: read with the lanes along whichever of the two is contiguous, staged in shared
// memory, written as 16-byte chunks of eight channels.
__global__ void __launch_bounds__(256) split_kernel(const FactorParams p, uint32_t pixels, int ones_at, int header_words, Parts out_a, Parts out_b) {
  __shared__ __align__(16) float t[32][68];
  begin_factor(p, header_words);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t px0 = blockIdx.x * 32u;
  const int c0 = blockIdx.y * 64;
  const float* x = reinterpret_cast<const float*>(p.x);
  const int hw = p.h * p.w;        // pixels of an image
  auto offset = [&](uint32_t px) {
    const uint32_t n = px / (uint32_t)hw;
    const int rem = (int)(px - n * hw), y = rem / p.w;
    return n * p.sn + y * p.sh + (rem - y * p.w) * p.sw;
  };
  if (p.sc <= (p.w > 1 ? p.sw : p.h > 1 ? p.sh : p.sn)) {      // lanes along the channels
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t px = px0 + warp + 8 * i;
      if (px >= pixels) break;
      const float* row = x + offset(px);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int c = c0 + lane + 32 * u;
        t[warp + 8 * i][lane + 32 * u] = c < p.c ? __ldg(row + c * p.sc) : (c == ones_at ? 1.f : 0.f);
      }
    }
  } else {                         // lanes along the pixels
    const uint32_t px = px0 + lane;
    const float* col = x + (px < pixels ? offset(px) : 0);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int c = c0 + warp + 8 * i;
      t[lane][warp + 8 * i] = c < p.c ? (px < pixels ? __ldg(col + c * p.sc) : 0.f) : (c == ones_at ? 1.f : 0.f);
    }
  }
  __syncthreads();
  const int r = tid >> 3, o = (tid & 7) * 8;
  const uint32_t px = px0 + r;
  if (px >= pixels || c0 + o >= out_a.c8) return;
  const float w = p.weight ? p.weight[px / hw] : 1.f;
  for (int side = 0; side < (p.weight ? 2 : 1); ++side) {
    const float f = side == 0 ? w : 1.f;
    uint32_t hi[4], mid[4], lo[4];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float4 v = *reinterpret_cast<const float4*>(&t[r][o + 4 * i]);
      split2(f * v.x, f * v.y, hi[2 * i], mid[2 * i], lo[2 * i]);
      split2(f * v.z, f * v.w, hi[2 * i + 1], mid[2 * i + 1], lo[2 * i + 1]);
    }
    __nv_bfloat16* d = const_cast<__nv_bfloat16*>(side == 0 ? out_a.a : out_b.b) + (int64_t)px * out_a.c8 + c0 + o;
    *reinterpret_cast<uint4*>(d) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(d + out_a.stride) = make_uint4(mid[0], mid[1], mid[2], mid[3]);
    *reinterpret_cast<uint4*>(d + 2 * out_a.stride) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
}

// With few channels the kernel's columns are folded into them: channel kx*c + ch of pixel (y, ox) is
// x[ch][y][ox*stride + kx*dil - pad], so that three channels under a 7x7 window are 7 x 24 columns and not 49 x 8.  A thread takes
// eight of a pixel's folded channels from global memory to global memory; neighbouring pixels read the same lines
// (staged in shared memory, 32 pixels x 64 channels per CTA, the stem of ResNet-50 left most threads without a channel).
__global__ void __launch_bounds__(256) split_folded_kernel(const FactorParams p, uint32_t pixels, int width, int fold, int header_words, Parts out_a, Parts out_b) {
  begin_factor(p, header_words);
  const int oct = out_a.c8 / 8, hw = p.h * width;
  const uint32_t i = blockIdx.x * 256u + threadIdx.x, px = i / (uint32_t)oct;
  if (px >= pixels) return;
  const int cf0 = (int)(i - px * oct) * 8;
  const uint32_t n = px / (uint32_t)hw;
  const int rem = (int)(px - n * hw), y = rem / width, x0 = (rem - y * width) * p.stride_w - p.pad_w;
  const float* src = reinterpret_cast<const float*>(p.x) + n * p.sn + y * p.sh;
  int kx = cf0 / p.c, ch = cf0 - kx * p.c;
  float v[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int ix = x0 + kx * p.dil_w;
    v[k] = kx < fold && (unsigned)ix < (unsigned)p.w ? __ldg(src + ix * p.sw + ch * p.sc) : 0.f;
    if (++ch == p.c) { ch = 0; ++kx; }
  }
  const float w = p.weight ? p.weight[n] : 1.f;
  for (int side = 0; side < (p.weight ? 2 : 1); ++side) {
    const float f = side == 0 ? w : 1.f;
    uint32_t hi[4], mid[4], lo[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) split2(f * v[2 * k], f * v[2 * k + 1], hi[k], mid[k], lo[k]);
    __nv_bfloat16* d = const_cast<__nv_bfloat16*>(side == 0 ? out_a.a : out_b.b) + (int64_t)px * out_a.c8 + cf0;
    *reinterpret_cast<uint4*>(d) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(d + out_a.stride) = make_uint4(mid[0], mid[1], mid[2], mid[3]);
    *reinterpret_cast<uint4*>(d + 2 * out_a.stride) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
}

// The same for NCHW planes whose pixels come in aligned runs of four: a CTA turns 64 pixels x 64 channels, four 16-byte loads
// per thread in flight.  Quad q of a channel's pixels lies at place q ^ (channel / 8), so that neither the 16-byte stores
// nor the loads of eight channels of a pixel (lanes: octets, then four pixels) meet a bank conflict.
__global__ void __launch_bounds__(256) split_planes_kernel(const FactorParams p, uint32_t pixels, int ones_at, int header_words, Parts out_a, Parts out_b) {
  __shared__ __align__(16) float t[64 * 64];
  begin_factor(p, header_words);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t px0 = blockIdx.x * 64u, hw = (uint32_t)(p.h * p.w);
  const int c0 = blockIdx.y * 64;
  {
    const int q = tid & 15, c = tid >> 4;
    const uint32_t px = px0 + 4 * q, n = px / hw;
    const float* src = reinterpret_cast<const float*>(p.x) + n * p.sn + (px - n * hw) + (c0 + c) * p.sc;
    float4 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int ch = c0 + c + 16 * i;
      const float fill = ch == ones_at ? 1.f : 0.f;
      v[i] = make_float4(fill, fill, fill, fill);
      if (px < pixels && ch < p.c) v[i] = __ldg(reinterpret_cast<const float4*>(src + 16 * i * p.sc));
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int ch = c + 16 * i;
      *reinterpret_cast<float4*>(&t[ch * 64 + ((q ^ (ch >> 3)) << 2)]) = v[i];
    }
  }
  __syncthreads();
  const int o = lane & 7;
  if (c0 + 8 * o >= out_a.c8) return;
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const int r = it * 32 + warp * 4 + (lane >> 3);
    const uint32_t px = px0 + r;
    if (px >= pixels) return;
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = t[(8 * o + i) * 64 + (((r >> 2) ^ o) << 2) + (r & 3)];
    const float w = p.weight ? p.weight[px / hw] : 1.f;
    for (int side = 0; side < (p.weight ? 2 : 1); ++side) {
      const float f = side == 0 ? w : 1.f;
      uint32_t hi[4], mid[4], lo[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) split2(f * v[2 * i], f * v[2 * i + 1], hi[i], mid[i], lo[i]);
      __nv_bfloat16* d = const_cast<__nv_bfloat16*>(side == 0 ? out_a.a : out_b.b) + (int64_t)px * out_a.c8 + c0 + 8 * o;
      *reinterpret_cast<uint4*>(d) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
      *reinterpret_cast<uint4*>(d + out_a.stride) = make_uint4(mid[0], mid[1], mid[2], mid[3]);
      *reinterpret_cast<uint4*>(d + 2 * out_a.stride) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
  }
}

// The same where the channels are contiguous, 16-byte aligned and a multiple of four: a thread takes eight channels of
// a pixel straight from global memory to global memory.
__global__ void __launch_bounds__(256) split_direct_kernel(const FactorParams p, uint32_t pixels, int ones_at, int header_words, Parts out_a, Parts out_b) {
  begin_factor(p, header_words);
  const int oct = out_a.c8 / 8, hw = p.h * p.w;
  const uint32_t i = blockIdx.x * 256u + threadIdx.x, px = i / (uint32_t)oct;
  if (px >= pixels) return;
  const int c = (int)(i - px * oct) * 8;
  const uint32_t n = px / (uint32_t)hw;
  const int rem = (int)(px - n * hw), y = rem / p.w;
  const float* src = reinterpret_cast<const float*>(p.x) + (n * p.sn + y * p.sh + (rem - y * p.w) * p.sw + c);
  const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 u = c < p.c ? __ldg(reinterpret_cast<const float4*>(src)) : z, v = c + 4 < p.c ? __ldg(reinterpret_cast<const float4*>(src) + 1) : z;
  if (ones_at == c) u.x = 1.f;      // a multiple of four, so the first of either half
  if (ones_at == c + 4) v.x = 1.f;
  const float w = p.weight ? p.weight[n] : 1.f;
  for (int side = 0; side < (p.weight ? 2 : 1); ++side) {
    const float f = side == 0 ? w : 1.f;
    uint32_t hi[4], mid[4], lo[4];
    split2(f * u.x, f * u.y, hi[0], mid[0], lo[0]);
    split2(f * u.z, f * u.w, hi[1], mid[1], lo[1]);
    split2(f * v.x, f * v.y, hi[2], mid[2], lo[2]);
    split2(f * v.z, f * v.w, hi[3], mid[3], lo[3]);
    __nv_bfloat16* d = const_cast<__nv_bfloat16*>(side == 0 ? out_a.a : out_b.b) + (int64_t)px * out_a.c8 + c;
    *reinterpret_cast<uint4*>(d) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(d + out_a.stride) = make_uint4(mid[0], mid[1], mid[2], mid[3]);
    *reinterpret_cast<uint4*>(d + 2 * out_a.stride) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
}

// The loads of one thread: 16-byte chunk l8 of the four 64-column blocks (A0 A1 B0 B1) of one row of every stage; a warp
// instruction covers four rows of one block and part, i.e. four whole lines.
struct Gather {
  int koff[4];             // element offset of this thread's chunk in block b
  int kpos[4];             // kernel position dh | dw << 16; -1: the ones column; -2: nothing
  int left;                // rows of the split that remain from this one on (<= 0: past the end)
  int n, y, x;             // image and output pixel

  __device__ __forceinline__ void init(const FactorParams& p, int col_a, int col_b, int64_t r_begin, int rows, int k, int l8) {
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int j0 = (b < 2 ? col_a : col_b) + (b & 1) * 64 + l8 * 8;
      koff[b] = 0;
      kpos[b] = (j0 == p.dcols && j0 < p.d) ? -1 : -2;
      if (j0 < p.dcols) {
        const int pos = j0 / p.c, c0 = j0 - pos * p.c;
        const int ky = pos / p.kw, kx = pos - ky * p.kw;
        const int dh = ky * p.dil_h, dw = kx * p.dil_w;
        koff[b] = (int)(dh * p.sh + dw * p.sw) + c0;
        kpos[b] = dh | (dw << 16);
      }
    }
    const int hw = p.ho * p.wo;
    left = rows - k;
    const int64_t r = r_begin + k;
    n = (int)(r / hw);
    const int rem = (int)(r - (int64_t)n * hw);
    y = rem / p.wo;
    x = rem - y * p.wo;
  }
  // copies of this row of one stage, then on to the row 32 further
  __device__ __forceinline__ void stage(const FactorParams& p, const Parts& q, uint32_t dst, uint32_t blocks, bool no_halo, int step_n, int step_y, int step_x) {
    const bool rvalid = left > 0;
    const int ih = y * p.stride_h - p.pad_h, iw = x * p.stride_w - p.pad_w;
    const int64_t pix = n * p.sn + ih * p.sh + iw * p.sw;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      if (!((blocks >> b) & 1u)) continue;
      const int kp = kpos[b];
      const uint32_t d = dst + (b >> 1) * SIDE + (b & 1) * BLK;
      if (kp == -1) {                              // like any other column, the row side takes the weight
        uint32_t one[3];
        split2(!rvalid ? 0.f : b < 2 && p.weight ? __ldg(p.weight + n) : 1.f, 0.f, one[0], one[1], one[2]);
#pragma unroll
        for (int t = 0; t < 3; ++t)
          asm volatile("st.shared.v4.b32 [%0], {%1,%2,%2,%2};" ::"r"(d + t * OPB), "r"(one[t]), "r"(0u) : "memory");
        continue;
      }
      bool in = rvalid && kp >= 0;
      if (!no_halo) in = in && (unsigned)(ih + (kp & 0xFFFF)) < (unsigned)p.h && (unsigned)(iw + (kp >> 16)) < (unsigned)p.w;
      const __nv_bfloat16* src = (b < 2 ? q.a : q.b) + (in ? pix + koff[b] : 0);
      const int bytes = in ? 16 : 0;
#pragma unroll
      for (int t = 0; t < 3; ++t)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d + t * OPB), "l"(src + t * q.stride), "r"(bytes) : "memory");
    }
    left -= KS;
    x += step_x;
    if (x >= p.wo) { x -= p.wo; ++y; }
    y += step_y;
    if (y >= p.ho) { y -= p.ho; ++n; }
    n += step_n;
  }
};

template <bool PAIR, bool BOX>
__global__ void __launch_bounds__(THREADS, 1) factor_f32_kernel(const FactorParams p, const Parts parts, const __grid_constant__ Boxes boxes) {
  static_assert(PAIR || !BOX, "one CTA gathers");
  // a box brings the three parts of 64 columns in one piece; the gather keeps the 128 columns of a part together
  constexpr uint32_t BLK_STRIDE = BOX ? 3 * BLK : BLK, PART_STRIDE = BOX ? BLK : OPB;
  constexpr int NACC = PAIR ? 128 : 64;          // accumulator columns per accumulate warp
  constexpr int ACC_COLS = 2 * NACC;             // TMEM columns of one accumulator
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bars[2 * STAGES + 4];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int fin_flag;

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;      // uniform, for setmaxnreg
  const uint32_t rank = PAIR ? cluster_ctarank() : 0u;
  const bool fused = p.tickets != nullptr;
  const int last_n = BOX ? boxes.narrow : 0;
  int bI, bJ;                                    // block (PAIR: 256 wide) row and column
  int split = blockIdx.y;
  if (BOX) {
    // the blocks of a narrow last block row come behind all others, whatever their split: short work last
    const int nb2 = ceil_div(p.d, 256), units = nb2 * (nb2 + 1) / 2;
    const int whole = last_n ? units - nb2 : units, narrow = units - whole;
    int id = blockIdx.x >> 1, unit;
    if (id < whole * p.splits) {
      split = id / whole;
      unit = id - split * whole;
    } else {
      id -= whole * p.splits;
      split = id / narrow;
      unit = whole + id - split * narrow;
    }
    tri_decode(unit, bI, bJ);
  } else {
    tri_decode(PAIR ? blockIdx.x >> 1 : blockIdx.x, bI, bJ);
  }
  const int64_t r_begin = (int64_t)split * p.rows_per_split;
  const int nrows = (int)max((int64_t)0, min((int64_t)p.rows_per_split, p.rows - r_begin));
  const int nstages = ceil_div(nrows, KS);
  const int nchunks = ceil_div(nstages, FLUSH);
  int* status = p.status;
  // The last block row, if it is at most 128 wide, takes the column side: N is that width (halves of it per CTA) and the
  // block it meets fills the 256 rows, so that its MMAs and loads shrink with it.  The tile comes out transposed.
  const bool ragged = last_n != 0 && bI == (p.d - 1) / 256, swapped = ragged && bI != bJ;
  const int col_a = (swapped ? bJ : bI) * (PAIR ? 256 : 128) + (int)rank * TILE;
  const int col_b = !ragged ? bJ * (PAIR ? 256 : 128) + (int)rank * TILE : rank == 0 ? bI * 256 : last_n == 128 ? bI * 256 + 64 : p.d + 255;
  // 64-column blocks A0 A1 B0 B1 that hold columns of the matrix and are needed; a box leaves a ones column
  // that is not among the channels out (it has a block to itself, written once below)
  const int loaded_cols = BOX ? p.dcols : p.d;
  const bool share = bI == bJ && p.weight == nullptr && !ragged;
  const uint32_t used = share ? 3u : ragged ? 7u : 15u;
  uint32_t blocks = 0;
#pragma unroll
  for (int b = 0; b < 4; ++b)
    if ((b < 2 ? col_a : col_b) + (b & 1) * 64 < loaded_cols && ((used >> b) & 1u)) blocks |= 1u << b;

  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (STAGES + s); };
  auto accfull_bar = [&](int b) { return bar0 + 8u * (2 * STAGES + b); };
  auto accempty_bar = [&](int b) { return bar0 + 8u * (2 * STAGES + 2 + b); };
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      // a pair's gather warps all arrive at the leader; of boxes the leader's producer, which announces the bytes of both
      // CTAs, and the peer's once it has issued its own
      mbar_init(full_bar(s), BOX ? 2 : (PAIR ? 2 : 1) * LOAD_WARPS);
      mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(accfull_bar(b), 1);
      mbar_init(accempty_bar(b), (PAIR ? 2 : 1) * EPI_WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // blocks past the matrix edge are never written: they stay zero
  const uint32_t idle = ~blocks & used;
  if (idle) {
    for (int b = 0; b < 4; ++b) {
      if (!((idle >> b) & 1u)) continue;
      for (uint32_t o = tid * 16u; o < 3 * STAGES * BLK; o += THREADS * 16u) {
        const uint32_t part = o / BLK;
        const uint32_t at = smem0 + (part / 3) * SLOT_BYTES + (b >> 1) * SIDE + (part % 3) * PART_STRIDE + (b & 1) * BLK_STRIDE + o % BLK;
        // the ones column, first of its block: hi is 1, in chunk 0 of every row (at its swizzled place)
        const bool one = BOX && p.d > p.dcols && (b < 2 ? col_a : col_b) + (b & 1) * 64 == p.dcols && part % 3 == 0 &&
                         ((o >> 4) & 7u) == ((o >> 7) & 7u);
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%2,%2};" ::"r"(at), "r"(one ? 0x3F80u : 0u), "r"(0u) : "memory");
      }
    }
  }
  fence_async_smem();
  if (warp == MMA_WARP) {
    if (PAIR) tmem_alloc2(smem_u32(&tmem_base_slot), 2 * ACC_COLS);
    else tmem_alloc(smem_u32(&tmem_base_slot), 2 * ACC_COLS);
  }
  tc_fence_before();
  if (PAIR) cluster_sync_all();
  else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  asm volatile("griddepcontrol.wait;" ::: "memory");                 // the parts are written, the header is clear
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  if (warp < EPI_WARPS) {
    // ------------------------------------------------------------------ accumulate warps
    asm volatile("setmaxnreg.inc.sync.aligned.u32 168;");
    // warp = 4*half + q: rows 32q.. of the CTA's 128, columns [NACC*half, +NACC)
    const int q = warp & 3, half = warp >> 2;
    float acc[NACC];
#pragma unroll
    for (int i = 0; i < NACC; ++i) acc[i] = 0.f;
    const uint32_t accempty0 = PAIR ? map_to_cta(accempty_bar(0), 0u) : accempty_bar(0);
    for (int c = 0; c < nchunks; ++c) {
      const int b = c & 1;
      if (!mbar_wait(accfull_bar(b), (c >> 1) & 1, status, 63)) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * ACC_COLS + half * NACC);
#pragma unroll
      for (int part = 0; part < NACC / 32; ++part) {
        uint32_t v[32];
        tmem_ld32(taddr + part * 32, v);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[part * 32 + i] += __uint_as_float(v[i]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (PAIR) mbar_arrive_cluster(accempty0 + 8u * b);
        else mbar_arrive(accempty0 + 8u * b);
      }
    }
    const int ti = PAIR ? 2 * bI + (int)rank : bI, tj = PAIR ? 2 * bJ + half : bJ;
    const int col0 = PAIR ? 0 : half * NACC;     // first column inside the 128x128 tile
    if (BOX && swapped) {
      // column i of the last block row, row jr of this CTA's 128: transposed into tile (2 bI, 2 bJ + rank)
      const int tr = 2 * bI, tc = 2 * bJ + (int)rank, jr = q * 32 + lane, width = p.d - 256 * bI;
      float* dst = p.partial + ((int64_t)(tr * (tr + 1) / 2 + tc) * p.splits + split) * (TILE * TILE) + part_at(0, jr);
      if (half == 0) {
#pragma unroll
        for (int i = 0; i < NACC; ++i)
          if (i < width) dst[4 * i] = p.accumulate ? dst[4 * i] + acc[i] : acc[i];
      }
    } else if (ti < ceil_div(p.d, TILE) && tj <= ti) {
      float* dst = p.partial + ((int64_t)(ti * (ti + 1) / 2 + tj) * p.splits + split) * (TILE * TILE) + part_at(q * 32 + lane, col0);
      if (p.accumulate) {
#pragma unroll
        for (int i = 0; i < NACC; i += 4) {
          const float4 v = *reinterpret_cast<const float4*>(dst + i * TILE);
          acc[i] += v.x; acc[i + 1] += v.y; acc[i + 2] += v.z; acc[i + 3] += v.w;
        }
      }
      if (fused && p.splits == 1) {
        // shared memory is free: every MMA has read its operands before the last accumulator was published
        float* ct = reinterpret_cast<float*>(smem_raw + (smem0 - smem_u32(smem_raw))) + (PAIR ? half * (TILE * fin::CT_LD) : 0) +
                    (q * 32 + lane) * fin::CT_LD + col0;
#pragma unroll
        for (int i = 0; i < NACC; ++i) ct[i] = acc[i];
      } else {
#pragma unroll
        for (int i = 0; i < NACC; i += 4)
          *reinterpret_cast<float4*>(dst + i * TILE) = make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
        if (fused) __threadfence();
      }
    }
    // the common tail has equal shares again; nobody may take registers back before these warps have given theirs
    asm volatile("setmaxnreg.dec.sync.aligned.u32 96;");
    asm volatile("bar.sync 2, %0;" ::"n"(THREADS) : "memory");
  } else if (warp < LOAD_WARP0) {
    // ------------------------------------------------------------------ MMA issuer (of a pair: the leader's)
    asm volatile("setmaxnreg.dec.sync.aligned.u32 24;");
    if (warp == MMA_WARP && lane == 0 && rank == 0) {
      // a narrow tile multiplies only the columns that exist (N in steps of 16)
      const int n_cols = min(TILE, (p.d - bJ * TILE + 15) / 16 * 16);
      const uint32_t idesc = PAIR ? (instr_desc_pair(1u, 1u) & ~(0x3Fu << 17)) | ((uint32_t)((ragged ? last_n : 256) >> 3) << 17)
                                  : ((instr_desc(1u, 1u) & ~(0x3Fu << 17)) | ((uint32_t)(n_cols >> 3) << 17));
      bool ok = true;
      int s = 0;
      for (; s < nstages && ok; ++s) {
        const int slot = s % STAGES, c = s / FLUSH, b = c & 1;
        const bool first_of_chunk = (s % FLUSH) == 0;
        if (first_of_chunk && c >= 2) ok = mbar_wait(accempty_bar(b), ((c >> 1) - 1) & 1, status, 62);
        if (!ok) break;
        ok = mbar_wait(full_bar(slot), (s / STAGES) & 1, status, 61);
        if (!ok) break;
        tc_fence_after();
        const uint32_t a0 = smem0 + slot * SLOT_BYTES, b0 = share ? a0 : a0 + SIDE;
        const uint32_t d_tmem = tmem_base + (uint32_t)(b * ACC_COLS);
        uint32_t on = first_of_chunk ? 0u : 1u;
        for (int ks = 0; ks < KS / 16; ++ks) {
          // 16 rows = two 1024-byte swizzle atoms; the next 64 columns start BLK further on
          const uint64_t a_d = smem_desc_sw128(a0 + ks * 2048u, BLK_STRIDE, 1024u), b_d = smem_desc_sw128(b0 + ks * 2048u, BLK_STRIDE, 1024u);
          constexpr uint64_t P = PART_STRIDE >> 4;       // from one part to the next, in descriptor units
          auto mma = [&](int pa, int pb) {
            if (PAIR) umma2<false>(d_tmem, a_d + pa * P, b_d + pb * P, idesc, on);
            else umma<false>(d_tmem, a_d + pa * P, b_d + pb * P, idesc, on);
            on = 1u;
          };
          mma(2, 0); mma(0, 2); mma(1, 1); mma(1, 0); mma(0, 1); mma(0, 0);
        }
        const bool publish = (s % FLUSH) == FLUSH - 1 || s == nstages - 1;
        if (PAIR) {
          umma2_commit_both(empty_bar(slot));
          if (publish) umma2_commit_both(accfull_bar(b));
        } else {
          umma_commit(empty_bar(slot));
          if (publish) umma_commit(accfull_bar(b));
        }
      }
      mmas_done<STAGES>(s, empty_bar, status, 68);
    }
    __syncwarp();
    asm volatile("bar.sync 2, %0;" ::"n"(THREADS) : "memory");
    asm volatile("setmaxnreg.inc.sync.aligned.u32 96;");
  } else {
    // ------------------------------------------------------------------ gather warps
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (BOX) {
      if (warp == LOAD_WARP0 && lane == 0 && !g_inject_stall) {
        int c0[4], x0[4], y0[4];
        uint32_t pair_blocks = 0;      // blocks that both CTAs load
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const int j0 = (b < 2 ? col_a : col_b) + (b & 1) * 64, pos = j0 / p.c, ky = pos / p.kw;
          c0[b] = j0 - pos * p.c;
          x0[b] = (pos - ky * p.kw) * p.dil_w - p.pad_w;
          y0[b] = ky * p.dil_h - p.pad_h;
          const int first = j0 - (int)rank * TILE;
          if (!((used >> b) & 1u)) continue;
          if (ragged && b == 2) pair_blocks += (bI * 256 < loaded_cols ? 1u : 0u) + (last_n == 128 && bI * 256 + 64 < loaded_cols ? 1u : 0u);
          else pair_blocks += (first < loaded_cols ? 1u : 0u) + (first + TILE < loaded_cols ? 1u : 0u);
        }
        const uint64_t map = reinterpret_cast<uint64_t>(&boxes.map);
        const uint32_t fulls = map_to_cta(full_bar(0), 0u);
        const int first_box = (int)(r_begin / KS), per_image = boxes.across * boxes.down;
        int n = first_box / per_image, iy = (first_box - n * per_image) / boxes.across;
        int ix = first_box - n * per_image - iy * boxes.across;
        int s = 0;
        for (; s < nstages; ++s) {
          const int slot = s % STAGES;
          if (s >= STAGES && !mbar_wait(empty_bar(slot), ((s / STAGES) - 1) & 1, status, 64)) break;
          const uint32_t fb = fulls + 8u * slot;
          if (rank == 0)
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full_bar(slot)), "r"(pair_blocks * 3 * BLK) : "memory");
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            if (!((blocks >> b) & 1u)) continue;
            const uint32_t dst = smem0 + slot * SLOT_BYTES + (b >> 1) * SIDE + (b & 1) * BLK_STRIDE;
            asm volatile(
                "cp.async.bulk.tensor.5d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];"
                ::"r"(dst), "l"(map), "r"(c0[b]), "r"(ix * boxes.bw + x0[b]), "r"(iy * boxes.bh + y0[b]), "r"(n * boxes.bn), "r"(0), "r"(fb)
                : "memory");
          }
          if (rank != 0) mbar_arrive_cluster(fb);
          if (++ix == boxes.across) { ix = 0; if (++iy == boxes.down) { iy = 0; ++n; } }
        }
        // the copies of both CTAs complete on the leader's barriers, and the cluster leaves together
        if (rank == 0) ring_landed<STAGES>(s, full_bar, status, 65);
      }
      __syncwarp();
      asm volatile("bar.sync 2, %0;" ::"n"(THREADS) : "memory");
      asm volatile("setmaxnreg.inc.sync.aligned.u32 96;");
    } else {
    const int w = warp - LOAD_WARP0;
    const int l8 = lane & 7, row = 4 * w + (lane >> 3);
    Gather g;
    g.init(p, col_a, col_b, r_begin, nrows, row, l8);
    const uint32_t dst0 = smem0 + (uint32_t)row * 128u + (uint32_t)((l8 ^ (row & 7)) << 4);
    const uint32_t full0 = PAIR ? map_to_cta(full_bar(0), 0u) : full_bar(0);
    const bool no_halo = p.kh == 1 && p.kw == 1 && p.pad_h == 0 && p.pad_w == 0;
    const int step_n = KS / (p.ho * p.wo), step_rem = KS - step_n * (p.ho * p.wo);
    const int step_y = step_rem / p.wo, step_x = step_rem - step_y * p.wo;
    for (int s = g_inject_stall ? nstages + LAG : 0; s < nstages + LAG; ++s) {      // stalled: nothing is loaded or handed over
      // a stage is handed over before the wait for the next free slot, which depends on an MMA further back
      if (s >= LAG) {
        asm volatile("cp.async.wait_group %0;" ::"n"(LAG - 1) : "memory");
        fence_async_smem();
        __syncwarp();
        if (lane == 0) {
          const uint32_t bar = full0 + 8u * ((s - LAG) % STAGES);
          if (PAIR) mbar_arrive_cluster(bar);
          else mbar_arrive(bar);
        }
      }
      if (s < nstages) {
        const int slot = s % STAGES;
        if (s >= STAGES && !mbar_wait(empty_bar(slot), ((s / STAGES) - 1) & 1, status, 64)) break;
        g.stage(p, parts, dst0 + slot * SLOT_BYTES, blocks, no_halo, step_n, step_y, step_x);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    asm volatile("bar.sync 2, %0;" ::"n"(THREADS) : "memory");
    asm volatile("setmaxnreg.inc.sync.aligned.u32 96;");
    }
  }
  tc_fence_before();
  if (PAIR) cluster_sync_all();          // neither CTA leaves while its peer's MMAs may still read its shared memory
  else __syncthreads();
  if (warp == MMA_WARP) {
    __syncwarp();
    tc_fence_after();
    if (PAIR) tmem_dealloc2(tmem_base, 2 * ACC_COLS);
    else tmem_dealloc(tmem_base, 2 * ACC_COLS);
  }
  if (fused) {
    const int nb = ceil_div(p.d, TILE);
    const int ti = PAIR ? 2 * bI + (int)rank : bI;
    float* ct0 = reinterpret_cast<float*>(smem_raw + (smem0 - smem_u32(smem_raw)));
    for (int hh = 0; hh < (PAIR ? 2 : 1); ++hh) {
      const int tj = PAIR ? 2 * bJ + hh : bJ;
      if (ti < nb && tj <= ti)
        fin::finish_tile<THREADS>(p, ti * (ti + 1) / 2 + tj, ti, tj, split, ct0 + (p.splits == 1 ? hh * (TILE * fin::CT_LD) : 0),
                                  &fin_flag, tid);
      __syncthreads();
    }
  }
}

// Blocks x splits of the rows over the 74 pairs (148 SMs), with rough costs: a stage (`stage_us`), the fixed cost of a CTA
// (set-up, pipeline fill, drain, tile: 5 us), a partial tile's way to memory and back (0.03 us).
// `narrow` of the units take `part` of the others' time and run behind them.
// Of these only the stage of boxes is a measurement (1.05 of the 1.1 us above); the others are estimates that were not
// measured by themselves.  They weigh splits against each other, nothing else.
static int choose_splits(int64_t rows, int units, int narrow, double part, int slots, int tiles, double stage_us, int max_splits,
                         int& rows_per_split) {
  const int64_t stages = ceil_div64(rows, KS);
  const int most = (int)std::max<int64_t>(1, std::min<int64_t>({stages / 4, 148, max_splits}));
  double best = 1e30;
  int64_t best_sps = stages;
  for (int s = 1; s <= most; ++s) {
    const int64_t sps = ceil_div64(stages, s), real = ceil_div64(stages, sps);
    const int64_t whole = (units - narrow) * real, rest = whole % slots;
    double rounds = (double)(whole / slots);
    int64_t left = narrow * real;
    if (rest) {
      rounds += 1.0;
      left -= (slots - rest) * (int64_t)(1.0 / part);      // beside the last round of the others
    }
    if (left > 0) rounds += part * (double)ceil_div64(left, slots);
    const double cost = rounds * ((double)sps * stage_us + 5.0) + 0.03 * (double)(tiles * real);
    if (cost < best - 1e-9) { best = cost; best_sps = sps; }
  }
  rows_per_split = (int)(best_sps * KS);
  return (int)ceil_div64(stages, best_sps);
}

template <bool PAIR, bool BOX>
static int launch(const FactorParams& p, const Parts& parts, const Boxes& boxes, int units, int splits, cudaStream_t st) {
  SSO_ENSURE_SMEM((factor_f32_kernel<PAIR, BOX>), SMEM);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = BOX ? dim3(2 * units * splits) : dim3(PAIR ? 2 * units : units, splits);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = SMEM;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = PAIR ? 2 : 1;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = 2;
  cudaLaunchKernelEx(&cfg, factor_f32_kernel<PAIR, BOX>, p, parts, boxes);
  SSO_LAUNCH_OK("factor_f32_kernel");
  return 0;
}

// ------------------------------------------------------------------------------------------------
// Tall and narrow: rows of at most 128 columns at one stride (Linear layers, 1x1 factors of channels_last
// activations).  There is one tile, so an element is converted once wherever that happens, and a pass over memory
// for the parts would cost more than the factor: the raw rows come into shared memory with cp.async (three stages of
// 32 KB in flight per SM), the warp that loaded a row splits it into the operand slots.  A stage is 64 rows of 128
// columns or 128 rows of 64.  Bound: instructions of the split (d = 64 from 802816 rows: 105 us against 355 us
// through the parts and 434 us for 3xTF32 with one stage of loads).
// ------------------------------------------------------------------------------------------------
namespace narrow {
constexpr int RAW = 4, SLOTS = 2, CHUNK = 64;      // rows between drains of the accumulator
constexpr uint32_t RAW_BYTES = 32768, SLOT_BYTES = 49152;
constexpr size_t SMEM = RAW * RAW_BYTES + SLOTS * SLOT_BYTES + 1024;

template <int NBLK, bool VEC>
__global__ void __launch_bounds__(THREADS, 1) narrow_kernel(const FactorParams p, int64_t row_stride) {
  constexpr int K = 128 / NBLK, R = K / LOAD_WARPS;            // rows of a stage, of a warp
  constexpr uint32_t PBLK = K * 128u, PART = NBLK * PBLK;      // 64 columns, one part
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bars[2 * SLOTS + 4];
  __shared__ uint32_t tmem_base_slot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t r_begin = (int64_t)blockIdx.x * p.rows_per_split;
  const int nrows = (int)max((int64_t)0, min((int64_t)p.rows_per_split, p.rows - r_begin));
  const int nstages = ceil_div(nrows, K), nchunks = nstages * (K / CHUNK);
  int* status = p.status;
  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t raw0 = smem0 + SLOTS * SLOT_BYTES;
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (SLOTS + s); };
  auto accfull_bar = [&](int b) { return bar0 + 8u * (2 * SLOTS + b); };
  auto accempty_bar = [&](int b) { return bar0 + 8u * (2 * SLOTS + 2 + b); };
  if (tid == 0) {
    for (int s = 0; s < SLOTS; ++s) {
      mbar_init(full_bar(s), LOAD_WARPS);
      mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(accfull_bar(b), 1);
      mbar_init(accempty_bar(b), EPI_WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) tmem_alloc(smem_u32(&tmem_base_slot), 256);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;

  if (warp < EPI_WARPS) {
    const int q = warp & 3, half = warp >> 2;
    float acc[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) acc[i] = 0.f;
    for (int c = 0; c < nchunks; ++c) {
      const int b = c & 1;
      if (!mbar_wait(accfull_bar(b), (c >> 1) & 1, status, 73)) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * 128 + half * 64);
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        uint32_t v[32];
        tmem_ld32(taddr + part * 32, v);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[part * 32 + i] += __uint_as_float(v[i]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(accempty_bar(b));
    }
    if (half < NBLK && q < 2 * NBLK) {
      float* dst = p.partial + (int64_t)blockIdx.x * (TILE * TILE) + part_at(q * 32 + lane, half * 64);
#pragma unroll
      for (int i = 0; i < 64; i += 4) *reinterpret_cast<float4*>(dst + i * TILE) = make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
    }
  } else if (warp == MMA_WARP) {
    if (lane == 0) {
      const int n_cols = (p.d + 15) / 16 * 16;
      const uint32_t idesc = (instr_desc(1u, 1u) & ~(0x3Fu << 17)) | ((uint32_t)(n_cols >> 3) << 17);
      bool ok = true;
      int c = 0;
      for (int s = 0; s < nstages && ok; ++s) {
        const int slot = s % SLOTS;
        ok = mbar_wait(full_bar(slot), (s / SLOTS) & 1, status, 71);
        if (!ok) break;
        tc_fence_after();
        const uint32_t a0 = smem0 + slot * SLOT_BYTES;
        for (int ks = 0; ks < K / 16; ++ks) {
          const int b = c & 1;
          uint32_t on = (ks % (CHUNK / 16)) == 0 ? 0u : 1u;
          if (!on && c >= 2) ok = mbar_wait(accempty_bar(b), ((c >> 1) - 1) & 1, status, 72);
          if (!ok) break;
          const uint32_t d_tmem = tmem_base + (uint32_t)(b * 128);
          // with one block the 64 rows behind it (M is 128) are whatever follows in shared memory: they only reach
          // accumulator rows that nobody reads
          const uint64_t desc = smem_desc_sw128(a0 + ks * 2048u, PBLK, 1024u);
          constexpr uint64_t P = PART >> 4;
          auto mma = [&](int pa, int pb) { umma<false>(d_tmem, desc + pa * P, desc + pb * P, idesc, on); on = 1u; };
          mma(2, 0); mma(0, 2); mma(1, 1); mma(1, 0); mma(0, 1); mma(0, 0);
          if ((ks % (CHUNK / 16)) == CHUNK / 16 - 1) {
            if (ks == K / 16 - 1) umma_commit(empty_bar(slot));
            umma_commit(accfull_bar(b));
            ++c;
          }
        }
      }
      mmas_done<2>(c, accfull_bar, status, 78);      // a chunk is begun only when its accumulator is free
    }
  } else if (warp >= LOAD_WARP0) {
    const int w = warp - LOAD_WARP0;
    // 16-byte chunk c of a row's 256 bytes sits at position c ^ (c >> 3): the copies of consecutive chunks and the
    // loads of every other chunk below both touch eight different bank groups
    auto pos = [](int c) { return (uint32_t)(c ^ (c >> 3)) * 16u; };
    const int chunk = lane & 15, row_l = w * R + (lane >> 4);
    const uint32_t raw_w = raw0 + (uint32_t)row_l * 256u + pos(chunk);
    const float* src0 = reinterpret_cast<const float*>(p.x) + (r_begin + row_l) * row_stride + chunk * 4;
    int have[NBLK];
#pragma unroll
    for (int b = 0; b < NBLK; ++b) have[b] = max(0, min(4, p.dcols - b * 64 - chunk * 4));
    auto load = [&](int s) {
      const float* src = src0 + (int64_t)s * K * row_stride;
      const uint32_t dst = raw_w + (s % RAW) * RAW_BYTES;
#pragma unroll
      for (int j = 0; j < R / 2; ++j) {
        const bool rv = s * K + row_l + 2 * j < nrows;
#pragma unroll
        for (int b = 0; b < NBLK; ++b) {
          const float* g = src + (int64_t)(2 * j) * row_stride + b * 64;
          const uint32_t d = dst + b * (K * 256u) + j * 512u;
          if (VEC) {
            const bool in = rv && have[b] > 0;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(in ? g : reinterpret_cast<const float*>(p.x)), "r"(in ? 16 : 0) : "memory");
          } else {
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              const bool in = rv && t < have[b];
              asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d + 4 * t), "l"(in ? g + t : reinterpret_cast<const float*>(p.x)), "r"(in ? 4 : 0) : "memory");
            }
          }
        }
      }
    };
    const int l8 = lane & 7, k0 = w * R + (lane >> 3);           // this lane splits columns 8*l8 .. of rows k0, k0 + 4, ..
    const int ones = p.d > p.dcols ? p.dcols - 8 * l8 : -1;      // the ones column, relative to this lane's first
    for (int s = 0; s < RAW - 1; ++s) {
      if (s < nstages) load(s);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int s = g_inject_stall ? nstages : 0; s < nstages; ++s) {      // stalled: no stage is handed over
      if (s + RAW - 1 < nstages) load(s + RAW - 1);
      asm volatile("cp.async.commit_group;" ::: "memory");
      asm volatile("cp.async.wait_group %0;" ::"n"(RAW - 1) : "memory");
      __syncwarp();                              // the whole warp's copies of stage s have landed
      const int slot = s % SLOTS;
      if (s >= SLOTS && !mbar_wait(empty_bar(slot), ((s / SLOTS) - 1) & 1, status, 74)) break;
#pragma unroll
      for (int j = 0; j < R / 4; ++j)
#pragma unroll
        for (int b = 0; b < NBLK; ++b) {
          const int k = k0 + 4 * j;
          float v[8];
          const uint32_t src = raw0 + (s % RAW) * RAW_BYTES + (uint32_t)(b * K + k) * 256u;
          asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(src + pos(2 * l8)) : "memory");
          asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "r"(src + pos(2 * l8 + 1)) : "memory");
          const int at = ones - 64 * b;
          if (ones >= 0 && at >= 0 && at < 8) {
            const float one = s * K + k < nrows ? 1.f : 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i)
              if (i == at) v[i] = one;
          }
          uint32_t hi[4], mid[4], lo[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) split2(v[2 * i], v[2 * i + 1], hi[i], mid[i], lo[i]);
          const uint32_t dst = smem0 + slot * SLOT_BYTES + b * PBLK + (uint32_t)k * 128u + (uint32_t)((l8 ^ (k & 7)) << 4);
          asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst), "r"(hi[0]), "r"(hi[1]), "r"(hi[2]), "r"(hi[3]) : "memory");
          asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst + PART), "r"(mid[0]), "r"(mid[1]), "r"(mid[2]), "r"(mid[3]) : "memory");
          asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst + 2 * PART), "r"(lo[0]), "r"(lo[1]), "r"(lo[2]), "r"(lo[3]) : "memory");
        }
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(full_bar(slot));
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 256);
  }
}
}  // namespace narrow

// What a problem looks like to the gather: its channels padded (or folded) to c8, its factor of width d.
struct Shape {
  int fold, c8, width, dcols, d, tiles, blocks;
  bool plain;                // columns are the channels as they lie, the ones column one of them
  int64_t image_bytes;       // parts of one image
};
static Shape shape_of(const FactorParams& p) {
  Shape s;
  const int kk = p.kh * p.kw, ones = p.d - p.dcols;
  // a row of a padded 1x1 window may lie outside the image, where every channel is zero and the ones column is not
  s.plain = kk == 1 && (ones == 0 || (p.pad_h == 0 && p.pad_w == 0));
  s.fold = (p.c < 8 && p.kw > 1) ? p.kw : 0;
  s.c8 = ceil_div(s.fold ? p.c * p.kw : p.c + (s.plain ? ones : 0), 8) * 8;
  s.width = s.fold ? p.wo : p.w;
  s.dcols = s.plain ? p.d : s.c8 * (s.fold ? p.kh : kk);
  s.d = s.plain ? p.d : s.dcols + ones;
  const int nb = ceil_div(s.d, 128), nb2 = ceil_div(s.d, 256);
  s.tiles = nb * (nb + 1) / 2;
  s.blocks = nb2 * (nb2 + 1) / 2;
  s.image_bytes = (int64_t)p.h * s.width * s.c8 * 6 * (p.weight ? 2 : 1);
  return s;
}
// Boxes of 32 whole pixels that cover the output exactly: no pixel is computed twice or for padding, and no row of a
// stage is left to be cleared.  Every other geometry (strides, odd image sizes, per-sample weights, channel counts
// below 64 columns of one kernel position) keeps the gather, which takes any.
static bool choose_boxes(const FactorParams& p, const Shape& s, Boxes& b) {
  if (p.weight || s.fold || p.stride_h != 1 || p.stride_w != 1 || (!s.plain && s.c8 % 64 != 0)) return false;
  b.bw = std::gcd(p.wo, KS);
  b.bh = std::gcd(p.ho, KS / b.bw);
  b.bn = KS / (b.bw * b.bh);
  b.across = p.wo / b.bw;
  b.down = p.ho / b.bh;
  return p.n % b.bn == 0 && tensor_map_encoder() != nullptr;
}
static bool encode_boxes(Boxes& b, const Parts& parts, const Shape& s, int h, int n) {
  const cuuint64_t row = (cuuint64_t)s.c8 * 2;
  const cuuint64_t dims[5] = {(cuuint64_t)s.c8, (cuuint64_t)s.width, (cuuint64_t)h, (cuuint64_t)n, 3};
  const cuuint64_t strides[4] = {row, row * s.width, row * s.width * h, (cuuint64_t)parts.stride * 2};
  const cuuint32_t box[5] = {64, (cuuint32_t)b.bw, (cuuint32_t)b.bh, (cuuint32_t)b.bn, 3}, step[5] = {1, 1, 1, 1, 1};
  return tensor_map_encoder()(&b.map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<__nv_bfloat16*>(parts.a), dims, strides, box, step,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
constexpr int64_t PARTS_TARGET = (int64_t)256 << 20;     // parts of one run of images
// Columns that the MMAs of the last block row compute if it is a narrow one: 32 (at most sixteen columns, all of them
// from one CTA; a pair's N is a multiple of 32), 128, or 0 for an ordinary block.  Its blocks run behind all others and
// read the parts once more, from L2 if they are small: the line lies between 50 MB (d = 577 from 131072 rows, 391 us
// without, 363 with) and 256 MB (d = 333 from 401408 rows, 1153 without, 1267 with), nearer to the size of L2.
constexpr int64_t NARROW_PARTS = (int64_t)96 << 20;
static int narrow_columns(int d) {
  const int width = d - (d - 1) / 256 * 256;
  return d <= 256 || width > 128 ? 0 : width <= 16 ? 32 : 128;
}
constexpr int64_t PARTIAL_TARGET = (int64_t)148 * 2 * 65536;

}  // namespace f32

// Scratch: header, partial tiles (at least one split), parts of at least one image.
static size_t f32_min_bytes(const FactorParams& p, const f32::Shape& s) {
  return factor_header_bytes(s.tiles) + (size_t)s.tiles * 65536 + (size_t)s.image_bytes + 512;
}
size_t factor_f32_workspace_bytes(const FactorParams& p) {
  const f32::Shape s = f32::shape_of(p);
  const int64_t all = s.image_bytes * p.n;
  const int64_t partial = std::max<int64_t>(f32::PARTIAL_TARGET, 4 * (int64_t)s.tiles * 65536);
  return factor_header_bytes(s.tiles) + (size_t)partial + (size_t)std::max<int64_t>(s.image_bytes, std::min<int64_t>(all, f32::PARTS_TARGET)) + 512;
}

bool factor_f32_supported(const FactorParams& p, size_t workspace_bytes) {
  const f32::Shape s = f32::shape_of(p);
  return (int64_t)p.h * s.width * s.c8 < ((int64_t)1 << 30) && (int64_t)p.n * p.h * s.width < ((int64_t)1 << 31) && workspace_bytes >= f32_min_bytes(p, s);
}

// Rows at one stride with contiguous columns, at most 128 of them: the stride, else 0.
static int64_t narrow_stride(const FactorParams& p) {
  if (p.d > 128 || p.kh != 1 || p.kw != 1 || p.pad_h || p.pad_w || p.stride_h != 1 || p.stride_w != 1 || p.weight || (p.sc != 1 && p.c > 1)) return 0;
  const int64_t rs = p.w > 1 ? p.sw : p.h > 1 ? p.sh : p.sn;
  const bool even = (p.w == 1 || p.h == 1 || p.sh == p.w * p.sw) && (p.h * p.w == 1 || p.n == 1 || p.sn == (int64_t)p.h * p.w * rs);
  return even && rs > 0 ? rs : 0;
}

template <int NBLK, bool VEC>
static int narrow_launch(const FactorParams& p, int64_t row_stride, cudaStream_t st) {
  SSO_ENSURE_SMEM((f32::narrow::narrow_kernel<NBLK, VEC>), f32::narrow::SMEM);
  f32::narrow::narrow_kernel<NBLK, VEC><<<p.splits, f32::THREADS, f32::narrow::SMEM, st>>>(p, row_stride);
  SSO_LAUNCH_OK("narrow_kernel");
  return factor_tc_run_reduce(p, 1, st);
}

static int factor_narrow_launch(FactorParams p, int64_t row_stride, void* workspace, size_t workspace_bytes, cudaStream_t st) {
  const size_t hdr = factor_header_bytes(1);
  const int64_t stages = ceil_div64(p.rows, 128);      // a CTA needs about four to pay for its set-up
  const int64_t most = std::max<int64_t>(1, std::min<int64_t>({148, stages / 4, (int64_t)((workspace_bytes - hdr) / 65536)}));
  p.rows_per_split = (int)(ceil_div64(stages, most) * 128);
  p.splits = (int)ceil_div64(p.rows, p.rows_per_split);
  p.status = reinterpret_cast<int*>(workspace);
  p.partial = reinterpret_cast<float*>(reinterpret_cast<char*>(workspace) + hdr);
  p.perm_c = 0; p.perm_kk = 1; p.tickets = nullptr;
  SSO_CUDA_OK(cudaMemsetAsync(p.status, 0, sizeof(int), st));
  const bool vec = p.c % 4 == 0 && row_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(p.x) & 15) == 0;
  if (p.d <= 64) return vec ? narrow_launch<1, true>(p, row_stride, st) : narrow_launch<1, false>(p, row_stride, st);
  return vec ? narrow_launch<2, true>(p, row_stride, st) : narrow_launch<2, false>(p, row_stride, st);
}

int factor_f32_launch(FactorParams p, void* workspace, size_t workspace_bytes, cudaStream_t st) {
  if (const int64_t rs = narrow_stride(p)) return factor_narrow_launch(p, rs, workspace, workspace_bytes, st);
  const f32::Shape s = f32::shape_of(p);
  SSO_CHECK_ARG(workspace != nullptr && workspace_bytes >= f32_min_bytes(p, s), "factor workspace too small: need %zu bytes, got %zu",
                f32_min_bytes(p, s), workspace_bytes);
  // images per run: as many as their parts fit next to one split's partial tiles, at most PARTS_TARGET
  const size_t hdr = factor_header_bytes(s.tiles);
  const int64_t room = (int64_t)(workspace_bytes - hdr - 512) - (int64_t)s.tiles * 65536;
  const int64_t per_run = std::max<int64_t>(1, std::min<int64_t>({(int64_t)p.n, f32::PARTS_TARGET / std::max<int64_t>(1, s.image_bytes), room / std::max<int64_t>(1, s.image_bytes)}));
  // a pair's block is 256 wide: up to 128 columns one CTA's tile is all there is to compute
  const bool pair = s.d > 128;
  f32::Boxes boxes{};
  bool box = pair && f32::choose_boxes(p, s, boxes) && per_run >= boxes.bn;
  const int whole = box ? boxes.bn : 1;      // images per run are a multiple of a box's
  const int runs = (int)ceil_div64(p.n, per_run / whole * whole);
  const int n_run = (int)ceil_div64(ceil_div64(p.n, runs), whole) * whole;
  const int64_t parts_bytes = n_run * s.image_bytes;
  const int max_splits = (int)(((int64_t)(workspace_bytes - hdr - 512) - (parts_bytes + 255) / 256 * 256) / ((int64_t)s.tiles * 65536));
  char* base = reinterpret_cast<char*>(workspace);
  FactorParams q = p;
  q.status = reinterpret_cast<int*>(base);
  f32::Parts parts;
  parts.a = reinterpret_cast<const __nv_bfloat16*>(base + (hdr + 255) / 256 * 256);
  parts.stride = (int64_t)n_run * p.h * s.width * s.c8;
  parts.b = p.weight ? parts.a + 3 * parts.stride : parts.a;
  parts.c8 = s.c8;
  q.partial = reinterpret_cast<float*>(base + (hdr + 255) / 256 * 256 + (parts_bytes + 255) / 256 * 256);
  const int64_t hw = (int64_t)p.ho * p.wo;
  int rps = 0;
  boxes.narrow = box && parts_bytes <= f32::NARROW_PARTS ? f32::narrow_columns(s.d) : 0;
  q.splits = f32::choose_splits(n_run * hw, pair ? s.blocks : s.tiles, boxes.narrow ? ceil_div(s.d, 256) : 0, boxes.narrow == 32 ? 0.6 : 0.75,
                                pair ? 74 : 148, s.tiles, box ? 1.05 : pair ? 0.85 : 0.6, max_splits, rps);
  q.rows_per_split = rps;
  const int kk = p.kh * p.kw;
  q.perm_c = s.plain ? 0 : s.c8;
  q.perm_kk = kk;
  q.perm_pub = s.plain ? 0 : p.c;
  q.perm_fold = s.fold;
  q.c = s.c8; q.dcols = s.dcols; q.d = s.d; q.w = s.width;
  q.sn = (int64_t)p.h * s.width * s.c8; q.sh = (int64_t)s.width * s.c8; q.sw = s.c8; q.sc = 1;
  if (s.fold) { q.kw = 1; q.stride_w = 1; q.pad_w = 0; q.dil_w = 1; }
  const bool fused = s.plain && q.splits == 1;
  if (fused) boxes.narrow = 0;      // its tiles come out transposed, which the finishing in the kernel does not expect
  q.ticket_tiles = s.tiles;
  const bool direct = !s.fold && p.sc == 1 && p.c % 4 == 0 && (reinterpret_cast<uintptr_t>(p.x) & 15) == 0 && p.sn % 4 == 0 &&
                      (p.h == 1 || p.sh % 4 == 0) && (p.w == 1 || p.sw % 4 == 0) && (int64_t)n_run * p.h * s.width * (s.c8 / 8) < ((int64_t)1 << 31);
  // planes (of more than one pixel) that a thread reads four pixels at a time
  const bool planes = !s.fold && !direct && p.sw == 1 && p.sh == p.w && p.h * p.w % 4 == 0 && p.sc % 4 == 0 && p.sn % 4 == 0 &&
                      (reinterpret_cast<uintptr_t>(p.x) & 15) == 0;
  const int header_words = fused ? (int)(hdr / sizeof(int)) : 1;
  for (int r = 0, n0 = 0; r < runs; ++r, n0 += n_run) {
    const int n = std::min(n_run, p.n - n0);
    FactorParams in = p;
    in.x = reinterpret_cast<const float*>(p.x) + n0 * p.sn;
    in.status = q.status;
    in.weight = p.weight ? p.weight + n0 : nullptr;
    const int64_t pixels = (int64_t)n * p.h * s.width;
    const int ones_at = s.plain && p.d > p.dcols ? p.c : -1;
    if (direct)
      f32::split_direct_kernel<<<(unsigned)ceil_div64(pixels * (s.c8 / 8), 256), 256, 0, st>>>(in, (uint32_t)pixels, ones_at,
                                                                                                            r == 0 ? header_words : 0, parts, parts);
    else if (planes)
      f32::split_planes_kernel<<<dim3((unsigned)ceil_div64(pixels, 64), ceil_div(s.c8, 64)), 256, 0, st>>>(in, (uint32_t)pixels, ones_at, r == 0 ? header_words : 0, parts, parts);
    else if (s.fold)
      f32::split_folded_kernel<<<(unsigned)ceil_div64(pixels * (s.c8 / 8), 256), 256, 0, st>>>(in, (uint32_t)pixels, s.width, s.fold, r == 0 ? header_words : 0, parts, parts);
    else
      f32::split_kernel<<<dim3((unsigned)ceil_div64(pixels, 32), ceil_div(s.c8, 64)), 256, 0, st>>>(in, (uint32_t)pixels, ones_at, r == 0 ? header_words : 0, parts, parts);
    SSO_LAUNCH_OK("split_kernel");
    q.n = n;
    q.weight = in.weight;
    q.rows = n * hw;
    q.accumulate = r > 0;
    q.tickets = fused && r == runs - 1 ? reinterpret_cast<int*>(base + 256) : nullptr;
    if (box && !f32::encode_boxes(boxes, parts, s, p.h, n)) return fail(-5, "cuTensorMapEncodeTiled failed for the parts of a factor");
    const int rc = box    ? f32::launch<true, true>(q, parts, boxes, s.blocks, q.splits, st)
                   : pair ? f32::launch<true, false>(q, parts, boxes, s.blocks, q.splits, st)
                          : f32::launch<false, false>(q, parts, boxes, s.tiles, q.splits, st);
    if (rc) return rc;
  }
  if (fused) return 0;
  return factor_tc_run_reduce(q, s.tiles, st);
}

int factor_f32_set_wait_controls(long long cycles, int stall) { return tc::set_wait_controls(cycles, stall); }

}  // namespace sso
