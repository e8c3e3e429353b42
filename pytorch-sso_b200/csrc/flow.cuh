// Records of the dataflow kernel (flow.cu), shared with the plan builder (engine.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace sso {
namespace flow {

enum Kind : int32_t {
  DIAG = 0,      // (p, -): factor the diagonal block of panel p and invert it
  PANEL = 1,     // (i, p): L(i, p) = (M(i, p) - sum_{k < p} L(i, k) L(p, k)^T) Linv(p)^T
  INVT = 2,      // (j, i): X(j, i) = -(sum_{j <= k < i} X(j, k) L(i, k)^T) Linv(i)^T,  X = L^-T
  PROD = 3       // (i, j): T(i, j) = sum_{k >= i} X(i, k) X(j, k)^T, and its mirror
};

struct Task {
  int16_t kind, mat;
  int16_t a, b;
};

struct alignas(64) Mat {
  unsigned char map_w[128];      // tensor maps (box 32 columns x 128 rows, SWIZZLE_128B) of the scratch matrix and of Linv
  unsigned char map_li[128];
  unsigned char map_box[128];    // the scratch matrix again, for stores of 32x32
  const float* src;              // M before damping
  float* W;                      // scratch matrix: L in the blocks below the diagonal
  float* X;                      // the same matrix, L^-T in the others; null: factorisation only
  float* Li;                     // [panels][128][128]: inverses of the diagonal blocks
  float* T;                      // the inverse, or null (factorisation only)
  float* U;                      // upper Cholesky factor (of M, or with X of the inverse), or null
  int32_t ld_src, ldw, ldt, ldu;
  int32_t d, np;
  int32_t pub;                   // size of M; d is larger by the padding rows of a reversed matrix
  int32_t mat;                   // index into the shift and info tables
  int32_t shifted;               // whether the damping shift is added
  int32_t partner, role, d_partner;
  int32_t info_slot;
  int32_t flag_w, flag_x, flag_d;      // first ready flag of the W tiles [np][np], X tiles [np][np], diagonal blocks [np]
};

struct Args {
  const Mat* mats;
  const Task* tasks;
  int n_tasks;
  int* sync;                 // [0] task counter (never reset), [1] epoch of this run, [2] value of the counter at its start
  int* flags;
  const float* traces;
  const float* damp_r;
  int* info;                 // nullable
  int* status;
  int with_u;                // whether U is written
  const float* src;          // nullable: the one matrix of the plan lies here this time, and its result goes to out
  float* out;
  int ld_src, ld_out;
  int rev;                   // the matrices are taken from the last row and column to the first
};

}  // namespace flow
int flow_launch(const flow::Args& a, int n_mats, int clear_info, int with_traces, cudaStream_t st);

}  // namespace sso
