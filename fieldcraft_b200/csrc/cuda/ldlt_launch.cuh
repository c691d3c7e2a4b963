// The device LDL^T's tasks and launchers (kernels in ldlt.cu, the panel's source in
// ldlt_panel.cuh).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "cuda/kernels.cuh"
#include "cuda/ldlt_panel.cuh"

namespace fc {
namespace ldlt {

// One front's panel step: the front and its state (Front), where its columns start in the
// analysis' postorder (`first`, for the failing column's name), and the GEMM tasks of the update
// of its later own columns (`slots`, `nslots` of them: update_tiles for the earliest end).
struct PanelTask {
  Front front;
  int64_t first;
  fc::GemmTask *slots;
  int32_t nslots;
  int32_t s;
};

// After a level's panels: rows [r0, r1) of a front's W21 = L21 D into w21 (leading dimension
// m - w, for the update-matrix GEMM). A CTA takes W21_ROWS rows.
constexpr int W21_ROWS = 32;
struct AfterTask {
  Front front;
  double *w21;
  int64_t r0, r1;
};

// After that, for the columns [c0, c0 + nb) of a front (nb <= 64): D out of them into d / e
// (split_d), which leaves the own block unit lower, and the solve's inverse of the diagonal block
// into X (leading dimension ldx) in the inverse arena.
struct InverseTask {
  Front front;
  double *d, *e;
  double *X;
  int64_t ldx;
  int32_t c0, nb;
};

void launch_inverse(const InverseTask *tasks, int count, cudaStream_t st);
// `tallest`, `widest`: the largest m and w of the launch's fronts (they size its grid and its CTAs);
// pos, from, twos: a number a supernode (see the kernel).
void launch_panel(const PanelTask *tasks, int count, int tallest, int widest, int32_t *pos, int32_t *from,
                  int32_t *twos, unsigned long long *failed, cudaStream_t st);
void launch_after(const AfterTask *tasks, int count, cudaStream_t st);
void launch_scale(int64_t nnz, const int64_t *a_src, const int32_t *a_row, const int32_t *a_col, const double *val,
                  unsigned long long *scale_bits, cudaStream_t st);
void launch_reset(int64_t n, const int32_t *local, int32_t *order, int8_t *pivots, cudaStream_t st);
// The solve's view of the pivots (after the last panel): own[j] is the place of column j of the
// structure's postorder in the solve's vectors (its supernode's columns in pivot order), perm_out
// the input permutation to that order, rows_out the row lists through `own`. local[j]: column j's
// place in its supernode.
void launch_fold(int64_t n, const int32_t *local, const int32_t *order, const int64_t *perm, int32_t *own,
                 int64_t *perm_out, int64_t rows_len, const int32_t *rows, int32_t *rows_out, cudaStream_t st);
void launch_d_inverse(int64_t n, int R, const double *d, const double *e, const int8_t *pivots, double *y,
                      cudaStream_t st);

}  // namespace ldlt
}  // namespace fc
