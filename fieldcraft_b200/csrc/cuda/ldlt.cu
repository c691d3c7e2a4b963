// The device LDL^T's pivoted panel step (ldlt_panel.cuh on CUDA threads): one CTA per front of
// a level on its own rows, each taking its next panel from where the previous one ended, then the
// rows below spread over the GPU. The source of the first is the one the CPU emulation checks
// against the oracle bit for bit; this file gives it the device's block (threads, __syncthreads)
// and its per-supernode state.
#include <cstdint>

#include "cuda/ldlt_launch.cuh"

namespace fc {
namespace ldlt {

struct DeviceBlock {
  __device__ int tid() const { return threadIdx.x; }
  __device__ int size() const { return blockDim.x; }
  __device__ void sync() { __syncthreads(); }
};

// Per supernode s: pos[s] is where its next panel starts (w when done), from[s] where the last one
// did (pos[s] when there was none), twos[s] counts its 2 x 2 pivots. A singular column lowers *failed to its postorder index (the first failing column in
// postorder is the one reported) and ends the supernode. After the panel the CTA writes the
// update of the later own columns as GEMM tasks (C -= L_panel W^T on the lower tiles, for the
// launch that follows); the slots it does not need stay empty (M = N = K = 0: no work).
constexpr int PANEL_THREADS = 512;
__global__ void __launch_bounds__(PANEL_THREADS) ldlt_panel_kernel(const PanelTask *__restrict__ tasks,
                                                                 int32_t *__restrict__ pos,
                                                                 int32_t *__restrict__ from,
                                                                 int32_t *__restrict__ twos,
                                                                 unsigned long long *__restrict__ failed) {
  extern __shared__ __align__(16) unsigned char panel_sm[];
  Shared &sh = *reinterpret_cast<Shared *>(panel_sm);
  const PanelTask &task = tasks[blockIdx.x];
  const Front &f = task.front;
  const int c0 = pos[task.s];
  int end = f.w;
  bool ok = false;
  if (c0 < f.w) {
    DeviceBlock blk;
    int made = 0;
    end = c0;
    const int singular = panel_own(blk, sh, f, c0, &end, &made);
    if (singular >= 0) {
      if (threadIdx.x == 0) {
        atomicMin(failed, (unsigned long long)(task.first + singular));
        pos[task.s] = f.w;
      }
      end = f.w;
    } else {
      ok = true;
      if (threadIdx.x == 0) twos[task.s] += made;
    }
  }
  // the update tasks (every slot written, so a finished or failed front leaves only empty ones)
  for (int q = threadIdx.x; q < task.nslots; q += blockDim.x) {
    fc::GemmTask g{};
    Tile t;
    if (ok && update_tile(f.m, f.w, end, q, t)) {
      g.C = f.F + t.i0 + (int64_t)t.j0 * f.m;
      g.c_si = 1, g.c_sj = f.m;
      g.A = f.F + t.i0 + (int64_t)c0 * f.m;
      g.a_si = 1, g.a_sk = f.m;
      g.B = f.W + (t.j0 - end);
      g.b_sj = 1, g.b_sk = f.ld_w;
      g.M = t.M, g.N = t.N, g.K = end - c0;
      g.flags = t.lower ? 1 : 0;
    } else {
      g.C = f.F, g.A = f.F, g.B = f.F;
      g.c_si = g.a_si = g.b_sj = 1;
      g.c_sj = g.a_sk = g.b_sk = 1;
    }
    task.slots[q] = g;
  }
  if (threadIdx.x == 0) {
    from[task.s] = ok ? c0 : end;
    if (ok) pos[task.s] = end;
  }
}

// After it: L of the rows below the own columns, and L D of the own rows past the panel (the update's
// coefficients). Eight threads a row, thread t of them the columns t, t + 8, ... in registers: as soon
// as a column's entry is divided the later ones take its product, so a row is a chain of 64 divisions
// and not of 2 000 subtractions, and its entries see panel_below's operations in panel_below's order.
constexpr int BELOW_ROWS = 32, BELOW_THREADS = 8 * BELOW_ROWS, BELOW_HELD = (PANEL + 8) / 8;
__global__ void __launch_bounds__(BELOW_THREADS) ldlt_below_kernel(const PanelTask *__restrict__ tasks,
                                                                   const int32_t *__restrict__ pos,
                                                                   const int32_t *__restrict__ from) {
  __shared__ double coef[PANEL + 1][8 * BELOW_HELD];  // L D at (row j, column q) of the panel's block: [q][j]
  __shared__ double d[PANEL + 1], e[PANEL + 1];
  __shared__ double by[PANEL + 1], inv[PANEL + 1];  // what a pivot's columns are divided by, and its reciprocal
  __shared__ int8_t kind[PANEL + 1];
  const PanelTask &task = tasks[blockIdx.x];
  const Front f = task.front;
  const int c0 = from[task.s], c1 = pos[task.s], kw = c1 - c0;
  const int64_t r0 = c0 + (int64_t)blockIdx.y * BELOW_ROWS;
  if (kw <= 0 || r0 >= f.m || r0 + BELOW_ROWS <= c1) return;
  for (int k = threadIdx.x; k < kw; k += BELOW_THREADS) {
    d[k] = at(f, c0 + k, c0 + k);
    kind[k] = f.pivots[c0 + k];
    e[k] = kind[k] == PIVOT_FIRST ? at(f, c0 + k + 1, c0 + k) : 0.0;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < kw; k += BELOW_THREADS) {
    by[k] = kind[k] == PIVOT_FIRST ? sub(mul(d[k], d[k + 1]), mul(e[k], e[k])) : d[k];
    inv[k] = reciprocal(by[k]);
  }
  const int lane = threadIdx.x & 7;
  const int64_t r = r0 + (threadIdx.x >> 3);
  // times_d for any row past the panel's columns q
  auto product = [&](int64_t row, int q) {
    const double x = at(f, row, c0 + q);
    if (kind[q] == PIVOT_FIRST) return add(mul(x, d[q]), mul(at(f, row, c0 + q + 1), e[q]));
    if (kind[q] == PIVOT_SECOND) return add(mul(at(f, row, c0 + q - 1), e[q - 1]), mul(x, d[q]));
    return mul(x, d[q]);
  };
  if (r >= c1 && r < f.w)
    for (int q = lane; q < kw; q += 8) f.W[(r - c1) + q * f.ld_w] = product(r, q);
  if (r0 + BELOW_ROWS <= f.w || f.m == f.w) return;
  const bool mine = r >= f.w && r < f.m;
  double g[BELOW_HELD];
#pragma unroll
  for (int t = 0; t < BELOW_HELD; ++t) g[t] = mine && 8 * t + lane < kw ? at(f, r, c0 + 8 * t + lane) : 0.0;
  // the panel's block below the pivots (no entry of a 2 x 2 pivot's own is read), six loads at a time
  constexpr int ENTRIES = (PANEL + 1) * 8 * BELOW_HELD, TOGETHER = 6;
  for (int x0 = threadIdx.x; x0 < ENTRIES; x0 += TOGETHER * BELOW_THREADS) {
    double v[TOGETHER];
#pragma unroll
    for (int u = 0; u < TOGETHER; ++u) {
      const int x = x0 + u * BELOW_THREADS, q = x / (8 * BELOW_HELD), j = x % (8 * BELOW_HELD);
      v[u] = j < kw && q < j && !(kind[q] == PIVOT_FIRST && j == q + 1) ? product(c0 + j, q) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < TOGETHER; ++u)
      if (x0 + u * BELOW_THREADS < ENTRIES) (&coef[0][0])[x0 + u * BELOW_THREADS] = v[u];
  }
  __syncthreads();
#pragma unroll
  for (int t = 0; t < BELOW_HELD; ++t) {
    for (int o = 0; o < 8 && 8 * t + o < kw; ++o) {
      const int k = 8 * t + o;
      if (kind[k] == PIVOT_SECOND) continue;
      const double x = __shfl_sync(0xffffffffu, g[t], o, 8);
      if (kind[k] == PIVOT_FIRST) {
        double y = __shfl_sync(0xffffffffu, g[t], (o + 1) & 7, 8);
        if (t + 1 < BELOW_HELD) {
          const double z = __shfl_sync(0xffffffffu, g[t + 1 < BELOW_HELD ? t + 1 : t], 0, 8);
          if (o == 7) y = z;
        }
        const double d11 = d[k], d21 = e[k], d22 = d[k + 1];
        const double l0 = quotient(sub(mul(x, d22), mul(y, d21)), by[k], inv[k]);
        const double l1 = quotient(sub(mul(y, d11), mul(x, d21)), by[k], inv[k]);
#pragma unroll
        for (int u = t; u < BELOW_HELD; ++u) {
          const int j = 8 * u + lane;
          if (j > k + 1) g[u] = sub(sub(g[u], mul(l0, coef[k][j])), mul(l1, coef[k + 1][j]));
          if (j == k) g[u] = l0;
          if (j == k + 1) g[u] = l1;
        }
      } else {
        const double l = quotient(x, by[k], inv[k]);
#pragma unroll
        for (int u = t; u < BELOW_HELD; ++u) {
          const int j = 8 * u + lane;
          if (j > k) g[u] = sub(g[u], mul(l, coef[k][j]));
          if (j == k) g[u] = l;
        }
      }
    }
  }
#pragma unroll
  for (int t = 0; t < BELOW_HELD; ++t)
    if (mine && 8 * t + lane < kw) at(f, r, c0 + 8 * t + lane) = g[t];
}

// front_w21 with an element a thread at a time, eight threads a row (a thread a row, each column's
// loads waiting for the one before: 29 us a launch).
__global__ void __launch_bounds__(8 * W21_ROWS) ldlt_after_kernel(const AfterTask *__restrict__ tasks) {
  const AfterTask &task = tasks[blockIdx.x];
  const Front f = task.front;
  const int64_t r = task.r0 + threadIdx.x % W21_ROWS, ld = f.m - f.w;
  if (r >= task.r1) return;
  double *__restrict__ out = task.w21 + (r - f.w);
#pragma unroll 4
  for (int k = threadIdx.x / W21_ROWS; k < f.w; k += 8) {
    const int8_t kind = f.pivots[k];
    const double x = at(f, r, k), d = at(f, k, k);
    double v = mul(x, d);
    if (kind == PIVOT_FIRST) v = add(v, mul(at(f, r, k + 1), at(f, k + 1, k)));
    if (kind == PIVOT_SECOND) v = add(mul(at(f, r, k - 1), at(f, k, k - 1)), v);
    out[k * ld] = v;
  }
}

// y <- D^-1 y between the solve's forward and backward passes: n unknowns in postorder, R
// right-hand sides row-major; one thread per unknown (the second column of a 2 x 2 pivot idles).
__global__ void ldlt_d_inverse_kernel(int64_t n, int R, const double *__restrict__ d, const double *__restrict__ e,
                                      const int8_t *__restrict__ pivots, double *__restrict__ y) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    apply_d_inverse(i, R, d, e, pivots, y);
}

// Lower.scale (cholesky.rs:1392-1416): each entry's magnitude to its row's and its column's
// largest, as the bits of non-negative doubles (ordered as integers); a NaN changes nothing, as
// in f64::max. scale_bits starts at zero.
__global__ void ldlt_scale_kernel(int64_t nnz, const int64_t *__restrict__ a_src, const int32_t *__restrict__ a_row,
                                  const int32_t *__restrict__ a_col, const double *__restrict__ val,
                                  unsigned long long *__restrict__ scale_bits) {
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < nnz; q += (int64_t)gridDim.x * blockDim.x) {
    const double v = fabs(val[a_src[q]]);
    if (isnan(v)) continue;
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    atomicMax(scale_bits + a_row[q], b);
    atomicMax(scale_bits + a_col[q], b);
  }
}

// Each supernode's pivots start as its columns in order, every one a 1 x 1 pivot.
__global__ void ldlt_reset_kernel(int64_t n, const int32_t *__restrict__ local, int32_t *__restrict__ order,
                                  int8_t *__restrict__ pivots) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    order[i] = local[i];
    pivots[i] = PIVOT_ONE;
  }
}

// D out of a block of columns, then the inverse of its unit lower diagonal block, both sides in
// shared memory, a step of the substitution a pass over them (one thread a column of global memory
// took 43 us a launch, this 28 with the split).
constexpr int INVERSE_THREADS = 256, INVERSE_LD = PANEL + 1;
__global__ void __launch_bounds__(INVERSE_THREADS) ldlt_inverse_kernel(const InverseTask *__restrict__ tasks) {
  extern __shared__ double sm[];
  double *L = sm, *X = sm + PANEL * INVERSE_LD;
  const InverseTask &t = tasks[blockIdx.x];
  const Front &f = t.front;
  DeviceBlock blk;
  split_d(blk, f, t.d, t.e, t.c0, t.c0 + t.nb);
  for (int e = threadIdx.x; e < PANEL * t.nb; e += blockDim.x) {
    const int i = e % PANEL, j = e / PANEL;
    if (i < t.nb) L[i + j * INVERSE_LD] = i > j ? at(f, t.c0 + i, t.c0 + j) : 0.0;
  }
  __syncthreads();
  unit_lower_inverse(blk, L, INVERSE_LD, t.nb, X, INVERSE_LD);
  for (int e = threadIdx.x; e < PANEL * t.nb; e += blockDim.x) {
    const int i = e % PANEL, j = e / PANEL;
    if (i >= j && i < t.nb) t.X[i + (int64_t)j * t.ldx] = X[i + j * INVERSE_LD];
  }
}

__global__ void ldlt_fold_kernel(int64_t n, const int32_t *__restrict__ local, const int32_t *__restrict__ order,
                                 const int64_t *__restrict__ perm, int32_t *__restrict__ own,
                                 int64_t *__restrict__ perm_out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t j = i - local[i] + order[i];  // the column at pivot position i
    own[j] = (int32_t)i;
    perm_out[i] = perm[j];
  }
}
__global__ void ldlt_rows_kernel(int64_t count, const int32_t *__restrict__ rows, const int32_t *__restrict__ own,
                                 int32_t *__restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = own[rows[i]];
}

namespace {
int grid_for(int64_t count, int threads) {
  const int64_t blocks = (count + threads - 1) / threads;
  return (int)(blocks < 4096 ? (blocks > 0 ? blocks : 1) : 4096);
}
}  // namespace

void launch_inverse(const InverseTask *tasks, int count, cudaStream_t st) {
  constexpr size_t smem = sizeof(double) * 2 * PANEL * INVERSE_LD;
  if (count <= 0) return;
  cudaFuncSetAttribute(ldlt_inverse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  ldlt_inverse_kernel<<<count, INVERSE_THREADS, smem, st>>>(tasks);
}

void launch_fold(int64_t n, const int32_t *local, const int32_t *order, const int64_t *perm, int32_t *own,
                 int64_t *perm_out, int64_t rows_len, const int32_t *rows, int32_t *rows_out, cudaStream_t st) {
  if (n > 0) ldlt_fold_kernel<<<grid_for(n, 256), 256, 0, st>>>(n, local, order, perm, own, perm_out);
  if (rows_len > 0) ldlt_rows_kernel<<<grid_for(rows_len, 256), 256, 0, st>>>(rows_len, rows, own, rows_out);
}

// A thread an own row up to 512: a column step is a chain of loads and barriers, bound by their
// latency, and the rows below would make it longer (they are most of a front's rows, and a CTA has one
// SM's FP64 units): they come after it, all of a level's together. Panels of 16 x 14 x 13 elements:
// 12.1 ms on all rows with each column formed when it is looked at (3.3 us a column on the longest
// chain); 7.5 and 2.3 for the rows below with eight columns held ahead; 5.2 and 1.5 with their
// coefficients side by side and zeros kept from the division's slow way.
void launch_panel(const PanelTask *tasks, int count, int tallest, int widest, int32_t *pos, int32_t *from,
                  int32_t *twos, unsigned long long *failed, cudaStream_t st) {
  if (count <= 0) return;
  const int threads = widest >= PANEL_THREADS ? PANEL_THREADS : widest <= 64 ? 64 : (widest + 31) / 32 * 32;
  cudaFuncSetAttribute(ldlt_panel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Shared));
  ldlt_panel_kernel<<<count, threads, sizeof(Shared), st>>>(tasks, pos, from, twos, failed);
  const dim3 grid(count, (tallest + BELOW_ROWS - 1) / BELOW_ROWS);
  ldlt_below_kernel<<<grid, BELOW_THREADS, 0, st>>>(tasks, pos, from);
}

void launch_after(const AfterTask *tasks, int count, cudaStream_t st) {
  if (count > 0) ldlt_after_kernel<<<count, 8 * W21_ROWS, 0, st>>>(tasks);
}

void launch_scale(int64_t nnz, const int64_t *a_src, const int32_t *a_row, const int32_t *a_col, const double *val,
                  unsigned long long *scale_bits, cudaStream_t st) {
  if (nnz > 0) ldlt_scale_kernel<<<grid_for(nnz, 256), 256, 0, st>>>(nnz, a_src, a_row, a_col, val, scale_bits);
}

void launch_reset(int64_t n, const int32_t *local, int32_t *order, int8_t *pivots, cudaStream_t st) {
  if (n > 0) ldlt_reset_kernel<<<grid_for(n, 256), 256, 0, st>>>(n, local, order, pivots);
}

void launch_d_inverse(int64_t n, int R, const double *d, const double *e, const int8_t *pivots, double *y,
                      cudaStream_t st) {
  if (n > 0) ldlt_d_inverse_kernel<<<grid_for(n, 256), 256, 0, st>>>(n, R, d, e, pivots, y);
}

}  // namespace ldlt
}  // namespace fc
