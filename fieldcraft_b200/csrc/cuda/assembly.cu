// K_ff of a structured hex8 box assembled on the device (include/fieldcraft_fem.h): the element
// matrices (host/hex8.hpp's operations, 36 threads an element), then every entry as the sum over
// the elements holding both its nodes in element label order (host/assembly.hpp's order, a warp per
// row), the host builder's operations in its order, so the values are its bits. After the solve:
// the motion of every DOF, the reactions at the held ones, and the stresses (host/stress.hpp).
#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/fieldcraft_fem.h"
#include "device_buf.hpp"
#include "host/assembly.hpp"
#include "host/stress.hpp"

struct fc_fem_device {
  fc::assembly::Box box{};
  int64_t n = 0, nnz = 0, elements = 0;
  int device = 0;
  int64_t dofs = 0;  // 3 nodes
  int64_t held = 0;  // DOFs without an equation
  fc::host::DeviceBuf d_ptr, d_idx, d_node, d_eq, d_ke, d_bad;
  fc::host::DeviceBuf d_held;    // their DOF indices
  fc::host::DeviceBuf d_corner;  // stress recovery: each element's corner values (48 doubles)
};

namespace {

using fc::hex8::add;
using fc::hex8::mul;
using fc::hex8::sub;

__constant__ double CORNER[8][3] = {{-1, -1, -1}, {1, -1, -1}, {1, 1, -1}, {-1, 1, -1},
                                    {-1, -1, 1},  {1, -1, 1},  {1, 1, 1},  {-1, 1, 1}};
__constant__ int OFFSET[8][3] = {{0, 0, 0}, {1, 0, 0}, {1, 1, 0}, {0, 1, 0},
                                 {0, 0, 1}, {1, 0, 1}, {1, 1, 1}, {0, 1, 1}};
// the corner pairs i <= j of an element matrix's upper blocks
__constant__ unsigned char PAIR_I[36] = {0, 0, 1, 0, 1, 2, 0, 1, 2, 3, 0, 1, 2, 3, 4, 0, 1, 2,
                                         3, 4, 5, 0, 1, 2, 3, 4, 5, 6, 0, 1, 2, 3, 4, 5, 6, 7};
__constant__ unsigned char PAIR_J[36] = {0, 1, 1, 2, 2, 2, 3, 3, 3, 3, 4, 4, 4, 4, 4, 5, 5, 5,
                                         5, 5, 5, 6, 6, 6, 6, 6, 6, 6, 7, 7, 7, 7, 7, 7, 7, 7};

// The gradients dx[8][3] of element e's shape functions at Gauss point p (xi fastest) and the
// Jacobian's determinant, with hex8::stiffness's and stress::element_stresses's operations in
// their order. False for a Jacobian out of range.
__device__ __forceinline__ bool gauss_gradients(const fc::assembly::Box &box, int64_t e, int p, double (*dx)[3],
                                                double &det) {
  const double gauss = 0.5773502691896258;
  const double xi0 = p & 1 ? gauss : -gauss, xi1 = p & 2 ? gauss : -gauss, xi2 = p & 4 ? gauss : -gauss;
  const int64_t ex = e % box.nx, ey = (e / box.nx) % box.ny, ez = e / ((int64_t)box.nx * box.ny);
  // a corner's coordinates are those of its planes: two per axis
  double px[2], py[2], pz[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    px[q] = mul(box.lx, (double)(ex + q)) / (double)box.nx;
    py[q] = mul(box.ly, (double)(ey + q)) / (double)box.ny;
    pz[q] = mul(box.lz, (double)(ez + q)) / (double)box.nz;
  }
  double dn[8][3], jm[3][3] = {};
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int ox = (i & 3) == 1 || (i & 3) == 2, oy = (i & 3) >= 2, oz = i >> 2;
    const double c0 = ox ? 1.0 : -1.0, c1 = oy ? 1.0 : -1.0, c2 = oz ? 1.0 : -1.0;
    const double f0 = add(1.0, mul(xi0, c0)), f1 = add(1.0, mul(xi1, c1)), f2 = add(1.0, mul(xi2, c2));
    dn[i][0] = mul(mul(mul(c0, f1), f2), 0.125);  // a division by 8 is exact either way
    dn[i][1] = mul(mul(mul(c1, f0), f2), 0.125);
    dn[i][2] = mul(mul(mul(c2, f0), f1), 0.125);
    const double x[3] = {px[ox], py[oy], pz[oz]};
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) jm[a][b] = add(jm[a][b], mul(dn[i][a], x[b]));
  }
  const double t1 = mul(jm[0][0], sub(mul(jm[1][1], jm[2][2]), mul(jm[1][2], jm[2][1])));
  const double t2 = mul(jm[0][1], sub(mul(jm[1][0], jm[2][2]), mul(jm[1][2], jm[2][0])));
  const double t3 = mul(jm[0][2], sub(mul(jm[1][0], jm[2][1]), mul(jm[1][1], jm[2][0])));
  det = add(sub(t1, t2), t3);
  if (!(det > 0.0) || !isfinite(det)) return false;
  double inv[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int j1 = (j + 1) % 3, j2 = (j + 2) % 3, i1 = (i + 1) % 3, i2 = (i + 2) % 3;
      inv[i][j] = sub(mul(jm[j1][i1], jm[j2][i2]), mul(jm[j1][i2], jm[j2][i1])) / det;
    }
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int b = 0; b < 3; ++b)
      dx[i][b] = add(add(mul(inv[b][0], dn[i][0]), mul(inv[b][1], dn[i][1])), mul(inv[b][2], dn[i][2]));
  return true;
}

// One Gauss point's term of the 3 x 3 block (i, j) with every product of hex8::stiffness, the
// zeros of B and D included (an infinite modulus or gradient makes them NaN there too).
__device__ __noinline__ void dense_block(double lambda, double mu, const double *gi, const double *gj, double w,
                                         double (&k)[3][3]) {
  const double dd = add(lambda, mul(2.0, mu));
  auto D = [&](int s, int t) { return s < 3 && t < 3 ? (s == t ? dd : lambda) : (s == t ? mu : 0.0); };
  auto B = [](const double *g, int s, int c) {
    const int a = s == 5 ? 1 : 0, b = s == 3 ? 1 : 2;  // shear row s joins directions a and b
    return s < 3 ? (s == c ? g[c] : 0.0) : (c == a ? g[b] : c == b ? g[a] : 0.0);
  };
  for (int c = 0; c < 3; ++c) {
    double db[6];
    for (int s = 0; s < 6; ++s) {
      double acc = 0.0;
      for (int t = 0; t < 6; ++t) acc = add(acc, mul(D(s, t), B(gj, t, c)));
      db[s] = acc;
    }
    for (int r = 0; r < 3; ++r) {
      double acc = 0.0;
      for (int s = 0; s < 6; ++s) acc = add(acc, mul(B(gi, s, r), db[s]));
      k[r][c] = add(k[r][c], mul(w, acc));
    }
  }
}

// The element matrices, ELEMENTS to a block: 8 threads an element form the gradients at its Gauss
// points in shared memory, then 36 threads an element its 3 x 3 upper blocks in registers, point by
// point, and each block goes with its mirror image to the matrix in shared memory, which is stored
// as it lies. The terms with a structural zero of B or D add exactly nothing while everything is
// finite and are left out; an element whose D or gradients are not finite takes them all
// (dense_block). Bound by FP64 arithmetic and the 4.6 KB an element stores: 0.19 ms for 48 x 40 x 36
// elements (318 MB, 1.7 TB/s) with four blocks an SM, one's gradients beside another's products (0.28
// with two at the compiler's 128 registers a thread, 0.22 with three; five spill: 0.21). With
// entry_kernel and the kernels below, K, reactions and stresses of that box take 0.59 ms; with one
// thread an element, a row, a DOF and an element each, their matrices accumulated in global memory,
// they took 6.1 ms.
constexpr int ELEMENTS = 6, ELEMENT_THREADS = 36 * ELEMENTS;

__global__ void __launch_bounds__(ELEMENT_THREADS, 4) element_kernel(fc::assembly::Box box, int64_t elements,
                                                                  const double *__restrict__ young, double nu,
                                                                  double *__restrict__ ke, int *__restrict__ bad) {
  __shared__ double grad[ELEMENTS][8][8][3];
  __shared__ double2 whole[ELEMENTS * 288];
  __shared__ double weight[ELEMENTS][8];
  __shared__ double lame[ELEMENTS][2];
  __shared__ int dense[ELEMENTS];
  const int tid = threadIdx.x, el = tid / 36, pair = tid % 36, i = PAIR_I[pair], j = PAIR_J[pair];
  for (int64_t e0 = (int64_t)blockIdx.x * ELEMENTS; e0 < elements; e0 += (int64_t)gridDim.x * ELEMENTS) {
    __syncthreads();
    if (tid < ELEMENTS) {
      const double e = e0 + tid < elements ? young[e0 + tid] : 1.0;
      const bool ok = e > 0.0 && nu > -1.0 && nu < 0.5;
      lame[tid][0] = mul(e, nu) / mul(add(1.0, nu), sub(1.0, mul(2.0, nu)));
      lame[tid][1] = e / mul(2.0, add(1.0, nu));
      dense[tid] = 0;
      if (!ok) atomicExch(bad, 1);
    }
    __syncthreads();
    if (tid < 8 * ELEMENTS && e0 + tid / 8 < elements) {
      const int q = tid / 8, p = tid % 8;
      double dx[8][3], det;
      if (gauss_gradients(box, e0 + q, p, dx, det)) {
        const double dd = add(lame[q][0], mul(2.0, lame[q][1]));
        double sum = 0.0;
#pragma unroll
        for (int a = 0; a < 8; ++a)
#pragma unroll
          for (int b = 0; b < 3; ++b) {
            grad[q][p][a][b] = dx[a][b];
            sum = add(sum, fabs(dx[a][b]));  // at least the largest: a product of D with any is below dd * sum
          }
        weight[q][p] = det;
        if (!isfinite(mul(add(dd, fabs(lame[q][0])), sum))) dense[q] = 1;
      } else {
        atomicExch(bad, 1);
      }
    }
    __syncthreads();
    const double lambda = lame[el][0], mu = lame[el][1], dd = add(lambda, mul(2.0, mu));
    double k[3][3] = {};
    if (dense[el]) {
      double kd[3][3] = {};  // apart from k, which stays in registers
      for (int p = 0; p < 8; ++p) dense_block(lambda, mu, grad[el][p][i], grad[el][p][j], weight[el][p], kd);
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) k[r][c] = kd[r][c];
    } else {
#pragma unroll 2
      for (int p = 0; p < 8; ++p) {
        const double *gi = grad[el][p][i], *gj = grad[el][p][j];
        const double w = weight[el][p];
        const double a0 = gi[0], a1 = gi[1], a2 = gi[2], b0 = gj[0], b1 = gj[1], b2 = gj[2];
        const double l0 = mul(lambda, b0), l1 = mul(lambda, b1), l2 = mul(lambda, b2);
        const double m0 = mul(mu, b0), m1 = mul(mu, b1), m2 = mul(mu, b2);
        k[0][0] = add(k[0][0], mul(w, add(add(mul(a0, mul(dd, b0)), mul(a1, m1)), mul(a2, m2))));
        k[0][1] = add(k[0][1], mul(w, add(mul(a0, l1), mul(a1, m0))));
        k[0][2] = add(k[0][2], mul(w, add(mul(a0, l2), mul(a2, m0))));
        k[1][0] = add(k[1][0], mul(w, add(mul(a1, l0), mul(a0, m1))));
        k[1][1] = add(k[1][1], mul(w, add(add(mul(a1, mul(dd, b1)), mul(a0, m0)), mul(a2, m2))));
        k[1][2] = add(k[1][2], mul(w, add(mul(a1, l2), mul(a2, m1))));
        k[2][0] = add(k[2][0], mul(w, add(mul(a2, l0), mul(a0, m2))));
        k[2][1] = add(k[2][1], mul(w, add(mul(a2, l1), mul(a1, m2))));
        k[2][2] = add(k[2][2], mul(w, add(add(mul(a2, mul(dd, b2)), mul(a0, m0)), mul(a1, m1))));
      }
    }
    if (i == j) k[1][0] = k[0][1], k[2][0] = k[0][2], k[2][1] = k[1][2];  // the upper half, mirrored
    double *out = reinterpret_cast<double *>(whole) + el * 576;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        out[(3 * i + r) * 24 + 3 * j + c] = k[r][c];
        if (i != j) out[(3 * j + c) * 24 + 3 * i + r] = k[r][c];
      }
    __syncthreads();
    double2 *dst = reinterpret_cast<double2 *>(ke + e0 * 576);
    const int count = 288 * (int)min((int64_t)ELEMENTS, elements - e0);
    for (int q = tid; q < count; q += ELEMENT_THREADS) dst[q] = whole[q];
  }
}

// Entry (v, a; w, c) over the nodes' grid positions: assembly::entry's terms in its order, loaded
// together (at most two elements an axis hold both nodes; a term that is not there adds zero,
// which changes no sum that started from +0).
__device__ __forceinline__ double grid_entry(const fc::assembly::Box &box, int4 v, int a, int4 w, int c,
                                             const double *__restrict__ ke) {
  const int mx = max(v.x, w.x) - 1, my = max(v.y, w.y) - 1, mz = max(v.z, w.z) - 1;
  const int hx = min(min(v.x, w.x), box.nx - 1), hy = min(min(v.y, w.y), box.ny - 1),
            hz = min(min(v.z, w.z), box.nz - 1);
  double t[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int ex = mx + (q & 1), ey = my + (q >> 1 & 1), ez = mz + (q >> 2);
    t[q] = 0.0;
    if (ex >= 0 && ex <= hx && ey >= 0 && ey <= hy && ez >= 0 && ez <= hz) {
      const int64_t e = ex + box.nx * (ey + (int64_t)box.ny * ez);
      auto corner = [](int dx, int dy, int dz) { return 4 * dz + (dy ? 3 - dx : dx); };  // assembly::corner_of
      const int i = corner(v.x - ex, v.y - ey, v.z - ez), j = corner(w.x - ex, w.y - ey, w.z - ez);
      t[q] = ke[e * 576 + (3 * i + a) * 24 + 3 * j + c];
    }
  }
  double acc = 0.0;
#pragma unroll
  for (int q = 0; q < 8; ++q) acc = add(acc, t[q]);
  return acc;
}

// K's values, a warp per row, a lane per entry: a row's entries and the rows of the element
// matrices that they add up are contiguous, so both stream through whole sectors (0.23 ms for the
// 16.7 M entries of that box; one thread a row walked its entries alone, a sector for each).
__global__ void __launch_bounds__(256) entry_kernel(fc::assembly::Box box, int64_t n, const int64_t *__restrict__ ptr,
                                                    const int32_t *__restrict__ idx, const int4 *__restrict__ node,
                                                    const double *__restrict__ ke, double *__restrict__ val) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x / 32);
  for (int64_t r = blockIdx.x * (int64_t)(blockDim.x / 32) + threadIdx.x / 32; r < n; r += warps) {
    const int4 v = node[r / 3];
    const int a = (int)(r % 3);
    const int64_t q1 = ptr[r + 1];
    for (int64_t q = ptr[r] + lane; q < q1; q += 32) {
      const int32_t col = idx[q];
      val[q] = grid_entry(box, v, a, node[col / 3], col % 3, ke);
    }
  }
}

// The motion over every DOF, and the reactions' zeros at the free ones, one thread per DOF.
__global__ void motion_kernel(int64_t dofs, const int64_t *__restrict__ eq, const double *__restrict__ q,
                              double *__restrict__ r, double *__restrict__ u) {
  for (int64_t d = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; d < dofs; d += (int64_t)gridDim.x * blockDim.x) {
    const int64_t e = eq[d];
    if (u) u[d] = e >= 0 ? q[e] : 0.0;
    if (r && e >= 0) r[d] = 0.0;
  }
}

// The reactions at the held DOFs, a warp each (assembly::reaction): the lanes form the products of
// the row's at most 81 entries with the motion, then add them one by one in column order (an
// entry past the box's faces adds +0, which changes no sum that started from +0).
__global__ void __launch_bounds__(128) reaction_kernel(fc::assembly::Box box, int64_t held,
                                                       const int64_t *__restrict__ held_dofs,
                                                       const int64_t *__restrict__ eq, const double *__restrict__ q,
                                                       const double *__restrict__ f, const double *__restrict__ ke,
                                                       double *__restrict__ r) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x / 32);
  const int64_t px = box.nx + 1, py = box.ny + 1;
  for (int64_t h = blockIdx.x * (int64_t)(blockDim.x / 32) + threadIdx.x / 32; h < held; h += warps) {
    const int64_t d = held_dofs[h], v = d / 3;
    const int4 at = make_int4((int)(v % px), (int)((v / px) % py), (int)(v / (px * py)), 0);
    double t[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int s = lane + 32 * k, c = s % 3, o = s / 3;
      const int4 w = make_int4(at.x + o % 3 - 1, at.y + o / 3 % 3 - 1, at.z + o / 9 - 1, 0);
      if (s < 81 && w.x >= 0 && w.y >= 0 && w.z >= 0 && w.x <= box.nx && w.y <= box.ny && w.z <= box.nz)
        t[k] = mul(grid_entry(box, at, (int)(d % 3), w, c, ke),
                   fc::assembly::expanded(eq, q, 3 * (w.x + px * (w.y + py * (int64_t)w.z)) + c));
    }
    double ku = 0.0;
    for (int s = 0; s < 81; ++s) ku = add(ku, __shfl_sync(0xffffffffu, s < 32 ? t[0] : s < 64 ? t[1] : t[2], s & 31));
    if (lane == 0) r[d] = sub(ku, f ? f[d] : 0.0);
  }
}

// Stress recovery, 8 threads an element (stress::element_stresses's operations): thread p takes
// Gauss point p, leaves its stress in shared memory, then extrapolates to corner p; the points and
// the corners store 48 contiguous values an element. (One thread an element kept its 144 values in
// local memory and stored each with a stride of 384 bytes.)
constexpr int STRESS_ELEMENTS = 16;
__global__ void __launch_bounds__(8 * STRESS_ELEMENTS)
    stress_element_kernel(fc::assembly::Box box, int64_t elements, const double *__restrict__ young, double nu,
                          const double *__restrict__ u, double *__restrict__ points, double *__restrict__ corner,
                          int *__restrict__ bad) {
  __shared__ double ue[STRESS_ELEMENTS][24];
  __shared__ double sg[STRESS_ELEMENTS][8][6];
  const int64_t px = box.nx + 1, py = box.ny + 1;
  const int el = threadIdx.x / 8, p = threadIdx.x % 8;
  for (int64_t e0 = (int64_t)blockIdx.x * STRESS_ELEMENTS; e0 < elements; e0 += (int64_t)gridDim.x * STRESS_ELEMENTS) {
    const int64_t e = e0 + el;
    const bool on = e < elements;
    __syncthreads();
    if (on) {
      const int64_t ex = e % box.nx, ey = (e / box.nx) % box.ny, ez = e / ((int64_t)box.nx * box.ny);
      const int64_t v = (ex + OFFSET[p][0]) + px * ((ey + OFFSET[p][1]) + py * (ez + OFFSET[p][2]));
      for (int a = 0; a < 3; ++a) ue[el][3 * p + a] = u[3 * v + a];
    }
    __syncthreads();
    if (on) {
      const double E = young[e];
      double dx[8][3], det;
      if (!(E > 0.0) || !(nu > -1.0 && nu < 0.5) || !gauss_gradients(box, e, p, dx, det)) {
        atomicExch(bad, 1);
        for (int s = 0; s < 6; ++s) sg[el][p][s] = 0.0;
      } else {
        const double lambda = mul(E, nu) / mul(add(1.0, nu), sub(1.0, mul(2.0, nu)));
        const double mu = E / mul(2.0, add(1.0, nu)), dd = add(lambda, mul(2.0, mu));
        double grad[3][3] = {};
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int b = 0; b < 3; ++b) grad[c][b] = add(grad[c][b], mul(ue[el][3 * i + c], dx[i][b]));
        const double strain[6] = {grad[0][0], grad[1][1], grad[2][2], add(grad[0][1], grad[1][0]),
                                  add(grad[0][2], grad[2][0]), add(grad[1][2], grad[2][1])};
#pragma unroll
        for (int s = 0; s < 6; ++s) {
          double acc = 0.0;
#pragma unroll
          for (int t = 0; t < 6; ++t)
            acc = add(acc, mul(s < 3 && t < 3 ? (s == t ? dd : lambda) : (s == t ? mu : 0.0), strain[t]));
          sg[el][p][s] = acc;
          if (points) points[e * 48 + 6 * p + s] = acc;
        }
      }
    }
    __syncthreads();
    if (on) {
      const double r3 = 1.7320508075688772;
      double v[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        double w = 1.0;
#pragma unroll
        for (int a = 0; a < 3; ++a) w = mul(w, add(1.0, mul(mul(r3, CORNER[p][a]), CORNER[q][a])));
        w = mul(w, 0.125);  // a division by 8 is exact either way
#pragma unroll
        for (int s = 0; s < 6; ++s) v[s] = add(v[s], mul(w, sg[el][q][s]));
      }
#pragma unroll
      for (int s = 0; s < 6; ++s) corner[e * 48 + 6 * p + s] = v[s];
    }
  }
}

__global__ void stress_node_kernel(fc::assembly::Box box, int64_t nodes, const double *__restrict__ corner,
                                   double *__restrict__ nodal, double *__restrict__ von_mises) {
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < nodes; v += (int64_t)gridDim.x * blockDim.x) {
    double s[6];
    fc::stress::nodal_mean(box, v, corner, s);
    if (nodal)
      for (int k = 0; k < 6; ++k) nodal[v * 6 + k] = s[k];
    if (von_mises) von_mises[v] = fc::stress::von_mises(s);
  }
}

// Blocks for `count` items of which one block takes `per` at a time.
int blocks_for(int64_t count, int per = 128) {
  const int64_t b = (count + per - 1) / per;
  return (int)(b < 8192 ? (b > 0 ? b : 1) : 8192);
}

}  // namespace

extern "C" {

int fc_fem_device_create(int nx, int ny, int nz, double lx, double ly, double lz, int64_t n, const int64_t *ptr,
                         const int32_t *idx, const int64_t *eq, int device, fc_fem_device **out) {
  if (!out || nx <= 0 || ny <= 0 || nz <= 0 || n < 0 || n % 3 != 0 || (n > 0 && (!ptr || !idx || !eq)) ||
      !(lx > 0 && ly > 0 && lz > 0))
    return FC_FEM_INVALID;
  *out = nullptr;
  if (cudaSetDevice(device) != cudaSuccess) return FC_FEM_INVALID;
  auto d = new fc_fem_device();
  d->box = {nx, ny, nz, lx, ly, lz};
  d->n = n;
  d->nnz = n > 0 ? ptr[n] : 0;
  d->elements = (int64_t)nx * ny * nz;
  d->device = device;
  const int64_t nodes = (int64_t)(nx + 1) * (ny + 1) * (nz + 1);
  d->dofs = 3 * nodes;
  std::vector<int64_t> heq(eq, eq + 3 * nodes);
  std::vector<int4> node(n / 3, make_int4(-1, -1, -1, 0));  // each free node's place in the grid
  std::vector<int64_t> held, hptr(ptr, ptr + n + 1);
  std::vector<int32_t> hidx(idx, idx + d->nnz);
  bool ok = true;
  for (int64_t v = 0; v < nodes && ok; ++v) {
    const int64_t e = eq[3 * v];
    if (e < 0) continue;
    if (e % 3 != 0 || e / 3 >= n / 3 || eq[3 * v + 1] != e + 1 || eq[3 * v + 2] != e + 2) ok = false;
    else node[e / 3] = make_int4((int)(v % (nx + 1)), (int)(v / (nx + 1) % (ny + 1)),
                                 (int)(v / ((int64_t)(nx + 1) * (ny + 1))), 0);
  }
  for (int64_t k = 0; k < n / 3 && ok; ++k) ok = node[k].x >= 0;
  for (int64_t q = 0; q < d->dofs; ++q)
    if (eq[q] < 0) held.push_back(q);
  d->held = (int64_t)held.size();
  for (int64_t q = 0; q < d->nnz && ok; ++q) ok = hidx[q] >= 0 && hidx[q] < n;
  if (!ok) {
    delete d;
    return FC_FEM_INVALID;
  }
  cudaStream_t st = nullptr;
  if (fc::host::upload(d->d_ptr, hptr, st) != cudaSuccess || fc::host::upload(d->d_idx, hidx, st) != cudaSuccess ||
      fc::host::upload(d->d_node, node, st) != cudaSuccess || fc::host::upload(d->d_eq, heq, st) != cudaSuccess ||
      fc::host::upload(d->d_held, held, st) != cudaSuccess ||
      d->d_ke.alloc(sizeof(double) * 576 * (size_t)d->elements) != cudaSuccess ||
      d->d_bad.alloc(sizeof(int)) != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess) {
    delete d;
    return FC_FEM_NOMEM;
  }
  *out = d;
  return FC_FEM_OK;
}

int fc_fem_assemble_device(fc_fem_device *d, const double *d_young, double poisson, double *d_val, void *stream) {
  if (!d || !d_young || (d->nnz > 0 && !d_val)) return FC_FEM_INVALID;
  cudaSetDevice(d->device);
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaMemsetAsync(d->d_bad.p, 0, sizeof(int), st);
  element_kernel<<<blocks_for(d->elements, ELEMENTS), ELEMENT_THREADS, 0, st>>>(
      d->box, d->elements, d_young, poisson, d->d_ke.as<double>(), d->d_bad.as<int>());
  if (d->n > 0)
    entry_kernel<<<blocks_for(d->n, 8), 256, 0, st>>>(d->box, d->n, d->d_ptr.as<int64_t>(), d->d_idx.as<int32_t>(),
                                                      d->d_node.as<int4>(), d->d_ke.as<double>(), d_val);
  int bad = 0;
  if (cudaMemcpyAsync(&bad, d->d_bad.p, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess || cudaGetLastError() != cudaSuccess)
    return FC_FEM_INVALID;
  return bad ? FC_FEM_INVALID : FC_FEM_OK;
}

int fc_fem_reactions_device(fc_fem_device *d, const double *d_q, const double *d_f, double *d_r, double *d_u,
                            void *stream) {
  if (!d || (d->n > 0 && !d_q) || (!d_r && !d_u)) return FC_FEM_INVALID;
  cudaSetDevice(d->device);
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  motion_kernel<<<blocks_for(d->dofs), 128, 0, st>>>(d->dofs, d->d_eq.as<int64_t>(), d_q, d_r, d_u);
  if (d_r && d->held > 0)
    reaction_kernel<<<blocks_for(d->held, 4), 128, 0, st>>>(d->box, d->held, d->d_held.as<int64_t>(),
                                                            d->d_eq.as<int64_t>(), d_q, d_f, d->d_ke.as<double>(), d_r);
  return cudaStreamSynchronize(st) == cudaSuccess && cudaGetLastError() == cudaSuccess ? FC_FEM_OK : FC_FEM_INVALID;
}

int fc_fem_stresses_device(fc_fem_device *d, const double *d_young, double poisson, const double *d_u,
                           double *d_points, double *d_nodal, double *d_von_mises, void *stream) {
  if (!d || !d_young || !d_u) return FC_FEM_INVALID;
  cudaSetDevice(d->device);
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (!d->d_corner.p && d->d_corner.alloc(sizeof(double) * 48 * (size_t)d->elements) != cudaSuccess)
    return FC_FEM_NOMEM;
  cudaMemsetAsync(d->d_bad.p, 0, sizeof(int), st);
  stress_element_kernel<<<blocks_for(d->elements, STRESS_ELEMENTS), 8 * STRESS_ELEMENTS, 0, st>>>(
      d->box, d->elements, d_young, poisson, d_u, d_points, d->d_corner.as<double>(), d->d_bad.as<int>());
  stress_node_kernel<<<blocks_for(d->dofs / 3), 128, 0, st>>>(d->box, d->dofs / 3, d->d_corner.as<double>(), d_nodal,
                                                               d_von_mises);
  int bad = 0;
  if (cudaMemcpyAsync(&bad, d->d_bad.p, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess || cudaGetLastError() != cudaSuccess)
    return FC_FEM_INVALID;
  return bad ? FC_FEM_INVALID : FC_FEM_OK;
}

void fc_fem_device_free(fc_fem_device *d) {
  if (!d) return;
  cudaSetDevice(d->device);
  delete d;
}

}  // extern "C"
