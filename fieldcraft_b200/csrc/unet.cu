// The learned preconditioner's network (forward, backward, Adam) and flexible CG, behind the C ABI
// of include/fieldcraft_unet.h. The network's layers run on this library's own kernels
// (cuda/unet_kernels.cu); this file holds its buffers and the order of the passes.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <mutex>
#include <random>
#include <string>
#include <vector>

#include "../../include/fieldcraft_unet.h"
#include "cuda/kernels.cuh"
#include "cuda/unet_kernels.cuh"
#include "device_buf.hpp"
#include "host/pass_room.hpp"
#include "scratch.hpp"

using fc::host::DeviceBuf;
using fc::host::set_status;
using fc::unet::Grid;
using bf16 = __nv_bfloat16;

namespace {

constexpr int C = 32, CIO = 16;
constexpr int MAX_LEVELS = 8;
constexpr int MAX_LAYERS = 4 * MAX_LEVELS - 1;

__global__ void f32_to_bf16_kernel(int64_t n, const float *__restrict__ a, bf16 *__restrict__ b) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    b[i] = __float2bfloat16_rn(a[i]);
}
__global__ void bf16_to_f32_kernel(int64_t n, const bf16 *__restrict__ a, float *__restrict__ b) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    b[i] = __bfloat162float(a[i]);
}
// The vectors of a group of pairs: blockIdx.y is the pair, its column `ld` past the last.
// d = z - e
__global__ void sub_kernel(int64_t n, const double *__restrict__ z, const double *__restrict__ e, int64_t ld,
                           double *__restrict__ d) {
  z += blockIdx.y * n, d += blockIdx.y * n, e += blockIdx.y * ld;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    d[i] = z[i] - e[i];
}
// d *= 2 / den; loss = num / den (num, den = d.d, e.e, or d.Kd, e.r in the energy norm); the
// pairs' losses are added in order onto *loss (onto zero for the first of all)
__global__ void loss_grad_kernel(int64_t n, const double *__restrict__ num, const double *__restrict__ den,
                                 double *__restrict__ d, double *loss, int first) {
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && loss) {
    double sum = first ? 0.0 : *loss;
    for (int q = 0; q < (int)gridDim.y; ++q) sum += num[q] / (den[q] > 0.0 ? den[q] : 1.0);
    *loss = sum;
  }
  const double ee = den[blockIdx.y] > 0.0 ? den[blockIdx.y] : 1.0;
  const double c = 2.0 / ee;
  d += blockIdx.y * n;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    d[i] *= c;
}
__global__ void copy_kernel(int64_t n, const double *__restrict__ a, double *__restrict__ b) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    b[i] = a[i];
}
// t = b - t (t holds A x)
__global__ void residual_from_kernel(int64_t n, const double *__restrict__ b, double *__restrict__ t) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    t[i] = b[i] - t[i];
}
__global__ void residual_inplace_kernel(int64_t n, const double *__restrict__ b, double *__restrict__ r) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    r[i] = b[i] - r[i];
}
// Nodal block-Jacobi: per node k (equations 3k..3k+2) the inverse of K's 3 x 3 diagonal block,
// from the rows of K (columns sorted); ok[0] is cleared for a block that is not positive definite.
__global__ void block_jacobi_kernel(int64_t nodes, const int64_t *__restrict__ ptr, const int32_t *__restrict__ idx,
                                    const double *__restrict__ val, double *__restrict__ inv, int *ok) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nodes; k += (int64_t)gridDim.x * blockDim.x) {
    double a[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    for (int i = 0; i < 3; ++i) {
      const int64_t row = 3 * k + i;
      for (int64_t q = ptr[row]; q < ptr[row + 1]; ++q) {
        const int64_t c = idx[q] - 3 * k;
        if (c >= 0 && c < 3) a[i][c] = val[q];
      }
    }
    // the inverse by cofactors (a symmetric 3 x 3)
    const double c00 = a[1][1] * a[2][2] - a[1][2] * a[2][1], c01 = a[1][2] * a[2][0] - a[1][0] * a[2][2],
                 c02 = a[1][0] * a[2][1] - a[1][1] * a[2][0];
    const double det = a[0][0] * c00 + a[0][1] * c01 + a[0][2] * c02;
    double *o = inv + 9 * k;
    if (!(det > 0.0) || !(a[0][0] > 0.0)) {
      *ok = 0;
      for (int q = 0; q < 9; ++q) o[q] = 0.0;
      continue;
    }
    const double d = 1.0 / det;
    o[0] = c00 * d;
    o[1] = c01 * d;
    o[2] = c02 * d;
    o[3] = c01 * d;
    o[4] = (a[0][0] * a[2][2] - a[0][2] * a[2][0]) * d;
    o[5] = (a[0][2] * a[1][0] - a[0][0] * a[1][2]) * d;
    o[6] = c02 * d;
    o[7] = o[5];
    o[8] = (a[0][0] * a[1][1] - a[0][1] * a[1][0]) * d;
  }
}
// z = B r, B the nodal block-Jacobi inverse; blockIdx.y the vector
__global__ void block_jacobi_apply_kernel(int64_t nodes, const double *__restrict__ inv, const double *__restrict__ r,
                                          int64_t ld, double *__restrict__ z) {
  r += blockIdx.y * ld, z += blockIdx.y * 3 * nodes;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nodes; k += (int64_t)gridDim.x * blockDim.x) {
    const double *o = inv + 9 * k;
    const double r0 = r[3 * k], r1 = r[3 * k + 1], r2 = r[3 * k + 2];
    z[3 * k] = o[0] * r0 + o[1] * r1 + o[2] * r2;
    z[3 * k + 1] = o[3] * r0 + o[4] * r1 + o[5] * r2;
    z[3 * k + 2] = o[6] * r0 + o[7] * r1 + o[8] * r2;
  }
}

__global__ void add_f32_kernel(int64_t n, const float *__restrict__ a, float *__restrict__ z) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    z[i] += a[i];
}

int blocks(int64_t n) { return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 148 * 8)); }

Grid coarser(const Grid &g) { return Grid{(g.X + 1) / 2, (g.Y + 1) / 2, (g.Z + 1) / 2}; }

}  // namespace

// What a group of passes works in, all in one allocation of its owner's.
struct Activations {
  // BF16, channels last, per level: the (pooled) input, the two convolutions of the way down (s =
  // the skip), the way up: u = upsampled + skip, its two convolutions b, d
  bf16 *x = nullptr, *y = nullptr, *pin[MAX_LEVELS] = {}, *a[MAX_LEVELS] = {}, *s[MAX_LEVELS] = {},
       *u[MAX_LEVELS] = {}, *b[MAX_LEVELS] = {}, *d[MAX_LEVELS] = {};
  // gradients per level
  bf16 *dy = nullptr, *ga[MAX_LEVELS] = {}, *gb[MAX_LEVELS] = {}, *gs[MAX_LEVELS] = {};
  // training, a column per pair of a group: the output, its difference
  double *tz = nullptr, *td = nullptr;
};

struct fc_unet : Activations {  // those of the call that runs (choose_passes)
  int device = 0;
  cudaStream_t stream = nullptr;
  int64_t n = 0;
  double kref = 1.0;
  int levels = 3, layers = 11;
  Grid g[MAX_LEVELS];
  int lcin[MAX_LAYERS], lcout[MAX_LAYERS], llevel[MAX_LAYERS];
  int64_t w_off[MAX_LAYERS], b_off[MAX_LAYERS], wb_off[MAX_LAYERS];
  int64_t params = 0, wcount = 0;
  DeviceBuf p, grad, m, v;   // FP32 parameters, gradients and Adam moments
  DeviceBuf gacc;            // a minibatch's mean gradient
  DeviceBuf wb, wt;          // BF16 weights and their flipped transposes
  DeviceBuf eq, feat;
  DeviceBuf part;            // weight-gradient partials
  DeviceBuf scal, dotpart;   // device scalars: [0,1] input scales, [2..] dots; dot partials
  DeviceBuf bj;              // nodal block-Jacobi inverses (9 doubles a node), added to the output
  bool has_bj = false;
  bool net_on = true;         // false: the preconditioner is the block-Jacobi part alone
  bool safeguard = true;      // FCG drops a stalling network (fc_unet_enable 2: it never does)
  // odd: M(r) = B r + (net(r) - net(-r)) / 2, so that M(-r) = -M(r) and M(0) = 0 (a part of the
  // output that does not depend on r, from the biases and the modulus channel, cancels)
  bool odd = true;
  // the handle's own activations, made with it and kept to its end, and a larger group's
  fc::PassRoom room;
  Activations own, group;
  DeviceBuf own_mem, group_mem;
  int most_grown = INT32_MAX;  // larger groups find no memory (for tests)
  DeviceBuf gtmp;              // one pass's gradients, where a pair's two do not fit together
  fc::unet::LayerTable table{};
  int64_t last_net_iterations = 0, last_dropped = 0;
  bool weights_stale = true;
  std::unique_ptr<fc::host::ScratchUser> scratch_user;
  std::mutex lock;
};

namespace {

bf16 *B(const DeviceBuf &b) { return b.as<bf16>(); }

// A group of pairs runs through the network side by side, a pass each (two with the odd form): at
// most PAIRS_MOST pairs, and activations of at most WORKSPACE_MOST bytes beside the handle's own.
constexpr int PAIRS_MOST = 8;
constexpr size_t WORKSPACE_MOST = (size_t)2 << 30;
// the device scalars: the passes' scales, then a value per pair each
constexpr int S_SCALES = 64, S_NRM = 96, S_NUM = 104, S_DEN = 112, S_COUNT = 128;

// The activations and gradients of `passes` passes in `mem`, one allocation (two dozen of them took a
// millisecond). Null pointers and false when there is no memory for it.
bool alloc_passes(const fc_unet *u, int passes, DeviceBuf &mem, Activations &out) {
  const int pairs = std::min(passes, PAIRS_MOST);
  for (int round = 0; round < 2; ++round) {  // sizes, then places
    Activations a;
    unsigned char *base = mem.as<unsigned char>();
    size_t at = 0;
    auto take = [&](auto *&p, size_t count) {
      p = reinterpret_cast<std::decay_t<decltype(p)>>(base + at);
      at += (sizeof(*p) * count + 255) / 256 * 256;
    };
    auto grid = [&](bf16 *&p, const Grid &g, int c) { take(p, (size_t)g.voxels() * c * passes); };
    take(a.tz, (size_t)u->n * pairs);
    take(a.td, (size_t)u->n * pairs);
    grid(a.x, u->g[0], CIO);
    grid(a.y, u->g[0], CIO);
    grid(a.dy, u->g[0], CIO);
    for (int lv = 0; lv < u->levels; ++lv) {
      const Grid &g = u->g[lv];
      for (bf16 **b : {&a.a[lv], &a.s[lv], &a.ga[lv], &a.gb[lv]}) grid(*b, g, C);
      if (lv > 0) grid(a.pin[lv], g, C);
      if (lv < u->levels - 1)
        for (bf16 **b : {&a.u[lv], &a.b[lv], &a.d[lv], &a.gs[lv]}) grid(*b, g, C);
    }
    if (round == 1) {
      out = a;
    } else if (mem.alloc(at) != cudaSuccess) {
      out = Activations();
      return false;
    }
  }
  return true;
}

// The handle's own: a vector's passes together, or one where they find no memory.
bool alloc_own(fc_unet *u, int passes) {
  for (u->room.own = passes; u->room.own > 0; --u->room.own)
    if (alloc_passes(u, u->room.own, u->own_mem, u->own)) return true;
  return false;
}

void use(fc_unet *u, const Activations &a) { static_cast<Activations &>(*u) = a; }

// Room for the passes of `pairs` vectors, or for as many as there is memory for: returns how many run
// together (at least one; a vector's two then run after one another).
int choose_passes(fc_unet *u, int pairs, int per) {
  size_t pass = 0;
  for (int lv = 0; lv < u->levels; ++lv) pass += sizeof(bf16) * (size_t)u->g[lv].voxels() * C * 9;
  int want = per * std::min(pairs, PAIRS_MOST);
  while (want > per && pass * want > WORKSPACE_MOST) want -= per;
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  if (want > u->room.own && cudaStreamIsCapturing(u->stream, &capturing) != cudaSuccess) {
    cudaGetLastError();
    capturing = cudaStreamCaptureStatusActive;
  }
  const fc::PassRoom::Choice c = u->room.choose(want, per, capturing != cudaStreamCaptureStatusNone, [&](int passes) {
    // (an allocation is not part of a capture that runs on another stream)
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    cudaStreamSynchronize(u->stream);
    u->group_mem.release();
    const bool ok = passes <= u->most_grown && alloc_passes(u, passes, u->group_mem, u->group);
    cudaThreadExchangeStreamCaptureMode(&mode);
    return ok;
  });
  use(u, c.in_group ? u->group : u->own);
  return c.passes;
}

// BF16 copies of the weights (and the flipped ones for the input gradients) after a change: before
// a kernel that is not a convolution, which reads them before the kernel ahead of it is done.
void refresh_weights(fc_unet *u) {
  if (!u->weights_stale) return;
  fc::unet::refresh(u->table, u->p.as<float>(), B(u->wb), B(u->wt), u->stream);
  u->weights_stale = false;
}

const Grid &G(const fc_unet *u, int level) { return u->g[level]; }

void conv(fc_unet *u, int passes, int l, const bf16 *in, bf16 *out, bool relu) {
  fc::unet::conv3(G(u, u->llevel[l]), passes, u->lcin[l], u->lcout[l], in, B(u->wb) + u->wb_off[l],
                  u->p.as<float>() + u->b_off[l], relu, nullptr, out, u->stream);
}
// the input gradient of layer l from its output gradient: conv with the flipped weights, then
// the ReLU mask of the layer's input (mask null: no ReLU there)
void conv_t(fc_unet *u, int passes, int l, const bf16 *dout, const bf16 *mask, bf16 *din) {
  fc::unet::conv3(G(u, u->llevel[l]), passes, u->lcout[l], u->lcin[l], dout, B(u->wt) + u->wb_off[l], nullptr,
                  false, mask, din, u->stream);
}

// What backward() does with the parameters' gradients of the pairs it is given: the last pair's
// lands in u->grad, `scale` times each pair's is added to u->gacc when `acc` (from zero unless
// `more`).
struct Gradients {
  int pairs, per;
  bool acc;
  float scale;
  bool more;
};
void conv_dw(fc_unet *u, const Gradients &gr, int l, const bf16 *in, const bf16 *dout) {
  float *acc = gr.acc ? u->gacc.as<float>() : nullptr, *grad = u->grad.as<float>();
  fc::unet::conv3_dw(G(u, u->llevel[l]), u->lcin[l], u->lcout[l], gr.pairs, gr.per, in, dout,
                     u->part.as<float>(), gr.scale, gr.more, acc ? acc + u->w_off[l] : nullptr,
                     acc ? acc + u->b_off[l] : nullptr, grad + u->w_off[l], grad + u->b_off[l], u->stream);
}

// the level's input on the way down: x at the top, the pooled skip of the level above below it
const bf16 *input_of(const fc_unet *u, int lv) { return lv == 0 ? u->x : u->pin[lv]; }
// what the level returns upwards: the bottom's second convolution, or the way up's last one
bf16 *low_of(const fc_unet *u, int lv) { return lv == u->levels - 1 ? u->s[lv] : u->d[lv]; }

// y = net(x) for `P` passes: per level on the way down two convolutions (the second's output is the
// skip) and a 2x2x2 average pooling, two at the bottom, per level on the way up nearest upsampling
// plus the skip and two convolutions, then the output convolution (layers in this order).
void forward(fc_unet *u, int P) {
  cudaStream_t st = u->stream;
  const int D = u->levels;
  int l = 0;
  for (int lv = 0; lv < D; ++lv) {
    conv(u, P, l++, input_of(u, lv), u->a[lv], true);
    conv(u, P, l++, u->a[lv], u->s[lv], true);
    if (lv < D - 1) fc::unet::pool(u->g[lv], u->g[lv + 1], P, u->s[lv], u->pin[lv + 1], st);
  }
  for (int lv = D - 2; lv >= 0; --lv) {
    fc::unet::up_add(u->g[lv], u->g[lv + 1], P, low_of(u, lv + 1), u->s[lv], u->u[lv], st);
    conv(u, P, l++, u->u[lv], u->b[lv], true);
    conv(u, P, l++, u->b[lv], u->d[lv], true);
  }
  conv(u, P, l, low_of(u, 0), u->y, false);
}

// parameters' gradients from dL/dy (in u->dy), after forward() on the same input
void backward(fc_unet *u, const Gradients &gr) {
  cudaStream_t st = u->stream;
  const int D = u->levels, P = gr.pairs * gr.per;
  int l = u->layers - 1;
  conv_dw(u, gr, l, low_of(u, 0), u->dy);
  conv_t(u, P, l, u->dy, low_of(u, 0), u->ga[0]);  // dL/d(top output), through its activation
  for (int lv = 0; lv < D - 1; ++lv) {  // the way up, from the top level to the coarsest
    l -= 2;
    conv_dw(u, gr, l + 1, u->b[lv], u->ga[lv]);
    conv_t(u, P, l + 1, u->ga[lv], u->b[lv], u->gb[lv]);
    conv_dw(u, gr, l, u->u[lv], u->gb[lv]);
    conv_t(u, P, l, u->gb[lv], nullptr, u->gs[lv]);  // dL/du: to the skip and, upsampled, below
    fc::unet::up_adjoint(u->g[lv], u->g[lv + 1], P, u->gs[lv], low_of(u, lv + 1), u->ga[lv + 1], st);
  }
  for (int lv = D - 1; lv >= 0; --lv) {  // the way down, from the bottom up
    l -= 2;
    conv_dw(u, gr, l + 1, u->a[lv], u->ga[lv]);
    conv_t(u, P, l + 1, u->ga[lv], u->a[lv], u->gb[lv]);
    conv_dw(u, gr, l, input_of(u, lv), u->gb[lv]);
    if (lv == 0) break;
    conv_t(u, P, l, u->gb[lv], nullptr, u->ga[lv]);  // dL/d(pooled input)
    fc::unet::pool_adjoint(u->g[lv - 1], u->g[lv], P, u->ga[lv], u->gs[lv - 1], u->s[lv - 1],
                           u->ga[lv - 1], st);  // dL/d(skip of the level above), masked
  }
}

double *scal(fc_unet *u, int k) { return u->scal.as<double>() + k; }

// out[q] = a_q . b_q for the columns q of a group of pairs
void pair_dots(fc_unet *u, int pairs, const double *a, int64_t lda, const double *b, int64_t ldb, double *out) {
  const double *pa[PAIRS_MOST], *pb[PAIRS_MOST];
  for (int q = 0; q < pairs; ++q) pa[q] = a + q * lda, pb[q] = b + q * ldb;
  fc::unet::dots(u->n, pairs, pa, pb, u->dotpart.as<double>(), out, u->stream);
}

int passes_per_pair(const fc_unet *u) { return u->odd ? 2 : 1; }

// The network's passes [p0, p0 + count) of the group's pairs, forward: their input grids, the pass.
// A range of whole pairs, or one pass of a pair (count 1).
void forward_passes(fc_unet *u, const double *r, int64_t ld, int p0, int count) {
  const int per = passes_per_pair(u), pairs = std::max(1, count / per), each = count / pairs;
  fc::unet::scatter_input(u->g[0], pairs, each, u->eq.as<int64_t>(), r + p0 / per * ld, ld, u->feat.as<float>(),
                          scal(u, S_SCALES + 2 * p0), u->x, u->stream);
  forward(u, count);
}

// z_q = M(r_q) for the group's pairs (z contiguous), `together` passes at a time.
void apply(fc_unet *u, int pairs, const double *r, int64_t ld, double *z, int together) {
  cudaStream_t st = u->stream;
  const int per = passes_per_pair(u);
  refresh_weights(u);
  pair_dots(u, pairs, r, ld, r, ld, scal(u, S_NRM));
  fc::unet::input_scales(u->n, pairs, per, scal(u, S_NRM), u->kref, scal(u, S_SCALES), st);
  if (u->has_bj)
    block_jacobi_apply_kernel<<<dim3(blocks(u->n / 3), pairs), 256, 0, st>>>(u->n / 3, u->bj.as<double>(), r, ld, z);
  else
    cudaMemsetAsync(z, 0, sizeof(double) * (size_t)u->n * pairs, st);
  for (int p0 = 0, count; p0 < per * pairs; p0 += count) {
    count = std::min(per * pairs - p0, together);
    forward_passes(u, r, ld, p0, count);
    const int whole = std::max(1, count / per);
    fc::unet::gather_output(u->g[0], whole, count / whole, u->eq.as<int64_t>(), u->y,
                            scal(u, S_SCALES + 2 * p0), z + p0 / per * u->n, u->n, u->has_bj || p0 % per != 0, st);
  }
}

// z = B r alone (the network left out)
void apply_jacobi(fc_unet *u, const double *r, double *z) {
  block_jacobi_apply_kernel<<<blocks(u->n / 3), 256, 0, u->stream>>>(u->n / 3, u->bj.as<double>(), r, u->n, z);
}

// The losses of `count` pairs (r_q, e_q) added into *d_loss, the last pair's gradient into u->grad,
// and with `acc` their mean into u->gacc (forward and backward of the network, in groups of pairs).
void pair_gradients(fc_unet *u, const double *d_r, const double *d_e, int count, int64_t ld, const int64_t *d_ptr,
                    const int32_t *d_idx, const double *d_val, double *d_loss, bool acc) {
  cudaStream_t st = u->stream;
  const int per = passes_per_pair(u);
  const int together = choose_passes(u, count, per);
  const int most = std::max(1, together / per);
  double *z = u->tz, *d = u->td;
  const int64_t *eq = u->eq.as<int64_t>();
  for (int q0 = 0; q0 < count; q0 += most) {
    const int g = std::min(most, count - q0);
    const double *r = d_r + q0 * ld, *e = d_e + q0 * ld;
    apply(u, g, r, ld, z, together);
    sub_kernel<<<dim3(blocks(u->n), g), 256, 0, st>>>(u->n, z, e, ld, d);
    double *grad = d;
    if (d_ptr) {
      // energy norm: loss = d.Kd / e.r (e.r = e.K e), dL/dz = 2 Kd / e.r
      fc::launch_spmv(u->n, d_ptr, d_idx, d_val, d, u->n, z, u->n, g, st);
      pair_dots(u, g, d, u->n, z, u->n, scal(u, S_NUM));
      pair_dots(u, g, e, ld, r, ld, scal(u, S_DEN));
      grad = z;
    } else {
      pair_dots(u, g, d, u->n, d, u->n, scal(u, S_NUM));
      pair_dots(u, g, e, ld, e, ld, scal(u, S_DEN));
    }
    loss_grad_kernel<<<dim3(blocks(u->n), g), 256, 0, st>>>(u->n, scal(u, S_NUM), scal(u, S_DEN), grad, d_loss,
                                                            q0 == 0);
    const float scale = 1.f / (float)count;
    if (together >= per) {
      fc::unet::scatter_grad(u->g[0], g, per, eq, grad, u->n, scal(u, S_SCALES), u->dy, st);
      backward(u, {g, per, acc, scale, q0 > 0});
      continue;
    }
    // room for one pass only: the second pass's activations are live, its gradient first and kept
    // aside; then the first pass again, forward and backward, and the two added
    fc::unet::scatter_grad(u->g[0], 1, 1, eq, grad, u->n, scal(u, S_SCALES + 2), u->dy, st);
    backward(u, {1, 1, acc, scale, q0 > 0});
    cudaMemcpyAsync(u->gtmp.p, u->grad.p, sizeof(float) * (size_t)u->params, cudaMemcpyDeviceToDevice, st);
    forward_passes(u, r, ld, 0, 1);
    fc::unet::scatter_grad(u->g[0], 1, 1, eq, grad, u->n, scal(u, S_SCALES), u->dy, st);
    backward(u, {1, 1, acc, scale, true});
    add_f32_kernel<<<blocks(u->params), 256, 0, st>>>(u->params, u->gtmp.as<float>(), u->grad.as<float>());
  }
}

int cuda_fail(fc_status *st, cudaError_t e, const char *where) {
  set_status(st, FC_CUDA_ERROR, -1, 0, 0, std::string(where) + ": " + cudaGetErrorString(e));
  return FC_CUDA_ERROR;
}

}  // namespace

extern "C" {

int fc_unet_create_levels(int32_t nx, int32_t ny, int32_t nz, int64_t n, const int64_t *eq, const float *feat,
                          double kref, int32_t levels, uint64_t seed, int32_t device, fc_unet **out,
                          fc_status *status) {
  if (!out || nx < 1 || ny < 1 || nz < 1 || n < 1 || !eq || !feat || !(kref > 0) || levels < 1 ||
      levels > MAX_LEVELS) {
    set_status(status, FC_INVALID_ARGUMENT, -1, 0, 0, "bad network arguments");
    return FC_INVALID_ARGUMENT;
  }
  *out = nullptr;
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) return cuda_fail(status, e, "device");
  fc_unet *u = new fc_unet();
  u->device = device;
  u->scratch_user = std::make_unique<fc::host::ScratchUser>(device);
  u->n = n;
  u->kref = kref;
  u->levels = levels;
  u->g[0] = Grid{nx + 1, ny + 1, nz + 1};
  for (int lv = 1; lv < levels; ++lv) u->g[lv] = coarser(u->g[lv - 1]);
  // the layers in forward order: (cin, cout, level)
  int L = 0;
  for (int lv = 0; lv < levels; ++lv)
    for (int q = 0; q < 2; ++q) u->lcin[L] = (lv == 0 && q == 0) ? CIO : C, u->lcout[L] = C, u->llevel[L++] = lv;
  for (int lv = levels - 2; lv >= 0; --lv)
    for (int q = 0; q < 2; ++q) u->lcin[L] = C, u->lcout[L] = C, u->llevel[L++] = lv;
  u->lcin[L] = C, u->lcout[L] = CIO, u->llevel[L++] = 0;
  u->layers = L;
  int64_t off = 0, woff = 0;
  for (int l = 0; l < L; ++l) {
    const int64_t nw = (int64_t)27 * u->lcin[l] * u->lcout[l];
    u->w_off[l] = off;
    off += nw;
    u->b_off[l] = off;
    off += u->lcout[l];
    u->wb_off[l] = woff;
    woff += nw;
    u->table.cin[l] = u->lcin[l], u->table.cout[l] = u->lcout[l];
    u->table.param[l] = u->w_off[l], u->table.weight[l] = u->wb_off[l];
  }
  u->table.layers = L;
  u->params = off;
  u->wcount = woff;
  const int64_t nodes = u->g[0].voxels();
  std::vector<float> host(off, 0.f);
  std::mt19937_64 rng(seed);
  std::normal_distribution<float> normal(0.f, 1.f);
  for (int l = 0; l < L - 1; ++l) {  // the last layer starts at zero: M(r) = 0, a loss of one
    const float sd = std::sqrt(2.f / (27.f * (l == 0 ? 4 : u->lcin[l])));
    const int64_t nw = (int64_t)27 * u->lcin[l] * u->lcout[l];
    for (int64_t q = 0; q < nw; ++q) host[u->w_off[l] + q] = sd * normal(rng);
  }
  bool ok = u->p.alloc(sizeof(float) * off) == cudaSuccess && u->grad.alloc(sizeof(float) * off) == cudaSuccess &&
            u->m.alloc(sizeof(float) * off) == cudaSuccess && u->v.alloc(sizeof(float) * off) == cudaSuccess &&
            u->gacc.alloc(sizeof(float) * off) == cudaSuccess &&
            u->wb.alloc(sizeof(bf16) * woff) == cudaSuccess && u->wt.alloc(sizeof(bf16) * woff) == cudaSuccess &&
            u->eq.alloc(sizeof(int64_t) * 3 * nodes) == cudaSuccess &&
            u->feat.alloc(sizeof(float) * nodes) == cudaSuccess &&
            u->scal.alloc(sizeof(double) * S_COUNT) == cudaSuccess &&
            u->dotpart.alloc(sizeof(double) * 8 * 512) == cudaSuccess &&
            u->part.alloc(sizeof(float) * std::max(fc::unet::DW_PARTIALS, 2 * PAIRS_MOST) * 28 * C * C) == cudaSuccess &&
            u->gtmp.alloc(sizeof(float) * off) == cudaSuccess && alloc_own(u, passes_per_pair(u));
  if (!ok) {
    delete u;
    set_status(status, FC_OUT_OF_MEMORY, -1, 0, 0, "device memory for the network");
    return FC_OUT_OF_MEMORY;
  }
  cudaMemcpy(u->p.p, host.data(), sizeof(float) * off, cudaMemcpyHostToDevice);
  cudaMemset(u->m.p, 0, sizeof(float) * off);
  cudaMemset(u->v.p, 0, sizeof(float) * off);
  cudaMemset(u->grad.p, 0, sizeof(float) * off);
  cudaMemcpy(u->eq.p, eq, sizeof(int64_t) * 3 * nodes, cudaMemcpyHostToDevice);
  cudaMemcpy(u->feat.p, feat, sizeof(float) * nodes, cudaMemcpyHostToDevice);
  e = cudaDeviceSynchronize();
  if (e != cudaSuccess) {
    delete u;
    return cuda_fail(status, e, "network set-up");
  }
  *out = u;
  set_status(status, FC_OK);
  return FC_OK;
}

int fc_unet_create(int32_t nx, int32_t ny, int32_t nz, int64_t n, const int64_t *eq, const float *feat, double kref,
                   uint64_t seed, int32_t device, fc_unet **out, fc_status *status) {
  return fc_unet_create_levels(nx, ny, nz, n, eq, feat, kref, 3, seed, device, out, status);
}

int fc_unet_set_operator(fc_unet *u, const int64_t *d_ptr, const int32_t *d_idx, const double *d_val) {
  if (!u || u->n % 3 != 0) return FC_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> g(u->lock);
  cudaSetDevice(u->device);
  if (!d_ptr) {
    u->has_bj = false;
    return FC_OK;
  }
  if (!d_idx || !d_val) return FC_INVALID_ARGUMENT;
  const int64_t nodes = u->n / 3;
  if (!u->bj.p && u->bj.alloc(sizeof(double) * 9 * (size_t)nodes) != cudaSuccess) return FC_OUT_OF_MEMORY;
  int *ok = u->scal.as<int>() + 2 * 60;  // a flag in the last scalar slots
  int one = 1;
  cudaMemcpyAsync(ok, &one, sizeof(int), cudaMemcpyHostToDevice, u->stream);
  block_jacobi_kernel<<<blocks(nodes), 256, 0, u->stream>>>(nodes, d_ptr, d_idx, d_val, u->bj.as<double>(), ok);
  cudaMemcpyAsync(&one, ok, sizeof(int), cudaMemcpyDeviceToHost, u->stream);
  if (cudaStreamSynchronize(u->stream) != cudaSuccess) return FC_CUDA_ERROR;
  u->has_bj = one != 0;
  return one ? FC_OK : FC_NOT_POSITIVE_DEFINITE;
}

int fc_unet_set_odd(fc_unet *u, int32_t odd) {
  if (!u) return FC_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> g(u->lock);
  u->odd = odd != 0;
  return FC_OK;
}

int fc_unet_enable(fc_unet *u, int32_t on) {
  if (!u || on < 0 || on > 2 || (!on && !u->has_bj)) return FC_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> g(u->lock);
  u->net_on = on != 0;
  u->safeguard = on != 2;
  return FC_OK;
}

int64_t fc_unet_stat(const fc_unet *u, int32_t what) {
  if (!u) return -1;
  switch (what) {
    case 0: return u->levels;
    case 1: return u->last_net_iterations;
    case 2: return u->last_dropped;
    case 3: return u->has_bj ? 1 : 0;
    default: return -1;
  }
}

void fc_unet_destroy(fc_unet *u) {
  if (!u) return;
  cudaSetDevice(u->device);
  if (u->stream) cudaStreamSynchronize(u->stream);
  delete u;
}

int fc_unet_set_stream(fc_unet *u, void *stream) {
  if (!u) return FC_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> g(u->lock);
  u->stream = static_cast<cudaStream_t>(stream);
  return FC_OK;
}

int64_t fc_unet_param_count(const fc_unet *u) { return u ? u->params : -1; }

int fc_unet_get_params(fc_unet *u, float *host) {
  if (!u || !host) return FC_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> g(u->lock);
  cudaSetDevice(u->device);
  cudaStreamSynchronize(u->stream);
  return cudaMemcpy(host, u->p.p, sizeof(float) * u->params, cudaMemcpyDeviceToHost) == cudaSuccess ? FC_OK
                                                                                                    : FC_CUDA_ERROR;
}

int fc_unet_set_params(fc_unet *u, const float *host) {
  if (!u || !host) return FC_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> g(u->lock);
  cudaSetDevice(u->device);
  cudaStreamSynchronize(u->stream);
  u->weights_stale = true;
  return cudaMemcpy(u->p.p, host, sizeof(float) * u->params, cudaMemcpyHostToDevice) == cudaSuccess ? FC_OK
                                                                                                    : FC_CUDA_ERROR;
}

int fc_unet_get_grads(fc_unet *u, float *host) {
  if (!u || !host) return FC_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> g(u->lock);
  cudaSetDevice(u->device);
  cudaStreamSynchronize(u->stream);
  return cudaMemcpy(host, u->grad.p, sizeof(float) * u->params, cudaMemcpyDeviceToHost) == cudaSuccess
             ? FC_OK
             : FC_CUDA_ERROR;
}

// Not part of the public ABI, for tests: the handle's own activations for `own` passes, and no memory for
// groups of more than `group`. Returns what the own ones hold.
int fc_test_unet_room(fc_unet *u, int own, int group) {
  std::lock_guard<std::mutex> g(u->lock);
  cudaSetDevice(u->device);
  cudaStreamSynchronize(u->stream);
  u->group_mem.release();
  u->room = fc::PassRoom();
  u->most_grown = group;
  if (!alloc_own(u, own)) return 0;
  use(u, u->own);
  return u->room.own;
}

// Not part of the public ABI, for tests: the weight gradient of one layer on device arrays (conv3_dw); in
// and dy in BF16, pairs * passes grids each; gw and gb receive the sum over the pairs of scale g.
int fc_test_unet_dw(int32_t X, int32_t Y, int32_t Z, int32_t cin, int32_t cout, int32_t pairs, int32_t passes,
                    const void *d_in, const void *d_dy, float scale, float *d_gw, float *d_gb) {
  const Grid g{X, Y, Z};
  const size_t nw = (size_t)27 * cin * cout;
  DeviceBuf part, last;
  if (part.alloc(sizeof(float) * (size_t)pairs * passes * fc::unet::dw_chunks(g, pairs * passes) * 28 * cin * cout) != cudaSuccess ||
      last.alloc(sizeof(float) * (nw + cout)) != cudaSuccess)
    return FC_OUT_OF_MEMORY;
  fc::unet::conv3_dw(g, cin, cout, pairs, passes, static_cast<const bf16 *>(d_in), static_cast<const bf16 *>(d_dy),
                     part.as<float>(), scale, false, d_gw, d_gb, last.as<float>(), last.as<float>() + nw, nullptr);
  return cudaDeviceSynchronize() == cudaSuccess ? FC_OK : FC_CUDA_ERROR;
}

int fc_unet_forward_grid(fc_unet *u, const float *d_x, float *d_y) {
  if (!u || !d_x || !d_y) return FC_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> g(u->lock);
  cudaSetDevice(u->device);
  const int64_t nv = u->g[0].voxels() * CIO;
  use(u, u->own);
  refresh_weights(u);
  f32_to_bf16_kernel<<<blocks(nv), 256, 0, u->stream>>>(nv, d_x, u->x);
  forward(u, 1);
  bf16_to_f32_kernel<<<blocks(nv), 256, 0, u->stream>>>(nv, u->y, d_y);
  const cudaError_t e = cudaStreamSynchronize(u->stream);
  return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? FC_OK : FC_CUDA_ERROR;
}

int fc_unet_backward_grid(fc_unet *u, const float *d_dy) {
  if (!u || !d_dy) return FC_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> g(u->lock);
  cudaSetDevice(u->device);
  const int64_t nv = u->g[0].voxels() * CIO;
  use(u, u->own);
  f32_to_bf16_kernel<<<blocks(nv), 256, 0, u->stream>>>(nv, d_dy, u->dy);
  backward(u, {1, 1, false, 1.f, false});
  const cudaError_t e = cudaStreamSynchronize(u->stream);
  return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? FC_OK : FC_CUDA_ERROR;
}

int fc_unet_apply(fc_unet *u, const double *d_r, double *d_z) {
  if (!u || !d_r || !d_z) return FC_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> g(u->lock);
  cudaSetDevice(u->device);
  if (u->net_on) {
    apply(u, 1, d_r, u->n, d_z, choose_passes(u, 1, passes_per_pair(u)));
  } else
    apply_jacobi(u, d_r, d_z);
  return cudaGetLastError() == cudaSuccess ? FC_OK : FC_CUDA_ERROR;
}

int fc_unet_train_step(fc_unet *u, const double *d_r, const double *d_e, const int64_t *d_ptr, const int32_t *d_idx,
                       const double *d_val, float lr, int32_t step, double *d_loss) {
  if (!u || !d_r || !d_e || step < 1 || (d_ptr && (!d_idx || !d_val))) return FC_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> g(u->lock);
  cudaSetDevice(u->device);
  pair_gradients(u, d_r, d_e, 1, u->n, d_ptr, d_idx, d_val, d_loss, false);
  fc::unet::adam(u->params, u->p.as<float>(), u->grad.as<float>(), u->m.as<float>(), u->v.as<float>(), lr, 0.9f,
                 0.999f, 1e-8f, step, u->stream);
  u->weights_stale = true;
  return cudaGetLastError() == cudaSuccess ? FC_OK : FC_CUDA_ERROR;
}

int fc_unet_train_batch(fc_unet *u, const double *d_r, const double *d_e, int32_t count, int64_t ld,
                        const int64_t *d_ptr, const int32_t *d_idx, const double *d_val, float lr, int32_t step,
                        double *d_loss) {
  if (!u || !d_r || !d_e || count < 1 || ld < u->n || step < 1 || (d_ptr && (!d_idx || !d_val)))
    return FC_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> g(u->lock);
  cudaSetDevice(u->device);
  cudaStream_t st = u->stream;
  pair_gradients(u, d_r, d_e, count, ld, d_ptr, d_idx, d_val, d_loss, true);
  fc::unet::adam(u->params, u->p.as<float>(), u->gacc.as<float>(), u->m.as<float>(), u->v.as<float>(), lr, 0.9f,
                 0.999f, 1e-8f, step, st);
  u->weights_stale = true;
  return cudaGetLastError() == cudaSuccess ? FC_OK : FC_CUDA_ERROR;
}

int fc_fcg_solve(fc_unet *net, fc_chol *fallback, int64_t n, const int64_t *d_ptr, const int32_t *d_idx,
                 const double *d_val, const double *d_b, double *d_x, double tol, int32_t max_iter, int32_t keep,
                 int32_t *iterations, double *relres, int32_t *used_fallback, fc_status *status) {
  if (iterations) *iterations = 0;
  if (used_fallback) *used_fallback = 0;
  if (n < 1 || !d_ptr || !d_idx || !d_val || !d_b || !d_x || keep < 1 || keep > 8 || max_iter < 0 ||
      (net && net->n != n)) {
    set_status(status, FC_INVALID_ARGUMENT, -1, 0, 0, "bad solver arguments");
    return FC_INVALID_ARGUMENT;
  }
  std::unique_lock<std::mutex> guard;
  if (net) {
    guard = std::unique_lock<std::mutex>(net->lock);
    cudaSetDevice(net->device);
  }
  cudaStream_t st = net ? net->stream : nullptr;
  const int together = net ? choose_passes(net, 1, passes_per_pair(net)) : 0;
  // vectors: r, z, q and the ring of `keep` directions p_j and A p_j
  const int ring = keep;
  constexpr int CHECK = 8;
  static_assert(8 * 296 <= 2 * fc::unet::FCG_CTAS, "the dots write over p.r and p.q at most");
  constexpr size_t SCALARS = 64, PARTS = (size_t)(2 + fc::unet::MAX_KEPT + CHECK + 1) * fc::unet::FCG_CTAS;
  fc::host::Scratch scratch(sizeof(double) * (SCALARS + PARTS + (size_t)n * (3 + 2 * ring)), st);
  if (!scratch.p) {
    set_status(status, FC_OUT_OF_MEMORY, -1, 0, 0, "device memory for FCG");
    return FC_OUT_OF_MEMORY;
  }
  double *const s = static_cast<double *>(scratch.p), *const part = s + SCALARS;
  double *r = part + PARTS, *z = r + n, *tmp = z + n;
  std::vector<double *> P(ring), Q(ring);
  for (int j = 0; j < ring; ++j) P[j] = tmp + n * (1 + 2 * j), Q[j] = P[j] + n;
  // [0] b.b [1] r.r [5] b - A x squared [8..8+ring) z.q_j with the network [16..16+ring) p_j.q_j
  // [32..32+CHECK) the last iterations' r.r; part: the dots' partials, and flexible CG's: p.r and p.q,
  // z.q_j, and r.r of CHECK iterations and of a start
  double *const part_pq = part, *const part_zq = part + 2 * fc::unet::FCG_CTAS,
               *const part_rr = part_zq + fc::unet::MAX_KEPT * fc::unet::FCG_CTAS;
  cudaMemsetAsync(d_x, 0, sizeof(double) * n, st);
  copy_kernel<<<blocks(n), 256, 0, st>>>(n, d_b, r);
  {
    const double *a[1] = {d_b}, *b[1] = {d_b};
    fc::unet::dots(n, 1, a, b, part, s + 0, st);
  }
  double bb = 0.0, rr = 0.0;
  cudaMemcpyAsync(&bb, s, sizeof(double), cudaMemcpyDeviceToHost, st);
  cudaError_t e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return cuda_fail(status, e, "FCG set-up");
  const double target = tol * tol * bb;
  int it = 0, stored = 0;
  bool converged = bb == 0.0;
  // The safeguard: while the network is in use, from iteration 2 SAFE_WINDOW on, a window of
  // SAFE_WINDOW iterations that does not lower ||r||^2 by SAFE_DROP drops it for the rest of the
  // solve (the block-Jacobi part, when set, stays) and restarts from the true residual b - A x with
  // no kept directions: directions made with the network's outputs slow the rest of the solve
  // down (measured: more than 1 500 iterations after a drop at 50, against 864 for block Jacobi
  // from zero), while after a restart the rest is block-Jacobi PCG from the current x.
  constexpr int SAFE_WINDOW = 25;
  constexpr int MAX_REPLACEMENTS = 8;  // residual replacements at most (see below)
  int replacements = 0;
  constexpr double SAFE_DROP = 0.25;
  bool use_net = net != nullptr && net->net_on;
  std::vector<double> history;
  if (net) net->last_dropped = 0, net->last_net_iterations = 0;
  // ||r||^2 of each iteration lands in a ring of device scalars (s + 32 + it % CHECK); the host
  // reads them every CHECK iterations (one synchronisation per CHECK iterations), then decides on
  // convergence, the safeguard and a residual replacement in iteration order.
  int since = 0;
  double ring_rr[CHECK];
  // the kept directions' slots, the most recent first, at iteration `it` with `have` stored
  auto kept = [&](int at, int have, int *slot) {
    for (int j = 0; j < have; ++j) slot[j] = (at - 1 - j) % ring;
    return have;
  };
  // z = M(r) and its products with the kept directions, for iteration `at`; with `update` the last
  // direction's step on x and r first (rr_slot: where r.r's partials go). The network's z is formed
  // apart.
  auto step = [&](bool update, int at, int have, int rr_slot) {
    const bool jacobi = net && net->has_bj;
    fc::unet::FcgStep a{};
    a.n = n, a.update = update ? 1 : 0, a.product = part_pq, a.x = d_x, a.r = r, a.zq = part_zq;
    a.rr = part_rr + (int64_t)rr_slot * fc::unet::FCG_CTAS;
    if (update) a.p = P[(at - 1) % ring], a.q = Q[(at - 1) % ring], a.den = s + 16 + (at - 1) % ring;
    int slot[fc::unet::MAX_KEPT];
    if (!use_net) {
      a.z = z, a.inv = jacobi ? net->bj.as<double>() : nullptr;
      a.kept = kept(at, have, slot);
      for (int j = 0; j < a.kept; ++j) a.qj[j] = Q[slot[j]];
    }
    fc::unet::fcg_step(a, st);
  };
  bool have_z = false;
  while (!converged && it < max_iter) {
    double *p = P[it % ring], *q = Q[it % ring];
    int slot[fc::unet::MAX_KEPT];
    const int m = kept(it, stored, slot);
    const double *pj[fc::unet::MAX_KEPT], *qj[fc::unet::MAX_KEPT], *zz[fc::unet::MAX_KEPT];
    for (int j = 0; j < m; ++j) pj[j] = P[slot[j]], qj[j] = Q[slot[j]], zz[j] = z;
    if (use_net) {
      apply(net, 1, r, n, z, together);
      if (m > 0) fc::unet::dots(n, m, zz, qj, part, s + 8, st);
    } else if (!have_z) {
      step(false, it, m, CHECK);
    }
    // p = z - sum_j (z.q_j / p_j.q_j) p_j over the stored directions (the denominators were kept
    // in s + 16 + slot when each direction was made); q = A p, p.r, p.q
    fc::unet::fcg_direction(n, m, z, pj, slot, s + 8, use_net ? nullptr : part_zq, s + 16, p, st);
    fc::unet::fcg_product(n, d_ptr, d_idx, d_val, p, r, q, part_pq, st);
    // alpha = p.r / p.q, x += alpha p, r -= alpha q, and the next iteration's z
    step(true, it + 1, std::min(stored + 1, ring), it % CHECK);
    have_z = !use_net;
    ++it;
    stored = std::min(stored + 1, ring);
    if (++since < CHECK && it < max_iter) continue;
    fc::unet::fcg_norms(n, CHECK, part_rr, s + 32, st);
    cudaMemcpyAsync(ring_rr, s + 32, sizeof(double) * CHECK, cudaMemcpyDeviceToHost, st);
    e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_fail(status, e, "FCG");
    bool nan = false, dropped = false;
    for (int k = it - since; k < it && !converged; ++k) {
      rr = ring_rr[k % CHECK];
      if (!(rr == rr)) {
        nan = true;
        break;
      }
      converged = rr <= target;
      history.push_back(rr);
      if (use_net) {
        net->last_net_iterations = k + 1;
        const size_t h = history.size();
        if (net->safeguard && h >= 2 * SAFE_WINDOW && rr > SAFE_DROP * history[h - 1 - SAFE_WINDOW]) {
          use_net = false;
          net->last_dropped = 1;
          dropped = true;
        }
      }
    }
    since = 0;
    if (nan) break;  // NaN: give up on FCG
    if (dropped && !converged) {
      // the network is dropped: go on from the true residual with no kept directions
      fc::launch_spmv(n, d_ptr, d_idx, d_val, d_x, n, tmp, n, 1, st);
      residual_from_kernel<<<blocks(n), 256, 0, st>>>(n, d_b, tmp);
      copy_kernel<<<blocks(n), 256, 0, st>>>(n, tmp, r);
      stored = 0;
      have_z = false;
    }
    if (converged && replacements < MAX_REPLACEMENTS) {
      // the recurrence says converged: check b - A x itself; when rounding has let the two drift
      // apart, go on from the true residual (the kept directions restart)
      fc::launch_spmv(n, d_ptr, d_idx, d_val, d_x, n, tmp, n, 1, st);
      residual_from_kernel<<<blocks(n), 256, 0, st>>>(n, d_b, tmp);
      const double *a[1] = {tmp}, *b2[1] = {tmp};
      fc::unet::dots(n, 1, a, b2, part, s + 5, st);
      double tr = 0.0;
      cudaMemcpyAsync(&tr, s + 5, sizeof(double), cudaMemcpyDeviceToHost, st);
      e = cudaStreamSynchronize(st);
      if (e != cudaSuccess) return cuda_fail(status, e, "FCG");
      if (!(tr <= target)) {
        copy_kernel<<<blocks(n), 256, 0, st>>>(n, tmp, r);
        stored = 0;
        have_z = false;
        converged = false;
        ++replacements;
      }
    }
  }
  if (iterations) *iterations = it;
  // the true residual of the returned x
  auto true_relres = [&]() {
    fc::launch_spmv(n, d_ptr, d_idx, d_val, d_x, n, r, n, 1, st);
    residual_inplace_kernel<<<blocks(n), 256, 0, st>>>(n, d_b, r);
    const double *a[1] = {r}, *b[1] = {r};
    fc::unet::dots(n, 1, a, b, part, s + 1, st);
    cudaMemcpyAsync(&rr, s + 1, sizeof(double), cudaMemcpyDeviceToHost, st);
    cudaStreamSynchronize(st);
    return bb > 0.0 ? std::sqrt(rr / bb) : std::sqrt(rr);
  };
  double rel = true_relres();
  if (!(rel <= tol) && fallback) {
    cudaMemcpyAsync(d_x, d_b, sizeof(double) * n, cudaMemcpyDeviceToDevice, st);
    cudaStreamSynchronize(st);
    fc_status cs{};
    const int rc = fc_chol_solve_device(fallback, d_x, 1, n, &cs);
    if (rc != FC_OK) {
      if (status) *status = cs;
      return rc;
    }
    if (used_fallback) *used_fallback = 1;
    rel = true_relres();
  }
  if (relres) *relres = rel;
  if (!(rel <= tol)) {
    set_status(status, FC_TIMEOUT, -1, 0, 0, "FCG did not reach the tolerance");
    return FC_TIMEOUT;
  }
  set_status(status, FC_OK);
  return FC_OK;
}

}  // extern "C"
