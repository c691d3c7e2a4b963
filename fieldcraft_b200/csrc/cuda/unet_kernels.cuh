// Kernels of the learned preconditioner: a 3-level, 32-channel 3D-convolution U-Net on the node
// grid of a hex8 mesh, BF16 activations and weights with FP32 accumulation on the tensor pipe,
// and the vector kernels of flexible CG.
//
// Activations are channels-last: voxel v = x + X (y + Y z) holds C consecutive BF16 channels.
// Weights of a 3x3x3 convolution are [tap][cout][cin] BF16 (tap = dx+1 + 3 (dy+1 + 3 (dz+1))).
#pragma once

#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace fc {
namespace unet {

struct Grid {
  int X, Y, Z;
  __host__ __device__ int64_t voxels() const { return (int64_t)X * Y * Z; }
};

// Batches: the passes of a batch lie one after the other, each a whole grid.

// out = act(conv3x3x3(in, w) + bias) on the batch's grids g; CIN, COUT in {16, 32}. relu: the leaky ReLU
// (x for x > 0, 0.05 x otherwise). mask (optional, COUT channels): out *= (mask > 0 ? 1 : 0.05),
// the derivative of the leaky ReLU whose output is `mask`, applied to a gradient. bias may be null.
// Launched as a programmatic dependent: the weights are read before the stream's previous kernel is
// done, so that kernel must not be the one that writes them.
void conv3(const Grid &g, int batch, int cin, int cout, const __nv_bfloat16 *in, const __nv_bfloat16 *w,
           const float *bias, bool relu, const __nv_bfloat16 *mask, __nv_bfloat16 *out, cudaStream_t st);
// Weight gradient of conv3 over `pairs` pairs of `passes` passes each: per pair g_w[tap][cout][cin] =
// sum over its passes' voxels of dy[v][cout] in[v + tap][cin] and g_b[cout] = sum of dy[v][cout],
// in chunks of each pass's tiles whose partials are added in order, then the passes. gw and gb receive
// the last pair's; accw and accb (or null) the sum over the pairs of scale g, on top of what they hold
// when `more`. part must hold grids * dw_chunks(g, grids) * 28 * cin * cout floats with grids = pairs *
// passes: at most max(DW_PARTIALS, grids) * 28 * cin * cout.
constexpr int DW_PARTIALS = 148;
int dw_chunks(const Grid &g, int grids);
void conv3_dw(const Grid &g, int cin, int cout, int pairs, int passes, const __nv_bfloat16 *in,
              const __nv_bfloat16 *dy, float *part, float scale, bool more, float *accw, float *accb, float *gw,
              float *gb, cudaStream_t st);
// A network's layers: channels, where the FP32 weights start in the parameters and the BF16 ones
// in their arrays.
constexpr int LAYERS_MOST = 31;
struct LayerTable {
  int layers;
  int cin[LAYERS_MOST], cout[LAYERS_MOST];
  int64_t param[LAYERS_MOST], weight[LAYERS_MOST];
};
// BF16 weights w and, for the input gradients, wt[26 - tap][cin][cout] = w[tap][cout][cin], of
// every layer.
void refresh(const LayerTable &t, const float *p, __nv_bfloat16 *w, __nv_bfloat16 *wt, cudaStream_t st);

// 2x2x2 average (sum / 8) onto the coarse grid gc (ceil halves); C = 32.
void pool(const Grid &gf, const Grid &gc, int batch, const __nv_bfloat16 *fine, __nv_bfloat16 *coarse, cudaStream_t st);
// fine = coarse(x/2, y/2, z/2) + skip; C = 32.
void up_add(const Grid &gf, const Grid &gc, int batch, const __nv_bfloat16 *coarse, const __nv_bfloat16 *skip,
            __nv_bfloat16 *fine, cudaStream_t st);
// The adjoints, times the leaky ReLU's derivative at `mask` (1 where mask > 0, else 0.05):
// coarse = sum of the 8 children of dfine (nearest upsampling); fine = dcoarse(parent) / 8 + dskip
// (average pooling plus the skip path).
void up_adjoint(const Grid &gf, const Grid &gc, int batch, const __nv_bfloat16 *dfine, const __nv_bfloat16 *mask,
                __nv_bfloat16 *dcoarse, cudaStream_t st);
void pool_adjoint(const Grid &gf, const Grid &gc, int batch, const __nv_bfloat16 *dcoarse, const __nv_bfloat16 *dskip,
                  const __nv_bfloat16 *mask, __nv_bfloat16 *dfine, cudaStream_t st);

// Between the equations' vectors and the grids of `pairs` vectors (column q at q * ld), `per` passes
// each with their own scales (scale[2 p], scale[2 p + 1] of pass p): the 16 input channels of voxel
// v are (r_x, r_y, r_z) * scale[2 p] at the node's free DOFs (0 where held), feat[v] (a fixed
// feature: the node's log Young's modulus), and zeros. eq[3 v + a] is the equation of DOF a of
// node v, -1 when held. Out: z[eq] = the sum over the vector's passes of y[v][a] * scale[2 p + 1],
// on top of z when `add`.
void scatter_input(const Grid &g, int pairs, int per, const int64_t *eq, const double *r, int64_t ld,
                   const float *feat, const double *scale, __nv_bfloat16 *x, cudaStream_t st);
void gather_output(const Grid &g, int pairs, int per, const int64_t *eq, const __nv_bfloat16 *y, const double *scale,
                   double *z, int64_t ld, bool add, cudaStream_t st);
// dy[v][a] = dz[eq[3v + a]] * scale[2 p + 1] (a < 3; the other 13 channels zero), BF16.
void scatter_grad(const Grid &g, int pairs, int per, const int64_t *eq, const double *dz, int64_t ld,
                  const double *scale, __nv_bfloat16 *dy, cudaStream_t st);

// Adam on n FP32 parameters: m = b1 m + (1 - b1) g, v = b2 v + (1 - b2) g^2,
// p -= lr (m / (1 - b1^t)) / (sqrt(v / (1 - b2^t)) + eps).
void adam(int64_t n, float *p, const float *g, float *m, float *v, float lr, float b1, float b2, float eps, int t,
          cudaStream_t st);

// ---- vector kernels (FP64) of flexible CG, scalars on the device --------------------------------
// out[k] = sum_i a_k[i] b_k[i] for the pairs (a, b) given; a fixed-order two-pass reduction
// (partials per CTA, then one CTA), so results are the same on every run.
void dots(int64_t n, int pairs, const double *const *a, const double *const *b, double *partial, double *out,
          cudaStream_t st);
// An iteration of flexible CG in three launches. A kernel leaves its sums as one partial a CTA, and
// the kernel that needs them adds the partials itself, every CTA in the same fixed order: no pass
// and no last CTA in between.
constexpr int MAX_KEPT = 8, FCG_CTAS = 148 * 8;
struct FcgStep {
  int64_t n;
  int update;                    // x += alpha p, r -= alpha q with alpha = p.r / p.q (0 when p.q is 0)
  const double *product;         // the product's partials (fcg_product)
  double *den;                   // receives p.q
  const double *p, *q;
  double *x, *r;
  double *z;                     // null: no preconditioner here; else z = B r, inv B's blocks (null: z = r)
  const double *inv;
  int kept;                      // partials of z . qj[j], j < kept
  const double *qj[MAX_KEPT];
  double *zq;                    // kept x fcg_step_ctas(n) partials
  double *rr;                    // fcg_step_ctas(n) partials of r . r
};
int fcg_step_ctas(int64_t n);
void fcg_step(const FcgStep &a, cudaStream_t st);
// p = z - sum_j beta_j p_j with beta_j = (z . q_j) / den[slot[j]], the numerators given as device
// scalars (num) or as fcg_step's partials (zq); p may be one of the p_j
void fcg_direction(int64_t n, int m, const double *z, const double *const *pj, const int *slot, const double *num,
                   const double *zq, const double *den, double *p, cudaStream_t st);
// q = A p (A by rows); the partials of p . r, then of p . q, in `sums` (2 x FCG_CTAS doubles)
void fcg_product(int64_t n, const int64_t *ptr, const int32_t *idx, const double *val, const double *p,
                 const double *r, double *q, double *sums, cudaStream_t st);
// out[k] = the sum of the partials of r . r at rr + k * FCG_CTAS, k < count
void fcg_norms(int64_t n, int count, const double *rr, double *out, cudaStream_t st);
// The passes' scales of `pairs` vectors from their nrm2 = ||r||^2 (dots): s[2 p] = sqrt(n) / ||r||,
// s[2 p + 1] = ||r|| / (sqrt(n) kref); with per = 2 (the odd network) the pass on r halves its
// output scale and the pass on -r has both negated.
void input_scales(int64_t n, int pairs, int per, const double *nrm2, double kref, double *s, cudaStream_t st);

}  // namespace unet
}  // namespace fc
