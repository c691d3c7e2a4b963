// Kernels of the learned preconditioner (see unet_kernels.cuh): 3x3x3 convolutions as implicit
// GEMMs on the BF16 tensor pipe (ldmatrix fragments, mma m16n8k16, FP32 accumulation), their
// weight gradients as GEMMs over voxels with a fixed-order reduction, grid transfers, Adam, and
// the FP64 vector kernels of flexible CG.
#include <algorithm>
#include <cstdint>

#include "spmv.cuh"
#include "unet_kernels.cuh"

namespace fc {
namespace unet {

namespace {

using bf16 = __nv_bfloat16;
// Programmatic dependent launch, as in kernels.cuh: a convolution loads its weights, which no
// kernel of a pass writes, before it waits for the kernel whose output it reads.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
constexpr float SLOPE = 0.05f;  // leaky ReLU: x for x > 0, SLOPE x otherwise
__device__ __forceinline__ float gate(float mask) { return mask > 0.f ? 1.f : SLOPE; }
// A weight gradient's tile: tx x ty voxels of a z plane, DW_VOXELS at most (DwTile); with the input's
// halo, a plane more on either side in z too, DW_HALO voxels at most.
constexpr int DW_VOXELS = 128, DW_HALO = 560, DW_TOGETHER = 4;
__host__ __device__ constexpr int dw_threads(int cout) { return 9 * (cout / 16) * 32; }
// A convolution's CTA: twelve warps of one or two groups of 16 voxels, so that a tile is 384 voxels at
// most (ConvTile), and the most voxels of a tile with its halo: two of them and the weights in 227 KB.
constexpr int CONV_WARPS = 12, CONV_THREADS = 32 * CONV_WARPS;
constexpr int CONV_VOXELS = 2 * 16 * CONV_WARPS, CONV_HALO = 1000;

__device__ __forceinline__ void cp16(void *smem, const void *gmem, bool ok) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(ok ? 16 : 0));
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;\n" ::); }

__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], const void *p) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(s));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], const void *p) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(s));
}
// D = A B + D, A 16 x 16 (row major), B 16 x 8 (column major), BF16 in, FP32 accumulate.
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
               "{%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__host__ __device__ constexpr int cstride(int c) { return c + 8; }  // shared-memory channel stride
// A convolution's tile: tx x ty x tz voxels, `halo` with a voxel more on every side, in one buffer or
// two.
struct ConvTile {
  int tx, ty, tz, halo, buffers;
};
template <int CIN, int COUT>
__host__ __device__ constexpr size_t conv_smem(int buffers, int halo) {
  return sizeof(bf16) * cstride(CIN) * ((size_t)27 * COUT + (size_t)buffers * halo);
}

// The halo of the tile at (x0, y0, z0), hx x hy x planes voxels from one before each, into shared
// memory, zero outside the grid: a row of hx voxels a warp at a time.
template <int CIN, int WARPS>
__device__ __forceinline__ void load_halo(bf16 *ts, const Grid &g, const bf16 *in, int x0, int y0, int z0, int hx,
                                          int hy, int planes) {
  constexpr int CS = cstride(CIN);
  for (int row = threadIdx.x >> 5; row < hy * planes; row += WARPS) {
    const int gy = y0 - 1 + row % hy, gz = z0 - 1 + row / hy;
    const bool in_grid = gy >= 0 && gy < g.Y && gz >= 0 && gz < g.Z;
    const int64_t v = in_grid ? ((int64_t)gz * g.Y + gy) * g.X : 0;
    for (int e = threadIdx.x & 31; e < hx * (CIN / 8); e += 32) {
      const int x = e / (CIN / 8), c8 = e % (CIN / 8), gx = x0 - 1 + x;
      const bool ok = in_grid && gx >= 0 && gx < g.X;
      cp16(ts + (row * hx + x) * CS + c8 * 8, in + (ok ? (v + gx) * CIN + c8 * 8 : 0), ok);
    }
  }
}

// NG groups of 16 voxels (group h's A rows at ts + at[h]) by COUT channels over the 27 taps; wl: this
// lane's row of the weights.
template <int CIN, int COUT, int NG>
__device__ __forceinline__ void conv_groups(float (&acc)[2][COUT / 8][4], const bf16 *ts, const int (&at)[2],
                                            const bf16 *wl, int hx, int hy) {
  constexpr int CS = cstride(CIN);
#pragma unroll
  for (int h = 0; h < NG; ++h)
#pragma unroll
    for (int nt = 0; nt < COUT / 8; ++nt) acc[h][nt][0] = acc[h][nt][1] = acc[h][nt][2] = acc[h][nt][3] = 0.f;
#pragma unroll 1
  for (int zy = 0; zy < 9; ++zy) {
    const bf16 *row = ts + (zy / 3 * hy + zy % 3) * hx * CS;
#pragma unroll
    for (int dx = 0; dx < 3; ++dx) {
#pragma unroll
      for (int ks = 0; ks < CIN / 16; ++ks) {
        uint32_t a[NG][4];
#pragma unroll
        for (int h = 0; h < NG; ++h) ldsm_x4(a[h], row + at[h] + dx * CS + ks * 16);
#pragma unroll
        for (int np = 0; np < COUT / 16; ++np) {
          uint32_t b[4];
          ldsm_x4(b, wl + ((3 * zy + dx) * COUT + np * 16) * CS + ks * 16);
#pragma unroll
          for (int h = 0; h < NG; ++h) {
            mma_bf16(acc[h][2 * np], a[h], b[0], b[1]);
            mma_bf16(acc[h][2 * np + 1], a[h], b[2], b[3]);
          }
        }
      }
    }
  }
}

// One CTA per tile of one of the batch's grids (persistent over tiles, the next one's halo in flight);
// all 27 taps' weights stay in shared memory. The tile's voxels, x fastest, are taken 16 by 16 as an
// MMA's rows wherever they lie in it (a fragment's rows are addressed lane by lane), so a tile fits the
// grid: a warp takes group `warp` and, where there are more, group warp + 12, by COUT channels. Bound by
// the fragments' shared-memory reads and the tensor pipe together: with one group a warp three fragments
// are read for four MMAs, with two four for eight. In tiles of 8 x 8 x 2, one group a warp, 39% of the
// MMAs on a 33 x 33 x 9 grid fell outside it (16 passes: 33 us, with tiles that fit 23). The passes of a
// batch run side by side: alone, a pass on a plate's grid has about one tile an SM and a launch is mostly
// the weights' load, which with one CTA an SM no longer runs beside the launch before (an application on
// 65 x 65 x 9 nodes 0.172 ms, 0.155 with two CTAs an SM; a training step on eight pairs 1.67 ms against 1.88).
template <int CIN, int COUT>
__global__ void __launch_bounds__(CONV_THREADS, 1)
    conv3_kernel(Grid g, int batch, ConvTile tile, const bf16 *__restrict__ in, const bf16 *__restrict__ w,
                 const float *__restrict__ bias, int relu, const bf16 *__restrict__ mask, bf16 *__restrict__ out) {
  constexpr int CS = cstride(CIN);
  extern __shared__ __align__(16) unsigned char smem[];
  bf16 *ws = reinterpret_cast<bf16 *>(smem);
  bf16 *buffers = ws + 27 * COUT * CS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gq = lane >> 2, tg = lane & 3, q = lane >> 3, r = lane & 7;
  for (int e = tid; e < 27 * COUT * (CIN / 8); e += CONV_THREADS) {
    const int row = e / (CIN / 8), c8 = e % (CIN / 8);
    cp16(ws + row * CS + c8 * 8, w + row * CIN + c8 * 8, true);
  }
  const int hx = tile.tx + 2, hy = tile.ty + 2, voxels_here = tile.tx * tile.ty * tile.tz;
  const int groups = (voxels_here + 15) / 16;
  const int mine = warp >= groups ? 0 : warp + CONV_WARPS >= groups ? 1 : 2;
  int at[2], place[2][2];  // A rows; and the voxels (x, y, z) this lane stores, -1 past the tile's
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int first = (warp + h * CONV_WARPS) * 16;
    int m = first + (q & 1) * 8 + r;
    if (m >= voxels_here) m = 0;
    at[h] = ((m / (tile.tx * tile.ty) * hy + m / tile.tx % tile.ty) * hx + m % tile.tx) * CS + (q >> 1) * 8;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      m = first + gq + 8 * e;
      place[h][e] = m < voxels_here ? m % tile.tx | m / tile.tx % tile.ty << 10 | m / (tile.tx * tile.ty) << 20 : -1;
    }
  }
  const bf16 *wl = ws + ((q >> 1) * 8 + r) * CS + (q & 1) * 8;
  const int ntx = (g.X + tile.tx - 1) / tile.tx, nty = (g.Y + tile.ty - 1) / tile.ty,
            ntz = (g.Z + tile.tz - 1) / tile.tz;
  const int ntiles = ntx * nty * ntz;
  const int64_t total = (int64_t)ntiles * batch, voxels = g.voxels();
  auto load = [&](int64_t t, bf16 *ts) {
    const int i = (int)(t % ntiles);
    load_halo<CIN, CONV_WARPS>(ts, g, in + t / ntiles * voxels * CIN, i % ntx * tile.tx, i / ntx % nty * tile.ty,
                               i / (ntx * nty) * tile.tz, hx, hy, tile.tz + 2);
  };
  pdl_wait();
  pdl_trigger();
  if (blockIdx.x < total) load(blockIdx.x, buffers);
  commit();
  int buffer = 0;
  for (int64_t t = blockIdx.x; t < total; t += gridDim.x) {
    const bf16 *ts = buffers + buffer * tile.halo * CS;
    if (t + gridDim.x < total) load(t + gridDim.x, buffers + (buffer ^ 1) * tile.halo * CS);
    commit();
    buffer ^= 1;
    asm volatile("cp.async.wait_group 1;\n" ::);
    __syncthreads();
    float acc[2][COUT / 8][4];
    if (mine == 2)
      conv_groups<CIN, COUT, 2>(acc, ts, at, wl, hx, hy);
    else if (mine == 1)
      conv_groups<CIN, COUT, 1>(acc, ts, at, wl, hx, hy);
    const int i = (int)(t % ntiles);
    const int64_t base = t / ntiles * voxels;
    const int x0 = i % ntx * tile.tx, y0 = i / ntx % nty * tile.ty, z0 = i / (ntx * nty) * tile.tz;
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int p = place[h][e], gx = x0 + (p & 1023), gy = y0 + (p >> 10 & 1023), gz = z0 + (p >> 20);
        if (h >= mine || p < 0 || gx >= g.X || gy >= g.Y || gz >= g.Z) continue;
        const int64_t v = base + ((int64_t)gz * g.Y + gy) * g.X + gx;
#pragma unroll
        for (int nt = 0; nt < COUT / 8; ++nt) {
          const int co = nt * 8 + 2 * tg;
          float v0 = acc[h][nt][2 * e], v1 = acc[h][nt][2 * e + 1];
          if (bias) v0 += bias[co], v1 += bias[co + 1];
          if (relu) v0 = v0 > 0.f ? v0 : SLOPE * v0, v1 = v1 > 0.f ? v1 : SLOPE * v1;
          if (mask) {
            const __nv_bfloat162 mk = *reinterpret_cast<const __nv_bfloat162 *>(mask + v * COUT + co);
            v0 *= gate(__bfloat162float(mk.x));
            v1 *= gate(__bfloat162float(mk.y));
          }
          *reinterpret_cast<__nv_bfloat162 *>(out + v * COUT + co) = __floats2bfloat162_rn(v0, v1);
        }
      }
    __syncthreads();
  }
}

// Weight gradient: CTA blockIdx.x takes a chunk of one pass's tiles (every pass cut alike, so that what
// cancels between two passes, as an odd network's output biases do, cancels to the last bit), warp w
// sixteen output channels (w / 9) of the three taps along x at
// (dy, dz) = (w % 9 % 3 - 1, w % 9 / 3 - 1), each the GEMM dW_tap (COUT x CIN) += dY^T (COUT x voxels)
// X_tap (voxels x CIN), both operands read transposed by ldmatrix.trans from channels-last tiles and
// dY's fragments shared by the three. The fifth warp of each nine also multiplies dY^T by ones: the bias
// gradient. A chunk's partial is 28 blocks of COUT x CIN floats, the taps' and one whose first COUT are
// the bias's. A tile's voxels, x fastest, are taken 16 by 16 wherever they lie in it, so a tile fits the
// grid (8 x 8 voxels: on a 33 x 33 plane a third of the products were outside it); past its last one dY
// is zero. The next tile's copies are in flight while a tile is multiplied. Nine warps with all the
// channels, 100 accumulators a thread, left one of the four schedulers three warps and the others two:
// 16 passes on a 33 x 33 x 9 grid took 53 us with both, 30 so. The tensor pipe truncates what it adds to
// an accumulator, so its sums leave it every DW_TOGETHER steps (64 voxels) and are added rounded: kept in
// it over a chunk of 4 100 voxels a gradient was off by 4.7e-6, now by 2e-7 (2-norm, eight pairs on 65 x
// 65 x 9 nodes). Half of the input channels at a time, so that both sums fit the registers, for an eighth
// more fragment reads: 63 -> 67 us on 33 x 33 x 9 nodes. Bound by the fragments'
// shared-memory reads and the tensor pipe.
struct DwTile {
  int tx, ty, tiles;  // tiles: of one pass
};
template <int CIN, int COUT>
__host__ __device__ constexpr size_t dw_smem() {
  return 2 * sizeof(bf16) * ((size_t)DW_HALO * cstride(CIN) + (size_t)DW_VOXELS * cstride(COUT));
}

template <int CIN, int COUT>
__global__ void __launch_bounds__(dw_threads(COUT)) conv3_dw_kernel(Grid g, DwTile tile, int chunks,
                                                                   const bf16 *__restrict__ in,
                                                                   const bf16 *__restrict__ dy,
                                                                   float *__restrict__ part) {
  constexpr int CS = cstride(CIN), DS = cstride(COUT), THREADS = dw_threads(COUT);
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int BUFFER = DW_HALO * CS + DW_VOXELS * DS;
  bf16 *buffers = reinterpret_cast<bf16 *>(smem);
  __shared__ int place[DW_VOXELS];  // where a voxel of the tile lies in its halo
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, unit = warp % 9, mt = warp / 9;
  const int gq = lane >> 2, tg = lane & 3, q = lane >> 3, r = lane & 7;
  const int hx = tile.tx + 2, hy = tile.ty + 2, here = tile.tx * tile.ty, steps = (here + 15) / 16;
  const int ntx = (g.X + tile.tx - 1) / tile.tx, nty = (g.Y + tile.ty - 1) / tile.ty;
  const int ntiles = ntx * nty * g.Z;
  const int per = (ntiles + chunks - 1) / chunks, t0 = blockIdx.x % chunks * per, t1 = min(ntiles, t0 + per);
  const int64_t base = (int64_t)(blockIdx.x / chunks) * g.voxels();
  for (int m = tid; m < DW_VOXELS; m += THREADS) place[m] = m < here ? (m / tile.tx * hx + m % tile.tx) * CS : 0;
  float acc[3][CIN / 8][4], bias[2] = {0.f, 0.f};
#pragma unroll
  for (int t = 0; t < 3; ++t)
#pragma unroll
    for (int nt = 0; nt < CIN / 8; ++nt) acc[t][nt][0] = acc[t][nt][1] = acc[t][nt][2] = acc[t][nt][3] = 0.f;
  auto load = [&](int i) {
    bf16 *ts = buffers + ((i - t0) & 1) * BUFFER, *ds = ts + DW_HALO * CS;
    const int x0 = i % ntx * tile.tx, y0 = i / ntx % nty * tile.ty, z = i / (ntx * nty);
    load_halo<CIN, THREADS / 32>(ts, g, in + base * CIN, x0, y0, z, hx, hy, 3);
    for (int e = tid; e < 16 * steps * (COUT / 8); e += THREADS) {
      const int m = e / (COUT / 8), c8 = e % (COUT / 8);
      const int gx = x0 + m % tile.tx, gy = y0 + m / tile.tx;
      const bool ok = m < here && gx < g.X && gy < g.Y;
      const int64_t v = base + (ok ? ((int64_t)z * g.Y + gy) * g.X + gx : 0);
      cp16(ds + m * DS + c8 * 8, dy + v * COUT + c8 * 8, ok);
    }
  };
  if (t0 < t1) load(t0);
  commit();
  for (int t = t0; t < t1; ++t) {
    if (t + 1 < t1) load(t + 1);  // into the buffer that the barrier below the last tile freed
    commit();
    asm volatile("cp.async.wait_group 1;\n" ::);
    __syncthreads();
    const bf16 *ts = buffers + ((t - t0) & 1) * BUFFER, *ds = ts + DW_HALO * CS;
    const bf16 *rows = ts + (unit / 3 * hy + unit % 3) * hx * CS + (q >> 1) * 8;
    for (int k0 = 0; k0 < steps; k0 += DW_TOGETHER) {
      const int k1 = min(steps, k0 + DW_TOGETHER);
#pragma unroll
      for (int np = 0; np < CIN / 16; ++np) {
        float here[3][2][4] = {}, ones[4] = {};
#pragma unroll 2
        for (int ks = k0; ks < k1; ++ks) {
          uint32_t a[4];  // rows: voxel ks 16 + (q >> 1) 8 + r; columns: channel
          ldsm_x4_t(a, ds + (ks * 16 + (q >> 1) * 8 + r) * DS + mt * 16 + (q & 1) * 8);
          if (unit == 4 && np == 0) mma_bf16(ones, a, 0x3f803f80u, 0x3f803f80u);
          const bf16 *brow = rows + place[ks * 16 + (q & 1) * 8 + r] + np * 16;  // B row: the voxel, shifted by the tap
#pragma unroll
          for (int dx = 0; dx < 3; ++dx) {
            uint32_t b[4];
            ldsm_x4_t(b, brow + dx * CS);
            mma_bf16(here[dx][0], a, b[0], b[1]);
            mma_bf16(here[dx][1], a, b[2], b[3]);
          }
        }
#pragma unroll
        for (int dx = 0; dx < 3; ++dx)
#pragma unroll
          for (int e = 0; e < 8; ++e) acc[dx][2 * np + e / 4][e % 4] += here[dx][e / 4][e % 4];
        if (np == 0) bias[0] += ones[0], bias[1] += ones[2];
      }
    }
    __syncthreads();
  }
  float *chunk_part = part + (int64_t)blockIdx.x * 28 * COUT * CIN;
#pragma unroll
  for (int dx = 0; dx < 3; ++dx) {
    float *dst = chunk_part + (3 * unit + dx) * COUT * CIN;  // tap dx + 3 (dy + 3 dz)
#pragma unroll
    for (int nt = 0; nt < CIN / 8; ++nt) {
      const int co = mt * 16 + gq, ci = nt * 8 + 2 * tg;
      *reinterpret_cast<float2 *>(dst + co * CIN + ci) = make_float2(acc[dx][nt][0], acc[dx][nt][1]);
      *reinterpret_cast<float2 *>(dst + (co + 8) * CIN + ci) = make_float2(acc[dx][nt][2], acc[dx][nt][3]);
    }
  }
  if (unit == 4 && tg == 0) {
    chunk_part[27 * COUT * CIN + mt * 16 + gq] = bias[0];
    chunk_part[27 * COUT * CIN + mt * 16 + gq + 8] = bias[1];
  }
}

// The chunks' partials of each pass added in a fixed order (8 threads an element take every eighth
// chunk, then those 8 sums in order), a pair's passes after one another and the pairs too: gw and gb
// receive the last pair's gradient; accw and accb (null: not kept) the sum of the pairs' gradients times
// `scale`, added to what they hold when `more`. Bound by the loads' latency: all passes' are in flight at
// once (16 passes of 9 chunks: 11 us with a cold cache; eight passes at a time, one after another, 24).
constexpr int REDUCE_WAYS = 8, REDUCE_ELEMENTS = 32, REDUCE_GRIDS = 16;
__global__ void __launch_bounds__(REDUCE_WAYS * REDUCE_ELEMENTS)
    dw_reduce_kernel(int pairs, int passes, int chunks, int weights, int cout, int64_t stride,
                     const float *__restrict__ part, float scale, int more, float *__restrict__ accw,
                     float *__restrict__ accb, float *__restrict__ gw, float *__restrict__ gb) {
  __shared__ float s[REDUCE_GRIDS][REDUCE_WAYS][REDUCE_ELEMENTS], total[REDUCE_GRIDS][REDUCE_ELEMENTS];
  const int el = threadIdx.x % REDUCE_ELEMENTS, way = threadIdx.x / REDUCE_ELEMENTS;
  const int e = blockIdx.x * REDUCE_ELEMENTS + el, grids = pairs * passes;
  const bool on = e < weights + cout;
  float *acc = accw ? (e < weights ? accw + e : accb + (e - weights)) : nullptr;
  float *grad = e < weights ? gw + e : gb + (e - weights);
  float sum = on && way == 0 && acc && more ? *acc : 0.f, last = 0.f;
  for (int p0 = 0; p0 < grids; p0 += REDUCE_GRIDS) {
    const int np = min(REDUCE_GRIDS, grids - p0);
    __syncthreads();
    float v[REDUCE_GRIDS];
#pragma unroll
    for (int p = 0; p < REDUCE_GRIDS; ++p) v[p] = 0.f;
    if (on)
      for (int c = way; c < chunks; c += REDUCE_WAYS) {
        float x[REDUCE_GRIDS];  // every pass's loads in flight
#pragma unroll
        for (int p = 0; p < REDUCE_GRIDS; ++p)
          x[p] = p < np ? part[((int64_t)(p0 + p) * chunks + c) * stride + e] : 0.f;
#pragma unroll
        for (int p = 0; p < REDUCE_GRIDS; ++p) v[p] += x[p];
      }
#pragma unroll
    for (int p = 0; p < REDUCE_GRIDS; ++p) s[p][way][el] = v[p];
    __syncthreads();
    // the ways' sums of a pass, a warp a pass; then the passes
    for (int p = way; p < np; p += REDUCE_WAYS) {
      float t = 0.f;
#pragma unroll
      for (int k = 0; k < REDUCE_WAYS; ++k) t += s[p][k][el];
      total[p][el] = t;
    }
    __syncthreads();
    if (way == 0)
      for (int p = 0; p < np; ++p) {
        const int pass = (p0 + p) % passes;
        last = pass == 0 ? total[p][el] : last + total[p][el];
        if (pass == passes - 1) sum += last * scale;
      }
  }
  if (on && way == 0) {
    *grad = last;
    if (acc) *acc = sum;
  }
}

// Every layer's BF16 weights and their flipped transposes from the FP32 parameters, a layer a
// blockIdx.y.
__global__ void refresh_kernel(LayerTable t, const float *__restrict__ p, bf16 *__restrict__ w, bf16 *__restrict__ wt) {
  const int l = blockIdx.y, cin = t.cin[l], cout = t.cout[l], total = 27 * cin * cout;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
    const int ci = e % cin, co = (e / cin) % cout, tap = e / (cin * cout);
    const bf16 v = __float2bfloat16_rn(p[t.param[l] + e]);
    w[t.weight[l] + e] = v;
    wt[t.weight[l] + ((26 - tap) * cin + ci) * cout + co] = v;
  }
}

constexpr int C32 = 32;
// The grid transfers: blockIdx.y is the grid of the batch.
__global__ void pool_kernel(Grid gf, Grid gc, const bf16 *__restrict__ fine, bf16 *__restrict__ coarse) {
  fine += blockIdx.y * gf.voxels() * C32;
  coarse += blockIdx.y * gc.voxels() * C32;
  const int64_t total = gc.voxels() * (C32 / 2);
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(e % (C32 / 2)) * 2;
    const int64_t vc = e / (C32 / 2);
    const int x = (int)(vc % gc.X), y = (int)((vc / gc.X) % gc.Y), z = (int)(vc / ((int64_t)gc.X * gc.Y));
    float s0 = 0.f, s1 = 0.f;
    for (int k = 0; k < 8; ++k) {
      const int fx = 2 * x + (k & 1), fy = 2 * y + ((k >> 1) & 1), fz = 2 * z + (k >> 2);
      if (fx >= gf.X || fy >= gf.Y || fz >= gf.Z) continue;
      const __nv_bfloat162 f =
          *reinterpret_cast<const __nv_bfloat162 *>(fine + (((int64_t)fz * gf.Y + fy) * gf.X + fx) * C32 + c);
      s0 += __bfloat162float(f.x), s1 += __bfloat162float(f.y);
    }
    *reinterpret_cast<__nv_bfloat162 *>(coarse + vc * C32 + c) = __floats2bfloat162_rn(s0 * 0.125f, s1 * 0.125f);
  }
}

__global__ void up_add_kernel(Grid gf, Grid gc, const bf16 *__restrict__ coarse, const bf16 *__restrict__ skip,
                              bf16 *__restrict__ fine) {
  coarse += blockIdx.y * gc.voxels() * C32;
  skip += blockIdx.y * gf.voxels() * C32;
  fine += blockIdx.y * gf.voxels() * C32;
  const int64_t total = gf.voxels() * (C32 / 2);
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(e % (C32 / 2)) * 2;
    const int64_t v = e / (C32 / 2);
    const int x = (int)(v % gf.X), y = (int)((v / gf.X) % gf.Y), z = (int)(v / ((int64_t)gf.X * gf.Y));
    const int64_t vc = ((int64_t)(z / 2) * gc.Y + y / 2) * gc.X + x / 2;
    const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162 *>(coarse + vc * C32 + c);
    const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162 *>(skip + v * C32 + c);
    *reinterpret_cast<__nv_bfloat162 *>(fine + v * C32 + c) = __floats2bfloat162_rn(
        __bfloat162float(a.x) + __bfloat162float(b.x), __bfloat162float(a.y) + __bfloat162float(b.y));
  }
}

__global__ void up_adjoint_kernel(Grid gf, Grid gc, const bf16 *__restrict__ dfine, const bf16 *__restrict__ mask,
                                  bf16 *__restrict__ dcoarse) {
  dfine += blockIdx.y * gf.voxels() * C32;
  mask += blockIdx.y * gc.voxels() * C32;
  dcoarse += blockIdx.y * gc.voxels() * C32;
  const int64_t total = gc.voxels() * (C32 / 2);
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(e % (C32 / 2)) * 2;
    const int64_t vc = e / (C32 / 2);
    const int x = (int)(vc % gc.X), y = (int)((vc / gc.X) % gc.Y), z = (int)(vc / ((int64_t)gc.X * gc.Y));
    float s0 = 0.f, s1 = 0.f;
    for (int k = 0; k < 8; ++k) {
      const int fx = 2 * x + (k & 1), fy = 2 * y + ((k >> 1) & 1), fz = 2 * z + (k >> 2);
      if (fx >= gf.X || fy >= gf.Y || fz >= gf.Z) continue;
      const __nv_bfloat162 f =
          *reinterpret_cast<const __nv_bfloat162 *>(dfine + (((int64_t)fz * gf.Y + fy) * gf.X + fx) * C32 + c);
      s0 += __bfloat162float(f.x), s1 += __bfloat162float(f.y);
    }
    const __nv_bfloat162 mk = *reinterpret_cast<const __nv_bfloat162 *>(mask + vc * C32 + c);
    s0 *= gate(__bfloat162float(mk.x));
    s1 *= gate(__bfloat162float(mk.y));
    *reinterpret_cast<__nv_bfloat162 *>(dcoarse + vc * C32 + c) = __floats2bfloat162_rn(s0, s1);
  }
}

__global__ void pool_adjoint_kernel(Grid gf, Grid gc, const bf16 *__restrict__ dcoarse, const bf16 *__restrict__ dskip,
                                    const bf16 *__restrict__ mask, bf16 *__restrict__ dfine) {
  dcoarse += blockIdx.y * gc.voxels() * C32;
  dskip += blockIdx.y * gf.voxels() * C32;
  mask += blockIdx.y * gf.voxels() * C32;
  dfine += blockIdx.y * gf.voxels() * C32;
  const int64_t total = gf.voxels() * (C32 / 2);
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(e % (C32 / 2)) * 2;
    const int64_t v = e / (C32 / 2);
    const int x = (int)(v % gf.X), y = (int)((v / gf.X) % gf.Y), z = (int)(v / ((int64_t)gf.X * gf.Y));
    const int64_t vc = ((int64_t)(z / 2) * gc.Y + y / 2) * gc.X + x / 2;
    const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162 *>(dcoarse + vc * C32 + c);
    const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162 *>(dskip + v * C32 + c);
    const __nv_bfloat162 mk = *reinterpret_cast<const __nv_bfloat162 *>(mask + v * C32 + c);
    const float s0 = (__bfloat162float(a.x) * 0.125f + __bfloat162float(b.x)) * gate(__bfloat162float(mk.x));
    const float s1 = (__bfloat162float(a.y) * 0.125f + __bfloat162float(b.y)) * gate(__bfloat162float(mk.y));
    *reinterpret_cast<__nv_bfloat162 *>(dfine + v * C32 + c) = __floats2bfloat162_rn(s0, s1);
  }
}

constexpr int CIO = 16;  // channels of the network's input and output grids
// Pass p of a batch (blockIdx.y) belongs to pair p / per (per passes a pair: r, or r and -r); its
// scales are scale[2 p] (input) and scale[2 p + 1] (output).
__global__ void scatter_input_kernel(Grid g, int per, const int64_t *__restrict__ eq, const double *__restrict__ r,
                                     int64_t ld, const float *__restrict__ feat, const double *__restrict__ scale,
                                     bf16 *__restrict__ x) {
  const int64_t total = g.voxels();
  const double s = scale[2 * blockIdx.y];
  r += blockIdx.y / per * ld;
  x += blockIdx.y * total * CIO;
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < total; v += (int64_t)gridDim.x * blockDim.x) {
    float c[4];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const int64_t q = eq[3 * v + a];
      c[a] = q >= 0 ? (float)(r[q] * s) : 0.f;
    }
    c[3] = feat[v];
    const __nv_bfloat162 lo = __floats2bfloat162_rn(c[0], c[1]), hi = __floats2bfloat162_rn(c[2], c[3]);
    uint4 *dst = reinterpret_cast<uint4 *>(x + v * CIO);
    dst[0] = make_uint4(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi), 0u, 0u);
    dst[1] = make_uint4(0u, 0u, 0u, 0u);
  }
}

// z (+)= the passes' outputs of pair blockIdx.y, added in pass order: add != 0 adds them to z.
__global__ void gather_output_kernel(Grid g, int per, const int64_t *__restrict__ eq, const bf16 *__restrict__ y,
                                     const double *__restrict__ scale, double *__restrict__ z, int64_t ld, int add) {
  const int64_t voxels = g.voxels(), total = voxels * 3;
  z += blockIdx.y * ld;
  y += blockIdx.y * per * voxels * CIO;
  scale += 2 * blockIdx.y * per;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t v = e / 3;
    const int c = (int)(e % 3);
    const int64_t q = eq[3 * v + c];
    if (q < 0) continue;
    // products and sums rounded one by one: the odd network's output changes sign with r exactly
    double sum = 0.0;
    for (int p = 0; p < per; ++p)
      sum = __dadd_rn(sum, __dmul_rn((double)__bfloat162float(y[(p * voxels + v) * CIO + c]), scale[2 * p + 1]));
    z[q] = add ? z[q] + sum : sum;
  }
}

__global__ void scatter_grad_kernel(Grid g, int per, const int64_t *__restrict__ eq, const double *__restrict__ dz,
                                    int64_t ld, const double *__restrict__ scale, bf16 *__restrict__ dy) {
  const int64_t total = g.voxels();
  const double s = scale[2 * blockIdx.y + 1];
  dz += blockIdx.y / per * ld;
  dy += blockIdx.y * total * CIO;
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < total; v += (int64_t)gridDim.x * blockDim.x) {
    float c[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const int64_t q = eq[3 * v + a];
      c[a] = q >= 0 ? (float)(dz[q] * s) : 0.f;
    }
    const __nv_bfloat162 lo = __floats2bfloat162_rn(c[0], c[1]), hi = __floats2bfloat162_rn(c[2], 0.f);
    uint4 *dst = reinterpret_cast<uint4 *>(dy + v * CIO);
    dst[0] = make_uint4(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi), 0u, 0u);
    dst[1] = make_uint4(0u, 0u, 0u, 0u);
  }
}

__global__ void adam_kernel(int64_t n, float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m,
                            float *__restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const float gr = g[e];
    const float mm = b1 * m[e] + (1.f - b1) * gr;
    const float vv = b2 * v[e] + (1.f - b2) * gr * gr;
    m[e] = mm, v[e] = vv;
    p[e] -= lr * (mm / c1) / (sqrtf(vv / c2) + eps);
  }
}

// ---- FCG vectors --------------------------------------------------------------------------------
constexpr int DOT_CTAS = 296, MAX_PAIRS = 8;
struct PairPtrs {
  const double *a[MAX_PAIRS], *b[MAX_PAIRS];
};
struct DirPtrs {
  const double *p[MAX_KEPT];
  int slot[MAX_KEPT];  // where each direction's denominator p_j.q_j is kept
};
// The sum of a CTA's 256 values, in every thread of the first warp: a fixed tree.
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double s[8];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
  __syncthreads();
  double sum = 0.0;
#pragma unroll
  for (int w = 0; w < 8; ++w) sum += s[w];
  return sum;
}
// blockIdx.y is the pair
__global__ void __launch_bounds__(256) dot_part_kernel(int64_t n, PairPtrs pp, double *__restrict__ part) {
  const int64_t per = (n + gridDim.x - 1) / gridDim.x;
  const int64_t i0 = blockIdx.x * per, i1 = min(n, i0 + per);
  const double *a = pp.a[blockIdx.y], *b = pp.b[blockIdx.y];
  double acc = 0.0;
  for (int64_t i = i0 + threadIdx.x; i < i1; i += blockDim.x) acc += a[i] * b[i];
  acc = block_sum(acc);
  if (threadIdx.x == 0) part[blockIdx.y * gridDim.x + blockIdx.x] = acc;
}
__global__ void __launch_bounds__(256) dot_final_kernel(int ctas, const double *__restrict__ part,
                                                        double *__restrict__ out) {
  double acc = 0.0;
  for (int b = threadIdx.x; b < ctas; b += blockDim.x) acc += part[blockIdx.x * ctas + b];
  acc = block_sum(acc);
  if (threadIdx.x == 0) out[blockIdx.x] = acc;
}

// ---- an iteration of flexible CG, three launches ------------------------------------------------
// Each is a programmatic dependent of the one before it (its CTAs are there when that one ends). Bound
// by the latency of three launches and by K from L2. As eleven launches, with a second launch for
// every sum, an iteration on 48 x 48 x 8 elements took 95 us; with each sum finished by the last CTA
// of the kernel that forms it (a fence, an atomic and another pass at the end of two kernels) 36; with
// the partials added where they are read 28. 64 threads a CTA in the step: 20 000 nodes are then 306
// CTAs, two an SM, and not 77.
constexpr int FCG_THREADS = 256, STEP_THREADS = 64;

// The CTA's sums of v[k] into part[k * ctas + blockIdx.x], k < count: a fixed tree.
template <int K, int THREADS>
__device__ __forceinline__ void cta_partials(double (&v)[K], int count, double *const (&part)[K]) {
  constexpr int WARPS = THREADS / 32;
  __shared__ double s[K][WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    if (lane == 0) s[k][warp] = v[k];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < K; ++k)
    if (k < count && (int)threadIdx.x == k) {
      double sum = 0.0;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) sum += s[k][w];
      part[k][blockIdx.x] = sum;
    }
}

// out[k] (shared) = the sum of part[k * stride + b], b < ctas, k < count, on every CTA the same: warps
// take sums in turn, each lane every 32nd partial, eight loads in flight.
template <int THREADS>
__device__ __forceinline__ void add_partials(const double *part, int64_t stride, int ctas, int count, double *out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int k = warp; k < count; k += THREADS / 32) {
    double sum = 0.0;
#pragma unroll 8
    for (int b = lane; b < ctas; b += 32) sum += part[k * stride + b];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) out[k] = sum;
  }
  __syncthreads();
}

__host__ __device__ inline int step_ctas(int64_t n) {
  const int64_t c = ((n + 2) / 3 + STEP_THREADS - 1) / STEP_THREADS;
  return (int)(c < 1 ? 1 : c > FCG_CTAS ? FCG_CTAS : c);
}
// The product's CTAs, all resident at once, every one the same number of rounds of rows: a CTA's partial
// sums follow its last round, and a second wave of CTAs started its rounds after the first one's end
// (912 CTAs, 740 of them resident: 32.2 us an iteration on 48 x 48 x 8 elements; four an SM 30.3, five
// 30.7, six with fewer registers 31.9).
constexpr int PRODUCT_PER_SM = 4;
__host__ __device__ inline int product_ctas(int64_t n) {
  constexpr int ROWS = FCG_THREADS / SPMV_LANES;
  const int64_t groups = (n + ROWS - 1) / ROWS, rounds = (groups + 148 * PRODUCT_PER_SM - 1) / (148 * PRODUCT_PER_SM);
  return groups < 1 ? 1 : (int)((groups + rounds - 1) / rounds);
}

// A thread a node (three equations), 64 a CTA: with `update`, x += alpha p and r -= alpha q; then, with
// `z`, z = B r (inv: B's 3 x 3 blocks; null: z = r) and its products with the kept directions' q_j;
// always r.r.
__global__ void __launch_bounds__(STEP_THREADS) fcg_step_kernel(FcgStep a) {
  __shared__ double pr_pq[2];
  pdl_wait();
  pdl_trigger();
  double v[1 + MAX_KEPT];
#pragma unroll
  for (int k = 0; k <= MAX_KEPT; ++k) v[k] = 0.0;
  double alpha = 0.0;
  if (a.update) {
    add_partials<STEP_THREADS>(a.product, FCG_CTAS, product_ctas(a.n), 2, pr_pq);
    alpha = pr_pq[1] != 0.0 ? pr_pq[0] / pr_pq[1] : 0.0;
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.den = pr_pq[1];
  }
  const int64_t nodes = (a.n + 2) / 3;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nodes; k += (int64_t)gridDim.x * blockDim.x) {
    double r[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int64_t i = 3 * k + c;
      r[c] = i < a.n ? a.r[i] : 0.0;
      if (a.update && i < a.n) {
        a.x[i] += alpha * a.p[i];
        r[c] -= alpha * a.q[i];
        a.r[i] = r[c];
      }
      v[0] += r[c] * r[c];
    }
    if (!a.z) continue;
    double z[3] = {r[0], r[1], r[2]};
    if (a.inv) {
      const double *o = a.inv + 9 * k;
#pragma unroll
      for (int c = 0; c < 3; ++c) z[c] = o[3 * c] * r[0] + o[3 * c + 1] * r[1] + o[3 * c + 2] * r[2];
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int64_t i = 3 * k + c;
      if (i >= a.n) continue;
      a.z[i] = z[c];
#pragma unroll
      for (int j = 0; j < MAX_KEPT; ++j)
        if (j < a.kept) v[1 + j] += z[c] * a.qj[j][i];
    }
  }
  double *part[1 + MAX_KEPT];
  part[0] = a.rr;
#pragma unroll
  for (int j = 0; j < MAX_KEPT; ++j) part[1 + j] = a.zq + (int64_t)j * gridDim.x;
  cta_partials<1 + MAX_KEPT, STEP_THREADS>(v, 1 + (a.z ? a.kept : 0), part);
}

__global__ void __launch_bounds__(FCG_THREADS) fcg_direction_kernel(int64_t n, int m, const double *z, DirPtrs pj,
                                                                    const double *num, const double *zq,
                                                                    const double *den, double *p) {
  __shared__ double sums[MAX_KEPT];
  pdl_wait();
  pdl_trigger();
  if (zq && m > 0) {
    const int ctas = step_ctas(n);
    add_partials<FCG_THREADS>(zq, ctas, ctas, m, sums);
    num = sums;
  }
  double beta[MAX_KEPT];
#pragma unroll
  for (int j = 0; j < MAX_KEPT; ++j) {
    const double d = j < m ? den[pj.slot[j]] : 0.0;
    beta[j] = d != 0.0 ? num[j] / d : 0.0;
  }
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double old[MAX_KEPT], v = z[i];
#pragma unroll
    for (int j = 0; j < MAX_KEPT; ++j) old[j] = j < m ? pj.p[j][i] : 0.0;
#pragma unroll
    for (int j = 0; j < MAX_KEPT; ++j)
      if (j < m) v -= beta[j] * old[j];
    p[i] = v;
  }
}

__global__ void __launch_bounds__(FCG_THREADS, PRODUCT_PER_SM)
    fcg_product_kernel(int64_t n, const int64_t *__restrict__ ptr, const int32_t *__restrict__ idx,
                       const double *__restrict__ val, const double *p, const double *r, double *q, double *sums) {
  pdl_wait();
  pdl_trigger();
  double v[2] = {0.0, 0.0};
  constexpr int ROWS = FCG_THREADS / SPMV_LANES;
  const int lane = threadIdx.x % SPMV_LANES;
  // every lane of a warp goes round as often as its last row: the sums are taken by shuffles
  const int64_t step = (int64_t)gridDim.x * ROWS;
  int64_t row = blockIdx.x * (int64_t)ROWS + threadIdx.x / SPMV_LANES;
  int64_t e0 = row < n ? ptr[row] : 0, e1 = row < n ? ptr[row + 1] : 0;
  for (int64_t base = blockIdx.x * (int64_t)ROWS; base < n; base += step, row += step) {
    // where the next row lies is read beside this one
    const int64_t f0 = row + step < n ? ptr[row + step] : 0, f1 = row + step < n ? ptr[row + step + 1] : 0;
    const double sum = spmv_entries(e0, e1, idx, val, p, lane);
    e0 = f0, e1 = f1;
    if (row < n && lane == 0) {
      q[row] = sum;
      const double pr = p[row];
      v[0] += pr * r[row];
      v[1] += pr * sum;
    }
  }
  double *const part[2] = {sums, sums + FCG_CTAS};
  cta_partials<2, FCG_THREADS>(v, 2, part);
}

__global__ void __launch_bounds__(FCG_THREADS) fcg_norms_kernel(int count, int ctas, const double *rr, double *out) {
  __shared__ double sums[8];
  add_partials<FCG_THREADS>(rr, FCG_CTAS, ctas, count, sums);
  if ((int)threadIdx.x < count) out[threadIdx.x] = sums[threadIdx.x];
}

// The passes' scales of pair threadIdx.x from nrm2 = ||r||^2: (sqrt(n) / ||r||, ||r|| / (sqrt(n) kref)),
// for the two passes of an odd network (s0, s1 / 2) and (-s0, -s1 / 2).
__global__ void input_scales_kernel(int64_t n, const double *__restrict__ nrm2, double kref, int per,
                                    double *__restrict__ s) {
  const double nr = sqrt(nrm2[threadIdx.x]);
  const double sn = sqrt((double)n);
  const double s0 = nr > 0.0 ? sn / nr : 0.0, s1 = nr / (sn * kref);
  s += 2 * per * threadIdx.x;
  s[0] = s0;
  s[1] = per == 2 ? 0.5 * s1 : s1;
  if (per == 2) s[2] = -s0, s[3] = -0.5 * s1;
}

int grid_for(int64_t work) { return (int)std::max<int64_t>(1, std::min<int64_t>((work + 255) / 256, 148 * 8)); }

// The sides of n voxels cut in equal parts, the last one shorter: `most` at most, 3 at least.
int sides(int n, int most, int (&out)[64]) {
  int count = 0;
  for (int parts = (n + most - 1) / most; parts <= n && count < 64; ++parts) {
    const int side = (n + parts - 1) / parts;
    if (count > 0 && side < 3) break;
    if (count == 0 || out[count - 1] != side) out[count++] = side;
  }
  return count;
}

// The tile of a convolution over `batch` grids: the sides divide the grid's evenly, and of those the
// one with the least work for the busiest SM, in groups of 16 voxels: its rounds of tiles, each its
// groups (six at least, a lone group being latency) and about one and a half for its barriers and
// stores, and the first halo's load, which nothing covers.
ConvTile conv_tile(const Grid &g, int batch, int sms) {
  ConvTile best{};
  double least = 0.0;
  int xs[64], ys[64], zs[64];
  const int nx = sides(g.X, 24, xs), ny = sides(g.Y, 24, ys), nz = sides(g.Z, 16, zs);
  for (int k = 0; k < nz; ++k)
    for (int j = 0; j < ny; ++j)
      for (int i = 0; i < nx; ++i) {
        const int tx = xs[i], ty = ys[j], tz = zs[k], halo = (tx + 2) * (ty + 2) * (tz + 2);
        if (tx * ty * tz > CONV_VOXELS || halo > CONV_HALO) continue;
        const int64_t tiles = (int64_t)batch * ((g.X + tx - 1) / tx) * ((g.Y + ty - 1) / ty) * ((g.Z + tz - 1) / tz);
        const int64_t rounds = (tiles + sms - 1) / sms;
        const int groups = std::max(6, (tx * ty * tz + 15) / 16);
        const double cost = rounds * (groups + 1.5) + halo / 250.0;
        if (best.tx == 0 || cost < least) least = cost, best = ConvTile{tx, ty, tz, halo, rounds > 1 ? 2 : 1};
      }
  return best;
}

template <int CIN, int COUT>
void conv3_launch(const Grid &g, int batch, const bf16 *in, const bf16 *w, const float *bias, bool relu,
                  const bf16 *mask, bf16 *out, cudaStream_t st) {
  static const int sms = [] {
    cudaFuncSetAttribute(conv3_kernel<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)conv_smem<CIN, COUT>(2, CONV_HALO));
    int dev = 0, count = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev);
    return std::max(count, 1);
  }();
  // the last sizes' tiles: a network's passes go over the same few grids
  struct Known {
    int X, Y, Z, batch;
    ConvTile tile;
  };
  static thread_local Known known[32] = {};
  Known &k = known[(uint32_t)(g.X * 31 + g.Y * 17 + g.Z * 7 + batch) % 32];
  if (k.X != g.X || k.Y != g.Y || k.Z != g.Z || k.batch != batch)
    k = Known{g.X, g.Y, g.Z, batch, conv_tile(g, batch, sms)};
  const ConvTile tile = k.tile;
  const int64_t tiles = (int64_t)batch * ((g.X + tile.tx - 1) / tile.tx) * ((g.Y + tile.ty - 1) / tile.ty) *
                        ((g.Z + tile.tz - 1) / tile.tz);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)std::max<int64_t>(1, std::min<int64_t>(tiles, sms)));
  cfg.blockDim = dim3(CONV_THREADS);
  cfg.dynamicSmemBytes = conv_smem<CIN, COUT>(tile.buffers, tile.halo);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, conv3_kernel<CIN, COUT>, g, batch, tile, in, w, bias, relu ? 1 : 0, mask, out);
}

// The chunks of a pass: at most one a CTA over all passes, and a CTA an SM (18 warps of 96 registers a
// thread), so that they run in one wave.
int chunks_of(int64_t tiles, int grids) {
  return (int)std::max<int64_t>(1, std::min<int64_t>(tiles, DW_PARTIALS / grids));
}

// A weight gradient's tile: the one with the least steps of 16 voxels in its longest chunk, a tile's
// barriers about a step.
DwTile dw_tile(const Grid &g, int grids) {
  struct Known {
    int X, Y, Z, grids;
    DwTile tile;
  };
  static thread_local Known known[32] = {};
  Known &k = known[(uint32_t)(g.X * 31 + g.Y * 17 + g.Z * 7 + grids) % 32];
  if (k.X == g.X && k.Y == g.Y && k.Z == g.Z && k.grids == grids) return k.tile;
  DwTile best{};
  double least = 0.0;
  int xs[64], ys[64];
  const int nx = sides(g.X, 24, xs), ny = sides(g.Y, 24, ys);
  for (int j = 0; j < ny; ++j)
    for (int i = 0; i < nx; ++i) {
      const int tx = xs[i], ty = ys[j];
      if (tx * ty > DW_VOXELS || (tx + 2) * (ty + 2) * 3 > DW_HALO) continue;
      const int64_t tiles = (int64_t)((g.X + tx - 1) / tx) * ((g.Y + ty - 1) / ty) * g.Z;
      const int chunks = chunks_of(tiles, grids);
      const double cost = (double)((tiles + chunks - 1) / chunks) * ((tx * ty + 15) / 16 + 1.0);
      if (best.tx == 0 || cost < least) least = cost, best = DwTile{tx, ty, (int)tiles};
    }
  k = Known{g.X, g.Y, g.Z, grids, best};
  return best;
}

template <int CIN, int COUT>
void dw_launch(const Grid &g, int pairs, int passes, const bf16 *in, const bf16 *dy, float *part, float scale,
               bool more, float *accw, float *accb, float *gw, float *gb, cudaStream_t st) {
  constexpr size_t smem = dw_smem<CIN, COUT>();
  static const bool configured =
      cudaFuncSetAttribute(conv3_dw_kernel<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) ==
      cudaSuccess;
  (void)configured;
  const int grids = pairs * passes;
  const DwTile tile = dw_tile(g, grids);
  const int chunks = chunks_of(tile.tiles, grids);
  conv3_dw_kernel<CIN, COUT><<<grids * chunks, dw_threads(COUT), smem, st>>>(g, tile, chunks, in, dy, part);
  const int elements = 27 * CIN * COUT + COUT;
  dw_reduce_kernel<<<(elements + REDUCE_ELEMENTS - 1) / REDUCE_ELEMENTS, REDUCE_WAYS * REDUCE_ELEMENTS, 0, st>>>(
      pairs, passes, chunks, 27 * CIN * COUT, COUT, (int64_t)28 * CIN * COUT, part, scale, more ? 1 : 0, accw, accb, gw, gb);
}

}  // namespace

void conv3(const Grid &g, int batch, int cin, int cout, const __nv_bfloat16 *in, const __nv_bfloat16 *w,
           const float *bias, bool relu, const __nv_bfloat16 *mask, __nv_bfloat16 *out, cudaStream_t st) {
  if (cin == 32 && cout == 32)
    conv3_launch<32, 32>(g, batch, in, w, bias, relu, mask, out, st);
  else if (cin == 16 && cout == 32)
    conv3_launch<16, 32>(g, batch, in, w, bias, relu, mask, out, st);
  else if (cin == 32 && cout == 16)
    conv3_launch<32, 16>(g, batch, in, w, bias, relu, mask, out, st);
  else
    conv3_launch<16, 16>(g, batch, in, w, bias, relu, mask, out, st);
}

int dw_chunks(const Grid &g, int grids) { return chunks_of(dw_tile(g, grids).tiles, grids); }

void conv3_dw(const Grid &g, int cin, int cout, int pairs, int passes, const __nv_bfloat16 *in,
              const __nv_bfloat16 *dy, float *part, float scale, bool more, float *accw, float *accb, float *gw,
              float *gb, cudaStream_t st) {
  if (cin == 32 && cout == 32)
    dw_launch<32, 32>(g, pairs, passes, in, dy, part, scale, more, accw, accb, gw, gb, st);
  else if (cin == 16 && cout == 32)
    dw_launch<16, 32>(g, pairs, passes, in, dy, part, scale, more, accw, accb, gw, gb, st);
  else if (cin == 32 && cout == 16)
    dw_launch<32, 16>(g, pairs, passes, in, dy, part, scale, more, accw, accb, gw, gb, st);
  else
    dw_launch<16, 16>(g, pairs, passes, in, dy, part, scale, more, accw, accb, gw, gb, st);
}

void refresh(const LayerTable &t, const float *p, __nv_bfloat16 *w, __nv_bfloat16 *wt, cudaStream_t st) {
  refresh_kernel<<<dim3(27, t.layers), 256, 0, st>>>(t, p, w, wt);
}

void pool(const Grid &gf, const Grid &gc, int batch, const __nv_bfloat16 *fine, __nv_bfloat16 *coarse,
          cudaStream_t st) {
  pool_kernel<<<dim3(grid_for(gc.voxels() * 16), batch), 256, 0, st>>>(gf, gc, fine, coarse);
}
void up_add(const Grid &gf, const Grid &gc, int batch, const __nv_bfloat16 *coarse, const __nv_bfloat16 *skip,
            __nv_bfloat16 *fine, cudaStream_t st) {
  up_add_kernel<<<dim3(grid_for(gf.voxels() * 16), batch), 256, 0, st>>>(gf, gc, coarse, skip, fine);
}
void up_adjoint(const Grid &gf, const Grid &gc, int batch, const __nv_bfloat16 *dfine, const __nv_bfloat16 *mask,
                __nv_bfloat16 *dcoarse, cudaStream_t st) {
  up_adjoint_kernel<<<dim3(grid_for(gc.voxels() * 16), batch), 256, 0, st>>>(gf, gc, dfine, mask, dcoarse);
}
void pool_adjoint(const Grid &gf, const Grid &gc, int batch, const __nv_bfloat16 *dcoarse,
                  const __nv_bfloat16 *dskip, const __nv_bfloat16 *mask, __nv_bfloat16 *dfine, cudaStream_t st) {
  pool_adjoint_kernel<<<dim3(grid_for(gf.voxels() * 16), batch), 256, 0, st>>>(gf, gc, dcoarse, dskip, mask, dfine);
}

void scatter_input(const Grid &g, int pairs, int per, const int64_t *eq, const double *r, int64_t ld,
                   const float *feat, const double *scale, __nv_bfloat16 *x, cudaStream_t st) {
  scatter_input_kernel<<<dim3(grid_for(g.voxels()), pairs * per), 256, 0, st>>>(g, per, eq, r, ld, feat, scale, x);
}
void gather_output(const Grid &g, int pairs, int per, const int64_t *eq, const __nv_bfloat16 *y, const double *scale,
                   double *z, int64_t ld, bool add, cudaStream_t st) {
  gather_output_kernel<<<dim3(grid_for(g.voxels() * 3), pairs), 256, 0, st>>>(g, per, eq, y, scale, z, ld,
                                                                              add ? 1 : 0);
}
void scatter_grad(const Grid &g, int pairs, int per, const int64_t *eq, const double *dz, int64_t ld,
                  const double *scale, __nv_bfloat16 *dy, cudaStream_t st) {
  scatter_grad_kernel<<<dim3(grid_for(g.voxels()), pairs * per), 256, 0, st>>>(g, per, eq, dz, ld, scale, dy);
}

void adam(int64_t n, float *p, const float *g, float *m, float *v, float lr, float b1, float b2, float eps, int t,
          cudaStream_t st) {
  const float c1 = 1.f - powf(b1, (float)t), c2 = 1.f - powf(b2, (float)t);
  adam_kernel<<<grid_for(n), 256, 0, st>>>(n, p, g, m, v, lr, b1, b2, eps, c1, c2);
}

void dots(int64_t n, int pairs, const double *const *a, const double *const *b, double *partial, double *out,
          cudaStream_t st) {
  PairPtrs pp{};
  for (int k = 0; k < pairs && k < MAX_PAIRS; ++k) pp.a[k] = a[k], pp.b[k] = b[k];
  if (pairs < 1) return;
  dot_part_kernel<<<dim3(DOT_CTAS, pairs), 256, 0, st>>>(n, pp, partial);
  dot_final_kernel<<<pairs, 256, 0, st>>>(DOT_CTAS, partial, out);
}

// A launch that may start while the stream's previous kernel ends (its kernel waits for it).
template <class... P, class... A>
static void launch_dependent(void (*kernel)(P...), int64_t grid, int threads, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)std::max<int64_t>(grid, 1));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, args...);
}

int fcg_step_ctas(int64_t n) { return step_ctas(n); }

void fcg_step(const FcgStep &a, cudaStream_t st) {
  launch_dependent(fcg_step_kernel, step_ctas(a.n), STEP_THREADS, st, a);
}

void fcg_direction(int64_t n, int m, const double *z, const double *const *pj, const int *slot, const double *num,
                   const double *zq, const double *den, double *p, cudaStream_t st) {
  DirPtrs dp{};
  for (int j = 0; j < m && j < MAX_KEPT; ++j) dp.p[j] = pj[j], dp.slot[j] = slot[j];
  launch_dependent(fcg_direction_kernel, std::min<int64_t>((n + FCG_THREADS - 1) / FCG_THREADS, FCG_CTAS),
                   FCG_THREADS, st, n, m, z, dp, num, zq, den, p);
}

void fcg_product(int64_t n, const int64_t *ptr, const int32_t *idx, const double *val, const double *p,
                 const double *r, double *q, double *sums, cudaStream_t st) {
  launch_dependent(fcg_product_kernel, product_ctas(n), FCG_THREADS, st, n, ptr, idx, val, p, r, q, sums);
}

void fcg_norms(int64_t n, int count, const double *rr, double *out, cudaStream_t st) {
  fcg_norms_kernel<<<1, FCG_THREADS, 0, st>>>(count, step_ctas(n), rr, out);
}

void input_scales(int64_t n, int pairs, int per, const double *nrm2, double kref, double *s, cudaStream_t st) {
  input_scales_kernel<<<1, pairs, 0, st>>>(n, nrm2, kref, per, s);
}

}  // namespace unet
}  // namespace fc
