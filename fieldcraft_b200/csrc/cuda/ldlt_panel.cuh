// The pivoted panel of the symmetric indefinite LDL^T (crates/solver/src/ldlt.rs:250-335) on one
// front, written once for a thread block: the device kernel runs panel_own with CUDA threads; the tests
// run the same source with host threads and a barrier, against the oracle, bit for bit. What follows a
// panel (the rows below, W, W21, the rows' order) the device has in forms of its own (ldlt.cu);
// panel_below, panel, panel_w, front_w21 and permute_rows_below here are the plain statement of it, which
// the tests complete a front with. split_d, unit_lower_inverse and D^-1 are shared again.
//
// The front holds a supernode's own columns: m rows x w columns, column-major with leading
// dimension m, entries (r, c) with r >= c meaningful. Columns before the panel are final (L below
// the pivots, D on them); the panel's and later columns hold the front after the earlier panels'
// updates. The panel chooses its pivots among all of the supernode's remaining own columns by
// the bounded Bunch-Kaufman (rook) search, interchanging the front's own rows and columns
// symmetrically, and stores 1 x 1 and 2 x 2 pivots; a 2 x 2 pivot may end it one column late.
// Every product and sum is rounded on its own (no fused multiply-add), in the reference's order,
// so a front's pivots and values are the reference's exactly.
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define FC_LDLT_FN __device__ __forceinline__
#define FC_LDLT_HD __host__ __device__ __forceinline__  // arithmetic the host plan shares
#define FC_LDLT_ONCE __device__ __forceinline__
#define FC_LDLT_UNROLL _Pragma("unroll")
#else
#include <cmath>
#include <cstring>
#define FC_LDLT_FN inline
#define FC_LDLT_HD inline
#define FC_LDLT_ONCE __attribute__((noinline, noclone))  // its barrier stays one call site
#define FC_LDLT_UNROLL
#endif
#ifndef FC_LDLT_HELD_ROWS
#define FC_LDLT_HELD_ROWS 1024
#endif

namespace fc {
namespace ldlt {

constexpr double ALPHA = 0.6403882032022076;  // (1 + sqrt 17) / 8, ldlt.rs:77
constexpr int ROOK_STEPS = 64;                // ldlt.rs:81
constexpr int PANEL = 64;                     // cholesky.rs:54
constexpr double PIVOT_TOLERANCE = 1e-10;     // cholesky.rs:48
constexpr int MAX_THREADS = 1024;
// Columns held up to date ahead of the search, and the own rows there is room for (see panel_own).
constexpr int HELD = 8, HELD_ROWS = FC_LDLT_HELD_ROWS;
constexpr int8_t PIVOT_ONE = 0, PIVOT_FIRST = 1, PIVOT_SECOND = 2;

#if defined(__CUDACC__)
FC_LDLT_FN double mul(double a, double b) { return __dmul_rn(a, b); }
FC_LDLT_FN double add(double a, double b) { return __dadd_rn(a, b); }
FC_LDLT_FN double sub(double a, double b) { return __dsub_rn(a, b); }
FC_LDLT_FN double fused(double a, double b, double c) { return __fma_rn(a, b, c); }
FC_LDLT_FN double magnitude(double x) { return fabs(x); }
FC_LDLT_FN bool finite(double x) { return isfinite(x); }
FC_LDLT_FN bool not_a_number(double x) { return isnan(x); }
#else
FC_LDLT_FN double mul(double a, double b) { return a * b; }
FC_LDLT_FN double add(double a, double b) { return a + b; }
FC_LDLT_FN double sub(double a, double b) { return a - b; }
FC_LDLT_FN double fused(double a, double b, double c) { return std::fma(a, b, c); }
FC_LDLT_FN double magnitude(double x) { return std::fabs(x); }
FC_LDLT_FN bool finite(double x) { return std::isfinite(x); }
FC_LDLT_FN bool not_a_number(double x) { return std::isnan(x); }
#endif

// x / d, correctly rounded, for many x and one d, from y = reciprocal(d) (Markstein, IBM J. Res. Dev. 34,
// 1990: with y the correctly rounded 1 / d and q within a unit of x / d in the last place, q plus the
// exact remainder x - q d times y rounds to x / d; one such step brings x y that close, the second ends
// it). Five dependent operations in place of a division's. Not for a significand of all ones (the
// theorem's exception) nor where a step could leave the normal range: there the division itself.
FC_LDLT_FN double reciprocal(double d) {
  const double size = magnitude(d), most = 2.037035976334486e90;  // 2^300
  if (!(size < most && size > 1.0 / most)) return 0.0;
#if defined(__CUDACC__)
  const unsigned long long bits = (unsigned long long)__double_as_longlong(d);
#else
  unsigned long long bits;
  std::memcpy(&bits, &d, sizeof(bits));
#endif
  return (bits << 12) == 0xfffffffffffff000ull ? 0.0 : 1.0 / d;
}
FC_LDLT_FN double quotient(double x, double d, double y) {
  const double size = magnitude(x), most = 4.149515568880993e180;  // 2^600
  if (!(y != 0.0 && size < most && (size > 1.0 / most || size == 0.0))) return x / d;
  const double first = mul(x, y);
  double q = fused(fused(-first, d, x), y, first);
  q = fused(fused(-q, d, x), y, q);
  return size == 0.0 ? first : q;  // (the zero's sign)
}

// x / d for a finite d other than zero: a zero's quotient apart, which the division takes its slow way
// for (a front has many, and one lane's is its warp's).
FC_LDLT_FN double divided(double x, double d) { return x == 0.0 ? mul(x, d) : x / d; }

// One front and its per-column state.
struct Front {
  double *F;            // m x w, column-major, leading dimension m
  int64_t m;
  int w;
  const double *scale;  // [w] the largest |A| of each own column (in the structure's order)
  int32_t *order;       // [w] order[c]: the own column (structure's order) at pivot position c
  int8_t *pivots;       // [w] PIVOT_ONE / PIVOT_FIRST / PIVOT_SECOND
  double *a, *b;        // [m] each: the searched column and a candidate (scratch)
  double *W;            // rows [c1, w) of L D over the panel's columns, ld_w x (c1 - c0)
  int64_t ld_w;         // >= w - c0 - PANEL
};

// Block-shared scratch. The panel's own D is kept here too: a column's update reads all of it, and
// one by one from the front every element was a load of its own.
struct Shared {
  double row[PANEL + 1];   // a row of L D over the panel's factored columns
  double d[PANEL + 1];     // D's diagonal at the panel's factored columns
  double e[PANEL + 1];     // its subdiagonal at the first column of a 2 x 2 pivot
  int8_t kind[PANEL + 1];  // PIVOT_ONE / PIVOT_FIRST / PIVOT_SECOND
  alignas(16) double rows[PANEL][HELD];  // rows of L D for the columns to hold: [column of L][row]
  double next[HELD];              // L D of the newest column at the held columns' rows
  double held[HELD][HELD_ROWS];   // the held columns, own rows from the panel's start
  double ab[2][HELD_ROWS];        // Front's a and b, own rows from the panel's start
#if defined(__CUDACC__)
  double best_v[32];  // a warp each
  int best_i[32];
  int nan[32];
#else
  double best_v[MAX_THREADS];
  int best_i[MAX_THREADS];
  int nan[MAX_THREADS];
#endif
};

FC_LDLT_FN double &at(const Front &f, int64_t r, int64_t c) { return f.F[r + c * f.m]; }

template <class T>
FC_LDLT_FN void exchange(T &x, T &y) {
  const T t = x;
  x = y;
  y = t;
}

// Element q of row c of L D over the panel's factored columns (times_d, cholesky.rs:458-481).
FC_LDLT_FN double times_d(const Shared &sh, const Front &f, int c0, int c, int q) {
  const double x = at(f, c, c0 + q);
  if (sh.kind[q] == PIVOT_FIRST) return add(mul(x, sh.d[q]), mul(at(f, c, c0 + q + 1), sh.e[q]));
  if (sh.kind[q] == PIVOT_SECOND) return add(mul(at(f, c, c0 + q - 1), sh.e[q - 1]), mul(x, sh.d[q]));
  return mul(x, sh.d[q]);
}

// The block's largest value bv and its lowest index bi (lo when every value is zero), from each
// thread's; false when any thread met a NaN. Every thread gets the same answer; a barrier in it
// comes after the threads' writes before the call.
template <class Block>
FC_LDLT_ONCE bool block_best(Block &blk, Shared &sh, double bv, int bi, int bn, int lo, int none, int &index,
                             double &value) {
#if defined(__CUDACC__)
  const int lane = blk.tid() & 31, warps = (blk.size() + 31) >> 5;
  // Magnitudes order as their bits do: the warp's largest in three integer reductions (the two
  // halves' largest, then the lowest index that has both) instead of five rounds of FP64 comparisons.
  auto warp_best = [&]() {
    const unsigned long long bits = (unsigned long long)__double_as_longlong(bv);
    const unsigned high = (unsigned)(bits >> 32), top = __reduce_max_sync(0xffffffffu, high);
    const unsigned low = high == top ? (unsigned)bits : 0u, below = __reduce_max_sync(0xffffffffu, low);
    bi = __reduce_min_sync(0xffffffffu, high == top && low == below ? bi : 0x7fffffff);
    bv = __longlong_as_double((long long)((unsigned long long)top << 32 | below));
    bn = __any_sync(0xffffffffu, bn);
  };
  warp_best();
  if (lane == 0) {
    sh.best_v[blk.tid() >> 5] = bv;
    sh.best_i[blk.tid() >> 5] = bi;
    sh.nan[blk.tid() >> 5] = bn;
  }
  blk.sync();
  bv = lane < warps ? sh.best_v[lane] : 0.0;
  bi = lane < warps ? sh.best_i[lane] : none;
  bn = lane < warps ? sh.nan[lane] : 0;
  warp_best();
#else
  auto better = [](double x, int i, double y, int j) { return x > y || (x == y && i < j); };
  sh.best_v[blk.tid()] = bv;
  sh.best_i[blk.tid()] = bi;
  sh.nan[blk.tid()] = bn;
  blk.sync();
  for (int t = 0; t < blk.size(); ++t) {
    bn |= sh.nan[t];
    if (better(sh.best_v[t], sh.best_i[t], bv, bi)) bv = sh.best_v[t], bi = sh.best_i[t];
  }
#endif
  index = bv > 0.0 ? bi : lo;
  value = bv;
  return bn == 0;
}

// Column c (local, >= k) of the part still to factor, own rows [k, w), into out: the front's entries
// less the products with the panel's factored columns [c0, k) (Block::current, ldlt.rs:173-192),
// a row a thread, 16 columns' loads in flight; and the largest magnitude of it over [lo, w) except
// row `skip`, with the lowest such index (largest, ldlt.rs:145-163; lo when all are zero). Returns
// false when one of those entries is not a number (the reference's NaN, which its callers treat
// as a singular column). Every thread gets the same answer.
template <class Block>
FC_LDLT_FN bool current(Block &blk, Shared &sh, const Front &f, int c0, int k, int c, double *out, int lo, int skip,
                        int &index, double &value) {
  const int len = k - c0;
  for (int q = blk.tid(); q < len; q += blk.size()) sh.row[q] = times_d(sh, f, c0, c, q);
  blk.sync();
  double bv = 0.0;
  int bi = lo, bn = 0;
  for (int r = k + blk.tid(); r < f.w; r += blk.size()) {
    double v = r >= c ? at(f, r, c) : at(f, c, r);
    const double *L = &at(f, r, c0);
    int q = 0;
    for (; q + 16 <= len; q += 16) {
      double l[16];
#if defined(__CUDACC__)
#pragma unroll
#endif
      for (int t = 0; t < 16; ++t) l[t] = L[(q + t) * f.m];
#if defined(__CUDACC__)
#pragma unroll
#endif
      for (int t = 0; t < 16; ++t) v = sub(v, mul(l[t], sh.row[q + t]));
    }
#if defined(__CUDACC__)
#pragma unroll 4
#endif
    for (; q < len; ++q) v = sub(v, mul(L[q * f.m], sh.row[q]));
    out[r] = v;
    if (r >= lo && r != skip) {
      const double x = magnitude(v);
      if (not_a_number(x)) {
        bn = 1;
      } else if (x > bv) {
        bv = x;
        bi = r;
      }
    }
  }
  return block_best(blk, sh, bv, bi, bn, lo, f.w, index, value);
}

// The columns [k, k + count), count <= COUNT, into sh.held: their own rows less the products with the
// panel's factored columns [c0, k), each entry's in order, the columns side by side (one column's
// subtractions are a chain, 64 at most). Row r is always held by the same thread.
template <int COUNT, class Block>
FC_LDLT_FN void hold(Block &blk, Shared &sh, const Front &f, int c0, int k, int count) {
  const int len = k - c0;
  for (int e = blk.tid(); e < COUNT * PANEL; e += blk.size()) {
    const int j = e % COUNT, q = e / COUNT;
    if (q < len) sh.rows[q][j] = j < count ? times_d(sh, f, c0, k + j, q) : 0.0;
  }
  blk.sync();
  for (int r = c0 + blk.tid(); r < f.w; r += blk.size()) {
    if (r < k) continue;
    double v[COUNT];
    FC_LDLT_UNROLL
    for (int j = 0; j < COUNT; ++j) v[j] = j < count && r >= k + j ? at(f, r, k + j) : 0.0;
    const double *L = &at(f, r, c0);
    int q = 0;
    for (; q + 16 <= len; q += 16) {
      double l[16];
      FC_LDLT_UNROLL
      for (int t = 0; t < 16; ++t) l[t] = L[(q + t) * f.m];
      FC_LDLT_UNROLL
      for (int t = 0; t < 16; ++t)
        FC_LDLT_UNROLL
        for (int j = 0; j < COUNT; ++j) v[j] = sub(v[j], mul(l[t], sh.rows[q + t][j]));
    }
#if defined(__CUDACC__)
#pragma unroll 4
#endif
    for (; q < len; ++q) {
      const double l = L[q * f.m];
      FC_LDLT_UNROLL
      for (int j = 0; j < COUNT; ++j) v[j] = sub(v[j], mul(l, sh.rows[q][j]));
    }
    FC_LDLT_UNROLL
    for (int j = 0; j < COUNT; ++j)
      if (j < count) sh.held[j][r - c0] = v[j];
  }
}

// current() for the held column k = base + j: into out, and the largest below the diagonal.
template <class Block>
FC_LDLT_FN bool held_column(Block &blk, Shared &sh, const Front &f, int c0, int k, int base, double *out, int &index,
                            double &value) {
  double bv = 0.0;
  int bi = k + 1, bn = 0;
  for (int r = c0 + blk.tid(); r < f.w; r += blk.size()) {
    if (r < k) continue;
    const double v = sh.held[k - base][r - c0];
    out[r] = v;
    const double x = magnitude(v);
    if (r == k) continue;
    if (not_a_number(x)) {
      bn = 1;
    } else if (x > bv) {
      bv = x;
      bi = r;
    }
  }
  return block_best(blk, sh, bv, bi, bn, k + 1, f.w, index, value);
}

// Symmetric interchange of local columns p and q (both at pivot positions >= k) in the front,
// the order and the scratch columns (interchange and Block::swap, ldlt.rs:128-143, 194-204).
// Every thread has read what the pivot decision needs (the scratch columns' entries) before
// any thread moves them: the first barrier.
template <class Block>
FC_LDLT_FN void interchange(Block &blk, const Front &f, int p, int q, double *a, double *b) {
  if (p == q) return;
  if (p > q) exchange(p, q);
  blk.sync();
  const int t = blk.tid(), T = blk.size();
  for (int c = t; c < p; c += T) exchange(at(f, p, c), at(f, q, c));
  for (int c = p + 1 + t; c < q; c += T) exchange(at(f, c, p), at(f, q, c));
  for (int64_t r = q + 1 + t; r < f.m; r += T) exchange(at(f, r, p), at(f, r, q));
  if (t == 0) {
    exchange(at(f, p, p), at(f, q, q));
    exchange(f.order[p], f.order[q]);
    exchange(a[p], a[q]);
    exchange(b[p], b[q]);
  }
  blk.sync();
}

// A 1 x 1 pivot at k from the current column (Block::one, ldlt.rs:206-221).
template <class Block>
FC_LDLT_FN void one(Block &blk, Shared &sh, const Front &f, int c0, int k, const double *col) {
  const double d = col[k];
  for (int r = k + 1 + blk.tid(); r < f.w; r += blk.size()) at(f, r, k) = divided(col[r], d);
  if (blk.tid() == 0) {
    at(f, k, k) = d;
    f.pivots[k] = PIVOT_ONE;
    sh.d[k - c0] = d;
    sh.kind[k - c0] = PIVOT_ONE;
  }
  blk.sync();
}

// The same for the held column k, which stayed in its place: the held columns after it, [k + 1, stop),
// take its product.
template <class Block>
FC_LDLT_FN void one_held(Block &blk, Shared &sh, const Front &f, int c0, int k, int base, int stop, double *col) {
  const double d = col[k];
  for (int r = c0 + blk.tid(); r < f.w; r += blk.size()) {
    if (r <= k) continue;
    const double l = divided(col[r], d);
    at(f, r, k) = l;
    col[r] = l;
    if (r < stop) sh.next[r - base] = mul(l, d);
  }
  if (blk.tid() == 0) {
    at(f, k, k) = d;
    f.pivots[k] = PIVOT_ONE;
    sh.d[k - c0] = d;
    sh.kind[k - c0] = PIVOT_ONE;
  }
  blk.sync();
  for (int r = c0 + blk.tid(); r < f.w; r += blk.size()) {
    if (r <= k) continue;
    const double l = col[r];
    double v[HELD], y[HELD];  // every load before the stores: one after the other they are a chain
    FC_LDLT_UNROLL
    for (int j = 0; j < HELD; ++j) v[j] = sh.held[j][r - c0], y[j] = sh.next[j];
    FC_LDLT_UNROLL
    for (int j = 0; j < HELD; ++j)
      if (j > k - base && j < stop - base) sh.held[j][r - c0] = sub(v[j], mul(l, y[j]));
  }
}

// A 2 x 2 pivot at k, k + 1 from the current columns a (k) and b (k + 1) (Block::two,
// ldlt.rs:223-248).
template <class Block>
FC_LDLT_FN void two(Block &blk, Shared &sh, const Front &f, int c0, int k, const double *a, const double *b) {
  const double d11 = a[k], d21 = a[k + 1], d22 = b[k + 1];
  const double det = sub(mul(d11, d22), mul(d21, d21));
  for (int r = k + 2 + blk.tid(); r < f.w; r += blk.size()) {
    const double x = a[r], y = b[r];
    at(f, r, k) = sub(mul(x, d22), mul(y, d21)) / det;
    at(f, r, k + 1) = sub(mul(y, d11), mul(x, d21)) / det;
  }
  if (blk.tid() == 0) {
    at(f, k, k) = d11;
    at(f, k + 1, k) = d21;
    at(f, k + 1, k + 1) = d22;
    f.pivots[k] = PIVOT_FIRST;
    f.pivots[k + 1] = PIVOT_SECOND;
    sh.d[k - c0] = d11;
    sh.e[k - c0] = d21;
    sh.d[k - c0 + 1] = d22;
    sh.kind[k - c0] = PIVOT_FIRST;
    sh.kind[k - c0 + 1] = PIVOT_SECOND;
  }
  blk.sync();
}

// The panel from column c0 on the own rows (Block::panel, ldlt.rs:250-335): its pivots, L of the rows
// [c0, w), and the interchanges of all rows. Returns -1, or the own column (the structure's order) found
// singular; *end receives where the panel ended and *twos the 2 x 2 pivots it made. Every thread returns
// the same.
//
// The next HELD columns are kept up to date in `held`, so that a column which is a pivot where it stands
// (the usual one) is there when its turn comes: formed when it is looked at, its chain of up to 64
// subtractions and the loads for it were most of a column's time. An interchange may move any of them:
// the columns after it are formed anew, first two of them, then four, then HELD.
template <class Block>
FC_LDLT_FN int panel_own(Block &blk, Shared &sh, const Front &f, int c0, int *end_out, int *twos) {
  const int w = f.w;
  const int end = c0 + PANEL < w ? c0 + PANEL : w;
  const bool holds = w - c0 <= HELD_ROWS;
  double *a = holds ? sh.ab[0] - c0 : f.a, *b = holds ? sh.ab[1] - c0 : f.b;
  int k = c0, base = c0, stop = c0, ahead = HELD;
  *twos = 0;
  while (k < end) {
    int r0;
    double omega_k;
    bool numbers;
    const double limit = PIVOT_TOLERANCE * f.scale[f.order[k]];  // column k's, read while it is looked at
    if (holds) {
      if (k >= stop) {
        const int count = end - k < ahead ? end - k : ahead;
        if (count > 4)
          hold<8>(blk, sh, f, c0, k, count);
        else if (count > 2)
          hold<4>(blk, sh, f, c0, k, count);
        else
          hold<2>(blk, sh, f, c0, k, count);
        base = k, stop = k + count, ahead = HELD < 2 * ahead ? HELD : 2 * ahead;
      }
      numbers = held_column(blk, sh, f, c0, k, base, a, r0, omega_k);
    } else {
      numbers = current(blk, sh, f, c0, k, k, a, k + 1, -1, r0, omega_k);
    }
    const double akk = magnitude(a[k]);
    if (!finite(akk) || !numbers || !finite(omega_k)) return f.order[k];
    bool pair = false;
    int p = k, pi = k, pr = k;
    if (!(akk >= ALPHA * omega_k)) {
      // the rook search: `a` holds column i, `b` the candidate r
      int i = k, r = r0, step = 0;
      double omega_i = omega_k;
      for (;;) {
        int s;
        double omega_r;
        const bool fine = current(blk, sh, f, c0, k, r, b, k, r, s, omega_r);
        const double arr = magnitude(b[r]);
        if (!finite(arr) || !fine || !finite(omega_r)) return f.order[k];
        step += 1;
        if (arr >= ALPHA * omega_r) {
          exchange(a, b);
          p = r;
          break;
        }
        if (omega_r <= omega_i || step >= ROOK_STEPS) {
          pair = true;
          pi = i;
          pr = r;
          break;
        }
        exchange(a, b);
        i = r;
        omega_i = omega_r;
        r = s;
      }
    }
    if (!pair) {
      interchange(blk, f, k, p, a, b);
      if (!(magnitude(a[k]) > (p == k ? limit : PIVOT_TOLERANCE * f.scale[f.order[k]]))) return f.order[k];
      if (holds && p == k) {
        one_held(blk, sh, f, c0, k, base, stop, a);
      } else {
        one(blk, sh, f, c0, k, a);
        stop = k, ahead = 2;
      }
      k += 1;
    } else {
      // i to k, then r to k + 1 (r was at k if i took its place)
      interchange(blk, f, k, pi, a, b);
      interchange(blk, f, k + 1, pr == k ? pi : pr, a, b);
      const double offdiagonal = magnitude(a[k + 1]);
      const double s0 = f.scale[f.order[k]], s1 = f.scale[f.order[k + 1]];
      const double size = s0 < s1 ? s1 : s0;
      if (!(offdiagonal > PIVOT_TOLERANCE * size)) return f.order[k];
      two(blk, sh, f, c0, k, a, b);
      *twos += 1;
      stop = k, ahead = 2;
      k += 2;
    }
  }
  *end_out = k;
  return -1;
}

// L of the rows [max(r0, w), r1) over the panel's columns [c0, c1), from panel_own's pivots (sh.d, e and
// kind): each row's entries by themselves, with the operations and the order of one(), two() and
// current(). (The device's kernel, which keeps a row in registers, is in ldlt.cu.)
template <class Block>
FC_LDLT_FN void panel_below(Block &blk, const Shared &sh, const Front &f, int c0, int c1, int64_t r0, int64_t r1) {
  for (int64_t r = (r0 > f.w ? r0 : f.w) + blk.tid(); r < r1; r += blk.size()) {
    auto value = [&](int k, int len) {
      double v = at(f, r, c0 + k);
      for (int q = 0; q < len; ++q) v = sub(v, mul(at(f, r, c0 + q), times_d(sh, f, c0, c0 + k, q)));
      return v;
    };
    for (int k = 0; k < c1 - c0; ++k) {
      const double x = value(k, k);
      if (sh.kind[k] == PIVOT_FIRST) {
        const double y = value(k + 1, k), d11 = sh.d[k], d21 = sh.e[k], d22 = sh.d[k + 1];
        const double det = sub(mul(d11, d22), mul(d21, d21)), inv = reciprocal(det);
        at(f, r, c0 + k) = quotient(sub(mul(x, d22), mul(y, d21)), det, inv);
        at(f, r, c0 + k + 1) = quotient(sub(mul(y, d11), mul(x, d21)), det, inv);
        ++k;
      } else {
        at(f, r, c0 + k) = quotient(x, sh.d[k], reciprocal(sh.d[k]));
      }
    }
  }
  blk.sync();
}

// Both: the whole panel on one block.
template <class Block>
FC_LDLT_FN int panel(Block &blk, Shared &sh, const Front &f, int c0, int *end_out, int *twos) {
  const int singular = panel_own(blk, sh, f, c0, end_out, twos);
  if (singular < 0) panel_below(blk, sh, f, c0, *end_out, f.w, f.m);
  return singular;
}

// W = L D for the rows [c1, w) over the panel's columns [c0, c1): the coefficients of the update
// of the later own columns by the panel (products' Y, cholesky.rs:531-548).
template <class Block>
FC_LDLT_FN void panel_w(Block &blk, const Front &f, int c0, int c1) {
  const int kw = c1 - c0;
  for (int64_t r = c1 + blk.tid(); r < f.w; r += blk.size()) {
    double *wr = f.W + (r - c1);
    int k = 0;
    while (k < kw) {
      const int c = c0 + k;
      if (f.pivots[c] == PIVOT_FIRST) {
        const double x = at(f, r, c), y = at(f, r, c + 1);
        const double d11 = at(f, c, c), d21 = at(f, c + 1, c), d22 = at(f, c + 1, c + 1);
        wr[k * f.ld_w] = add(mul(x, d11), mul(y, d21));
        wr[(k + 1) * f.ld_w] = add(mul(x, d21), mul(y, d22));
        k += 2;
      } else {
        wr[k * f.ld_w] = mul(at(f, r, c), at(f, c, c));
        k += 1;
      }
    }
  }
  blk.sync();
}

// W21 = L21 D: the rows [r0, r1) of the front, of those past its columns, times its block diagonal,
// row r at out[r - w], leading dimension ld_out, for the update
// matrix U = -L21 W21^T the parent assembles (products' Y for a descendant, cholesky.rs:531-548,
// with times_d's operations).
template <class Block>
FC_LDLT_FN void front_w21(Block &blk, const Front &f, double *out, int64_t ld_out, int64_t r0, int64_t r1) {
  for (int64_t r = r0 + blk.tid(); r < r1; r += blk.size()) {
    double *o = out + (r - f.w);
    int k = 0;
    while (k < f.w) {
      if (f.pivots[k] == PIVOT_FIRST) {
        const double x = at(f, r, k), y = at(f, r, k + 1);
        const double d11 = at(f, k, k), d21 = at(f, k + 1, k), d22 = at(f, k + 1, k + 1);
        o[k * ld_out] = add(mul(x, d11), mul(y, d21));
        o[(k + 1) * ld_out] = add(mul(x, d21), mul(y, d22));
        k += 2;
      } else {
        o[k * ld_out] = mul(at(f, r, k), at(f, k, k));
        k += 1;
      }
    }
  }
  blk.sync();
}

// All of W21.
template <class Block>
FC_LDLT_FN void front_w21(Block &blk, const Front &f, double *out, int64_t ld_out) {
  front_w21(blk, f, out, ld_out, f.w, f.m);
}

// D out of a factored front's columns [c0, c1): d[c] receives D's diagonal and e[c] its
// subdiagonal (the 2 x 2 pivots' d21 at their first column, else 0); the front's own block becomes
// unit lower (ones on the diagonal, zeros where a 2 x 2 pivot's d21 was), the form the triangular
// solve reads.
template <class Block>
FC_LDLT_FN void split_d(Block &blk, const Front &f, double *d, double *e, int c0, int c1) {
  for (int c = c0 + blk.tid(); c < c1; c += blk.size()) {
    d[c] = at(f, c, c);
    e[c] = 0.0;
    at(f, c, c) = 1.0;
    if (f.pivots[c] == PIVOT_FIRST) {
      e[c] = at(f, c + 1, c);
      at(f, c + 1, c) = 0.0;
    }
  }
  blk.sync();
}
template <class Block>
FC_LDLT_FN void split_d(Block &blk, const Front &f, double *d, double *e) {
  split_d(blk, f, d, e, 0, f.w);
}

// y <- D^-1 y for the unknowns [0, n) of R right-hand sides (row-major, y[i * R + j]), D given by
// its diagonal d, subdiagonal e and the pivot kinds (the solve's block step, cholesky.rs:946-974).
// One thread per pivot group: a 1 x 1 pivot or the first column of a 2 x 2 one.
FC_LDLT_FN void apply_d_inverse(int64_t i, int R, const double *d, const double *e, const int8_t *pivots, double *y) {
  if (pivots[i] == PIVOT_SECOND) return;
  if (pivots[i] == PIVOT_FIRST) {
    const double d11 = d[i], d21 = e[i], d22 = d[i + 1];
    const double det = sub(mul(d11, d22), mul(d21, d21));
    for (int j = 0; j < R; ++j) {
      const double p = y[i * R + j], q = y[(i + 1) * R + j];
      y[i * R + j] = sub(mul(d22, p), mul(d21, q)) / det;
      y[(i + 1) * R + j] = sub(mul(d11, q), mul(d21, p)) / det;
    }
  } else {
    for (int j = 0; j < R; ++j) y[i * R + j] = y[i * R + j] / d[i];
  }
}

// X = L^-1 for an nb x nb unit lower block of a front (nb <= 64; L's diagonal is not read),
// column-major with leading dimension ldx: column j by forward substitution, x_i = -sum over
// k in [j, i) of L(i, k) x_k, summed in k order from zero. Step k adds its term to every sum
// still open (rows past k, columns up to k), so a step is parallel over up to 1024 entries and
// each entry's terms still come in k order; until the end X holds the sums themselves. The
// strictly upper part of X is left as it is (zero in the solve's inverse arena).
template <class Block>
FC_LDLT_FN void unit_lower_inverse(Block &blk, const double *Lb, int64_t ldl, int nb, double *X, int64_t ldx) {
  for (int e = blk.tid(); e < nb * nb; e += blk.size())
    if (e % nb > e / nb) X[e % nb + (int64_t)(e / nb) * ldx] = 0.0;
  blk.sync();
  for (int k = 0; k < nb; ++k) {
    const int rows = nb - 1 - k;
    for (int e = blk.tid(); e < rows * (k + 1); e += blk.size()) {
      const int i = k + 1 + e % rows, j = e / rows;
      const double x = j == k ? 1.0 : -X[k + (int64_t)j * ldx];
      X[i + (int64_t)j * ldx] = add(X[i + (int64_t)j * ldx], mul(Lb[i + (int64_t)k * ldl], x));
    }
    blk.sync();
  }
  for (int e = blk.tid(); e < nb * nb; e += blk.size()) {
    const int i = e % nb, j = e / nb;
    if (i == j) X[i + (int64_t)j * ldx] = 1.0;
    if (i > j) X[i + (int64_t)j * ldx] = -X[i + (int64_t)j * ldx];
  }
  blk.sync();
}

// Rows [w, m) of every own column of a front put in a new order: row w + i takes the old row
// w + from[i] (from: a permutation of [0, m - w)). One column at a time through `tmp` (m - w
// entries), threads over its rows.
template <class Block>
FC_LDLT_FN void permute_rows_below(Block &blk, const Front &f, const int32_t *from, double *tmp) {
  const int64_t u = f.m - f.w;
  for (int c = 0; c < f.w; ++c) {
    double *col = f.F + f.w + (int64_t)c * f.m;
    for (int64_t i = blk.tid(); i < u; i += blk.size()) tmp[i] = col[from[i]];
    blk.sync();
    for (int64_t i = blk.tid(); i < u; i += blk.size()) col[i] = tmp[i];
    blk.sync();
  }
}

// The update of the later own columns by a panel that ended at c1, as tiles of at most 64 x 64:
// the front's rows [c1, m) of its columns [c1, w), lower part only; column blocks of 64 from c1,
// in each the row blocks from the diagonal down. Tile `slot` of that list, or false past its end.
struct Tile {
  int64_t i0;   // first row
  int j0;       // first column
  int M, N;     // rows, columns
  bool lower;   // a diagonal tile: only rows >= columns
};
constexpr int TILE_ROWS = 64;

FC_LDLT_HD bool update_tile(int64_t m, int w, int c1, int64_t slot, Tile &t) {
  for (int j0 = c1; j0 < w; j0 += TILE_ROWS) {
    const int64_t rows = (m - j0 + TILE_ROWS - 1) / TILE_ROWS;
    if (slot < rows) {
      t.i0 = j0 + slot * TILE_ROWS;
      t.j0 = j0;
      t.M = (int)(m - t.i0 < TILE_ROWS ? m - t.i0 : TILE_ROWS);
      t.N = w - j0 < TILE_ROWS ? w - j0 : TILE_ROWS;
      t.lower = slot == 0;
      return true;
    }
    slot -= rows;
  }
  return false;
}

// The tiles of that update: at most this many for a panel that ends at c1 or later (the count
// falls as c1 grows), so a plan sized for the earliest end holds every case.
FC_LDLT_HD int64_t update_tiles(int64_t m, int w, int c1) {
  int64_t count = 0;
  for (int j0 = c1; j0 < w; j0 += TILE_ROWS) count += (m - j0 + TILE_ROWS - 1) / TILE_ROWS;
  return count;
}

}  // namespace ldlt
}  // namespace fc
