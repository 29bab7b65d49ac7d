// Space transforms of windows of any shape (the reference's per-window FFT
// along the space axes, src/fk.c:307-373 forward, src/fk.c:375-443 adjoint):
// surveys whose sizes their windows do not divide (18 x 35 for a nominal
// 16 x 32, padded 23 x 44), prime padded lengths (23, 43, 83, 127) and
// windows without a shape-specialised kernel.
//
// A DFT of length P over many lines is a product with a small real cosine /
// sine table.  Inputs j and P - j and outputs k and P - k share their terms:
//
//   s_j = x_j + x_{P-j},  d_j = x_j - x_{P-j},  j = 1 .. H = (P - 1) / 2
//   A_k = x_0 + (-1)^k x_{P/2} [P even] + sum_j s_j cos(2 pi j k / P)
//   B_k = sum_j d_j sin(2 pi j k / P),          k = 0 .. P / 2
//   forward (inverse DFT, first L outputs kept):  y_k = A_k + i B_k
//   adjoint (L inputs, zero-padded, all outputs): y_k = A_k - i B_k
//   y_{P-k}: the other sign
//
// which is P^2 real multiply-adds per line in both directions, for any P.
// It is bound by the FP32 pipe and the issue slots around it (37 x 101
// traces of 873 samples, planes of 23 x 44: 1.1 G multiply-adds, 30 us at
// 36.7 T/s, against 37 us of memory traffic forward and 60 us adjoint;
// measured 152 and 193 us, and 730 and 826 us by the generic block FFTs), so:
//
//  * a thread accumulates 4 lines x 4 output pairs in registers (packed
//    f32x2 multiply-adds on the (re, im) pairs: the same rate as scalar
//    ones at half the issue slots); eight threads share the table values,
//    so the shared memory delivers half of what it could;
//  * one running sum of P / 2 terms loses more than the stages of radix
//    passes do where P is composite (relative L2 error of the operators on
//    80 x 80 planes 1.19 times theirs, on 44 x 44 1.06).  Such axes sum in
//    runs of four or eight terms whose sums are then added up; the totals
//    take the registers of half the tile's lines (2 lines x 4 output pairs).
//    0.98 and 0.97 times the radix passes' error then, at 1.2 times the time
//    of one sum (planes of 60 x 60, 28.9 M values: forward 320 -> 364 us,
//    adjoint 370 -> 433; radix passes 718 and 873);
//  * the raw planes of the next batch are copied (cp.async) into a staging
//    buffer behind the products of this one; a thread forms the pairs s, d
//    as it reads the lines, and the contiguous axis is transformed in place,
//    so that the planes of a batch take 15 KB each (23 x 44): keeping the
//    pairs in shared memory saves a quarter of the adds but leaves room for
//    two planes instead of three, and was slower;
//  * the last two axes of a window are one kernel (plane_dft): the planes
//    go axis by axis through shared memory, and the adjoint applies the
//    ISTA update to the model rows on the way out.  Other axes (the first
//    of a 3-D window; of two axes too long for three planes to fit in an
//    SM's shared memory, the first) are one pass each over memory
//    (axis_dft);
//  * persistent blocks of 128 threads, up to four per SM (registers), so
//    that one block's barriers are covered by the others;
//  * windows with one axis (line_dft): a batch is as many lines as the
//    block's threads have tiles for; long axes run blocks of 256 threads,
//    which share one table (33 KB for P = 88).
#pragma once

#include "fast.cuh"

namespace agd {

constexpr int kDftThreads = 128;
constexpr int kDftMaxP = 128;  // longest axis served

// One axis of a window: table rows j = 1 .. H over outputs k < kpad
// (cosines, then sines), kpad = P / 2 + 1 rounded up to a multiple of the
// output tile.
template <typename R>
struct DftAxis {
  const R *tab;
  int P, H, kpad, n_in, n_out;
  int lines;  // lines of a thread's tile: 4 (one sum), 2 (runs) or 1 (runs of runs)
  int run;    // terms of a run
};

// One window's planes: rows along axis b (contiguous), columns along axis a
// (line_dft: no axis a, a plane is one line).
template <typename R>
struct PlaneDftJob {
  const Cx<R> *src;  // [planes][a.n_in][b.n_in]
  Cx<R> *dst;        // [planes][a.n_out][b.n_out]
  long planes;
  DftAxis<R> a, b;
  int np;   // planes (lines) per batch
  int pid;  // problem of the window
};

// One window's lines along a strided axis: [outer][n_in][inner] ->
// [outer][n_out][inner].
template <typename R>
struct AxisDftJob {
  const Cx<R> *src;
  Cx<R> *dst;
  long outer;
  int inner;
  DftAxis<R> a;
  int nl;  // lines per batch
};

// output pairs per thread: registers for 4 x 4 packed floats, 4 x 2 doubles
template <typename R>
constexpr int kDftTk = sizeof(R) == sizeof(float) ? 4 : 2;

__host__ __device__ inline int dft_round4(int n) { return (n + 3) & ~3; }

// Shared memory of a batch of planes, in reals, in this order: tables of b
// and a, the staged input planes, the rows between the axes and before the
// store (odd stride: columns hit distinct banks).
template <typename R>
__host__ __device__ inline int dft_table_reals(const DftAxis<R> &x) {
  return 2 * x.H * x.kpad;
}
template <typename R>
__host__ __device__ inline int plane_stage_reals(const DftAxis<R> &a, const DftAxis<R> &b,
                                                 int np) {
  return 2 * dft_round4(np * a.n_in * b.n_in);
}
template <typename R>
__host__ __device__ inline int dft_row_stride(const DftAxis<R> &x) {
  return (x.n_in > x.n_out ? x.n_in : x.n_out) | 1;
}
template <typename R>
inline size_t plane_dft_smem(const DftAxis<R> &a, const DftAxis<R> &b, int np) {
  return ((size_t)dft_table_reals(a) + dft_table_reals(b) + plane_stage_reals(a, b, np) +
          2L * np * a.n_out * dft_row_stride(b)) * sizeof(R);
}
// table, the lines
template <typename R>
inline size_t line_dft_smem(const DftAxis<R> &b, int nl) {
  return ((size_t)dft_table_reals(b) + 2L * nl * dft_row_stride(b)) * sizeof(R);
}
// tables, two staged batches of nl lines (nl a multiple of 4)
template <typename R>
inline size_t axis_dft_smem(const DftAxis<R> &a, int nl) {
  return ((size_t)dft_table_reals(a) + 4L * a.n_in * nl) * sizeof(R);
}

// ------------------------------------------------------------ arithmetic

// acc += x * w for a complex x and a real w
__device__ __forceinline__ void fma_real(float2 &acc, float2 x, float w) {
  unsigned long long a, b, c;
  asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "f"(acc.x), "f"(acc.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(b) : "f"(x.x), "f"(x.y));
  asm("mov.b64 %0, {%1, %1};" : "=l"(c) : "f"(w));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(a) : "l"(b), "l"(c));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(acc.x), "=f"(acc.y) : "l"(a));
}
__device__ __forceinline__ void fma_real(double2 &acc, double2 x, double w) {
  acc.x += x.x * w;
  acc.y += x.y * w;
}
// u + v and u - v
__device__ __forceinline__ void sum_diff(float2 u, float2 v, float2 &s, float2 &d) {
  unsigned long long a, b, c;
  asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "f"(u.x), "f"(u.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(b) : "f"(v.x), "f"(v.y));
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(c) : "l"(a), "l"(b));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(s.x), "=f"(s.y) : "l"(c));
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(c) : "l"(a), "l"(b));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(c));
}
__device__ __forceinline__ void sum_diff(double2 u, double2 v, double2 &s, double2 &d) {
  s = cadd(u, v);
  d = csub(u, v);
}

// two consecutive complex values (16-byte aligned for float)
__device__ __forceinline__ void load_pair(const float2 *p, float2 &u, float2 &v) {
  const float4 q = *reinterpret_cast<const float4 *>(p);
  u = make_float2(q.x, q.y);
  v = make_float2(q.z, q.w);
}
__device__ __forceinline__ void load_pair(const double2 *p, double2 &u, double2 &v) {
  u = p[0];
  v = p[1];
}
__device__ __forceinline__ void load_tab(const float *p, float (&v)[4]) {
  const float4 q = *reinterpret_cast<const float4 *>(p);
  v[0] = q.x;
  v[1] = q.y;
  v[2] = q.z;
  v[3] = q.w;
}
__device__ __forceinline__ void load_tab(const double *p, double (&v)[2]) {
  const double2 q = *reinterpret_cast<const double2 *>(p);
  v[0] = q.x;
  v[1] = q.y;
}

// Tables of one axis into shared memory (a multiple of 16 bytes).
template <typename R, int NT = kDftThreads>
__device__ __forceinline__ void dft_load_table(R *to, const DftAxis<R> &x) {
  constexpr int per = 16 / sizeof(R);
  const int n = dft_table_reals(x) / per;
  for (int e = threadIdx.x; e < n; e += NT) cp_async<16>(to + e * per, x.tab + e * per);
}

// Accumulators of a tile of TL lines x TK output pairs; with TL = 2, also the
// totals of the runs before this one; with TL = 1, those of this group of
// kDftGroup runs and of the groups before it.
constexpr int kDftGroup = 4;
template <typename R, int TL>
struct DftTile {
  static constexpr int TK = kDftTk<R>;
  static constexpr bool kRuns = TL < 4, kGroups = TL == 1;
  Cx<R> a[TL][TK], b[TL][TK];
  Cx<R> ta[kRuns ? TL : 1][TK], tb[kRuns ? TL : 1][TK];
  Cx<R> ga[TK], gb[TK];  // groups

  // from x_0 and x_{P/2} (k0 is even: the sign of x_{P/2} follows m)
  __device__ __forceinline__ void start(const Cx<R> (&u)[TL], const Cx<R> (&v)[TL]) {
#pragma unroll
    for (int i = 0; i < TL; ++i)
#pragma unroll
      for (int m = 0; m < TK; ++m) {
        a[i][m] = (m & 1) ? csub(u[i], v[i]) : cadd(u[i], v[i]);
        b[i][m] = cmake<Cx<R>>((R)0, (R)0);
        if constexpr (kRuns) ta[i][m] = tb[i][m] = b[i][m];
        if constexpr (kGroups) ga[m] = gb[m] = b[i][m];
      }
  }
  // one pair (s, d) of each line, with the table values at c, n
  __device__ __forceinline__ void add(const Cx<R> (&s)[TL], const Cx<R> (&d)[TL], const R *c,
                                      const R *n) {
    R cv[TK], nv[TK];
    load_tab(c, cv);
    load_tab(n, nv);
#pragma unroll
    for (int m = 0; m < TK; ++m)
#pragma unroll
      for (int i = 0; i < TL; ++i) {
        fma_real(a[i][m], s[i], cv[m]);
        fma_real(b[i][m], d[i], nv[m]);
      }
  }
  // the same as the first pair of a run: the last run's sums go to the totals
  __device__ __forceinline__ void add_new_run(const Cx<R> (&s)[TL], const Cx<R> (&d)[TL],
                                              const R *c, const R *n) {
    R cv[TK], nv[TK];
    load_tab(c, cv);
    load_tab(n, nv);
#pragma unroll
    for (int m = 0; m < TK; ++m)
#pragma unroll
      for (int i = 0; i < TL; ++i) {
        ta[i][m] = cadd(ta[i][m], a[i][m]);
        tb[i][m] = cadd(tb[i][m], b[i][m]);
        a[i][m] = cscale(s[i], cv[m]);
        b[i][m] = cscale(d[i], nv[m]);
      }
  }
  // the group's sums into the totals; a new group
  __device__ __forceinline__ void end_group() {
#pragma unroll
    for (int m = 0; m < TK; ++m) {
      ga[m] = cadd(ga[m], ta[0][m]);
      gb[m] = cadd(gb[m], tb[0][m]);
      ta[0][m] = tb[0][m] = cmake<Cx<R>>((R)0, (R)0);
    }
  }
  __device__ __forceinline__ void finish() {
#pragma unroll
    for (int i = 0; i < TL; ++i)
#pragma unroll
      for (int m = 0; m < TK; ++m) {
        a[i][m] = cadd(ta[i][m], a[i][m]);
        b[i][m] = cadd(tb[i][m], b[i][m]);
        if constexpr (kGroups) {
          a[i][m] = cadd(ga[m], a[i][m]);
          b[i][m] = cadd(gb[m], b[i][m]);
        }
      }
  }
  // outputs k0 .. of line i at out + k * ks, k < n_out
  template <bool FWD, typename I>
  __device__ __forceinline__ void store(int i, Cx<R> *out, I ks, int k0,
                                        const DftAxis<R> &x) const {
    const int ko = x.P / 2 + 1;
    Cx<R> *lo = out + k0 * ks;
    Cx<R> *hi = out + (x.P - k0) * ks;
#pragma unroll
    for (int m = 0; m < TK; ++m, lo += ks, hi -= ks) {
      const int k = k0 + m;
      const Cx<R> A = a[i][m], B = b[i][m];
      const Cx<R> plus = cmake<Cx<R>>(A.x - B.y, A.y + B.x);   // A + i B
      const Cx<R> minus = cmake<Cx<R>>(A.x + B.y, A.y - B.x);  // A - i B
      if (k < min(ko, x.n_out)) *lo = FWD ? plus : minus;
      if (k > 0 && 2 * k < x.P && x.P - k < x.n_out) *hi = FWD ? minus : plus;
    }
  }
};

// The thread's tile number -> line tile and output tile: blocks of eight
// line tiles of tl lines (fewer in the last), in a block output tile by
// output tile.  Lines of the tile: line0 + at + i * w with w the block's line
// tiles.
struct DftTileAt {
  int line0, w, k;
  __device__ __forceinline__ DftTileAt(int tile, int lt_n, int kt_n, int tl) {
    const int blk = tile / (8 * kt_n);
    const int rem = tile - blk * 8 * kt_n;
    w = min(8, lt_n - 8 * blk);
    k = rem / w;
    line0 = 8 * tl * blk;
    at = rem - k * w;
  }
  int at;
};

// Accumulates a tile from raw lines in shared memory: element e of line i at
// lo[i] + e * es, zero from n_in on.
template <typename R, int TL>
__device__ __forceinline__ void dft_accumulate_raw(DftTile<R, TL> &acc,
                                                   const Cx<R> *const (&lo)[TL], int es,
                                                   const DftAxis<R> &x, const R *tab, int k0) {
  using C = Cx<R>;
  constexpr bool kRuns = TL < 4;
  const int mid = x.P / 2;
  const bool has_mid = x.P % 2 == 0 && mid < x.n_in;
  const int both = min(x.P - x.n_in, x.H);  // pairs 1 .. both have one member
  C u[TL], v[TL];
#pragma unroll
  for (int i = 0; i < TL; ++i) {
    u[i] = lo[i][0];
    v[i] = has_mid ? lo[i][mid * es] : cmake<C>((R)0, (R)0);
  }
  acc.start(u, v);
  const R *cj = tab + k0;
  const R *nj = cj + x.H * x.kpad;
  int j = 1, e = es, f = (x.P - 1) * es;
  // one pair of each line: elements e and, with both members present, f
  auto term = [&](bool both_in, bool new_run) {
#pragma unroll
    for (int i = 0; i < TL; ++i) {
      if (both_in)
        sum_diff(lo[i][e], lo[i][f], u[i], v[i]);
      else
        u[i] = v[i] = lo[i][e];
    }
    if constexpr (kRuns) {
      if (new_run)
        acc.add_new_run(u, v, cj, nj);
      else
        acc.add(u, v, cj, nj);
    } else {
      acc.add(u, v, cj, nj);
    }
    ++j;
    e += es;
    f -= es;
    cj += x.kpad;
    nj += x.kpad;
  };
  if constexpr (kRuns) {
    int end = x.run;  // last pair of the run
    bool fresh = false;
    [[maybe_unused]] int runs = 0;
    // the pairs up to last, in runs
    auto terms = [&](int last, bool both_in) {
      while (j <= last) {
        const int stop = min(last, end);
        if constexpr (TL == 1) {
          if (fresh && runs % kDftGroup == 1 && runs > 1) acc.end_group();
        }
        term(both_in, fresh);
        fresh = false;
#pragma unroll 2
        while (j <= stop) term(both_in, false);
        if (j > end) {
          end += x.run;
          ++runs;
          fresh = true;
        }
      }
    };
    terms(both, false);
    terms(x.H, true);
    acc.finish();
  } else {
#pragma unroll 1
    while (j <= both) term(false, false);
#pragma unroll 1
    while (j <= x.H) term(true, false);
  }
}

// All outputs of n_lines raw lines in shared memory: element e of line q at
// raw + in_at(q) + e * es; outputs to out_at(q) + k * ks.  Lines past n_lines
// take the last line's place and are not stored.
template <typename R, bool FWD, int TL, typename InAt, typename OutAt, typename I>
__device__ __forceinline__ void dft_tiles_from_raw(const Cx<R> *raw, int es, int n_lines,
                                                   const DftAxis<R> &x, const R *tab, InAt in_at,
                                                   OutAt out_at, I ks) {
  const int kt_n = x.kpad / kDftTk<R>;
  const int lt_n = (n_lines + TL - 1) / TL;
  for (int tile = threadIdx.x; tile < lt_n * kt_n; tile += kDftThreads) {
    const DftTileAt t(tile, lt_n, kt_n, TL);
    const int k0 = kDftTk<R> * t.k;
    const Cx<R> *lo[TL];
#pragma unroll
    for (int i = 0; i < TL; ++i)
      lo[i] = raw + in_at(min(t.line0 + t.at + i * t.w, n_lines - 1));
    DftTile<R, TL> acc;
    dft_accumulate_raw<R, TL>(acc, lo, es, x, tab, k0);
#pragma unroll
    for (int i = 0; i < TL; ++i) {
      const int q = t.line0 + t.at + i * t.w;
      if (q < n_lines) acc.template store<FWD>(i, out_at(q), ks, k0, x);
    }
  }
}
template <typename R, bool FWD, typename InAt, typename OutAt, typename I>
__device__ __forceinline__ void dft_from_raw(const Cx<R> *raw, int es, int n_lines,
                                             const DftAxis<R> &x, const R *tab, InAt in_at,
                                             OutAt out_at, I ks) {
  if (x.lines == 4)
    dft_tiles_from_raw<R, FWD, 4>(raw, es, n_lines, x, tab, in_at, out_at, ks);
  else if (x.lines == 2)
    dft_tiles_from_raw<R, FWD, 2>(raw, es, n_lines, x, tab, in_at, out_at, ks);
  else
    dft_tiles_from_raw<R, FWD, 1>(raw, es, n_lines, x, tab, in_at, out_at, ks);
}

// The transforms of n rows of shared memory (elements side by side, rows rs
// apart) in place: as many rows at a time as the block's threads have tiles
// for, all read before any is overwritten.  Every warp meets the block's
// barrier once per step, with tiles or without (the two places are separate
// so that the accumulators need no values in idle warps).
template <typename R, bool FWD, int NT, int TL>
__device__ __forceinline__ void dft_tiles_in_place(Cx<R> *rows, int rs, int n,
                                                   const DftAxis<R> &x, const R *tab) {
  const int kt_n = x.kpad / kDftTk<R>;
  const int per = TL * (NT / kt_n);
  for (int r0 = 0; r0 < n; r0 += per, rows += per * rs) {
    const int m = min(per, n - r0);
    const int lt_n = (m + TL - 1) / TL;
    const int tiles = lt_n * kt_n;
    if ((int)(threadIdx.x & ~31) >= tiles) {  // a warp without tiles
      asm volatile("barrier.sync 0;" ::: "memory");
      continue;
    }
    const DftTileAt t(min((int)threadIdx.x, tiles - 1), lt_n, kt_n, TL);
    const int k0 = kDftTk<R> * t.k;
    DftTile<R, TL> acc;
    const Cx<R> *lo[TL];
#pragma unroll
    for (int i = 0; i < TL; ++i) lo[i] = rows + min(t.line0 + t.at + i * t.w, m - 1) * rs;
    dft_accumulate_raw<R, TL>(acc, lo, 1, x, tab, k0);
    asm volatile("barrier.sync 0;" ::: "memory");
#pragma unroll
    for (int i = 0; i < TL; ++i) {
      const int q = t.line0 + t.at + i * t.w;
      if ((int)threadIdx.x < tiles && q < m) acc.template store<FWD>(i, rows + q * rs, 1, k0, x);
    }
  }
}
template <typename R, bool FWD, int NT>
__device__ __forceinline__ void dft_rows_in_place(Cx<R> *rows, int rs, int n,
                                                  const DftAxis<R> &x, const R *tab) {
  if (x.lines == 4)
    dft_tiles_in_place<R, FWD, NT, 4>(rows, rs, n, x, tab);
  else if (x.lines == 2)
    dft_tiles_in_place<R, FWD, NT, 2>(rows, rs, n, x, tab);
  else
    dft_tiles_in_place<R, FWD, NT, 1>(rows, rs, n, x, tab);
}

// Finished rows of shared memory (stride rs) to n rows of n_out values at
// dst, with the update (epilogues as axis_pass); returns the largest |x|^2
// of kUpdateMax.  A fixed thread -> (row, column) map (no index division),
// four model loads in flight per thread.
template <typename R, int NT>
__device__ __forceinline__ R dft_rows_out(const Cx<R> *rows, int rs, int n, int n_out,
                                          Cx<R> *dst, int epilogue, R step, R lamb) {
  using C = Cx<R>;
  const R lamb_sq = lamb * lamb;
  const int cpr = min(n_out, NT);
  const int tr = NT / cpr;
  const int r0 = threadIdx.x / cpr;
  const int c0 = threadIdx.x - r0 * cpr;
  const bool need_x = epilogue != kStore;
  R most = (R)0;
  for (int c = r0 < tr ? c0 : n_out; c < n_out; c += cpr)
    for (int r = r0; r < n; r += 4 * tr) {
      C x[4];
      if (need_x) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (r + u * tr < n) x[u] = dst[(r + u * tr) * n_out + c];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int ru = r + u * tr;
        if (ru >= n) break;
        const C g = rows[ru * rs + c];
        C xn = g;
        if (need_x) {
          xn = cmake<C>(sub_rn<R>(x[u].x, mul_rn<R>(step, g.x)),
                        sub_rn<R>(x[u].y, mul_rn<R>(step, g.y)));
          if (epilogue == kUpdateThreshold) {
            xn = soft_threshold<R>(xn, lamb, lamb_sq);
          } else {
            const R a2 = abs_sq<R>(xn);
            most = a2 > most ? a2 : most;
          }
        }
        dst[ru * n_out + c] = xn;
      }
    }
  return most;
}

// One atomic maximum per warp (every lane takes part).
template <typename R>
__device__ __forceinline__ void warp_atomic_max(R *out, R v) {
  for (int o = 16; o > 0; o >>= 1) {
    const R w = __shfl_xor_sync(0xffffffffu, v, o);
    v = w > v ? w : v;
  }
  if ((threadIdx.x & 31) == 0) atomic_max_nonneg(out, v);
}

// ------------------------------------------------------------ kernels

// A job's record into shared memory (the threads of one warp, or fewer
// words than threads): its fields are then read where they are used instead
// of held in registers through the products.
template <typename J>
__device__ __forceinline__ void dft_job_in(J *to, const J *from) {
  static_assert(sizeof(J) % 4 == 0 && sizeof(J) / 4 <= kDftThreads, "a word per thread");
  if (threadIdx.x < sizeof(J) / 4)
    reinterpret_cast<int *>(to)[threadIdx.x] = reinterpret_cast<const int *>(from)[threadIdx.x];
}

// The last two space axes of windows, forward (FWD: model planes -> cropped
// planes) or adjoint with the ISTA update (epilogues as axis_pass; kStore
// only in the forward direction).  Persistent blocks walk batches of up to
// job.np planes: batch b is planes [batch_plane[b], + np) of job
// batch_job[b].
template <typename R, bool FWD>
__global__ void __launch_bounds__(kDftThreads, sizeof(R) == sizeof(float) ? 4 : 3)
    plane_dft(const PlaneDftJob<R> *__restrict__ jobs, const int *__restrict__ batch_job,
              const long *__restrict__ batch_plane, int n_batch, int epilogue, R step_arg,
              R lamb_arg, const R *step_dev, const R *lamb_dev, R *max_out) {
  using C = Cx<R>;
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const bool multi = step_dev != nullptr;
  R *const smem = reinterpret_cast<R *>(smem_raw);
  R local_max = (R)0;
  // a batch's input planes into its staging buffer (which starts after the
  // tables of its job)
  auto fetch = [&](int bi) {
    const PlaneDftJob<R> &job = jobs[batch_job[bi]];
    const long p0 = batch_plane[bi];
    const int np = (int)min((long)job.np, job.planes - p0);
    C *stage = reinterpret_cast<C *>(smem + dft_table_reals(job.b) + dft_table_reals(job.a));
    const C *src = job.src + p0 * ((long)job.a.n_in * job.b.n_in);
    const int n = np * job.a.n_in * job.b.n_in;
    // the model rows that the update will read
    if (!FWD && epilogue != kStore && threadIdx.x == 0) {
      const long plane = (long)job.a.n_out * job.b.n_out;
      prefetch_l2(job.dst + p0 * plane, np * plane * (long)sizeof(C));
    }
    if (sizeof(C) == 8 && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
      for (int e = threadIdx.x; e < n / 2; e += kDftThreads)
        cp_async<16>(stage + 2 * e, src + 2 * e);
      if ((n & 1) && threadIdx.x == 0) cp_async<sizeof(C)>(stage + n - 1, src + n - 1);
    } else {
      for (int e = threadIdx.x; e < n; e += kDftThreads) cp_async<sizeof(C)>(stage + e, src + e);
    }
  };
  __shared__ PlaneDftJob<R> records[2];  // of this batch and the last
  const R *tab_a = nullptr, *tab_b = nullptr;  // tables now in shared memory
  bool fetched = false;                        // this batch is already on its way
  int half = 0;
  for (int bi = blockIdx.x; bi < n_batch; bi += gridDim.x, half ^= 1) {
    const PlaneDftJob<R> &job = records[half];
    dft_job_in(&records[half], jobs + batch_job[bi]);
    if (!fetched) {
      // first batch, or one of other tables: nothing of the last is in use
      __syncthreads();
      dft_load_table<R>(smem, job.b);
      dft_load_table<R>(smem + dft_table_reals(job.b), job.a);
      tab_a = job.a.tab;
      tab_b = job.b.tab;
      fetch(bi);
      cp_async_commit();
    }
    cp_async_wait<0>();
    __syncthreads();
    const long p0 = batch_plane[bi];
    const int np = (int)min((long)job.np, job.planes - p0);
    R *tb = smem;
    R *ta = tb + dft_table_reals(job.b);
    C *stage = reinterpret_cast<C *>(ta + dft_table_reals(job.a));
    C *rows = stage + plane_stage_reals(job.a, job.b, job.np) / 2;
    const int rs = dft_row_stride(job.b);
    {
      const int nb = job.b.n_in;
      const int skip = (job.a.n_in - 1) * nb;  // between the planes' columns
      const int plane_rows = job.a.n_out * rs;
      dft_from_raw<R, FWD>(
          stage, nb, np * nb, job.a, ta, [&](int q) { return q + q / nb * skip; },
          [&](int q) {
            const int p = q / nb;
            return rows + p * plane_rows + (q - p * nb);
          },
          rs);
    }
    __syncthreads();
    // the staging buffer is free: the next batch, if its tables are the same
    // (equal padded lengths have equal window lengths, so the same layout)
    const int next = bi + gridDim.x;
    fetched = false;
    if (next < n_batch) {
      const PlaneDftJob<R> &nj = jobs[batch_job[next]];
      if (nj.a.tab == tab_a && nj.b.tab == tab_b) {
        fetch(next);
        fetched = true;
      }
    }
    cp_async_commit();
    dft_rows_in_place<R, FWD, kDftThreads>(rows, rs, np * job.a.n_out, job.b, tb);
    __syncthreads();
    const R most = dft_rows_out<R, kDftThreads>(
        rows, rs, np * job.a.n_out, job.b.n_out,
        job.dst + p0 * ((long)job.a.n_out * job.b.n_out), FWD ? (int)kStore : epilogue,
        multi ? step_dev[job.pid] : step_arg,
        lamb_dev != nullptr ? lamb_dev[multi ? job.pid : 0] : lamb_arg);
    if (!FWD && epilogue == kUpdateMax) {
      if (multi)  // one maximum per problem
        warp_atomic_max(max_out + job.pid, most);
      else
        local_max = most > local_max ? most : local_max;
    }
  }
  if (!FWD && epilogue == kUpdateMax && !multi) warp_atomic_max(max_out, local_max);
}

// Windows with one space axis (or the last axis of windows whose planes do
// not fit): as plane_dft, a batch being job.np lines whose tiles are at most
// one per thread.
template <typename R, bool FWD, int NT>
__global__ void __launch_bounds__(NT, (sizeof(R) == sizeof(float) ? 512 : 384) / NT)
    line_dft(const PlaneDftJob<R> *__restrict__ jobs, const int *__restrict__ batch_job,
             const long *__restrict__ batch_line, int n_batch, int epilogue, R step_arg,
             R lamb_arg, const R *step_dev, const R *lamb_dev, R *max_out) {
  using C = Cx<R>;
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const bool multi = step_dev != nullptr;
  R *const tab = reinterpret_cast<R *>(smem_raw);
  R local_max = (R)0;
  const R *tab_b = nullptr;
  for (int bi = blockIdx.x; bi < n_batch; bi += gridDim.x) {
    const PlaneDftJob<R> &job = jobs[batch_job[bi]];
    const DftAxis<R> b = job.b;
    const long l0 = batch_line[bi];
    const int n = (int)min((long)job.np, job.planes - l0);
    const int rs = dft_row_stride(b);
    C *rows = reinterpret_cast<C *>(tab + dft_table_reals(b));
    __syncthreads();  // the last batch is stored
    if (tab_b != b.tab) {
      dft_load_table<R, NT>(tab, b);
      tab_b = b.tab;
    }
    const C *src = job.src + l0 * b.n_in;
    if (threadIdx.x == 0) {
      // into L2: the model lines that the update will read, and the next
      // batch's lines
      if (!FWD && epilogue != kStore)
        prefetch_l2(job.dst + l0 * b.n_out, n * b.n_out * (long)sizeof(C));
      if (bi + gridDim.x < n_batch) {
        const PlaneDftJob<R> &nj = jobs[batch_job[bi + gridDim.x]];
        const long m0 = batch_line[bi + gridDim.x];
        prefetch_l2(nj.src + m0 * nj.b.n_in,
                    min((long)nj.np, nj.planes - m0) * nj.b.n_in * (long)sizeof(C));
      }
    }
    const int cpr = min(b.n_in, NT);
    const int tr = NT / cpr;
    const int r0 = threadIdx.x / cpr;
    for (int r = r0; r0 < tr && r < n; r += tr)
      for (int c = threadIdx.x - r0 * cpr; c < b.n_in; c += cpr)
        cp_async<sizeof(C)>(rows + r * rs + c, src + r * b.n_in + c);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    dft_rows_in_place<R, FWD, NT>(rows, rs, n, b, tab);
    __syncthreads();
    const R most = dft_rows_out<R, NT>(
        rows, rs, n, b.n_out, job.dst + l0 * b.n_out, FWD ? (int)kStore : epilogue,
        multi ? step_dev[job.pid] : step_arg,
        lamb_dev != nullptr ? lamb_dev[multi ? job.pid : 0] : lamb_arg);
    if (!FWD && epilogue == kUpdateMax) {
      if (multi)  // one maximum per problem
        warp_atomic_max(max_out + job.pid, most);
      else
        local_max = most > local_max ? most : local_max;
    }
  }
  if (!FWD && epilogue == kUpdateMax && !multi) warp_atomic_max(max_out, local_max);
}

// One strided space axis of windows; batch b is lines [batch_line[b], + nl)
// of job batch_job[b], line q = outer index * inner + inner index.  Two
// staged batches: the next one is copied in behind this one's products.
template <typename R, bool FWD>
__global__ void __launch_bounds__(kDftThreads, sizeof(R) == sizeof(float) ? 4 : 3)
    axis_dft(const AxisDftJob<R> *__restrict__ jobs, const int *__restrict__ batch_job,
             const long *__restrict__ batch_line, int n_batch) {
  using C = Cx<R>;
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  R *const smem = reinterpret_cast<R *>(smem_raw);
  auto fetch = [&](int bi, int half) {
    const AxisDftJob<R> &job = jobs[batch_job[bi]];
    const long q0 = batch_line[bi];
    const int inner = job.inner;
    const int n = (int)min((long)job.nl, job.outer * inner - q0);
    const int n_in = job.a.n_in;
    C *to = reinterpret_cast<C *>(smem + dft_table_reals(job.a)) + half * n_in * job.nl;
    const long o0 = q0 / inner;
    const int i0 = (int)(q0 - o0 * inner);
    for (int q = threadIdx.x; q < n; q += kDftThreads) {
      const int o = (i0 + q) / inner;
      const C *src = job.src + (o0 + o) * n_in * inner + (i0 + q - o * inner);
      C *d = to + q;
      for (int e = 0; e < n_in; ++e, src += inner, d += job.nl) cp_async<sizeof(C)>(d, src);
    }
  };
  const R *tab_a = nullptr;
  bool fetched = false;
  int half = 0;
  for (int bi = blockIdx.x; bi < n_batch; bi += gridDim.x, half ^= 1) {
    const AxisDftJob<R> &job = jobs[batch_job[bi]];
    const DftAxis<R> a = job.a;
    const long q0 = batch_line[bi];
    const int inner = job.inner;
    const int n = (int)min((long)job.nl, job.outer * inner - q0);
    if (!fetched) {
      __syncthreads();
      dft_load_table<R>(smem, a);
      tab_a = a.tab;
      fetch(bi, half);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    const int next = bi + gridDim.x;
    fetched = false;
    if (next < n_batch && jobs[batch_job[next]].a.tab == tab_a) {
      // the other half was last read before the barrier above
      fetch(next, half ^ 1);
      fetched = true;
    }
    cp_async_commit();
    const long o0 = q0 / inner;
    const int i0 = (int)(q0 - o0 * inner);
    C *dst = job.dst + o0 * a.n_out * inner;
    const C *raw = reinterpret_cast<const C *>(smem + dft_table_reals(a)) + half * a.n_in * job.nl;
    dft_from_raw<R, FWD>(
        raw, job.nl, n, a, smem, [](int q) { return q; },
        [&](int q) {
          const int o = (i0 + q) / inner;
          return dst + (long)o * a.n_out * inner + (i0 + q - o * inner);
        },
        (long)inner);
  }
}

}  // namespace agd
