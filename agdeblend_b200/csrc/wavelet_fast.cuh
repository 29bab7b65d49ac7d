// Wavelet convolution / correlation of window traces (reference
// src/wavelet.c:239-301) by a transform of length N that splits into
// pairwise coprime prime powers of at most 32: the trace length C itself
// where it does (e.g. 2431 = 11 * 13 * 17), else a longer N >= 2 C - 1 (see
// "Other trace lengths" below).
//
// Per trace the reference computes y <- c2r(r2c(y) * S) with S the
// 1/C-scaled phase spectrum (conjugated for the adjoint), or the bare
// transform pair for traces without a spectrum.  Here two traces a, b of a
// window travel as one complex sequence z = a + i b:
//
//  * prime-factor (Good-Thomas) FFT in shared memory: with C = f_0 f_1 ...
//    and s_i = C / f_i, sample t has the coordinates n_i = t mod f_i, and
//    the load copies it to position sum_i n_i g_i of a dense array with
//    extents (f_0, f_1, ...) and strides g_i (qmap, built on the host).  As
//    exp(-2 pi i t k / C) factors over the axes for k = sum_i k_i s_i mod C,
//    a pass along axis i is a plain f_i-point DFT over lines of stride g_i,
//    with no twiddles and no index wrap; after the forward passes frequency
//    k sits at sum_i (k s_i^-1 mod f_i) g_i (kpos), and the inverse passes
//    return the dense array to the sample layout, which the store reads
//    back through qmap.  Consecutive samples lie sum_i g_i apart, an odd
//    stride, so the copies in and out are free of bank conflicts.
//  * the outermost axis is the turning point: a thread transforms a line
//    forward, multiplies it by the spectrum (kept in the dense frequency
//    order) and transforms it back, where the traces of every pair of the
//    block share a spectrum.  Otherwise, with Z' the product spectrum,
//      Z'_k = ((Z_k + conj Z_{C-k}) S_a + (Z_k - conj Z_{C-k}) S_b) / 2,
//    in a step of its own (Z_k S when both use the same).  The real and
//    imaginary parts of the inverse are the two filtered traces.  A trace
//    without a spectrum (bare transform pair, i.e. C times the trace) stays
//    out of the transform, as zeros, and is scaled when the pair is stored:
//    C times the rounding of its partner would swamp it.
//
// Other trace lengths.  The operator is a circular convolution of length C
// with the real sequence g = c2r(S), so for a C with a large prime (1791 =
// 9 * 199) the trace is zero-padded to the N >= 2 C - 1 of least arithmetic,
// multiplied by the length-N spectrum of the zero-padded g, and sample
// t + C of the linear convolution (t + N - C of the correlation) is added
// back to sample t.  The cost is that of a transform of twice the length;
// a length-C transform would need a direct DFT of its prime factor (199
// products per sample).  13,230 traces of 1791 samples, both directions:
// 59.8 ms with the direct factor-199 passes, 0.47 ms padded to N = 3696.
// Lengths whose radix passes sum directly over no prime above 19 keep them:
// they are the more accurate there (engine.cuh, pick_wavelet_shapes).
//
// The adjoint reads its traces straight from the blended record (the blend
// adjoint gather of src/blend.c:1262-1292), so the traces are not written
// and re-read between the two steps.  Loads are cp.async copies (zero-filled
// outside a trace's blended samples), all in flight at once.
#pragma once

#include "fast.cuh"

namespace agd {

constexpr int kPfaMaxFactors = 4;
constexpr int kWavThreads = 256;
constexpr int kWavMaxPairs = 4;  // pairs of a block at most

struct PfaShape {
  int N;                          // transform length
  int nf;                         // number of factors (axes)
  int f[kPfaMaxFactors];          // pairwise coprime prime powers, outermost axis first
  int g[kPfaMaxFactors];          // dense stride of each axis (product of the later f)
  float inv_g[kPfaMaxFactors];    // 1 / g (quotients by the float reciprocal)
  float inv_lines[kPfaMaxFactors];  // f / N: 1 / (lines of a pass)
};

template <typename R>
struct WaveletFastJob {
  R *y;                        // window traces [n_traces][C]
  const int *src;              // per trace spectrum index, or -1 (transform pair only)
  const unsigned short *qmap;  // [N] dense position of sample t
  const unsigned short *kpos;  // [N] dense position of frequency k after the forward passes
  const long *blend_rec;       // per trace: flat record start, or -1 (adjoint gather)
  const int *blend_ts;         // per trace: first blended sample
  const int *blend_n;          // per trace: number of blended samples
  int n_traces;
  int C;                       // trace length: N, or at most (N + 1) / 2
  PfaShape sh;
};

// floor(x / d) for 0 <= x < 2^22 from the rounded reciprocal r = 1 / d:
// (x + 1/2) / d lies at least 1/(2d) from an integer and the product's
// relative error is below 2^-23, so truncation gives the exact quotient.
__device__ __forceinline__ int div_small(int x, float r) {
  return __float2int_rz(((float)x + 0.5f) * r);
}

// One pass along an axis of extent F and stride g over np dense arrays of
// N elements: line l of a pair starts at l + (l / g) (F - 1) g.
template <typename R, int F, bool INV>
__device__ __forceinline__ void pfa_pass(Cx<R> *buf, int np, int N, int g, float inv_g,
                                         float inv_lines) {
  using C = Cx<R>;
  const int lines = N / F;
  const int total = np * lines;
  for (int idx = threadIdx.x; idx < total; idx += kWavThreads) {
    const int pr = div_small(idx, inv_lines);
    const int l = idx - pr * lines;
    const int hi = div_small(l, inv_g);
    C *b = buf + pr * N + l + hi * (F - 1) * g;
    C v[F];
#pragma unroll
    for (int m = 0; m < F; ++m) v[m] = b[m * g];
    dft<R, F, INV>(v);
#pragma unroll
    for (int m = 0; m < F; ++m) b[m * g] = v[m];
  }
}

// The turning point of the transform along the outermost axis, where the two
// traces of every pair share a spectrum: the forward DFT of a line, its
// products with the spectrum (stored in the dense frequency order, so that
// the values of neighbouring lines lie side by side) and the inverse DFT,
// without leaving the registers.  spec_of(pair): the pair's spectrum.
template <typename R, int F, typename Spec>
__device__ __forceinline__ void pfa_turn(Cx<R> *buf, int np, int N, int g, float inv_lines,
                                         bool adjoint, Spec spec_of) {
  using C = Cx<R>;
  const int lines = N / F;  // = g
  const int total = np * lines;
  for (int idx = threadIdx.x; idx < total; idx += kWavThreads) {
    const int pr = div_small(idx, inv_lines);
    const int l = idx - pr * lines;
    C *b = buf + pr * N + l;
    const C *sp = spec_of(pr) + l;
    C v[F];
#pragma unroll
    for (int m = 0; m < F; ++m) v[m] = b[m * g];
    dft<R, F, false>(v);
#pragma unroll
    for (int m = 0; m < F; ++m) {
      C w = __ldg(sp + m * g);
      if (adjoint) w.y = -w.y;
      v[m] = cmul(v[m], w);
    }
    dft<R, F, true>(v);
#pragma unroll
    for (int m = 0; m < F; ++m) b[m * g] = v[m];
  }
}

// Factors above FMAX are compiled out (their register DFTs would raise the
// register demand of every pass); the host picks an instantiation whose
// FMAX covers the shape.
template <typename R, bool INV, int FMAX>
__device__ void pfa_pass_any(int F, Cx<R> *buf, int np, int N, int g, float inv_g,
                             float inv_lines) {
#define AGD_PFA_CASE(n) \
  case n: \
    if constexpr (n <= FMAX) pfa_pass<R, n, INV>(buf, np, N, g, inv_g, inv_lines); \
    break;
  switch (F) {
    AGD_PFA_CASE(2)
    AGD_PFA_CASE(3)
    AGD_PFA_CASE(4)
    AGD_PFA_CASE(5)
    AGD_PFA_CASE(7)
    AGD_PFA_CASE(8)
    AGD_PFA_CASE(9)
    AGD_PFA_CASE(11)
    AGD_PFA_CASE(13)
    AGD_PFA_CASE(16)
    AGD_PFA_CASE(17)
    AGD_PFA_CASE(19)
    AGD_PFA_CASE(23)
    AGD_PFA_CASE(25)
    AGD_PFA_CASE(27)
    AGD_PFA_CASE(32)
    default: break;  // the host only builds shapes from the factors above
  }
#undef AGD_PFA_CASE
}

template <typename R, int FMAX, typename Spec>
__device__ void pfa_turn_any(int F, Cx<R> *buf, int np, int N, int g, float inv_lines,
                             bool adjoint, Spec spec_of) {
#define AGD_PFA_CASE(n) \
  case n: \
    if constexpr (n <= FMAX) pfa_turn<R, n>(buf, np, N, g, inv_lines, adjoint, spec_of); \
    break;
  switch (F) {
    AGD_PFA_CASE(2)
    AGD_PFA_CASE(3)
    AGD_PFA_CASE(4)
    AGD_PFA_CASE(5)
    AGD_PFA_CASE(7)
    AGD_PFA_CASE(8)
    AGD_PFA_CASE(9)
    AGD_PFA_CASE(11)
    AGD_PFA_CASE(13)
    AGD_PFA_CASE(16)
    AGD_PFA_CASE(17)
    AGD_PFA_CASE(19)
    AGD_PFA_CASE(23)
    AGD_PFA_CASE(25)
    AGD_PFA_CASE(27)
    AGD_PFA_CASE(32)
    default: break;
  }
#undef AGD_PFA_CASE
}

// Input sample t of trace tr: from the record through its blend coordinates
// (adjoint), or from the traces themselves.
template <typename R>
__device__ __forceinline__ R wavelet_input(const WaveletFastJob<R> &job, const R *record, int tr,
                                           int t) {
  if (record == nullptr) return job.y[(long)tr * job.C + t];
  const long r0 = job.blend_rec[tr];
  const int s0 = job.blend_ts[tr];
  return r0 >= 0 && t >= s0 && t < s0 + job.blend_n[tr] ? record[r0 + (t - s0)] : (R)0;
}

// Each CTA transforms np_max pairs of traces of one window (fewer in the
// window's last CTA).  direction +1: convolution in place on the traces;
// -1: correlation of the traces gathered from `record`, written to y.
// MINB blocks per SM (the register budget of the largest DFT decides which
// is faster; the engine times the candidates); factors up to FMAX.
// PADDED: some window's transform is longer than its traces.
template <typename R, int MINB, int FMAX, bool PADDED>
__global__ void __launch_bounds__(kWavThreads, MINB)
    wavelet_fast(const WaveletFastJob<R> *__restrict__ jobs, const int *__restrict__ cta_job,
                 const int *__restrict__ cta_pair0, int np_max,
                 const Cx<R> *__restrict__ spectra, const long *__restrict__ spec_off,
                 int direction, const R *__restrict__ record) {
  using C = Cx<R>;
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *buf = reinterpret_cast<C *>(smem_raw);
  const WaveletFastJob<R> &job = jobs[cta_job[blockIdx.x]];
  const PfaShape &sh = job.sh;  // read per pass (a local copy would sit in local memory)
  const int N = sh.N;
  const int Ct = PADDED ? job.C : N;
  const int n_tr = job.n_traces;
  const int pair0 = cta_pair0[blockIdx.x];
  const int np = min(np_max, ((n_tr + 1) >> 1) - pair0);
  const unsigned short *__restrict__ qmap = job.qmap;
  const unsigned short *__restrict__ kpos = job.kpos;

  // ---- load: trace a -> real part, trace b -> imaginary part, each sample
  // to its dense position; thread u copies half u & 1 of sample u >> 1, so a
  // warp fills 16 whole complex slots; every copy of the block in flight
  // together, one position look-up for all pairs
  {
    const R *from[kWavMaxPairs];  // this thread's trace of each pair, sample 0
    int lo[kWavMaxPairs], hi[kWavMaxPairs];
#pragma unroll
    for (int pr = 0; pr < kWavMaxPairs; ++pr) {
      const int tr = 2 * (pair0 + pr) + (threadIdx.x & 1);
      from[pr] = job.y;
      lo[pr] = hi[pr] = 0;
      if (pr >= np || tr >= n_tr || job.src[tr] < 0) continue;
      if (record != nullptr) {
        const long r0 = job.blend_rec[tr];
        if (r0 < 0) continue;
        lo[pr] = job.blend_ts[tr];
        hi[pr] = lo[pr] + job.blend_n[tr];  // a span ends within the trace
        from[pr] = record + r0 - lo[pr];
      } else {
        hi[pr] = Ct;
        from[pr] = job.y + (long)tr * Ct;
      }
    }
    R *to = reinterpret_cast<R *>(buf) + (threadIdx.x & 1);
    for (int t = threadIdx.x >> 1; t < N; t += kWavThreads / 2) {
      R *slot = to + 2 * __ldg(qmap + t);
#pragma unroll
      for (int pr = 0; pr < kWavMaxPairs; ++pr)
        if (pr < np) {
          const bool v = t >= lo[pr] && t < hi[pr];
          cp_async<sizeof(R)>(slot + 2 * pr * N, v ? from[pr] + t : job.y, v);
        }
    }
  }
  cp_async_commit();
  // spectrum of each pair's traces (a half without one holds zeros: any
  // spectrum serves it)
  __shared__ long at[kWavMaxPairs][2];
  if (threadIdx.x < np) {
    const int ta = 2 * (pair0 + threadIdx.x);
    const int sa = job.src[ta];
    const int sb = ta + 1 < n_tr ? job.src[ta + 1] : sa;
    at[threadIdx.x][0] = sa >= 0 ? spec_off[sa] : sb >= 0 ? spec_off[sb] : 0;
    at[threadIdx.x][1] = sb >= 0 ? spec_off[sb] : sa >= 0 ? spec_off[sa] : 0;
  }
  cp_async_wait<0>();
  __syncthreads();
  bool shared = true;
  for (int pr = 0; pr < np; ++pr) shared = shared && at[pr][0] == at[pr][1];

  const bool adjoint = direction < 0;
  for (int i = sh.nf - 1; i > 0; --i) {
    pfa_pass_any<R, false, FMAX>(sh.f[i], buf, np, N, sh.g[i], sh.inv_g[i], sh.inv_lines[i]);
    __syncthreads();
  }
  if (shared) {
    pfa_turn_any<R, FMAX>(sh.f[0], buf, np, N, sh.g[0], sh.inv_lines[0], adjoint,
                          [&](int pr) { return spectra + at[pr][0]; });
    __syncthreads();
  } else {
    pfa_pass_any<R, false, FMAX>(sh.f[0], buf, np, N, sh.g[0], sh.inv_g[0], sh.inv_lines[0]);
    __syncthreads();
    // spectrum product (frequencies k and N - k together)
    for (int pr = 0; pr < np; ++pr) {
      const C *spa = spectra + at[pr][0];
      const C *spb = spectra + at[pr][1];
      C *b = buf + pr * N;
      for (int k = threadIdx.x; k < N / 2 + 1; k += kWavThreads) {
        const int p = __ldg(kpos + k);
        const int q = __ldg(kpos + (k ? N - k : 0));
        C fa = spa[p], fb = spb[p];
        if (adjoint) {
          fa.y = -fa.y;
          fb.y = -fb.y;
        }
        const C zp = b[p];
        const C zq = b[q];
        const C u = cmake<C>(zp.x + zq.x, zp.y - zq.y);  // Z_k + conj Z_{N-k}
        const C d = cmake<C>(zp.x - zq.x, zp.y + zq.y);  // Z_k - conj Z_{N-k}
        const C ua = cmul(u, fa);
        const C db = cmul(d, fb);
        b[p] = cmake<C>((R)0.5 * (ua.x + db.x), (R)0.5 * (ua.y + db.y));
        // Z'_{N-k} = conj((u S_a - d S_b) / 2)
        if (q != p) b[q] = cmake<C>((R)0.5 * (ua.x - db.x), (R)-0.5 * (ua.y - db.y));
      }
    }
    __syncthreads();
    pfa_pass_any<R, true, FMAX>(sh.f[0], buf, np, N, sh.g[0], sh.inv_g[0], sh.inv_lines[0]);
    __syncthreads();
  }
  for (int i = 1; i < sh.nf; ++i) {
    pfa_pass_any<R, true, FMAX>(sh.f[i], buf, np, N, sh.g[i], sh.inv_g[i], sh.inv_lines[i]);
    __syncthreads();
  }

  // ---- store both traces of each pair; a padded transform's samples past
  // the trace end wrap onto sample t
  [[maybe_unused]] const int wrap = adjoint ? N - Ct : Ct;
  [[maybe_unused]] const int w_lo = adjoint ? 1 : 0;  // samples [w_lo, w_hi) take one
  [[maybe_unused]] const int w_hi = adjoint ? Ct : Ct - 1;
  {
    bool live[kWavMaxPairs][2];
#pragma unroll
    for (int pr = 0; pr < kWavMaxPairs; ++pr)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int tr = 2 * (pair0 + pr) + h;
        live[pr][h] = pr < np && tr < n_tr && job.src[tr] >= 0;
      }
    R *y0 = job.y + 2L * pair0 * Ct;
    for (int t = threadIdx.x; t < Ct; t += kWavThreads) {
      const C *b = buf + __ldg(qmap + t);
      const C *u = nullptr;
      if constexpr (PADDED) {
        if (N != Ct && t >= w_lo && t < w_hi) u = buf + __ldg(qmap + t + wrap);
      }
#pragma unroll
      for (int pr = 0; pr < kWavMaxPairs; ++pr)
        if (pr < np) {
          C v = b[pr * N];
          if constexpr (PADDED) {
            if (u != nullptr) v = cadd(v, u[pr * N]);
          }
          R *y = y0 + 2L * pr * Ct + t;
          if (live[pr][0]) y[0] = v.x;
          if (live[pr][1]) y[Ct] = v.y;
        }
    }
  }
  for (int tr = 2 * pair0; tr < min(2 * (pair0 + np), n_tr); ++tr) {  // without a spectrum
    if (job.src[tr] >= 0) continue;
    for (int t = threadIdx.x; t < Ct; t += kWavThreads)
      job.y[(long)tr * Ct + t] = wavelet_input<R>(job, record, tr, t) * (R)Ct;
  }
}

// ------------------------------------------------- padded spectra (set-up)

// Taps g of the circular convolution whose 1/C-scaled length-C half spectrum
// is sp (c2r: the imaginary parts of the zero and Nyquist bins are ignored):
// g[n] = sum_k S_k e^{+2 pi i n k / C} over all k, in double precision.  One
// block per tap.
__global__ void __launch_bounds__(kWavThreads)
    wavelet_taps(const double2 *__restrict__ sp, int C, double *__restrict__ g) {
  __shared__ double red[32];
  const long n = blockIdx.x;
  double acc = 0.0;
  for (int k = threadIdx.x; k <= C / 2; k += kWavThreads) {
    double s, c;
    sincospi(2.0 * (double)((n * k) % C) / (double)C, &s, &c);
    if (k == 0 || 2 * k == C)
      acc += sp[k].x * c;
    else
      acc += 2.0 * (sp[k].x * c - sp[k].y * s);
  }
  const double t = block_sum(acc, red);
  if (threadIdx.x == 0) g[n] = t;
}

// Spectrum of the taps zero-padded to length N, scaled by 1/N, in the dense
// frequency order: out[kpos[k]] = (1/N) sum_{n<C} g[n] e^{-2 pi i n k / N},
// and its conjugate at kpos[N - k].  One block per k <= N / 2.
template <typename R>
__global__ void __launch_bounds__(kWavThreads)
    wavelet_pad_spectrum(const double *__restrict__ g, int C, int N,
                         const unsigned short *__restrict__ kpos, Cx<R> *__restrict__ out) {
  __shared__ double red_c[32], red_s[32];
  const long k = blockIdx.x;
  double re = 0.0, im = 0.0;
  for (int n = threadIdx.x; n < C; n += kWavThreads) {
    double s, c;
    sincospi(2.0 * (double)((n * k) % N) / (double)N, &s, &c);
    re += g[n] * c;
    im -= g[n] * s;
  }
  const double tr = block_sum(re, red_c);
  const double ti = block_sum(im, red_s);
  if (threadIdx.x == 0) {
    out[kpos[k]] = cmake<Cx<R>>((R)(tr / N), (R)(ti / N));
    if (k > 0 && 2 * k != N) out[kpos[N - k]] = cmake<Cx<R>>((R)(tr / N), (R)(-ti / N));
  }
}

}  // namespace agd
