// Time axis of windows whose time length is Lt = 16 NA and padded length
// N = Pt = 20 NA (NA = 16: 256 samples, padded 320; NA = 8: 128, 160), the
// forward c2r with taper and overlap-add (src/fk.c:307-373) and the adjoint
// gather, taper and r2c (src/fk.c:375-452).
//
// Two traces a, b of a window travel as one complex sequence z = a + i b of
// length N, so no half-length split with its twiddles is needed:
// Z_k = A_k + i B_k and Z_{N-k} = conj A_k + i conj B_k.  The transform is
// four-step with N = NA * 20, and sample n = n2 + NA n1 (n2 < NA, n1 < 20)
// in both directions:
//
//   forward  Z_k, k = 20 k1 + k2: DFT-NA over k1 per k2, twiddle
//            W_N^(n2 k2), DFT-20 over k2 per n2.  Thread n2 then holds the
//            samples n2 + NA n1; the window keeps n1 < 16, and as the hop is
//            8 NA, samples n1 and n1 + 8 are one hop apart: taper,
//            overlap-add and carry stay in the thread's registers.
//   adjoint  DFT-20 over n1 per n2 (n1 >= 16 is padding; the thread keeps
//            the half of its samples that the next window shares), twiddle
//            W_N^(n2 k1), DFT-NA over n2 per k1, k = k1 + 20 k2.  A bin
//            needs Z_k and Z_{N-k} = line 20 - k1, entry NA - 1 - k2: only
//            the upper half of the entries crosses threads.
//
// Bins [f][trace] of a trace pair are 16 consecutive bytes in single
// precision: one copy, one store.  Bound by instruction issue; per trace and
// window about a third of the instructions of half-length transforms of
// single traces.  50,176 traces of 9 windows of 256 samples: forward 320 ->
// 186 us, adjoint 362 -> 182 us (double, 6144 traces: 188 -> 82 and
// 184 -> 72 us).  Blocks own 8 pairs (the loads and
// stores of 8 pairs fill a 128-byte line); a grid that leaves the device
// idle is split over the windows as well (gridDim.y), the forward direction
// repeating one window per split for its carry.
#pragma once

#include "fast.cuh"

namespace agd {

constexpr int kPairs = 8;                    // trace pairs per block
constexpr int kPairThreads = 20 * kPairs;

// work buffer: entry (line 0..19 of pair p, index n2 < NA) at n2 * kPairStride +
// line * kPairs + p; the odd stride keeps threads of consecutive n2 on
// distinct banks
constexpr int kPairStride = 20 * kPairs + 1;

template <typename R, int NA>
struct TimePair {
  static constexpr int N = 20 * NA;
  static constexpr int F = 10 * NA + 1;
  static constexpr int H = 8 * NA;
  static constexpr int kWork = NA * kPairStride;        // complex
  static constexpr int kBins = F * kPairs * 2;          // complex
  static constexpr size_t kFwdSmem = (size_t)(kBins + kWork + N) * sizeof(Cx<R>);
  static constexpr size_t kAdjSmem = (size_t)(2 * kWork + N) * sizeof(Cx<R>);
};

template <typename R>
struct CxPair {  // one bin of two traces
  Cx<R> a, b;
};

// Windows [begin, end) of this block's share of T
__device__ __forceinline__ void pair_range(int T, int &begin, int &end) {
  begin = (int)((long)T * blockIdx.y / gridDim.y);
  end = (int)((long)T * (blockIdx.y + 1) / gridDim.y);
}

template <typename R, int NA, int MINB>
__global__ void __launch_bounds__(kPairThreads, MINB)
    time_fwd_pair(const TimeJob<R> *__restrict__ jobs, const int *__restrict__ cta_job,
                  const int *__restrict__ cta_trace0) {
  using C = Cx<R>;
  using S = TimePair<R, NA>;
  constexpr int N = S::N, F = S::F, H = S::H;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  CxPair<R> *bins = reinterpret_cast<CxPair<R> *>(smem_raw);  // [f][pair]
  C *work = reinterpret_cast<C *>(bins + F * kPairs);
  C *tw = work + S::kWork;  // W_N^(m k) at 20 m + k
  __shared__ R taper[16 * NA];
  const TimeJob<R> &job = jobs[cta_job[blockIdx.x]];
  const int t0 = cta_trace0[blockIdx.x];
  const int ntr = job.n_traces;
  const int nb = min(2 * kPairs, ntr - t0);
  int t_begin, t_end;
  pair_range(job.T, t_begin, t_end);
  for (int k = threadIdx.x; k < N; k += kPairThreads) {
    tw[k] = ctw<R>(tw_offset(N) + (k / 20) * (k % 20));
    if (k < 16 * NA) taper[k] = job.time_taper[k];
  }
  pdl_enter();
  if (t_begin == t_end) return;
  // copies in: pair cp, bins cf, cf + 20, ...
  const int cp = threadIdx.x % kPairs;
  const int cf = threadIdx.x / kPairs;
  const C *z0 = job.z + t0 + 2 * cp + (long)cf * ntr;
  const bool has_a = 2 * cp < nb, has_b = 2 * cp + 1 < nb;
  const bool vec = sizeof(C) == 8 && has_b && ntr % 2 == 0 &&
                   (reinterpret_cast<uintptr_t>(z0) & 15) == 0;
  auto fetch = [&](int t) {
    const C *z = z0 + (long)t * F * ntr;
    CxPair<R> *d = bins + cf * kPairs + cp;
    for (int f = cf; f < F; f += 20, z += 20L * ntr, d += 20 * kPairs) {
      if (vec) {
        cp_async<16>(d, z);
      } else {
        cp_async<sizeof(C)>(&d->a, has_a ? z : job.z, has_a);
        cp_async<sizeof(C)>(&d->b, has_b ? z + 1 : job.z, has_b);
      }
    }
  };
  // the window before the first gives its carry
  const int t_first = t_begin > 0 ? t_begin - 1 : 0;
  fetch(t_first);
  cp_async_commit();
  // second pass: sample offset n2 of pair p, for NA * kPairs threads
  const int n2 = threadIdx.x % NA;
  const int p = threadIdx.x / NA;
  const bool second = threadIdx.x < NA * kPairs;
  const bool live_a = second && 2 * p < nb, live_b = second && 2 * p + 1 < nb;
  const R sca = live_a ? job.space_scale[t0 + 2 * p] : (R)0;
  const R scb = live_b ? job.space_scale[t0 + 2 * p + 1] : (R)0;
  R *ya = job.y + (long)(t0 + 2 * p) * job.C + n2;
  R *yb = ya + job.C;
  C carry[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) carry[q] = cmake<C>((R)0, (R)0);
  for (int t = t_first; t < t_end; ++t) {
    cp_async_wait<0>();
    __syncthreads();
    {  // first pass: line k2 = cf of pair cp
      C v[NA];
#pragma unroll
      for (int k1 = 0; k1 < NA; ++k1) {
        // bins past N / 2 are mirrored; Z_0 and Z_{N/2} take the real parts
        const bool mirror = k1 >= NA / 2;
        const CxPair<R> x = bins[(mirror ? N - 20 * k1 - cf : 20 * k1 + cf) * kPairs + cp];
        v[k1] = mirror ? cmake<C>(x.a.x + x.b.y, x.b.x - x.a.y)
                       : cmake<C>(x.a.x - x.b.y, x.b.x + x.a.y);
        if ((k1 == 0 || k1 == NA / 2) && cf == 0) v[k1] = cmake<C>(x.a.x, x.b.x);
      }
      dft<R, NA, true>(v);
      C *w = work + threadIdx.x;  // line cf, pair cp
#pragma unroll
      for (int m = 0; m < NA; ++m) {
        C u = v[m];
        if (m > 0) {
          const C f = tw[20 * m + cf];
          u = cmake<C>(u.x * f.x + u.y * f.y, u.y * f.x - u.x * f.y);  // times conj W
        }
        w[m * kPairStride] = u;
      }
    }
    __syncthreads();
    if (t + 1 < t_end) fetch(t + 1);  // the bins are free
    cp_async_commit();
    if (second) {
      C v[20];
      const C *w = work + n2 * kPairStride + p;
#pragma unroll
      for (int k = 0; k < 20; ++k) v[k] = w[k * kPairs];
      dft<R, 20, true>(v);
      const int s = t * H;
      const bool store = t >= t_begin;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const R w0 = taper[n2 + NA * q], w1 = taper[n2 + NA * (q + 8)];
        const R oa = carry[q].x + (v[q].x * sca) * w0;
        const R ob = carry[q].y + (v[q].y * scb) * w0;
        if (store && live_a) ya[s + NA * q] = oa;
        if (store && live_b) yb[s + NA * q] = ob;
        carry[q] = cmake<C>((v[q + 8].x * sca) * w1, (v[q + 8].y * scb) * w1);
      }
    }
  }
  if (t_end < job.T) return;
  // last half window, then zeros up to C
  const int s = t_end * H;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    if (live_a) ya[s + NA * q] = carry[q].x;
    if (live_b) yb[s + NA * q] = carry[q].y;
  }
  const int tail = job.C - (t_end + 1) * H;
  for (int idx = threadIdx.x; idx < nb * tail; idx += kPairThreads) {
    const int i = idx / tail;
    job.y[(long)(t0 + i) * job.C + (t_end + 1) * H + (idx - i * tail)] = (R)0;
  }
}

template <typename R, int NA, int MINB>
__global__ void __launch_bounds__(kPairThreads, MINB)
    time_adj_pair(const TimeJob<R> *__restrict__ jobs, const int *__restrict__ cta_job,
                  const int *__restrict__ cta_trace0, const R *__restrict__ record,
                  int from_record) {
  using C = Cx<R>;
  using S = TimePair<R, NA>;
  constexpr int N = S::N, F = S::F, H = S::H;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *tw = reinterpret_cast<C *>(smem_raw);  // W_N^(m k) at NA m + k: neighbouring threads
                                            // read neighbouring values
  C *work2 = tw + N;                        // two work buffers
  __shared__ R taper[16 * NA];
  const TimeJob<R> &job = jobs[cta_job[blockIdx.x]];
  const int t0 = cta_trace0[blockIdx.x];
  const int ntr = job.n_traces;
  const int nb = min(2 * kPairs, ntr - t0);
  int t_begin, t_end;
  pair_range(job.T, t_begin, t_end);
  for (int k = threadIdx.x; k < N; k += kPairThreads) {
    tw[k] = ctw<R>(tw_offset(N) + (k / NA) * (k % NA));
    if (k < 16 * NA) taper[k] = job.time_taper[k];
  }
  pdl_enter();
  if (t_begin == t_end) return;
  // first pass: samples n2 + NA n1 of pair p, for NA * kPairs threads
  const int n2 = threadIdx.x % NA;
  const int p = threadIdx.x / NA;
  const bool first = threadIdx.x < NA * kPairs;
  // per trace: source of trace sample n2, readable samples [lo, hi) - n2
  const R *src[2];
  int lo[2], hi[2];
  R sc[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int i = 2 * p + h;
    src[h] = job.y;
    lo[h] = hi[h] = 0;
    sc[h] = (R)0;
    if (first && i < nb) {
      const int tr = t0 + i;
      sc[h] = job.space_scale[tr];
      if (from_record) {
        const long rec = job.blend_rec[tr];
        const int ts = job.blend_ts[tr];
        if (rec >= 0) {
          src[h] = record + (rec - ts) + n2;
          lo[h] = ts - n2;
          hi[h] = ts + job.blend_n[tr] - n2;
        }
      } else {
        src[h] = job.y + (long)tr * job.C + n2;
        lo[h] = -n2;
        hi[h] = job.C - n2;
      }
    }
  }
  // half a window of both traces, scaled: samples s0 + n2 + NA q, q < 8
  auto load_half = [&](int s0, C (&x)[8]) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int s = s0 + NA * q;
      x[q].x = s >= lo[0] && s < hi[0] ? src[0][s] : (R)0;
      x[q].y = s >= lo[1] && s < hi[1] ? src[1][s] : (R)0;
    }
  };
  C head[8], next[8];
  load_half(t_begin * H, head);
  load_half((t_begin + 1) * H, next);
#pragma unroll
  for (int q = 0; q < 8; ++q) head[q] = cmake<C>(head[q].x * sc[0], head[q].y * sc[1]);
  // second pass: line k1 of pair sp
  const int sp = threadIdx.x % kPairs;
  const int k1 = threadIdx.x / kPairs;
  const int mate = k1 > 0 ? 20 - k1 : 0;  // line of Z_{N-k}
  const bool out_a = 2 * sp < nb, out_b = 2 * sp + 1 < nb;
  C *z0 = job.z + t0 + 2 * sp + (long)k1 * ntr;
  const bool vec = sizeof(C) == 8 && out_b && ntr % 2 == 0 &&
                   (reinterpret_cast<uintptr_t>(z0) & 15) == 0;
  auto put = [&](C *z, C a, C b) {
    if (vec) {
      *reinterpret_cast<float4 *>(z) = make_float4((float)a.x, (float)a.y, (float)b.x, (float)b.y);
    } else {
      if (out_a) z[0] = a;
      if (out_b) z[1] = b;
    }
  };
  __syncthreads();
  for (int t = t_begin; t < t_end; ++t) {
    C *work = work2 + (t & 1) * S::kWork;
    if (first) {
      C v[20];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const R w0 = taper[n2 + NA * q], w1 = taper[n2 + NA * (q + 8)];
        v[q] = cscale(head[q], w0);
        head[q] = cmake<C>(next[q].x * sc[0], next[q].y * sc[1]);
        v[q + 8] = cscale(head[q], w1);
      }
#pragma unroll
      for (int q = 16; q < 20; ++q) v[q] = cmake<C>((R)0, (R)0);
      if (t + 1 < t_end) load_half((t + 2) * H, next);
      dft<R, 20, false>(v);
      C *w = work + n2 * kPairStride + p;
#pragma unroll
      for (int m = 0; m < 20; ++m) w[m * kPairs] = m > 0 ? cmul(v[m], tw[NA * m + n2]) : v[m];
    }
    __syncthreads();
    C v[NA];
    C *w = work + threadIdx.x;  // line k1, pair sp
#pragma unroll
    for (int m = 0; m < NA; ++m) v[m] = w[m * kPairStride];
    dft<R, NA, false>(v);
#pragma unroll
    for (int m = NA / 2; m < NA; ++m) w[m * kPairStride] = v[m];
    __syncthreads();
    // bins k1 + 20 i from v[i] and the mate's entry NA - 1 - i (line 0: its
    // own entry NA - i), doubled as bins 1 .. N/2 - 1 are
    const C *u = work + (k1 > 0 ? NA - 1 : NA) * kPairStride + mate * kPairs + sp;
    C *z = z0 + (long)t * F * ntr;
    const long step = 20L * ntr;
#pragma unroll
    for (int i = 0; i < NA / 2; ++i, z += step) {
      if (i == 0 && k1 == 0) {
        put(z, cmake<C>(v[0].x, (R)0), cmake<C>(v[0].y, (R)0));
        continue;
      }
      const C m = u[-i * kPairStride];
      put(z, cmake<C>(v[i].x + m.x, v[i].y - m.y), cmake<C>(v[i].y + m.y, m.x - v[i].x));
    }
    if (k1 == 0) put(z, cmake<C>(v[NA / 2].x, (R)0), cmake<C>(v[NA / 2].y, (R)0));
  }
}

}  // namespace agd
