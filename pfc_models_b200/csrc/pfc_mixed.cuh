// Run-time mixed-radix engine: transforms of any length with factors up to 13, planned on
// the host as a sequence of radices, for the row and column kernels of the sizes without a
// compile-time kernel, for the observables of every plan, and for the one-CTA step.
//
// A CTA holds `count` equal transforms in shared memory. A pass of radix R takes the
// (transform, butterfly) pairs as one flat list of items dealt to all threads of the CTA,
// reads each butterfly's R values from one buffer and writes its outputs to the other, so a
// thread holds one butterfly at a time and a pass costs one barrier. What bounds these
// kernels is the latency of that chain (shared memory, a short dependent DFT, a barrier per
// pass) rather than HBM, so the passes that can share their registers are fused:
//  * a forward and an inverse transform that meet (row: inverse, N, forward; column:
//    forward, ETD1 update, inverse) run the radices of the second in reverse order: the last
//    pass of the first and the first pass of the second then hold the same elements, and
//    the pointwise work between them is applied in the registers (mixed_mid);
//  * the column's first pass reads and its last pass writes global memory directly, and the
//    real-packing twiddles of the rows are applied on the way from and to global memory.
// Radices run in descending order first, so that the fused middle pass, which carries the
// pointwise work, has the most and smallest butterflies to deal out.
// Measured on B200 against the one-buffer engine it replaces, which parked every value
// between the same phases in shared memory (16 barriers a row pass where this has 6): a step
// of 896 x 1568 FP64 87 -> 45 us, of 264 x 264 with an external potential 33 -> 24 us, a 28 x
// 24 cell in one CTA 8.0 -> 6.4 us; the 256^2 FP64 field 8.9 -> 5 us.
#pragma once
#include "pfc_kernels.cuh"

namespace pfc {

// j / d for d of the plan's tables (magic = floor(2^32 / d) + 1, 0 for d = 1); exact while
// j * d < 2^32.
__device__ __forceinline__ int mixed_div(int j, unsigned magic) {
  return magic ? (int)__umulhi((unsigned)j, magic) : j;
}

template <int R, bool INV, class T> __device__ __forceinline__ void mixed_dft(cplx<T>* v) {
  if constexpr (R == 5 || R == 7 || R == 11 || R == 13) dft_odd_c<R, INV>(v);
  else dft<R, INV>(v, (const cplx<T>*)nullptr);
}

// v[q] *= w^(q k) of a pass with stride ns (table [q - 1][k], conjugated for the inverse)
template <int R, bool INV, class T>
__device__ __forceinline__ void mixed_twiddle(cplx<T>* v, const cplx<T>* __restrict__ tw, int ns, int k) {
  const cplx<T>* w = tw + k;
#pragma unroll
  for (int q = 1; q < R; ++q) {
    cplx<T> x = w[(q - 1) * ns];
    if (INV) x.y = -x.y;
    v[q] = cmul(v[q], x);
  }
}

// One pass of radix R over `count` transforms: ld(f, i) and st(f, i, v) read and write
// element i of transform f.
template <int R, bool INV, class T, class Ld, class St>
__device__ __forceinline__ void mixed_items(const FftDesc& d, int p, int count, const cplx<T>* __restrict__ tw, Ld ld,
                                            St st) {
  const int nr = d.nr[p], ns = d.ns[p];
  const unsigned mnr = d.mag_nr[p], mns = d.mag_ns[p];
  const int items = count * nr;
  for (int i = threadIdx.x; i < items; i += blockDim.x) {
    const int f = mixed_div(i, mnr), j = i - f * nr;
    const int k = ns == 1 ? 0 : j - ns * mixed_div(j, mns);
    cplx<T> v[R];
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = ld(f, j + q * nr);
    if (ns > 1) mixed_twiddle<R, INV>(v, tw + d.twoff[p], ns, k);
    mixed_dft<R, INV>(v);
    const int base = (j - k) * R + k;
#pragma unroll
    for (int q = 0; q < R; ++q) st(f, base + q * ns, v[q]);
  }
}

// Calls f with the pass's radix as a compile-time constant. The radix sets are the ones of
// the plan (kRadixPow2, kRadixSmall: primes up to 7, kRadixAll).
template <int R> struct RadixC { static constexpr int value = R; };
template <int RSET, class T, class F>
__device__ __forceinline__ void mixed_switch(int radix, F f) {
  switch (radix) {
    case 2: f(RadixC<2>{}); break;
    case 4: f(RadixC<4>{}); break;
    case 8: f(RadixC<8>{}); break;
    case 16:
      if constexpr (sizeof(T) == 4) f(RadixC<16>{});   // FP64 plans run radix 8 and below
      break;
    default:
      if constexpr (RSET != kRadixPow2) {
        switch (radix) {
          case 3: f(RadixC<3>{}); break;
          case 5: f(RadixC<5>{}); break;
          case 7: f(RadixC<7>{}); break;
          default:
            if constexpr (RSET == kRadixAll) {
              if (radix == 11) f(RadixC<11>{});
              else if (radix == 13) f(RadixC<13>{});
            }
            break;
        }
      }
      break;
  }
}

template <bool INV, int RSET, class T, class Ld, class St>
__device__ __forceinline__ void mixed_pass(const FftDesc& d, int p, int count, const cplx<T>* __restrict__ tw, Ld ld,
                                           St st) {
  mixed_switch<RSET, T>(d.radix[p], [&](auto r) {
    mixed_items<decltype(r)::value, INV, T>(d, p, count, tw, ld, st);
  });
}

// The last pass of a transform (direction INV, description d), the pointwise work on its
// natural-order outputs, and the first pass of the opposite transform (the same radix, no
// twiddles). fn.load(f, i) returns what element i of transform f needs from global memory,
// fn.apply(f, i, aux, v) updates v; the loads of up to 4 elements are issued together, and
// before the butterfly's own reads where the whole butterfly fits.
template <int R, bool INV, class T, class Ld, class Fn, class St>
__device__ __forceinline__ void mixed_mid_items(const FftDesc& d, int f0, int count,
                                                const cplx<T>* __restrict__ tw, Ld ld, Fn fn, St st) {
  const int p = d.npass - 1, nr = d.nr[p];
  const unsigned mnr = d.mag_nr[p];
  const int items = (count - f0) * nr;
  constexpr int CH = R <= 5 ? R : 4;
  for (int i = threadIdx.x; i < items; i += blockDim.x) {
    const int g = mixed_div(i, mnr), j = i - g * nr, f = f0 + g;
    typename Fn::Aux aux[CH];
    if constexpr (CH == R) {
#pragma unroll
      for (int q = 0; q < R; ++q) aux[q] = fn.load(f, j + q * nr);
    }
    cplx<T> v[R];
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = ld(f, j + q * nr);
    if (nr > 1) mixed_twiddle<R, INV>(v, tw + d.twoff[p], nr, j);
    mixed_dft<R, INV>(v);
    if constexpr (CH == R) {
#pragma unroll
      for (int q = 0; q < R; ++q) fn.apply(f, j + q * nr, aux[q], v[q]);
    } else {
#pragma unroll
      for (int c = 0; c < R; c += CH) {
#pragma unroll
        for (int q = c; q < c + CH && q < R; ++q) aux[q - c] = fn.load(f, j + q * nr);
#pragma unroll
        for (int q = c; q < c + CH && q < R; ++q) fn.apply(f, j + q * nr, aux[q - c], v[q]);
      }
    }
    mixed_dft<R, !INV>(v);
#pragma unroll
    for (int q = 0; q < R; ++q) st(f, j * R + q, v[q]);
  }
}

// The same for transform 0 alone where the pointwise work pairs elements ky and n - ky (the
// packed DC / Nyquist column): a thread runs butterflies j and nr - j together, which hold
// both elements of every pair, and pair(ky, kyp, a, b) updates them (kyp == ky for 0 and n/2,
// a and b then the same element). The items are dealt from the last thread down, to the
// threads that the regular columns leave idle.
template <int R, bool INV, class T, class Ld, class Pair, class St>
__device__ __forceinline__ void mixed_mid_paired(const FftDesc& d, const cplx<T>* __restrict__ tw, Ld ld, Pair pair,
                                                 St st) {
  const int p = d.npass - 1, nr = d.nr[p];
  for (int j = (int)blockDim.x - 1 - (int)threadIdx.x; j <= nr / 2; j += blockDim.x) {
    const int jp = j == 0 ? 0 : nr - j;
    const bool two = jp != j;
    cplx<T> a[R], b[R];
#pragma unroll
    for (int q = 0; q < R; ++q) a[q] = ld(0, j + q * nr);
    if (nr > 1) mixed_twiddle<R, INV>(a, tw + d.twoff[p], nr, j);
    mixed_dft<R, INV>(a);
    if (two) {
#pragma unroll
      for (int q = 0; q < R; ++q) b[q] = ld(0, jp + q * nr);
      mixed_twiddle<R, INV>(b, tw + d.twoff[p], nr, jp);
      mixed_dft<R, INV>(b);
#pragma unroll
      for (int q = 0; q < R; ++q) pair(j + q * nr, jp + (R - 1 - q) * nr, a[q], b[R - 1 - q]);
      mixed_dft<R, !INV>(b);
#pragma unroll
      for (int q = 0; q < R; ++q) st(0, jp * R + q, b[q]);
    } else if (j == 0) {
#pragma unroll
      for (int q = 0; q <= R / 2; ++q) pair(q * nr, ((R - q) % R) * nr, a[q], a[(R - q) % R]);
    } else {
#pragma unroll
      for (int q = 0; q < (R + 1) / 2; ++q) pair(j + q * nr, j + (R - 1 - q) * nr, a[q], a[R - 1 - q]);
    }
    mixed_dft<R, !INV>(a);
#pragma unroll
    for (int q = 0; q < R; ++q) st(0, j * R + q, a[q]);
  }
}

// Pre-twiddle of the packed inverse real transform: Z[k] = S + U, Z[m - k] = conj(S - U),
// S = X[k] + conj X[m-k], U = i conj(r_k) (X[k] - conj X[m-k]); Z[0] from the packed DC.
template <class T>
__device__ __forceinline__ void real_pre(cplx<T> xk, cplx<T> xm, cplx<T> r, cplx<T>& zk, cplx<T>& zm) {
  const cplx<T> s = xk + conj(xm), u = mul_i(cmul(conj(r), xk - conj(xm)));
  zk = s + u;
  zm = conj(s - u);
}
// Post-twiddle of the forward: Y[k] = E + r_k O, Y[m - k] = conj(E - r_k O),
// E = (Z[k] + conj Z[m-k]) / 2, O = -i (Z[k] - conj Z[m-k]) / 2.
template <class T>
__device__ __forceinline__ void real_post(cplx<T> zk, cplx<T> zm, cplx<T> r, cplx<T>& yk, cplx<T>& ym) {
  const cplx<T> e = T(0.5) * (zk + conj(zm)), o = T(0.5) * rot4<false>(zk - conj(zm));
  const cplx<T> t = cmul(r, o);
  yk = e + t;
  ym = conj(e - t);
}
template <class T> __device__ __forceinline__ cplx<T> real_dc(cplx<T> p) { return mk(p.x + p.y, p.x - p.y); }

// The packed column's update of one (ky, -ky) pair: n_hat and N_hat of kx = 0 and kx = m are
// unpacked, updated with their own coefficients c0 and cm (and forcing) and repacked.
__device__ __forceinline__ void packed_update(cplx<double> pk, cplx<double> pkp, cplx<double> qk, cplx<double> qkp,
                                              cplx<double> c0, cplx<double> cm, const cplx<double>* f0,
                                              const cplx<double>* fm, cplx<double>& ok, cplx<double>& okp) {
  cplx<double> h0, hm, g0, gm;
  unpack_pair(pk, pkp, h0, hm);
  unpack_pair(qk, qkp, g0, gm);
  cplx<double> h0n = h0 + c0.x * h0 + c0.y * g0;
  cplx<double> hmn = hm + cm.x * hm + cm.y * gm;
  if (f0) {
    h0n = h0n + *f0;
    hmn = hmn + *fm;
  }
  ok = h0n + mul_i(hmn);
  okp = conj(h0n) + mul_i(conj(hmn));
}

// The external-potential decision by the row pass itself: the CTA that stores the last of the
// ranges reduces them all and applies the reference's rules (a kernel of its own cost 3.2 us
// and a launch gap a step). Out of line; every thread of the CTA calls it.
static __device__ __noinline__ void extv_decide_last(const double* minmax, int nparts, ExtvState* st, double g) {
  __shared__ bool last;
  __shared__ double range[2];
  if (threadIdx.x == 0) {
    __threadfence();   // this CTA's pair before the count
    last = atomicAdd(&st->done, 1u) == (unsigned)nparts - 1u;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double lo = INFINITY, hi = -INFINITY;
  for (int i = threadIdx.x; i < nparts; i += blockDim.x) {
    lo = fmin(lo, __ldcg(minmax + 2 * i));
    hi = fmax(hi, __ldcg(minmax + 2 * i + 1));
  }
  block_minmax_store(lo, hi, range);
  if (threadIdx.x == 0) {
    extv_apply(st, range[0], range[1], g);
    st->done = 0;
  }
}

// N of one site of the FP64 row kernel. The log model's is out of line: a thread's butterfly holds
// up to 26 sites, and as many inlined logarithms waited for their instructions (a step of 338 x 11
// 31.6 -> 28.1 us, 242 x 280 26.1 -> 23.3, 264 x 264 18.4 -> 17.7, 896 x 1568 49.9 -> 48.5).
static __device__ __noinline__ double nonlin_log_call(double n, double g, int clamp, double min_phi, double min_log) {
  return nonlin_plain<kModelLog>(n, g, clamp, min_phi, min_log);
}
template <int MODEL>
__device__ __forceinline__ double nonlin_site(double n, double g, int clamp, double min_phi, double min_log) {
  if constexpr (MODEL == kModelLog) return nonlin_log_call(n, g, clamp, min_phi, min_log);
  else return nonlin_plain<MODEL>(n, g, clamp, min_phi, min_log);
}

// ---------------------------------------------------------------- row kernel
// `rows` = 2^rows_log2 rows per CTA, two buffers of rows * ld values. Modes as row_kernel's
// (pfc_kernels.cuh).
template <class T, int MODE, int MODEL, int RSET>
__global__ void __launch_bounds__(256, 2) mixed_row_kernel(RowArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int m = a.m, ny = a.ny, rl2 = a.rows_log2, rows = 1 << rl2, ld = a.ld;
  cplx<T>* src = reinterpret_cast<cplx<T>*>(smem_raw);
  cplx<T>* dst = src + rows * ld;
  const int tid = threadIdx.x, nth = blockDim.x;
  const int y0 = blockIdx.x << rl2;
  const bool dev = (sizeof(T) == 4);
  const cplx<T>* in = a.in;
  cplx<T>* out = a.out;
  const double* scal = a.scal;
  double* out_real = a.out_real;
  double* partials = a.partials;
  if (a.batch) {
    const BatchBufs& bb = a.batch[blockIdx.y];
    in = static_cast<const cplx<T>*>(bb.w);
    out = static_cast<cplx<T>*>(bb.v);
    scal = bb.scal;
    if (partials) partials += (size_t)blockIdx.y * a.partials_stride;
  }
  auto ld_s = [&](int f, int i) { return src[f * ld + generic_pad(i)]; };
  auto st_s = [&](int f, int i, cplx<T> v) { dst[f * ld + generic_pad(i)] = v; };
  auto flip = [&]() {
    __syncthreads();
    cplx<T>* t = src;
    src = dst;
    dst = t;
  };
  const int np = a.fft.npass;

  if (MODE != kRowForward) {
    // packed spectra, column-major [kx][y]: consecutive threads take consecutive rows of one
    // pair (k, m - k); the pre-twiddle is applied on the way into shared memory
    const int n = (m / 2 + 1) << rl2;
#pragma unroll 4
    for (int i = tid; i < n; i += nth) {
      const int r = i & (rows - 1), k = i >> rl2, y = y0 + r;
      const bool valid = y < ny;
      cplx<T>* row = src + r * ld;
      if (k == 0) {
        row[0] = valid ? real_dc(in[y]) : mk(T(0), T(0));
      } else {
        cplx<T> zk = mk(T(0), T(0)), zm = zk;
        if (valid) real_pre(in[(size_t)k * ny + y], in[(size_t)(m - k) * ny + y], a.rtw[k], zk, zm);
        row[generic_pad(k)] = zk;
        if (m - k != k) row[generic_pad(m - k)] = zm;
      }
    }
  } else {
    // real FP64 field (ny, nx), row-major; deviation form subtracts the mean. The tile's values are
    // dealt to the threads as one list: with a loop over its rows, up to 32 narrow ones waited for
    // memory in turn (upload of 16 x 75 FP64: row kernel 24 us, now 7)
    const double mean = dev ? scal[kScalMean] : 0.0;
    const double2* s2 = reinterpret_cast<const double2*>(a.in_real) + (size_t)y0 * m;
    const int n = m << rl2, nvalid = (ny - y0) * m;
#pragma unroll 4
    for (int i = tid; i < n; i += nth) {
      const int r = i / m, j = i - r * m;
      cplx<T> v = mk(T(0), T(0));
      if (i < nvalid) {
        const double2 p = s2[i];
        v = mk((T)(p.x - mean), (T)(p.y - mean));
      }
      src[r * ld + generic_pad(j)] = v;
    }
  }
  __syncthreads();

  if constexpr (MODE == kRowStep) {
    double lo = INFINITY, hi = -INFINITY;
    struct Nonlin {
      struct Aux {};
      float c1, c2, inv, lmin;
      double inv_d, mphi_rel, g, min_phi, min_log;
      int clamp, nvalid;
      bool track;
      double *lo, *hi;
      __device__ __forceinline__ Aux load(int, int) const { return Aux{}; }
      __device__ __forceinline__ void apply(int f, int, Aux, cplx<T>& z) const {
        if constexpr (sizeof(T) == 4) {
          z = mk((T)nonlin_dev<MODEL>((float)z.x, c1, c2, inv, inv_d, clamp, mphi_rel, lmin),
                 (T)nonlin_dev<MODEL>((float)z.y, c1, c2, inv, inv_d, clamp, mphi_rel, lmin));
        } else {
          if (track && f < nvalid) {
            *lo = fmin(*lo, fmin((double)z.x, (double)z.y));
            *hi = fmax(*hi, fmax((double)z.x, (double)z.y));
          }
          z = mk((T)nonlin_site<MODEL>((double)z.x, g, clamp, min_phi, min_log),
                 (T)nonlin_site<MODEL>((double)z.y, g, clamp, min_phi, min_log));
        }
      }
    } fn;
    fn.c1 = fn.c2 = fn.inv = fn.lmin = 0.f;
    fn.inv_d = fn.mphi_rel = 0.0;
    if (dev) {
      fn.c1 = (float)scal[kScalC1];
      fn.c2 = (float)scal[kScalC2];
      fn.inv = (float)scal[kScalInvMean];
      fn.inv_d = scal[kScalInvMean];
      fn.mphi_rel = a.min_phi * fn.inv_d;
      fn.lmin = (float)scal[kScalLogMin];
    }
    fn.g = a.g; fn.min_phi = a.min_phi; fn.min_log = a.min_log;
    fn.clamp = a.clamp;
    fn.nvalid = ny - y0;
    fn.track = a.minmax != nullptr;
    fn.lo = &lo; fn.hi = &hi;
    for (int p = 0; p < np - 1; ++p) {
      mixed_pass<true, RSET, T>(a.fft, p, rows, a.tw, ld_s, st_s);
      flip();
    }
    mixed_switch<RSET, T>(a.fft.radix[np - 1], [&](auto r) {
      mixed_mid_items<decltype(r)::value, true, T>(a.fft, 0, rows, a.tw, ld_s, fn, st_s);
    });
    if (sizeof(T) == 8 && a.minmax) {
      block_minmax_store(lo, hi, a.minmax + 2 * blockIdx.x);
      if (MODEL == kModelLog && a.extv) extv_decide_last(a.minmax, gridDim.x, a.extv, a.g);
    }
    flip();
    for (int p = 1; p < np; ++p) {
      mixed_pass<false, RSET, T>(a.fft_b, p, rows, a.tw, ld_s, st_s);
      flip();
    }
  } else if constexpr (MODE == kRowForward) {
    for (int p = 0; p < np; ++p) {
      mixed_pass<false, RSET, T>(a.fft, p, rows, a.tw, ld_s, st_s);
      flip();
    }
  }

  if constexpr (MODE == kRowStep || MODE == kRowForward) {
    const int n = (m / 2 + 1) << rl2;
#pragma unroll 4
    for (int i = tid; i < n; i += nth) {
      const int r = i & (rows - 1), k = i >> rl2, y = y0 + r;
      if (y >= ny) continue;
      const cplx<T>* row = src + r * ld;
      if (k == 0) {
        out[y] = real_dc(row[0]);
      } else {
        cplx<T> yk, ym;
        real_post(row[generic_pad(k)], row[generic_pad(m - k)], a.rtw[k], yk, ym);
        out[(size_t)k * ny + y] = yk;
        if (m - k != k) out[(size_t)(m - k) * ny + y] = ym;
      }
    }
    return;
  }

  if constexpr (MODE == kRowMaterialize || MODE == kRowReduce) {
    // every pass but the last; the last one's outputs, in natural order, go straight to the
    // field or into the sums
    for (int p = 0; p < np - 1; ++p) {
      mixed_pass<true, RSET, T>(a.fft, p, rows, a.tw, ld_s, st_s);
      flip();
    }
    if constexpr (MODE == kRowMaterialize) {
      const double add = a.add ? *a.add : 0.0;
      KSum acc[1] = {{0.0, 0.0}};
      mixed_pass<true, RSET, T>(a.fft, np - 1, rows, a.tw, ld_s, [&](int f, int j, cplx<T> z) {
        if (y0 + f < ny) {
          reinterpret_cast<double2*>(out_real + (size_t)(y0 + f) * a.nx)[j] =
              make_double2(add + (double)z.x, add + (double)z.y);
          ksum_add(acc[0], (double)z.x);
          ksum_add(acc[0], (double)z.y);
        }
      });
      if (partials) block_reduce_store<1>(acc, partials + 2 * blockIdx.x);
    } else {
      // sums of: raw value (mean), free-energy polynomial, nonlinear mu
      const double mean = dev ? scal[kScalMean] : 0.0;
      const double eps = a.red ? a.red[blockIdx.y].epsilon : a.epsilon, g = a.g;
      KSum acc[3] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
      mixed_pass<true, RSET, T>(a.fft, np - 1, rows, a.tw, ld_s, [&](int f, int, cplx<T> z) {
        if (y0 + f >= ny) return;
        const double vv[2] = {(double)z.x, (double)z.y};
#pragma unroll
        for (int h = 0; h < 2; ++h) row_reduce_add<MODEL>(acc, mean, vv[h], eps, g, a.clamp, a.min_phi, a.min_log);
      });
      block_reduce_store<3>(acc, partials + 6 * blockIdx.x);
    }
  }
}

// ---------------------------------------------------------------- column kernel
// What a mode does with one element (load, apply) and with one pair of the packed column
// (pair), between the forward and the inverse transform of a column.
template <class T, int MODE>
struct ColWork {
  struct Aux {
    cplx<T> c, p;
  };
  const ColArgs<T>* a;
  const cplx<T>* coef;
  const cplx<double>* coef64;
  const void* nin;
  const cplx<float>* nin_lo;
  void* nout;
  cplx<float>* nout_lo;
  int c0;

  __device__ __forceinline__ Aux load(int f, int ky) const {
    Aux x{};
    if constexpr (MODE == kColStep) {
      const int kx = c0 + f, kh = ky <= a->ny / 2 ? ky : a->ny - ky;
      x.c = coef[(size_t)kx * a->nyh + kh];
      x.p = static_cast<const cplx<T>*>(nin)[(size_t)kx * a->ny + ky];
    }
    return x;
  }
  __device__ __forceinline__ void apply(int f, int ky, const Aux& x, cplx<T>& v) const {
    const int kx = c0 + f;
    const size_t i = (size_t)kx * a->ny + ky;
    if constexpr (MODE == kColStep) {
      const cplx<double> q = mk((double)v.x, (double)v.y);
      const bool slow = sizeof(T) == 8 || fabs((double)x.c.x) < (double)a->slow_tau;
      cplx<double> c = mk((double)x.c.x, (double)x.c.y), pk = mk((double)x.p.x, (double)x.p.y);
      if (sizeof(T) == 4 && slow) {
        c = coef64[(size_t)kx * a->nyh + (ky <= a->ny / 2 ? ky : a->ny - ky)];
        const cplx<float> l = nin_lo[i];
        pk.x += (double)l.x;
        pk.y += (double)l.y;
      }
      cplx<double> o = pk + c.x * pk + c.y * q;
      if (a->forcing) o = o + a->forcing[i];
      state_st<T>(nout, nout_lo, i, o, slow);
      v = mk((T)o.x, (T)o.y);
    } else if constexpr (MODE == kColInit) {
      if (a->dev_form && kx == 0 && ky == 0) v.x = T(0);
      state_st<T>(nout, nout_lo, i, mk((double)v.x, (double)v.y), true);   // lo = 0
    } else {
      double mn, mq;
      col_combine_factors(*a, kx, ky, mn, mq);
      const cplx<double> o = mn * state_ld<T>(nin, nin_lo, i, true) + mq * mk((double)v.x, (double)v.y);
      v = mk((T)o.x, (T)o.y);
    }
  }
  __device__ __forceinline__ void pair(int ky, int kyp, cplx<T>& v, cplx<T>& vp) const {
    const bool same = ky == kyp;
    const cplx<double> qk = mk((double)v.x, (double)v.y), qkp = mk((double)vp.x, (double)vp.y);
    const cplx<double> pk = state_ld<T>(nin, nin_lo, ky, true), pkp = state_ld<T>(nin, nin_lo, kyp, true);
    cplx<double> ok, okp;
    if constexpr (MODE == kColStep) {
      // the packed column holds kx = 0 (slow near ky = 0): always at full precision
      const int kh = ky <= kyp ? ky : kyp;
      bool s0, sm;
      const cplx<double> c0v = coef_ld<T>(coef, coef64, kh, a->slow_tau, true, s0);
      const cplx<double> cmv = coef_ld<T>(coef, coef64, (size_t)a->m * a->nyh + kh, a->slow_tau, true, sm);
      const cplx<double>*f0 = nullptr, *fm = nullptr;
      if (a->forcing) {
        f0 = a->forcing + ky;
        fm = a->forcing + (size_t)a->m * a->ny + ky;
      }
      packed_update(pk, pkp, qk, qkp, c0v, cmv, f0, fm, ok, okp);
      state_st<T>(nout, nout_lo, ky, ok, true);
      if (!same) state_st<T>(nout, nout_lo, kyp, okp, true);
    } else {
      double mn[2], mq[2];
      col_combine_factors(*a, 0, ky, mn[0], mq[0]);
      col_combine_factors(*a, a->m, ky, mn[1], mq[1]);
      cplx<double> h0, hm, g0, gm;
      unpack_pair(pk, pkp, h0, hm);
      unpack_pair(qk, qkp, g0, gm);
      const cplx<double> h0n = mn[0] * h0 + mq[0] * g0, hmn = mn[1] * hm + mq[1] * gm;
      ok = h0n + mul_i(hmn);
      okp = conj(h0n) + mul_i(conj(hmn));
    }
    v = mk((T)ok.x, (T)ok.y);
    if (!same) vp = mk((T)okp.x, (T)okp.y);
  }
};

// `cols` columns per CTA, two buffers of cols * ld values. Modes: step, init, combine.
template <class T, int MODE, int RSET>
__global__ void __launch_bounds__(256, 2) mixed_col_kernel(ColArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int ny = a.ny, m = a.m, ld = a.ld;
  const int c0 = blockIdx.x * a.cols, cols = min(a.cols, m - c0);
  cplx<T>* src = reinterpret_cast<cplx<T>*>(smem_raw);
  cplx<T>* dst = src + a.cols * ld;
  ColWork<T, MODE> w;
  w.a = &a;
  w.c0 = c0;
  w.coef = a.coef; w.coef64 = a.coef64;
  w.nin = a.nin; w.nin_lo = a.nin_lo; w.nout = a.nout; w.nout_lo = a.nout_lo;
  const cplx<T>* in = a.in;
  cplx<T>* wout = a.wout;
  if (a.batch) {
    const BatchBufs& bb = a.batch[blockIdx.y];
    in = static_cast<const cplx<T>*>(bb.v);
    wout = static_cast<cplx<T>*>(const_cast<void*>(bb.w));
    w.coef = static_cast<const cplx<T>*>(bb.coef);
    w.coef64 = static_cast<const cplx<double>*>(bb.coef64);
    w.nin = bb.nin; w.nout = bb.nout;
    w.nin_lo = static_cast<const cplx<float>*>(bb.nin_lo);
    w.nout_lo = static_cast<cplx<float>*>(bb.nout_lo);
  }
  const cplx<T>* in0 = in + (size_t)c0 * ny;
  cplx<T>* out0 = wout + (size_t)c0 * ny;
  const T s = (T)a.scale;
  auto ld_g = [&](int f, int i) { return in0[(size_t)f * ny + i]; };
  auto st_g = [&](int f, int i, cplx<T> v) { out0[(size_t)f * ny + i] = mk(s * v.x, s * v.y); };
  auto ld_s = [&](int f, int i) { return src[f * ld + generic_pad(i)]; };
  auto st_s = [&](int f, int i, cplx<T> v) { dst[f * ld + generic_pad(i)] = v; };
  auto flip = [&]() {
    __syncthreads();
    cplx<T>* t = src;
    src = dst;
    dst = t;
  };
  auto each = [&](auto f) {   // every element of the CTA's columns
    for (int i = threadIdx.x; i < cols * ny; i += blockDim.x) {
      const int c = i / ny;
      f(c, i - c * ny);
    }
  };
  const int np = a.fft.npass;

  if (MODE == kColCombine && a.combine == kCombineLocalN) {
    // nothing of V is needed: the filtered n_hat, then the inverse transform
    each([&](int c, int ky) {
      cplx<T> v = mk(T(0), T(0)), vp = v;
      if (c0 + c == 0) w.pair(ky, ky == 0 ? 0 : ny - ky, v, vp);
      else w.apply(c, ky, typename ColWork<T, MODE>::Aux{}, v);
      dst[c * ld + generic_pad(ky)] = v;
    });
    flip();
    for (int p = 0; p < np - 1; ++p) {
      mixed_pass<true, RSET, T>(a.fft, p, cols, a.tw, ld_s, st_s);
      flip();
    }
    mixed_pass<true, RSET, T>(a.fft, np - 1, cols, a.tw, ld_s, st_g);
    return;
  }
  if (MODE == kColStep) {
    // the columns' n_hat and coefficients set out for L2 while the forward transform runs
    // (whole 16-byte granules inside the arrays)
    const size_t se = sizeof(cplx<T>);
    const uintptr_t n0 = reinterpret_cast<uintptr_t>(w.nin) + (size_t)c0 * ny * se;
    const uintptr_t k0 = reinterpret_cast<uintptr_t>(w.coef + (size_t)c0 * a.nyh);
    const uintptr_t n1 = n0 + (size_t)cols * ny * se, k1 = k0 + (size_t)cols * a.nyh * sizeof(cplx<T>);
    const uintptr_t lim = ~(uintptr_t)15;
    const int half = blockDim.x >> 1;
    if ((int)threadIdx.x < half)
      l2_prefetch_range(reinterpret_cast<const void*>(n0 & lim), (unsigned)((n1 & lim) - (n0 & lim)), threadIdx.x, half);
    else
      l2_prefetch_range(reinterpret_cast<const void*>(k0 & lim), (unsigned)((k1 & lim) - (k0 & lim)),
                        threadIdx.x - half, blockDim.x - half);
  }
  if constexpr (MODE == kColStep && sizeof(T) == 8) {
    if (a.extv && a.extv->changed) {   // M or V changed: this CTA's coefficients and forcing
      const double M = a.extv->M;
      for (int c = 0; c < cols; ++c) extv_rebuild_column(*a.ec, M, c0 + c);
      if (c0 == 0) extv_rebuild_column(*a.ec, M, m);
      __syncthreads();
    }
  }
  // The CTA with the packed column, whose update pairs ky with ny - ky, parks its spectra in
  // shared memory between the two transforms; the others update in the middle pass.
  const bool packed = MODE != kColInit && c0 == 0;
  int p = 0;
  if (np == 1) {
    each([&](int c, int ky) { dst[c * ld + generic_pad(ky)] = ld_g(c, ky); });
  } else {
    mixed_pass<false, RSET, T>(a.fft, 0, cols, a.tw, ld_g, st_s);
    p = 1;
  }
  flip();
  for (; p < (packed ? np : np - 1); ++p) {
    mixed_pass<false, RSET, T>(a.fft, p, cols, a.tw, ld_s, st_s);
    flip();
  }
  p = 0;
  if (packed) {
    for (int i = threadIdx.x; i < cols * ny; i += blockDim.x) {
      const int c = i / ny, ky = i - c * ny, kyp = ky == 0 ? 0 : ny - ky;
      cplx<T>& v = src[c * ld + generic_pad(ky)];
      if (c > 0) w.apply(c, ky, w.load(c, ky), v);
      else if (ky <= kyp) w.pair(ky, kyp, v, src[generic_pad(kyp)]);
    }
    __syncthreads();
  } else {
    mixed_switch<RSET, T>(a.fft.radix[np - 1], [&](auto r) {
      mixed_mid_items<decltype(r)::value, false, T>(a.fft, 0, cols, a.tw, ld_s, w, st_s);
    });
    flip();
    p = 1;
  }
  for (; p < np - 1; ++p) {
    mixed_pass<true, RSET, T>(a.fft_b, p, cols, a.tw, ld_s, st_s);
    flip();
  }
  if (p < np) mixed_pass<true, RSET, T>(a.fft_b, np - 1, cols, a.tw, ld_s, st_g);
  else each([&](int c, int ky) { st_g(c, ky, ld_s(c, ky)); });
}

}  // namespace pfc
