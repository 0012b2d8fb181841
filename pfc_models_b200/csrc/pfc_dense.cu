// Whole-grid step kernel for the smallest FP64 mixed-radix cells: the step of pfc_onecta.cuh (one
// CTA per plan, `nsteps` steps a launch) with every transform as a small FP64 matrix product on
// the tensor cores (mma.sync m8n8k4). At these lengths the chain of FFT phases, not its
// arithmetic, is the step: the FFT passes run 12 % of the issue slots, waiting at barriers for
// the few threads with a butterfly and on instruction fetch of the unrolled butterflies. A
// product deals the work to all warps evenly, in a few instructions, and needs no packing
// twiddles. Folding halves each side of it: with e = x[i] + x[n - i] and o = x[i] - x[n - i] a
// real sequence transforms by a cosine and a sine matrix of n / 2 + 1 rows and columns,
//   X[k] = sum_i w_i (e_i cos(2 pi i k / n) - i o_i sin(2 pi i k / n)), X[n - k] its mirror,
// w = 1/2 where i is its own mirror (e counts it twice), so one warp tile yields both k and
// n - k, which the next fold and the packed column's update pair up in its registers. Four
// phases a step, each a product and its pointwise work, with a barrier between:
//   1  n(x), N(n), fold over x        2  row spectra V
//   3  fold over y, N_hat, the ETD1 update, fold over ky        4  W
// A fragment entry (out, in) is read as A[out][in] by the column products (out = rows of the
// tile) and as B[in][out] by the row products: the lane layouts of A (row lane / 4, column
// lane % 4) and B (row lane % 4, column lane / 4) make the two the same table.
// A sum of n / 2 terms in a chain rounds more than an FFT's log n levels, most of all by the mean
// density, which every partial sum would carry. So the step transforms n - nbar and N - N(nbar),
// the mean being constant: its error against 80-bit values, pooled over 11 sizes and both models
// after 1 and 10 steps, is 0.92 times that of the FFT passes (1.14 with the mean; two chains a sum
// beside it would give 0.90, and 3 % more time).
// A 28 x 24 step needs 224 products, 900 cycles of an SM's FP64 rate (one m8n8k4 per 16 cycles
// and scheduler); it takes 4000 (5600 with the log model's logarithms), bound by the
// instruction chain of its four phases: 2.1 us std, 2.9 us log, where the FFT passes take
// 6.0 and 6.7. tcgen05 has no FP64 form, so this is the FP64 tensor path of the chip.
// A translation unit of its own: the driver loads a unit's code as one, at its first kernel's first
// use, and a large unit slowly (24 ms of a process's first 28 x 24 plan with pfc_onecta.cuh's kernels).
#include <algorithm>
#include <cmath>

#include "pfc_mixed.cuh"
#include "pfc_registry.h"

namespace pfc {

namespace {

__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c0), "+d"(c1) : "d"(a), "d"(b));
}

template <int MODEL>
__global__ void __launch_bounds__(kOneCtaMaxThreads, 2) onecta_dense_kernel(DenseArgs a, const BatchBufs* table,
                                                                            long long nsteps) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int m = a.m, ny = a.ny, ys = a.ys, ks = a.ks, h = ny / 2;
  const int nrow = a.tr * a.kr * 32, ncol = a.tc * a.kc * 32;
  double2* rtab = reinterpret_cast<double2*>(smem_raw);
  double2* ctab = rtab + nrow;
  double2* S = ctab + ncol;                                 // n_hat, packed [kx][ky]
  double* areaA = reinterpret_cast<double*>(S + m * ny);
  double* areaB = areaA + a.size_a;
  // area A: 2 Re W and 2 Im W [k][y] (k <= m, the packed column's parts at 0 and m) in phases
  // 4 to 1, the real sequences of V [c][y] (c = 2 k + part) in phases 2 to 3
  double *wre = areaA, *wim = areaA + 4 * a.kr * ys, *rv = areaA;
  // area B: the folded N [x][y] in phases 1 to 2, the folded new spectrum [c][ky] in 3 to 4
  double *ne = areaB, *no = areaB + 4 * a.kr * ys, *xe = areaB, *xo = areaB + a.cpad * ks;
  const BatchBufs& bb = table[blockIdx.x];
  double2* W = static_cast<double2*>(const_cast<void*>(bb.w));
  double* V = static_cast<double*>(bb.v);
  double2* P[2] = {static_cast<double2*>(const_cast<void*>(bb.nin)), static_cast<double2*>(bb.nout)};
  const double2* coef = static_cast<const double2*>(bb.coef);
  const int tid = threadIdx.x, nth = blockDim.x, warp = tid >> 5, lane = tid & 31, nwarp = nth >> 5;
  const int lr = lane >> 2, lc = lane & 3;
  const double s2 = 2.0 * a.scale;
  // the mean density, which every step keeps (the k = 0 mode's coefficients are zero), and its N
  const double nbar = a.scale * P[0][0].x, nref = nonlin_plain<MODEL>(nbar, a.g, a.clamp, a.min_phi, a.min_log);

  // (the areas' padding is only ever multiplied by zero entries of the tables: any finite value)
  for (int i = tid; i < a.size_a + a.size_b; i += nth) areaA[i] = 0.0;
  for (int i = tid; i < nrow; i += nth) rtab[i] = a.row_tab[i];
  for (int i = tid; i < ncol; i += nth) ctab[i] = a.col_tab[i];
  __syncthreads();
  for (int i = tid; i < m * ny; i += nth) {
    const int k = i / ny, y = i - k * ny;
    const double2 w = W[i];
    S[i] = P[0][i];
    if (k == 0) {
      wre[y] = 2.0 * (w.x - nbar);
      wre[m * ys + y] = 2.0 * w.y;
    } else {
      wre[k * ys + y] = 2.0 * w.x;
      wim[k * ys + y] = 2.0 * w.y;
    }
  }
  __syncthreads();

  // tiles are dealt to the warps in turn: (slow, fast) tile indices of a warp's first tile, and
  // the stride to its next (no division inside the steps)
  const int ty = (ny + 7) >> 3, tcols = a.cpad >> 3;
  const int ry0 = warp / a.tr, rx0 = warp % a.tr, rdy = nwarp / a.tr, rdx = nwarp % a.tr;
  const int cc0 = warp / a.tc, ck0 = warp % a.tc, cdc = nwarp / a.tc, cdk = nwarp % a.tc;
  auto row_tiles = [&](auto f) {
    for (int i = ry0, x = rx0; i < ty;) {
      f(8 * i, x);
      i += rdy;
      x += rdx;
      if (x >= a.tr) { x -= a.tr; ++i; }
    }
  };
  auto col_tiles = [&](auto f) {
    for (int i = cc0, k = ck0; i < tcols;) {
      f(8 * i, k);
      i += cdc;
      k += cdk;
      if (k >= a.tc) { k -= a.tc; ++i; }
    }
  };
  for (long long step = 0; step < nsteps; ++step) {
    const bool last = step == nsteps - 1;
    // ---- 1: n - nbar = C - S at x, C + S at nx - x; N - nref of both; folded over x
    row_tiles([&](int y, int tx) {
      double c0 = 0.0, c1 = 0.0, s0 = 0.0, s1 = 0.0;
      const double *pr = wre + lc * ys + y + lr, *pi = wim + lc * ys + y + lr;
      const double2* f = rtab + (tx * a.kr) * 32 + lane;
#pragma unroll 4
      for (int q = 0; q < a.kr; ++q) {
        const double2 w = f[q * 32];
        dmma(c0, c1, pr[4 * q * ys], w.x);
        dmma(s0, s1, pi[4 * q * ys], w.y);
      }
      const double p0 = nonlin_plain<MODEL>(nbar + (c0 - s0), a.g, a.clamp, a.min_phi, a.min_log) - nref;
      const double q0 = nonlin_plain<MODEL>(nbar + (c0 + s0), a.g, a.clamp, a.min_phi, a.min_log) - nref;
      const double p1 = nonlin_plain<MODEL>(nbar + (c1 - s1), a.g, a.clamp, a.min_phi, a.min_log) - nref;
      const double q1 = nonlin_plain<MODEL>(nbar + (c1 + s1), a.g, a.clamp, a.min_phi, a.min_log) - nref;
      const int x = tx * 8 + 2 * lc, yy = y + lr;
      if (yy < ny) {
        if (x <= m) {
          ne[x * ys + yy] = p0 + q0;
          no[x * ys + yy] = p0 - q0;
        }
        if (x + 1 <= m) {
          ne[(x + 1) * ys + yy] = p1 + q1;
          no[(x + 1) * ys + yy] = p1 - q1;
        }
      }
    });
    __syncthreads();
    // ---- 2: V[k] = C - i S (of N - nref: V[0] lacks nx nref)
    row_tiles([&](int y, int tx) {
      double c0 = 0.0, c1 = 0.0, s0 = 0.0, s1 = 0.0;
      const double *pe = ne + lc * ys + y + lr, *po = no + lc * ys + y + lr;
      const double2* f = rtab + (tx * a.kr) * 32 + lane;
#pragma unroll 4
      for (int q = 0; q < a.kr; ++q) {
        const double2 w = f[q * 32];
        dmma(c0, c1, pe[4 * q * ys], w.x);
        dmma(s0, s1, po[4 * q * ys], w.y);
      }
      const int yy = y + lr;
      auto put = [&](int k, double re, double im) {
        if (yy >= ny || k > m) return;
        if (k == 0 || k == m) {
          rv[(k == 0 ? 0 : ys) + yy] = re;
          if (last) V[2 * yy + (k == 0 ? 0 : 1)] = k == 0 ? re + 2.0 * m * nref : re;
        } else {
          rv[2 * k * ys + yy] = re;
          rv[(2 * k + 1) * ys + yy] = im;
          if (last) reinterpret_cast<double2*>(V)[k * ny + yy] = make_double2(re, im);
        }
      };
      put(tx * 8 + 2 * lc, c0, -s0);
      put(tx * 8 + 2 * lc + 1, c1, -s1);
    });
    __syncthreads();
    // ---- 3: N_hat at ky and ny - ky, the update of both, folded over ky
    double2* p_old = P[step & 1];
    double2* p_new = P[(step + 1) & 1];
    col_tiles([&](int c, int tk) {
      const int ky = tk * 8 + lr, k = (c >> 1) + lc;
      const bool on = ky <= h && k < m;
      const int kyp = ky == 0 ? 0 : ny - ky;
      double2 cf = make_double2(0.0, 0.0), cm = cf, u = cf, v = cf;
      if (on) {
        cf = coef[k * a.nyh + ky];
        if (k == 0) cm = coef[m * a.nyh + ky];
        u = S[k * ny + ky];
        v = S[k * ny + kyp];
      }
      double p0 = 0.0, p1 = 0.0, q0 = 0.0, q1 = 0.0;
      const double2* f = ctab + (tk * a.kc) * 32 + lane;
      const double* col = rv + (c + lr) * ys;
#pragma unroll 4
      for (int q = 0; q < a.kc; ++q) {
        const int i = min(4 * q + lc, h);
        const double x = col[i], y = col[i == 0 ? 0 : ny - i];
        const double2 w = f[q * 32];
        dmma(p0, p1, w.x, x + y);
        dmma(q0, q1, w.y, x - y);
      }
      if (on) {
        const cplx<double> n0 = mk(p0 + q1, p1 - q0), n1 = mk(p0 - q1, p1 + q0);
        const cplx<double> pk = mk(u.x, u.y), pkp = mk(v.x, v.y);
        cplx<double> ok, okp;
        if (k == 0) {
          packed_update(pk, pkp, n0, n1, mk(cf.x, cf.y), mk(cm.x, cm.y), nullptr, nullptr, ok, okp);
        } else {
          ok = pk + cf.x * pk + cf.y * n0;
          okp = pkp + cf.x * pkp + cf.y * n1;
        }
        if (kyp == ky) okp = ok;
        const double2 o = make_double2(ok.x, ok.y), op = make_double2(okp.x, okp.y);
        S[k * ny + ky] = o;
        S[k * ny + kyp] = op;
        if (last) {
          p_old[k * ny + ky] = u;
          p_old[k * ny + kyp] = v;
          p_new[k * ny + ky] = o;
          p_new[k * ny + kyp] = op;
        }
        xe[2 * k * ks + ky] = k == 0 && ky == 0 ? 0.0 : ok.x + okp.x;   // (without the mean)
        xe[(2 * k + 1) * ks + ky] = ok.y + okp.y;
        xo[2 * k * ks + ky] = ok.x - okp.x;
        xo[(2 * k + 1) * ks + ky] = ok.y - okp.y;
      }
    });
    __syncthreads();
    // ---- 4: W at y and ny - y
    col_tiles([&](int c, int tk) {
      double p0 = 0.0, p1 = 0.0, q0 = 0.0, q1 = 0.0;
      const double2* f = ctab + (tk * a.kc) * 32 + lane;
      const double *pe = xe + (c + lr) * ks + lc, *po = xo + (c + lr) * ks + lc;
#pragma unroll 4
      for (int q = 0; q < a.kc; ++q) {
        const double2 w = f[q * 32];
        dmma(p0, p1, w.x, pe[4 * q]);
        dmma(q0, q1, w.y, po[4 * q]);
      }
      const int y = tk * 8 + lr, k = (c >> 1) + lc;
      if (y <= h && k < m) {
        // (column 0 is rounded with the mean, as it is kept in memory: where a launch ends is no
        // matter then)
        auto put = [&](int yy, double re, double im) {
          double w = a.scale * re;
          if (k == 0) {
            w += nbar;
            wre[yy] = 2.0 * (w - nbar);
            wre[m * ys + yy] = s2 * im;
          } else {
            wre[k * ys + yy] = s2 * re;
            wim[k * ys + yy] = s2 * im;
          }
          if (last) W[k * ny + yy] = make_double2(w, a.scale * im);
        };
        put(y, p0 - q1, p1 + q0);
        if (y != 0 && ny - y != y) put(ny - y, p0 + q1, p1 - q0);
      }
    });
    __syncthreads();
  }
}

}  // namespace

size_t dense_shape(int m, int ny, DenseArgs& a) {
  a.m = m; a.ny = ny; a.nyh = ny / 2 + 1;
  a.tr = m / 8 + 1; a.kr = m / 4 + 1;             // m + 1 outputs and inputs
  a.tc = ny / 2 / 8 + 1; a.kc = ny / 2 / 4 + 1;   // ny / 2 + 1
  // strides of 4 (mod 8) doubles: the fragment loads of a half warp (4 x 4 values) fall on
  // different banks
  auto stride = [](int n) { while (n % 8 != 4) ++n; return n; };
  a.ys = stride((ny + 7) / 8 * 8);
  a.ks = stride(4 * a.kc);
  a.cpad = (2 * m + 7) / 8 * 8;
  a.size_a = std::max(8 * a.kr, a.cpad) * a.ys;
  a.size_b = std::max(8 * a.kr * a.ys, 2 * a.cpad * a.ks);
  return 16 * ((size_t)32 * (a.tr * a.kr + a.tc * a.kc) + (size_t)m * ny) + 8 * (size_t)(a.size_a + a.size_b);
}

int dense_products(const DenseArgs& a) {
  return 4 * ((a.ny + 7) / 8 * a.tr * a.kr + a.cpad / 8 * a.tc * a.kc);
}

void dense_table(int n, const std::vector<long double>& root, std::vector<long double>& tw) {
  const int h = n / 2, tiles = h / 8 + 1, steps = h / 4 + 1;
  for (int t = 0; t < tiles; ++t)
    for (int q = 0; q < steps; ++q)
      for (int lane = 0; lane < 32; ++lane) {
        const int out = 8 * t + lane / 4, in = 4 * q + lane % 4;
        long double c = 0, s = 0;
        if (out <= h && in <= h) {
          const int k = out * in % n;
          const long double w = (in == 0 || 2 * in == n) ? 0.5L : 1.0L;
          c = w * root[2 * k];
          s = 2 * k % n == 0 ? 0.0L : -w * root[2 * k + 1];
        }
        tw.push_back(c);
        tw.push_back(s);
      }
}

cudaError_t dense_allow_smem(size_t bytes) {
  for (void* fn : {(void*)onecta_dense_kernel<kModelStd>, (void*)onecta_dense_kernel<kModelLog>}) {
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_dense_step(const DenseArgs& args, const BatchBufs* table, int count, long long nsteps, int model,
                              size_t smem, cudaStream_t stream) {
  void* fn = model == kModelLog ? (void*)onecta_dense_kernel<kModelLog> : (void*)onecta_dense_kernel<kModelStd>;
  DenseArgs a = args;
  void* p[] = {(void*)&a, (void*)&table, (void*)&nsteps};
  return cudaLaunchKernel(fn, dim3(count), dim3(kOneCtaMaxThreads), p, smem, stream);
}

}  // namespace pfc
