// Whole-grid step kernel for small FP64 mixed-radix plans (the phase-diagram cells,
// e.g. 28 x 24 or 32 x 56 sites).
//
// On such grids the two-kernel step (row pass, column pass) is bound by launch and
// barrier latency, not by HBM: a 28 x 24 step takes about 20 us while it moves 20 KB. Here
// one CTA holds one plan's whole grid in shared memory (the row buffers, the column
// buffers and the spectral state) and runs `nsteps` steps in a loop, so a block of steps
// is one launch; a batch of plans is one launch with one CTA per plan.
//
// Small cells run the transforms as matrix products (pfc_dense.cu). The others
// run the passes of mixed_row_kernel<kRowStep> followed by those of
// mixed_col_kernel<kColStep> (pfc_mixed.cuh) with the same arithmetic, every butterfly of all
// rows (or columns) dealt to the CTA's threads. What bounds a step is the chain of its phases,
// each a shared-memory read, a short dependent FP64 DFT and a barrier, so here the
// real-packing twiddles too are applied where the next phase reads: a cell whose sides need
// two passes each takes 6 phases and barriers a step (16 before), 28 x 24 log cells
// 8.0 -> 6.4 us a step. On the last step of a launch the kernel leaves in global memory what
// the two-kernel step leaves: V (the nonlinear spectrum of the state the step started
// from), that state, the new state and W (the new state's inverse column transforms).
#pragma once
#include "pfc_mixed.cuh"
#include "pfc_registry.h"

namespace pfc {

// MINB 1: all registers for one CTA per SM (single plans, small batches); MINB 2: two
// CTAs per SM (batches with more plans than SMs).
template <int MODEL, int RSET, int MINB>
__global__ void __launch_bounds__(kOneCtaMaxThreads, MINB) onecta_step_kernel(RowArgs<double> ra, ColArgs<double> ca,
                                                                         const BatchBufs* table, long long nsteps) {
  using T = double;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int m = ra.m, ny = ra.ny, ldr = ra.ld, ldc = ca.ld, nyh = ca.nyh;
  const int spec = m * ny, half = max(ny * ldr, m * ldc);
  cplx<T>* src = reinterpret_cast<cplx<T>*>(smem_raw);   // ny row buffers of ldr, or m column buffers of ldc
  cplx<T>* dst = src + half;
  cplx<T>* S = dst + half;                               // n_hat, packed [kx][y]
  const BatchBufs& bb = table[blockIdx.x];
  cplx<T>* W = static_cast<cplx<T>*>(const_cast<void*>(bb.w));
  cplx<T>* V = static_cast<cplx<T>*>(bb.v);
  cplx<T>* P[2] = {static_cast<cplx<T>*>(const_cast<void*>(bb.nin)), static_cast<cplx<T>*>(bb.nout)};
  const cplx<T>* coef = static_cast<const cplx<T>*>(bb.coef);
  const int tid = threadIdx.x, nth = blockDim.x;

  for (int i = tid; i < spec; i += nth) {
    const int kx = i / ny, y = i - kx * ny;
    src[kx * ldc + generic_pad(y)] = W[i];
    S[i] = P[0][i];
  }
  __syncthreads();
  const T s = (T)ca.scale;
  const FftDesc &ra_a = ra.fft, &ra_b = ra.fft_b, &ca_a = ca.fft, &ca_b = ca.fft_b;
  const int npr = ra_a.npass, npc = ca_a.npass;

  auto ld_r = [&](int f, int i) { return src[f * ldr + generic_pad(i)]; };
  auto st_r = [&](int f, int i, cplx<T> v) { dst[f * ldr + generic_pad(i)] = v; };
  auto ld_c = [&](int f, int i) { return src[f * ldc + generic_pad(i)]; };
  auto st_c = [&](int f, int i, cplx<T> v) { dst[f * ldc + generic_pad(i)] = v; };
  auto flip = [&]() {
    __syncthreads();
    cplx<T>* t = src;
    src = dst;
    dst = t;
  };
  // row y's element k of the inverse transform's input, from the columns of W
  auto ld_pre = [&](int y, int k) {
    if (k == 0) return real_dc(src[generic_pad(y)]);
    const int kk = min(k, m - k);
    cplx<T> zk, zm;
    real_pre(src[kk * ldc + generic_pad(y)], src[(m - kk) * ldc + generic_pad(y)], ra.rtw[kk], zk, zm);
    return k == kk ? zk : zm;
  };

  for (long long step = 0; step < nsteps; ++step) {
    const bool last = step == nsteps - 1;
    // ---- row pass
    if (npr == 1) {
      for (int i = tid; i < spec; i += nth) {
        const int y = i / m, k = i - y * m;
        st_r(y, k, ld_pre(y, k));
      }
      flip();
    } else {
      mixed_pass<true, RSET, T>(ra_a, 0, ny, ra.tw, ld_pre, st_r);
      flip();
      for (int p = 1; p < npr - 1; ++p) {
        mixed_pass<true, RSET, T>(ra_a, p, ny, ra.tw, ld_r, st_r);
        flip();
      }
    }
    struct Nonlin {
      struct Aux {};
      const RowArgs<double>* a;
      __device__ __forceinline__ Aux load(int, int) const { return Aux{}; }
      __device__ __forceinline__ void apply(int, int, Aux, cplx<T>& z) const {
        z = mk((T)nonlin_plain<MODEL>((double)z.x, a->g, a->clamp, a->min_phi, a->min_log),
               (T)nonlin_plain<MODEL>((double)z.y, a->g, a->clamp, a->min_phi, a->min_log));
      }
    } fn{&ra};
    mixed_switch<RSET, T>(ra_a.radix[npr - 1], [&](auto r) {
      mixed_mid_items<decltype(r)::value, true, T>(ra_a, 0, ny, ra.tw, ld_r, fn, st_r);
    });
    flip();
    for (int p = 1; p < npr; ++p) {
      mixed_pass<false, RSET, T>(ra_b, p, ny, ra.tw, ld_r, st_r);
      flip();
    }
    // ---- column pass: V[kx][y] from the rows' transforms
    auto ld_post = [&](int kx, int y) {
      const cplx<T>* row = src + y * ldr;
      cplx<T> v;
      if (kx == 0) {
        v = real_dc(row[0]);
      } else {
        const int kk = min(kx, m - kx);
        cplx<T> yk, ym;
        real_post(row[generic_pad(kk)], row[generic_pad(m - kk)], ra.rtw[kk], yk, ym);
        v = kx == kk ? yk : ym;
      }
      if (last) V[kx * ny + y] = v;
      return v;
    };
    if (npc == 1) {
      for (int i = tid; i < spec; i += nth) {
        const int kx = i / ny, y = i - kx * ny;
        st_c(kx, y, ld_post(kx, y));
      }
      flip();
    } else {
      mixed_pass<false, RSET, T>(ca_a, 0, m, ca.tw, ld_post, st_c);
      flip();
      for (int p = 1; p < npc - 1; ++p) {
        mixed_pass<false, RSET, T>(ca_a, p, m, ca.tw, ld_c, st_c);
        flip();
      }
    }
    // the last step leaves the state it starts from and the new one in global memory
    cplx<T>* p_old = last ? P[step & 1] : nullptr;
    cplx<T>* p_new = P[(step + 1) & 1];
    struct Update {
      struct Aux {
        cplx<T> c, p;
      };
      const cplx<T>* coef;
      cplx<T> *S, *p_old, *p_new;
      int ny, nyh;
      __device__ __forceinline__ Aux load(int kx, int ky) const {
        return Aux{coef[kx * nyh + (ky <= ny / 2 ? ky : ny - ky)], S[kx * ny + ky]};
      }
      __device__ __forceinline__ void put(int i, cplx<T> was, cplx<T> now) const {
        S[i] = now;
        if (p_old) {
          p_old[i] = was;
          p_new[i] = now;
        }
      }
      __device__ __forceinline__ void apply(int kx, int ky, const Aux& x, cplx<T>& v) const {
        const cplx<double> o = x.p + x.c.x * x.p + x.c.y * v;
        put(kx * ny + ky, x.p, o);
        v = o;
      }
    } up{coef, S, p_old, p_new, ny, nyh};
    mixed_switch<RSET, T>(ca_a.radix[npc - 1], [&](auto r) {
      constexpr int R = decltype(r)::value;
      mixed_mid_items<R, false, T>(ca_a, 1, m, ca.tw, ld_c, up, st_c);
      mixed_mid_paired<R, false, T>(ca_a, ca.tw, ld_c, [&](int ky, int kyp, cplx<T>& v, cplx<T>& vp) {
        const int kh = min(ky, kyp);
        const cplx<T> pk = S[ky], pkp = S[kyp];
        cplx<T> ok, okp;
        packed_update(pk, pkp, v, vp, coef[kh], coef[m * nyh + kh], nullptr, nullptr, ok, okp);
        up.put(ky, pk, ok);
        v = ok;
        if (kyp != ky) {
          up.put(kyp, pkp, okp);
          vp = okp;
        }
      }, st_c);
    });
    flip();
    // ---- inverse columns: W
    auto st_w = [&](int kx, int y, cplx<T> v) {
      const cplx<T> w = mk(s * v.x, s * v.y);
      dst[kx * ldc + generic_pad(y)] = w;
      if (last) W[kx * ny + y] = w;
    };
    if (npc == 1) {
      for (int i = tid; i < spec; i += nth) {
        const int kx = i / ny, y = i - kx * ny;
        st_w(kx, y, ld_c(kx, y));
      }
    } else {
      for (int p = 1; p < npc - 1; ++p) {
        mixed_pass<true, RSET, T>(ca_b, p, m, ca.tw, ld_c, st_c);
        flip();
      }
      mixed_pass<true, RSET, T>(ca_b, npc - 1, m, ca.tw, ld_c, st_w);
    }
    flip();
  }
}

}  // namespace pfc
