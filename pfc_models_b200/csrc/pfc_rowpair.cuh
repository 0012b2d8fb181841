// Row step kernels with paired butterflies for power-of-two rows.
//
// The same pass as row_step_fast (pfc_fast.cuh: packed inverse real transform of W, the
// nonlinearity, forward real transform to V, M = nx / 2 complex points a row), without the
// shared-memory phases around the transforms. There, a tile is staged through shared memory
// and the real-packing twiddles, which combine elements k and M - k, are applied in place
// before and after: 6 of the 10 (two Stockham passes) or 14 (three) shared-memory accesses per
// value, and what bounds the kernel is that L1 / shared-memory pipe (FP64 2048^2: 80 % of its
// throughput; FP32 8192^2: 73 % of its wavefronts). Here
//  * the first pass (and the last) has radix EE / 2, and a thread runs butterflies j and
//    NR - j of the NR = 2 M / EE: together they hold both elements of every pair (k, M - k),
//    so the real-packing twiddles are register arithmetic;
//  * the lanes run over the tile's rows first, so a pass's elements of ROWS rows are ROWS
//    consecutive values of the column-major W: the first pass reads global memory and the
//    last writes it directly, in runs of ROWS values (64 bytes).
// What is left is one shared-memory store and load per exchange between passes (8 accesses a
// value for three passes). B200, one-lane kernel (at 4096 and 8192 the two-lane packed one with
// the TMA tile) against this, us per row pass with its events: 2048^2 FP64 39.1 -> 31.1, FP32
// 20.9 -> 18.9; 8192^2 FP64 714 -> 596, FP32 322 -> 282; 4096^2 FP64 152 -> 122, FP32 79 -> 62;
// 1024^2 log FP64 19.2 -> 16.7; whole steps beside the launch rule in pfc_plan.cu.
//
// Exchange buffer: entry (idx, r) at pad(idx) * ROWS + r, pad(i) = i + (i >> a) + (i >> b) for
// the radices 2^a and 2^b of the first and the last pass of the sequence (one term when they
// are equal): a pass writing with stride 1, 2^a or 2^b over the lanes then puts the two 64-byte
// runs that a half warp (8-byte values; a quarter warp for 16-byte ones) serves at once on
// different halves of the banks. All index parts are disjoint bit fields, and pad adds over
// those, so every access is one run-time base plus compile-time offsets.
#pragma once
#include "pfc_fast.cuh"

namespace pfc {

// Radices of an N-point transform with EE values per thread: EE / 2, then the rest of N in as
// few passes of at most EE as it takes, split evenly. Sequence B runs them in reverse.
template <int N, int EE>
struct PairSeq {
  __host__ __device__ static constexpr int lg(int x) { return x <= 1 ? 0 : 1 + lg(x >> 1); }
  static constexpr int R0 = EE / 2, REST = lg(N / R0), LE = lg(EE);
  static constexpr int NREST = (REST + LE - 1) / LE, NP = 1 + NREST;
  __host__ __device__ static constexpr int radA(int p) {
    return p == 0 ? R0 : 1 << (REST / NREST + (p - 1 < REST % NREST ? 1 : 0));
  }
  __host__ __device__ static constexpr int radB(int p) { return radA(NP - 1 - p); }
  __host__ __device__ static constexpr int rad(bool b, int p) { return b ? radB(p) : radA(p); }
  __host__ __device__ static constexpr int ns(bool b, int p) { return p == 0 ? 1 : ns(b, p - 1) * rad(b, p - 1); }
  // offset of pass p's twiddle table ([q - 1][k], q < R, k < ns) within the sequence's
  __host__ __device__ static constexpr int tw(bool b, int p) {
    return p <= 1 ? 0 : tw(b, p - 1) + ns(b, p - 1) * (rad(b, p - 1) - 1);
  }
  static constexpr int TPF = N / EE, LAST = radA(NP - 1);
  static constexpr int A = lg(R0), B = lg(LAST);
  __host__ __device__ static constexpr int pad(int i) { return i + (i >> A) + (A != B ? (i >> B) : 0); }
  static constexpr int SLOTS = pad(N - 1) + 1;
};

// registers: 64 a thread where they hold the values beside the arithmetic, else 128
template <class T, int EE, int THREADS> struct PairMinBlocks {
  static constexpr int regs = 2 * EE * (int)(sizeof(T) / 4) <= 32 ? 64 : 128;
  static constexpr int value = 65536 / (THREADS * regs) > 0 ? 65536 / (THREADS * regs) : 1;
};

template <class T, int N, int EE, int ROWS, bool SEQB, int PASS>
struct PairPass {
  using S = PairSeq<N, EE>;
  static constexpr int R = S::rad(SEQB, PASS), NS = S::ns(SEQB, PASS), NR = N / R, NB = EE / R;
  static __device__ __forceinline__ void load(const cplx<T>* buf, cplx<T>* v, int t) {
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      const cplx<T>* p = buf + S::pad(t + b * S::TPF) * ROWS;
#pragma unroll
      for (int q = 0; q < R; ++q) v[b * R + q] = p[S::pad(q * NR) * ROWS];
    }
  }
  static __device__ __forceinline__ void store(cplx<T>* buf, const cplx<T>* v, int t) {
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      const int j = t + b * S::TPF, k = j & (NS - 1);
      cplx<T>* p = buf + (S::pad((j - k) * R) + S::pad(k)) * ROWS;
#pragma unroll
      for (int q = 0; q < R; ++q) p[S::pad(q * NS) * ROWS] = v[b * R + q];
    }
  }
  // one butterfly (index j): twiddles and DFT
  template <bool INV>
  static __device__ __forceinline__ void butterfly(cplx<T>* v, int j, const cplx<T>* __restrict__ tw) {
    if constexpr (NS > 1) {
      const cplx<T>* w = tw + S::tw(SEQB, PASS) + (j & (NS - 1));
      cplx<T> wq[R];
#pragma unroll
      for (int q = 1; q < R; ++q) wq[q] = ldkc(w + (q - 1) * NS);
#pragma unroll
      for (int q = 1; q < R; ++q) {
        cplx<T> x = wq[q];
        if (INV) x.y = -x.y;
        v[q] = cmul(v[q], x);
      }
    }
    dft_c<R, INV>(v);
  }
  template <bool INV>
  static __device__ __forceinline__ void compute(cplx<T>* v, int t, const cplx<T>* __restrict__ tw) {
#pragma unroll
    for (int b = 0; b < NB; ++b) butterfly<INV>(v + b * R, t + b * S::TPF, tw);
  }
};

// Barrier of the THREADS threads that run the body: the whole CTA in the step kernel, the first
// ones (whole warps) of a work-queue CTA, on the named barrier of body_sync.
template <int THREADS, bool QUEUE>
__device__ __forceinline__ void pair_sync() {
  if constexpr (QUEUE) asm volatile("bar.sync 15, %0;" ::"n"(THREADS) : "memory");
  else __syncthreads();
}

// Passes [PA, PB) of a sequence in place through buf.
template <class T, int N, int EE, int ROWS, bool SEQB, bool INV, bool QUEUE, int PA, int PB>
__device__ __forceinline__ void pair_mid(cplx<T>* buf, cplx<T>* v, int t, const cplx<T>* __restrict__ tw) {
  if constexpr (PA < PB) {
    using P = PairPass<T, N, EE, ROWS, SEQB, PA>;
    P::load(buf, v, t);
    pair_sync<ROWS * (N / EE), QUEUE>();
    P::template compute<INV>(v, t, tw);
    P::store(buf, v, t);
    pair_sync<ROWS * (N / EE), QUEUE>();
    pair_mid<T, N, EE, ROWS, SEQB, INV, QUEUE, PA + 1, PB>(buf, v, t, tw);
  }
}

// f(a, b, k) on every pair of elements k (in a) and M - k (in b) that a thread's two
// butterflies hold, va of index t, vb of NR - t (t = 0: 0 and NR / 2, each its own mirror);
// dc(a) on element 0 and mid(a) on element M / 2, which pair with themselves.
template <int R, int NR, class T, class F, class Dc, class Mid>
__device__ __forceinline__ void pair_elements(cplx<T>* va, cplx<T>* vb, int t, F f, Dc dc, Mid mid) {
  if (t != 0) {
#pragma unroll
    for (int q = 0; q < R; ++q) f(va[q], vb[R - 1 - q], t + q * NR);
  } else {
    dc(va[0]);
#pragma unroll
    for (int q = 1; q < R / 2; ++q) f(va[q], va[R - q], q * NR);
    mid(va[R / 2]);
#pragma unroll
    for (int q = 0; q < R / 2; ++q) f(vb[q], vb[R - 1 - q], NR / 2 + q * NR);
  }
}

template <class T, int M, int EE, int ROWS, int MODEL>
__global__ void __launch_bounds__(ROWS * (M / EE), PairMinBlocks<T, EE, ROWS * (M / EE)>::value)
row_step_pair(FastRowArgs<T> a) {
  constexpr bool QUEUE = false;
  const BatchBufs* batch = a.batch;
  const unsigned tile = blockIdx.x, member = blockIdx.y;
  const PdlSync sync;
#include "pfc_rowpair_body.cuh"
}

// Row tile `tile` of member `member` on the first ROWS * M / EE threads of a work-queue CTA, other
// CTAs of whose launch write W.
template <class T, int M, int EE, int ROWS, int MODEL>
__device__ __forceinline__ void row_pair_queue(const FastRowArgs<T>& a, const BatchBufs* batch, unsigned tile,
                                               unsigned member) {
  constexpr bool QUEUE = true;
  const NoSync sync;
#include "pfc_rowpair_body.cuh"
}

}  // namespace pfc
