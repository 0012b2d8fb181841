// The statements of row_step_pair and row_pair_queue (pfc_rowpair.cuh), which includes this file
// in both: as a function that the kernel inlines, the same statements compile to other code, with
// which a step took 0.4 (2048^2) to 1.5 % (256^2 FP64) longer.
// In scope: T, M, EE, ROWS, MODEL, QUEUE, a, batch, tile, member, sync.
  using S = PairSeq<M, EE>;
  constexpr int R0 = S::R0, NR = M / R0, NP = S::NP, THREADS = ROWS * S::TPF;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int r = threadIdx.x & (ROWS - 1), t = threadIdx.x / ROWS;
  cplx<T>* buf = reinterpret_cast<cplx<T>*>(smem_raw) + r;
  const size_t ny = a.ny;
  const int y = tile * ROWS + r;
  const cplx<T>* gin = a.in;
  cplx<T>* gout = a.out;
  const double* scal = a.scal;
  if (batch) {
    const BatchBufs& b = batch[member];
    gin = static_cast<const cplx<T>*>(b.w);
    gout = static_cast<cplx<T>*>(b.v);
    scal = b.scal;
  }
  const int jb = t == 0 ? NR / 2 : NR - t;   // the second butterfly

  sync();   // W is the previous column pass's output

  cplx<T> v[EE];
  {
    const cplx<T>* pa = gin + t * ny + y;
    const cplx<T>* pb = gin + jb * ny + y;
#pragma unroll
    for (int q = 0; q < R0; ++q) v[q] = ld_field<QUEUE>(pa + q * (NR * ny));
#pragma unroll
    for (int q = 0; q < R0; ++q) v[R0 + q] = ld_field<QUEUE>(pb + q * (NR * ny));
  }
  // Z[k] = S + U, Z[M - k] = conj(S - U), S = X[k] + conj X[M-k], U = i conj(r_k) (X[k] - conj X[M-k])
  pair_elements<R0, NR>(v, v + R0, t,
      [&](cplx<T>& x, cplx<T>& z, int k) {
        const cplx<T> s = x + conj(z), u = mul_i(cmul(conj(ldkc(a.rtw + k)), x - conj(z)));
        x = s + u;
        z = conj(s - u);
      },
      [](cplx<T>& x) { x = mk(x.x + x.y, x.x - x.y); },
      [](cplx<T>& x) { x = T(2) * conj(x); });   // r_{M/2} = -i: S + U = 2 conj X
  {
    dft_c<R0, true>(v);
    dft_c<R0, true>(v + R0);
    cplx<T>* p = buf + S::pad(t * R0) * ROWS;
    cplx<T>* q2 = buf + S::pad(jb * R0) * ROWS;
#pragma unroll
    for (int q = 0; q < R0; ++q) p[S::pad(q) * ROWS] = v[q];
#pragma unroll
    for (int q = 0; q < R0; ++q) q2[S::pad(q) * ROWS] = v[R0 + q];
    pair_sync<THREADS, QUEUE>();
  }
  pair_mid<T, M, EE, ROWS, false, true, QUEUE, 1, NP - 1>(buf, v, t, a.twA);
  {
    using PL = PairPass<T, M, EE, ROWS, false, NP - 1>;
    PL::load(buf, v, t);
    PL::template compute<true>(v, t, a.twA);
  }
  // ---- v holds n[2e] + i n[2e + 1]
  if constexpr (sizeof(T) == 4) {
    const float c1 = (float)scal[kScalC1], c2 = (float)scal[kScalC2], inv = (float)scal[kScalInvMean];
    const double inv_d = scal[kScalInvMean], mphi_rel = a.min_phi * inv_d;
    const float lmin = (float)scal[kScalLogMin];
#pragma unroll
    for (int e = 0; e < EE; ++e)
      v[e] = mk((T)nonlin_dev<MODEL>((float)v[e].x, c1, c2, inv, inv_d, a.clamp, mphi_rel, lmin),
                (T)nonlin_dev<MODEL>((float)v[e].y, c1, c2, inv, inv_d, a.clamp, mphi_rel, lmin));
  } else {
#pragma unroll
    for (int e = 0; e < EE; ++e)
      v[e] = mk((T)nonlin_plain<MODEL>((double)v[e].x, a.g, a.clamp, a.min_phi, a.min_log),
                (T)nonlin_plain<MODEL>((double)v[e].y, a.g, a.clamp, a.min_phi, a.min_log));
  }
  {
    using Q0 = PairPass<T, M, EE, ROWS, true, 0>;
    Q0::template compute<false>(v, t, a.twB);
    pair_sync<THREADS, QUEUE>();   // every thread has read the last exchange
    Q0::store(buf, v, t);
    pair_sync<THREADS, QUEUE>();
  }
  pair_mid<T, M, EE, ROWS, true, false, QUEUE, 1, NP - 1>(buf, v, t, a.twB);
  {
    using QL = PairPass<T, M, EE, ROWS, true, NP - 1>;
    static_assert(QL::R == R0 && QL::NS == NR, "sequence B ends with the radix that A begins with");
    const cplx<T>* p = buf + S::pad(t) * ROWS;
    const cplx<T>* q2 = buf + S::pad(jb) * ROWS;
#pragma unroll
    for (int q = 0; q < R0; ++q) v[q] = p[S::pad(q * NR) * ROWS];
#pragma unroll
    for (int q = 0; q < R0; ++q) v[R0 + q] = q2[S::pad(q * NR) * ROWS];
    QL::template butterfly<false>(v, t, a.twB);
    QL::template butterfly<false>(v + R0, jb, a.twB);
  }
  // Y[k] = E + r_k O, Y[M - k] = conj(E - r_k O), E = (Z[k] + conj Z[M-k]) / 2,
  // O = -i (Z[k] - conj Z[M-k]) / 2
  pair_elements<R0, NR>(v, v + R0, t,
      [&](cplx<T>& x, cplx<T>& z, int k) {
        const cplx<T> e = T(0.5) * (x + conj(z));
        const cplx<T> o = cmul(ldkc(a.rtw + k), T(0.5) * rot4<false>(x - conj(z)));
        x = e + o;
        z = conj(e - o);
      },
      [](cplx<T>& x) { x = mk(x.x + x.y, x.x - x.y); },
      [](cplx<T>& x) { x = conj(x); });
  {
    cplx<T>* pa = gout + t * ny + y;
    cplx<T>* pb = gout + jb * ny + y;
#pragma unroll
    for (int q = 0; q < R0; ++q) pa[q * (NR * ny)] = v[q];
#pragma unroll
    for (int q = 0; q < R0; ++q) pb[q * (NR * ny)] = v[R0 + q];
  }
