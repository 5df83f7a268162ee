// Large-block kernels (Hamiltonian blocks of kMaxBlock < b <= kMaxBigBlock), included by
// bl_engine.cu after DevSys and the complex helpers.  One CTA works on one crystallite's
// block with the matrices in shared memory; products are CTA-wide FP64 GEMMs with 2x2
// output tiles, one tile per thread (NT = 1) or two (NT = 2, blocks above 64), and CTAs of
// about one thread per tile so that registers stay low and several CTAs share an SM.
// Same arithmetic as the small-block kernels:
//   k_big_step      (c, step)   H_i, U_i = exp(-i 2pi tau H_i) by Taylor + squaring
//   k_big_dyson     (c, segment) A_{i+1} = U_i A_i within a segment (A stays in shared memory)
//   k_big_floquet   (c)         A_n = V diag(lam) V^H: Cayley transform, parallel Jacobi
//   k_big_seg_frame (c, segment) V_s = E_s V_F
//   k_big_eigframe  (c, segment) W_i = A_{i+1} V_F
//   k_big_qr        (c, step) per pair  Q = W_a^H M_ab W_b for block pairs with a big block
// and, for the mixed form, the same step and Dyson in double-float on the FP32 pipe:
//   k_big_step_df   (c, step)   U_i in double-float (the Taylor series term by term)
//   k_big_dyson_df  (c)         A_{i+1} = U_i A_i in double-float

constexpr int kMaxBigBlock = 74;   // 5 real b x b matrices fit 227 KB of shared memory
// k_big_floquet: a block from kFloqWide on has an SM's shared memory to itself and needs the warps
constexpr int kBigThreads = 512, kFloqWide = 40;
__host__ __device__ constexpr int floquet_threads(int b) { return b >= kFloqWide ? kBigThreads : 256; }
constexpr int kBigPSMax = 63;      // 7 real b x b matrices (Paterson-Stockmeyer step) fit
constexpr int kMaxInt = 128;       // interactions per system on the large-block path

// Element e of block (size b, packed offset bp) of crystallite c inside one step's A or W
// array: [item][c] as at(), or, for the large blocks of a crystallite-major job (s.clay), the
// block's region [bp Cpad, (bp + b^2) Cpad) taken as [c][e].
__device__ __forceinline__ size_t big_at(const DevSys &s, int b, int bp, int e, int c) {
  return (s.clay && b > kMaxBlock && b <= kMaxBigBlock) ? size_t(bp) * s.Cpad + size_t(c) * b * b + e
                                                        : size_t(bp + e) * s.Cpad + c;
}

__host__ __device__ constexpr int big_tiles(int m, int n) { return ((m + 1) / 2) * ((n + 1) / 2); }
// tiles per thread of an m x n product, and the CTA size that gives each thread NT tiles
__host__ __device__ constexpr int big_nt(int m, int n) { return big_tiles(m, n) <= 1024 ? 1 : 2; }
__host__ __device__ constexpr int big_threads(int m, int n) {
  return ((big_tiles(m, n) + big_nt(m, n) - 1) / big_nt(m, n) + 31) / 32 * 32;
}

// C (m x n) = alpha * A (m x k) * B (k x n) (+ epilogue), real, shared memory, row-major.
// ep(e, v) returns the value stored at C[e] for the product value v.
template <class EP>
__device__ void cta_mm_real(const double *A, int lda, const double *B, int ldb, double *C, int ldc, int m, int n,
                            int k, double alpha, EP ep) {
  const int tm = (m + 1) / 2, tn = (n + 1) / 2;
  for (int t = threadIdx.x; t < tm * tn; t += blockDim.x) {
    const int i0 = (t / tn) * 2, j0 = (t % tn) * 2;
    const int i1 = min(i0 + 1, m - 1), j1 = min(j0 + 1, n - 1);
    double c00 = 0, c01 = 0, c10 = 0, c11 = 0;
    for (int l = 0; l < k; ++l) {
      const double a0 = A[i0 * lda + l], a1 = A[i1 * lda + l];
      const double b0 = B[l * ldb + j0], b1 = B[l * ldb + j1];
      c00 = fma(a0, b0, c00), c01 = fma(a0, b1, c01), c10 = fma(a1, b0, c10), c11 = fma(a1, b1, c11);
    }
    C[i0 * ldc + j0] = ep(i0 * ldc + j0, alpha * c00);
    if (j0 + 1 < n) C[i0 * ldc + j0 + 1] = ep(i0 * ldc + j0 + 1, alpha * c01);
    if (i0 + 1 < m) {
      C[(i0 + 1) * ldc + j0] = ep((i0 + 1) * ldc + j0, alpha * c10);
      if (j0 + 1 < n) C[(i0 + 1) * ldc + j0 + 1] = ep((i0 + 1) * ldc + j0 + 1, alpha * c11);
    }
  }
}
__device__ __forceinline__ void cta_mm_real(const double *A, int lda, const double *B, int ldb, double *C, int ldc,
                                            int m, int n, int k, double alpha) {
  cta_mm_real(A, lda, B, ldb, C, ldc, m, n, k, alpha, [](int, double v) { return v; });
}

// Upper-triangle 2x2 tiles of an m x m matrix: tile t -> (ti, tj), ti <= tj, t < big_sym_tiles.
// Rows pr and tm-1-pr together hold tm+1 tiles; an odd tm's middle row comes last.
__host__ __device__ constexpr int big_sym_tiles(int m) { return ((m + 1) / 2) * ((m + 1) / 2 + 1) / 2; }
__device__ __forceinline__ void sym_tile(int t, int tm, int &ti, int &tj) {
  const int h = tm / 2, pr = t / (tm + 1), q = t % (tm + 1);
  if (pr < h) {
    if (q < tm - pr) ti = pr, tj = pr + q;
    else ti = tm - 1 - pr, tj = ti + (q - (tm - pr));
  } else {
    ti = h, tj = h + (t - h * (tm + 1));
  }
}

// C = alpha * A * B (+ epilogue) for m x m real A, B that are symmetric and commute, so
// that C is symmetric: only upper-triangle tiles are computed, each value stored at (i, j)
// and (j, i).  ep(e, v) gives the stored value for the upper element e = i*m + j (called
// once per upper element, by the thread that stores it and its mirror).
template <class EP>
__device__ void cta_mm_sym(const double *A, const double *B, double *C, int m, double alpha, EP ep) {
  const int tm = (m + 1) / 2;
  for (int t = threadIdx.x; t < big_sym_tiles(m); t += blockDim.x) {
    int ti, tj;
    sym_tile(t, tm, ti, tj);
    const int i0 = 2 * ti, j0 = 2 * tj;
    const int i1 = min(i0 + 1, m - 1), j1 = min(j0 + 1, m - 1);
    double c00 = 0, c01 = 0, c10 = 0, c11 = 0;
    for (int l = 0; l < m; ++l) {
      const double a0 = A[i0 * m + l], a1 = A[i1 * m + l];
      const double b0 = B[l * m + j0], b1 = B[l * m + j1];
      c00 = fma(a0, b0, c00), c01 = fma(a0, b1, c01), c10 = fma(a1, b0, c10), c11 = fma(a1, b1, c11);
    }
    auto put = [&](int i, int j, double v) {
      const double x = ep(i * m + j, alpha * v);
      C[i * m + j] = x;
      if (i != j) C[j * m + i] = x;
    };
    put(i0, j0, c00);
    if (j0 + 1 < m) put(i0, j0 + 1, c01);
    if (i0 + 1 < m) {
      if (ti != tj) put(i0 + 1, j0, c10);  // on a diagonal tile (i0+1, i0) mirrors c01
      if (j0 + 1 < m) put(i0 + 1, j0 + 1, c11);
    }
  }
}
__device__ __forceinline__ void cta_mm_sym(const double *A, const double *B, double *C, int m, double alpha) {
  cta_mm_sym(A, B, C, m, alpha, [](int, double v) { return v; });
}

// Complex 2x2-tiled product into per-thread registers: acc[q] for the tiles
// t = threadIdx.x + q*blockDim.x.  CONJ_A: use A^H (A stored k x m).
template <int NT, bool CONJ_A, class C>
__device__ void cta_mm_cplx_regs(const C *A, int lda, const C *B, int ldb, int m, int n, int k, C (&acc)[NT][4]) {
  const int tm = (m + 1) / 2, tn = (n + 1) / 2;
#pragma unroll
  for (int q = 0; q < NT; ++q) {
    const int t = threadIdx.x + q * blockDim.x;
    acc[q][0] = acc[q][1] = acc[q][2] = acc[q][3] = mkc<C>(0, 0);
    if (t >= tm * tn) continue;
    const int i0 = (t / tn) * 2, j0 = (t % tn) * 2;
    const int i1 = min(i0 + 1, m - 1), j1 = min(j0 + 1, n - 1);
    C c00 = mkc<C>(0, 0), c01 = c00, c10 = c00, c11 = c00;
    for (int l = 0; l < k; ++l) {
      C a0, a1;
      if (CONJ_A) {
        a0 = cconj(A[l * lda + i0]), a1 = cconj(A[l * lda + i1]);
      } else {
        a0 = A[i0 * lda + l], a1 = A[i1 * lda + l];
      }
      const C b0 = B[l * ldb + j0], b1 = B[l * ldb + j1];
      c00 = cfma(a0, b0, c00), c01 = cfma(a0, b1, c01), c10 = cfma(a1, b0, c10), c11 = cfma(a1, b1, c11);
    }
    acc[q][0] = c00, acc[q][1] = c01, acc[q][2] = c10, acc[q][3] = c11;
  }
}

// Visits this thread's tile outputs: f(row, col, value).
template <int NT, class C, class F>
__device__ void cta_tiles_store(int m, int n, const C (&acc)[NT][4], F f) {
  const int tm = (m + 1) / 2, tn = (n + 1) / 2;
#pragma unroll
  for (int q = 0; q < NT; ++q) {
    const int t = threadIdx.x + q * blockDim.x;
    if (t >= tm * tn) continue;
    const int i0 = (t / tn) * 2, j0 = (t % tn) * 2;
    f(i0, j0, acc[q][0]);
    if (j0 + 1 < n) f(i0, j0 + 1, acc[q][1]);
    if (i0 + 1 < m) {
      f(i0 + 1, j0, acc[q][2]);
      if (j0 + 1 < n) f(i0 + 1, j0 + 1, acc[q][3]);
    }
  }
}

// Shared memory of k_big_step for a block of size b.
__host__ __device__ constexpr size_t big_step_smem(int b) {
  return sizeof(double) * size_t(b <= kBigPSMax ? 7 : 5) * size_t(b) * size_t(b);
}

// One CTA per (crystallite, step): U_i of a large block, exp(-iX) with X = 2pi tau H_i / 2^sq
// (||X||_inf <= 1/2) by its Taylor polynomial, then sq squarings.  Blocks above kBigPSMax
// sum the series term by term up to the degree taylor_degree gives for the step's norm.
// Blocks up to kBigPSMax evaluate the polynomial as cos X = C(Y), sin X = X S(Y), Y = X^2,
// C and S by Paterson-Stockmeyer with the power of Y that the step's degree needs (5 to 7 real
// products; always 7 before: 5 spins, 320 crystallites, n = 157, step 2.58 -> 2.18 ms); larger
// blocks accumulate the terms one product at a time (up to 14).  All
// factors are polynomials in X, hence symmetric and commuting: products are symmetric
// and only their upper triangles are computed (cta_mm_sym).
__global__ void __launch_bounds__(1024) k_big_step(DevSys s, int k) {
  extern __shared__ double bsm[];
  __shared__ double fk[kMaxInt];
  __shared__ double red[kMaxBigBlock];
  __shared__ double scl[3];
  const int c = blockIdx.x % s.C, i = blockIdx.x / s.C;
  const int b = s.bs[k], bp = s.bpoff[k], bb = b * b;
  if (s.fk && !s.fk_df) {  // k_coef's coefficients (same arithmetic), read in parallel
    for (int kk = threadIdx.x; kk < s.nint; kk += blockDim.x) fk[kk] = s.fk[at(i * s.nint + kk, c, s.Cpad)];
  } else if (threadIdx.x == 0) {
    double t1 = s.t0[c] + double(i) * s.tau, t2 = t1 + s.tau;
    double tmid = (t2 - t1) / 2.0 + t1;
    double sp, cp;
    sincos(tmid * s.wr * kPi2, &sp, &cp);
    double m[3][3];
    orient_rows(s, c, sp, cp, m);
    for (int kk = 0; kk < s.nint; ++kk) fk[kk] = term_coef(s, kk, m);
  }
  __syncthreads();
  double *X = bsm;
  const double *Hcb = hc_of(s, i) + bp;
  for (int x = threadIdx.x; x < bb; x += blockDim.x) {  // each element's own terms, longest first
    const int e = s.tk_order[bp + x];
    double h = Hcb[e];
    for (int t = s.tk_ptr[bp + e]; t < s.tk_ptr[bp + e + 1]; ++t) h = fma(fk[s.tk_term[t]], s.tk_val64[t], h);
    X[e] = h;
  }
  __syncthreads();
  for (int p = threadIdx.x; p < b; p += blockDim.x) {
    double rs = 0;
    for (int q = 0; q < b; ++q) rs += fabs(X[p * b + q]);
    red[p] = rs;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double nrm = 0;
    for (int p = 0; p < b; ++p) nrm = fmax(nrm, red[p]);
    const double tp = s.tau * kPi2;
    nrm *= tp;
    int sq = 0;
    if (nrm > 0.5) {
      frexp(nrm / 0.5, &sq);
      sq = min(sq, 60);
    }
    scl[0] = ldexp(tp, -sq);
    scl[1] = double(sq);
    scl[2] = double(taylor_degree(ldexp(nrm, -sq), s.mixed != 0));  // terms the series needs
  }
  __syncthreads();
  const double sc = scl[0];
  const int sq = int(scl[1]), nterms = int(scl[2]);
  double *R, *I, *F0, *F1, *F2;  // result R + iI and three free b x b buffers for squaring
  if (b <= kBigPSMax) {
    double *Y = X + bb, *Y2 = Y + bb, *Y3 = Y2 + bb, *Y4 = Y3 + bb, *T = Y4 + bb;
    R = T + bb;
    for (int e = threadIdx.x; e < bb; e += blockDim.x) X[e] *= sc;
    __syncthreads();
    cta_mm_sym(X, X, Y, b, 1.0);
    __syncthreads();
    cta_mm_sym(Y, Y, Y2, b, 1.0);
    __syncthreads();
    // the polynomials to the degree this step's norm needs (cos X: nterms / 2 in Y), at the fewest
    // products: powers up to Y^2 serve degree 4 (5 products in all), Y^3 degree 6 (6), Y^4
    // degree 7 (7).  P(Y) = low(Y) + top(Y) Y^m, top evaluated into T.
    const int m = nterms <= 9 ? 2 : nterms <= 13 ? 3 : 4;
    double *Ym = m == 2 ? Y2 : m == 3 ? Y3 : Y4;
    if (m >= 3) cta_mm_sym(Y2, Y, Y3, b, 1.0);
    if (m == 4) cta_mm_sym(Y2, Y2, Y4, b, 1.0);
    __syncthreads();
    double *S = m == 4 ? Y3 : Y4;  // S(Y): over Y^3 in place when Y^4 is the factor (element e's
                                   // epilogue reads Y3[e] before the same thread writes it)
    for (int pass = 0; pass < 2; ++pass) {
      const bool sn = pass == 1;
      auto cf = [&](int j) { return sn ? sin_coef(j) : cos_coef(j); };
      const double t0 = cf(m), t1 = cf(m + 1), t2 = cf(m + 2), t3 = m >= 3 ? cf(m + 3) : 0.0;
      const double l0 = cf(0), l1 = cf(1), l2 = cf(2), l3 = cf(3);
      for (int e = threadIdx.x; e < bb; e += blockDim.x) {
        double v = fma(t2, Y2[e], fma(t1, Y[e], (e / b == e % b) ? t0 : 0.0));
        if (m >= 3) v = fma(t3, Y3[e], v);
        T[e] = v;
      }
      __syncthreads();
      cta_mm_sym(Ym, T, sn ? S : R, b, 1.0, [&](int e, double v) {
        v += fma(l1, Y[e], (e / b == e % b) ? l0 : 0.0);
        if (m >= 3) v = fma(l2, Y2[e], v);
        if (m == 4) v = fma(l3, Y3[e], v);
        return v;
      });
      __syncthreads();
    }
    I = Y;  // -sin X = -X S(Y)
    cta_mm_sym(X, S, I, b, -1.0);
    F0 = Y2, F1 = S == Y4 ? Y3 : Y4, F2 = T;
  } else {
    double *P = X + bb, *Q = P + bb;
    R = Q + bb, I = R + bb;
    for (int e = threadIdx.x; e < bb; e += blockDim.x) {
      const double x = sc * X[e];
      X[e] = x, P[e] = x;
      R[e] = (e / b == e % b) ? 1.0 : 0.0;
      I[e] = -x;
    }
    __syncthreads();
    for (int kt = 2; kt <= nterms; ++kt) {  // the degree the step's norm needs (<= 15)
      cta_mm_sym(P, X, Q, b, 1.0 / kt);
      __syncthreads();
      const int m4 = kt & 3;
      for (int e = threadIdx.x; e < bb; e += blockDim.x) {
        const double v = Q[e];
        if (m4 == 2) R[e] -= v;
        else if (m4 == 3) I[e] += v;
        else if (m4 == 0) R[e] += v;
        else I[e] -= v;
      }
      double *t = P;
      P = Q, Q = t;
      __syncthreads();
    }
    F0 = P, F1 = Q, F2 = X;
  }
  __syncthreads();
  for (int t = 0; t < sq; ++t) {  // (R + iI)^2 = (RR - II) + i 2RI
    cta_mm_sym(R, R, F0, b, 1.0);
    cta_mm_sym(I, I, F1, b, 1.0);
    cta_mm_sym(R, I, F2, b, 2.0);
    __syncthreads();
    for (int e = threadIdx.x; e < bb; e += blockDim.x) R[e] = F0[e] - F1[e], I[e] = F2[e];
    __syncthreads();
  }
  double2 *Ub = s.U + size_t(i) * s.S2 * s.Cpad;
  const double2 *fr = frame_of(s, i);
  if (fr) {  // lab frame of a chunk rf phase: U = R U' R^H
    const int bo = s.boff[k];
    for (int e = threadIdx.x; e < bb; e += blockDim.x)
      Ub[at(bp + e, c, s.Cpad)] = cmul(cmul(fr[bo + e / b], cmk(R[e], I[e])), cconj(fr[bo + e % b]));
  } else {
    for (int e = threadIdx.x; e < bb; e += blockDim.x) Ub[at(bp + e, c, s.Cpad)] = cmk(R[e], I[e]);
  }
}

// One CTA per (crystallite, segment): the segment's products P_i = U_i P_{i-1}, P in shared
// memory; or (prefix) one per crystallite, the chain over the segments' last products.
template <int NT>
__global__ void __launch_bounds__(NT == 1 ? 1024 : 768) k_big_dyson(DevSys s, int k, bool prefix) {
  extern __shared__ double2 bsc[];
  const int c = blockIdx.x % s.C;
  const int b = s.bs[k], bp = s.bpoff[k], bb = b * b;
  double2 *Us = bsc, *As = Us + bb;
  for (int e = threadIdx.x; e < bb; e += blockDim.x) As[e] = cmk(e / b == e % b ? 1.0 : 0.0, 0.0);
  double2 acc[NT][4];
  const Chain ch = seg_chain(s, b, blockIdx.x / s.C, prefix);
  for (int i = 0; i < ch.count; ++i) {
    const double2 *Ub = ch.from(s, i);
    for (int e = threadIdx.x; e < bb; e += blockDim.x) Us[e] = Ub[at(bp + e, c, s.Cpad)];
    __syncthreads();
    cta_mm_cplx_regs<NT, false, double2>(Us, b, As, b, b, b, b, acc);
    __syncthreads();
    double2 *Ab = ch.to(s, i);
    cta_tiles_store<NT>(b, b, acc, [&](int r, int q, double2 v) {
      As[r * b + q] = v;
      Ab[at(bp + r * b + q, c, s.Cpad)] = v;
    });
    __syncthreads();
  }
}

// One CTA per (crystallite, segment t): V_t = E_t V_F (k_seg_frame's for the large blocks): FP64
// over E_t, t >= 1; mixed form in double-float, rounded to float2, t = 0 (V_F itself) included.
template <bool MIX>
__global__ void __launch_bounds__(1024) k_big_seg_frame(DevSys s, int k) {
  extern __shared__ __align__(16) unsigned char bsr[];
  const int c = blockIdx.x % s.C, t = blockIdx.x / s.C + (MIX ? 0 : 1);
  const int b = s.bs[k], bp = s.bpoff[k], bb = b * b;
  if constexpr (MIX) {
    float2 *Vo = seg_Vf(s, t);
    float4 *Vs = reinterpret_cast<float4 *>(bsr), *Es = Vs + bb;
    if (t == 0) {
      for (int e = threadIdx.x; e < bb; e += blockDim.x)
        Vo[big_at(s, b, bp, e, c)] = cvt<float2>(s.VF[at(bp + e, c, s.Cpad)]);
      return;
    }
    const float4 *E = reinterpret_cast<const float4 *>(seg_E(s, t - 1));
    for (int e = threadIdx.x; e < bb; e += blockDim.x) {
      Vs[e] = df_store(s.VF[at(bp + e, c, s.Cpad)]);
      Es[e] = E[big_at(s, b, bp, e, c)];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < bb; e += blockDim.x) {
      const int r = e / b, q = e % b;
      CdfAcc a = {{0.f, 0.f}, {0.f, 0.f}};
      for (int l = 0; l < b; ++l) cdf_mac(a, Es[r * b + l], Vs[l * b + q]);
      const float4 w = cdf_fin(a);
      Vo[big_at(s, b, bp, e, c)] = make_float2(w.x, w.y);
    }
  } else {
    double2 *Vs = reinterpret_cast<double2 *>(bsr), *Es = Vs + bb, *E = seg_E(s, t - 1);
    for (int e = threadIdx.x; e < bb; e += blockDim.x) {
      Vs[e] = s.VF[at(bp + e, c, s.Cpad)];
      Es[e] = E[at(bp + e, c, s.Cpad)];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < bb; e += blockDim.x) {
      const int r = e / b, q = e % b;
      double2 acc = cmk(0, 0);
      for (int l = 0; l < b; ++l) acc = cfma(Es[r * b + l], Vs[l * b + q], acc);
      E[at(bp + e, c, s.Cpad)] = acc;
    }
  }
}

// One CTA per (crystallite, kSegLen steps): W_i = A_{i+1} V_F = P_i V_s (FP64, in place over A).
template <int NT, class C>
__global__ void __launch_bounds__(NT == 1 ? 1024 : 768) k_big_eigframe(DevSys s, int k) {
  extern __shared__ __align__(16) unsigned char bsr[];
  const int c = blockIdx.x % s.C, i0 = int(blockIdx.x / s.C) * kSegLen, i1 = min(s.n, i0 + kSegLen);
  const int b = s.bs[k], bp = s.bpoff[k], bb = b * b;
  C *Vs = reinterpret_cast<C *>(bsr), *As = Vs + bb;
  for (int e = threadIdx.x; e < bb; e += blockDim.x) Vs[e] = frame_elem<C>(s, segmented(s, b), i0, at(bp + e, c, s.Cpad));
  C acc[NT][4];
  for (int i = i0; i < i1; ++i) {
    const double2 *Ab = s.A + size_t(i) * s.S2 * s.Cpad;
    C *Wb = Bufs<C>::W(s) + size_t(i) * s.S2 * s.Cpad;
    for (int e = threadIdx.x; e < bb; e += blockDim.x) As[e] = cvt<C>(Ab[at(bp + e, c, s.Cpad)]);
    __syncthreads();
    cta_mm_cplx_regs<NT, false, C>(As, b, Vs, b, b, b, b, acc);
    cta_tiles_store<NT>(b, b, acc, [&](int r, int q, C v) { Wb[at(bp + r * b + q, c, s.Cpad)] = v; });
    __syncthreads();
  }
}

// One big Q/R block pair as the kernel sees it: blocks a, b, the output offset, and the
// non-zeros of M_ab (D or rho) by row: row l holds entries [rp[l], rp[l+1]) of (ci, cv).
struct BigPair {
  int a, b, off, nitems, isq, wchunk;
  int e2;  // |M_ab W_b| <= 2^e2: the larger of M_ab's row and column sums
  const int *rp, *ci;
  const double2 *cv;
  const float2 *cvf;  // mixed form: cv in single precision (a conversion is an FP64-pipe instruction)
};
__device__ __forceinline__ double2 pair_coef(const BigPair &P, int j, double2) { return __ldg(P.cv + j); }
__device__ __forceinline__ float2 pair_coef(const BigPair &P, int j, float2) { return __ldg(P.cvf + j); }

// Shared memory of k_big_qr: W_a, a column chunk of W_b and of X = M_ab W_b.
template <class C>
__host__ __device__ constexpr size_t big_qr_smem(int ba, int bb, int w) {
  return sizeof(C) * (size_t(ba) * ba + size_t(bb) * w + size_t(ba) * w);
}

// One CTA per (crystallite, step) of one block pair: Q^{ab} = W_a^H (M_ab W_b), M = D (or
// rho), over column chunks of width wchunk; M's non-zeros come from the host.
template <int NT, class C>
__global__ void __launch_bounds__(NT == 1 ? 1024 : 768) k_big_qr(DevSys s, BigPair bp2) {
  extern __shared__ __align__(16) unsigned char bsr[];
  const int c = blockIdx.x % s.C, i = blockIdx.x / s.C;
  const int ba = s.bs[bp2.a], bb = s.bs[bp2.b], pa = s.bpoff[bp2.a], pb = s.bpoff[bp2.b];
  const int w = bp2.wchunk;
  C *out = bp2.isq ? Bufs<C>::Q(s) : Bufs<C>::R(s);
  const C *W = Bufs<C>::W(s) + size_t(i) * s.S2 * s.Cpad;
  C *Wa = reinterpret_cast<C *>(bsr), *Wb = Wa + ba * ba, *X = Wb + bb * w;
  for (int e = threadIdx.x; e < ba * ba; e += blockDim.x) Wa[e] = W[big_at(s, ba, pa, e, c)];
  C *ob = out + size_t(i) * bp2.nitems * s.Cpad;
  C acc[NT][4];
  for (int q0 = 0; q0 < bb; q0 += w) {
    const int wc = min(w, bb - q0);
    for (int e = threadIdx.x; e < bb * wc; e += blockDim.x) {
      const int m = e / wc, q = e % wc;
      Wb[e] = W[big_at(s, bb, pb, m * bb + q0 + q, c)];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < ba * wc; e += blockDim.x) {
      const int l = e / wc, q = e % wc;
      C x = mkc<C>(0, 0);
      for (int j = __ldg(bp2.rp + l); j < __ldg(bp2.rp + l + 1); ++j)
        x = cfma(pair_coef(bp2, j, C()), Wb[__ldg(bp2.ci + j) * wc + q], x);
      X[e] = x;
    }
    __syncthreads();
    cta_mm_cplx_regs<NT, true, C>(Wa, ba, X, wc, ba, wc, ba, acc);
    cta_tiles_store<NT>(ba, wc, acc, [&](int r, int q, C v) { ob[at(bp2.off + r * bb + q0 + q, c, s.Cpad)] = v; });
    __syncthreads();
  }
}

// One CTA per crystallite: unitary eigen-decomposition of a block of A_n by the Cayley
// transform K = i (I+W)^{-1}(I-W), W = e^{ia} A_n, and a parallel (round-robin) complex
// Jacobi on K; a second pass moves -1 into the widest spectral gap when the first is ill
// conditioned.  Work arrays of floquet_cta: Mm, Xk (b x b each), rot and rpair ((b/2+1) x 2),
// fv and lam (b each), red (max(b, blockDim.x)); in shared memory for blocks up to
// kMaxBigBlock, Mm and Xk in global memory above.
struct FloqWork {
  double2 *Mm, *Xk, *rot, *fv, *lam;
  int *rpair;
  double *red;
  float2 *Kf;  // MIX: b x b single-precision K
};

// q = e / d and r = e - q d without an integer division: the FP32 quotient is at most one off
__device__ __forceinline__ int fdiv(int e, float invd, int d, int &r) {
  int q = __float2int_rz(float(e) * invd);
  r = e - q * d;
  if (r < 0) --q, r += d;
  if (r >= d) ++q, r -= d;
  return q;
}
// (i, j) with i <= j < n of the e-th of n (n + 1) / 2 pairs: rows i and n-1-i share a line of n + 1
__device__ __forceinline__ int tri_pair(int e, int n, float inv_n1, int &j) {
  int col;
  const int r = fdiv(e, inv_n1, n + 1, col);
  if (col < n - r) {
    j = r + col;
    return r;
  }
  j = col - 1;
  return n - 1 - r;
}

// c x - s y and s' x + c y of a rotation's two outputs
template <class C, class T>
__device__ __forceinline__ C rot_mix(T c, C x, C s, C y) {
  C v;
  v.x = fma(c, x.x, fma(s.x, y.x, -(s.y * y.y)));
  v.y = fma(c, x.y, fma(s.x, y.y, s.y * y.x));
  return v;
}

// The parallel Jacobi sweeps of floquet_cta over the Hermitian K with V accumulating the rotations;
// returns convergence.  The angles come from single precision; in FP64 each rotation is scaled to
// c^2 + |s|^2 = 1 and elements at the diagonal's rounding are set to zero, as in lanes_sweeps.  A round's pairs are disjoint, so K <- G^H K G splits into
// 2 x 2 blocks (pair t1's rows, pair t2's columns): only t1 <= t2 is computed and its conjugate
// stored with it, 24 FP64 operations per element pair against 48 for columns then rows of the
// whole of K, and one barrier less per round.
template <class C>
__device__ bool floquet_sweeps(C *K, C *V, int b, int max_sweeps, const FloqWork &wk) {
  using T = decltype(C::x);
  constexpr bool kF64 = sizeof(T) == 8;
  C *rot = reinterpret_cast<C *>(wk.rot);  // per pair: (c, 1 to set K_pq to zero), (s e^{i ph})
  auto rpair = [&](int t, int q) -> int & { return wk.rpair[2 * t + q]; };
  double *red = wk.red;
  const int bb = b * b;
  const float invb = 1.f / float(b);
  const int bq = b + (b & 1);  // players in the round-robin (one dummy when b is odd)
  const int np = bq / 2, nblk = np * (np + 1) / 2;
  const float inv_np = 1.f / float(np), inv_np1 = 1.f / float(np + 1);
  bool conv = false, polish = false;
  const int nw = (blockDim.x + 31) / 32, wid = threadIdx.x >> 5, lid = threadIdx.x & 31;
  for (int sweep = 0; sweep < max_sweeps && !conv; ++sweep) {
    // off(K)^2 and diag(K)^2: sums per thread, a fixed shuffle tree per warp, the warps' sums
    // added by one thread
    T off = 0, dg = 0;
    for (int e = threadIdx.x; e < bb; e += blockDim.x) {
      int q;
      const int r = fdiv(e, invb, b, q);
      const C v = K[e];
      if (r < q) off += v.x * v.x + v.y * v.y;
      else if (r == q) dg += v.x * v.x;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      off += __shfl_xor_sync(0xffffffffu, off, o);
      dg += __shfl_xor_sync(0xffffffffu, dg, o);
    }
    if (lid == 0) red[2 * wid] = off, red[2 * wid + 1] = dg;
    __syncthreads();
    if (threadIdx.x == 0) {
      double so = 0, sd = 0;
      for (int t = 0; t < nw; ++t) so += red[2 * t], sd += red[2 * t + 1];
      red[2 * nw] = so, red[2 * nw + 1] = sd;
    }
    __syncthreads();
    const double offs = red[2 * nw], dgs = red[2 * nw + 1];
    __syncthreads();
    if (kF64) {
      conv = offs <= 1e-34 * dgs || offs <= 1e-60;
    } else {  // single precision: once small, one more sweep reaches its rounding
      const bool small = offs <= 1e-10 * dgs;
      conv = (small && polish) || offs == 0.0;
      polish = small;
    }
    if (conv) break;
    for (int round = 0; round < bq - 1; ++round) {
      for (int t = threadIdx.x; t < np; t += blockDim.x) {
        auto player = [&](int j) { return j == 0 ? 0 : 1 + (j - 1 + round) % (bq - 1); };
        int p = player(t), q = player(bq - 1 - t);
        if (p > q) {
          int tmp = p;
          p = q, q = tmp;
        }
        rpair(t, 0) = p, rpair(t, 1) = q;
        C rc = mkc<C>(1, 0), rs = mkc<C>(0, 0);
        if (q < b) {
          const float hx = float(K[p * b + q].x), hy = float(K[p * b + q].y);
          const T kpp = K[p * b + p].x, kqq = K[q * b + q].x;
          const float ab = hypotf(hx, hy), dmax = kF64 ? fmaxf(fabsf(float(kpp)), fabsf(float(kqq))) : 0.f;
          if (kF64 && ab <= fmaxf(kSweepZero * dmax, kSweepTiny)) rc.y = 1;
          if (ab > fmaxf(kSweepRound * dmax, kSweepTiny)) {
            const float theta = 0.5f * float(kqq - kpp) / ab;
            float tt;
            if (fabsf(theta) > 1e18f) tt = 0.5f / theta;  // theta^2 stays finite
            else tt = copysignf(1.f, theta) / (fabsf(theta) + sqrtf(fmaf(theta, theta, 1.f)));
            const float cf = rsqrtf(fmaf(tt, tt, 1.f)), ts = tt * cf / ab;
            rc.x = cf;
            rs = mkc<C>(hx * ts, hy * ts);
            if (kF64) {
              const T d = fma(rc.x, rc.x, fma(rs.x, rs.x, fma(rs.y, rs.y, T(-1))));
              const T nn = fma(fma(T(0.375), d, T(-0.5)), d, T(1));
              rc.x *= nn;
              rs = cscale(rs, nn);
            }
          }
        }
        rot[2 * t] = rc, rot[2 * t + 1] = rs;
      }
      __syncthreads();
      // G = [[c, s], [-conj(s), c]] per pair: K's blocks, then the columns of V, the pair index
      // fastest (a warp's accesses to V stay within one row)
      for (int e = threadIdx.x; e < nblk + np * b; e += blockDim.x) {
        if (e < nblk) {
          int t2;
          const int t1 = tri_pair(e, np, inv_np1, t2);
          const int p1 = rpair(t1, 0), q1 = rpair(t1, 1), p2 = rpair(t2, 0), q2 = rpair(t2, 1);
          const bool h1 = q1 < b, h2 = q2 < b;
          const C zero = mkc<C>(0, 0);
          C kpp = K[p1 * b + p2], kpq = h2 ? K[p1 * b + q2] : zero, kqp = h1 ? K[q1 * b + p2] : zero,
            kqq = h1 && h2 ? K[q1 * b + q2] : zero;
          {
            const T c2 = rot[2 * t2].x;
            const C s2 = rot[2 * t2 + 1], m2 = mkc<C>(-s2.x, s2.y);
            const C x = rot_mix(c2, kpp, m2, kpq), y = rot_mix(c2, kqp, m2, kqq);
            kpq = rot_mix(c2, kpq, s2, kpp), kqq = rot_mix(c2, kqq, s2, kqp);
            kpp = x, kqp = y;
          }
          {
            const T c1 = rot[2 * t1].x;
            const C s1 = rot[2 * t1 + 1], m1 = mkc<C>(-s1.x, -s1.y), j1 = cconj(s1);
            const C x = rot_mix(c1, kpp, m1, kqp), y = rot_mix(c1, kpq, m1, kqq);
            kqp = rot_mix(c1, kqp, j1, kpp), kqq = rot_mix(c1, kqq, j1, kpq);
            kpp = x, kpq = y;
          }
          if (t1 == t2) {  // the diagonal stays real
            if (rot[2 * t1].y != 0) kpq = zero;
            kpp.y = 0, kqq.y = 0, kqp = cconj(kpq);
          }
          K[p1 * b + p2] = kpp;
          if (t1 != t2) K[p2 * b + p1] = cconj(kpp);
          if (h2) K[p1 * b + q2] = kpq;
          if (h2 && t1 != t2) K[q2 * b + p1] = cconj(kpq);
          if (h1) K[q1 * b + p2] = kqp;
          if (h1 && t1 != t2) K[p2 * b + q1] = cconj(kqp);
          if (h1 && h2) K[q1 * b + q2] = kqq;
          if (h1 && h2 && t1 != t2) K[q2 * b + q1] = cconj(kqq);
        } else {
          int t;
          const int kk = fdiv(e - nblk, inv_np, np, t);
          const int p = rpair(t, 0), q = rpair(t, 1);
          if (q >= b) continue;
          const T cc = rot[2 * t].x;
          const C sp = rot[2 * t + 1];
          const C vp = V[kk * b + p], vq = V[kk * b + q];
          V[kk * b + p] = rot_mix(cc, vp, mkc<C>(-sp.x, sp.y), vq);
          V[kk * b + q] = rot_mix(cc, vq, sp, vp);
        }
      }
      __syncthreads();
    }
  }
  return conv;
}

// x - f y, complex double-float
__device__ __forceinline__ float4 cdf_fms(float4 x, float4 f, float4 y) {
  CdfAcc a = {{x.x, x.z}, {x.y, x.w}};
  cdf_mac(a, make_float4(-f.x, -f.y, -f.z, -f.w), y);
  return cdf_fin(a);
}
__device__ __forceinline__ float4 cdf_mul(float4 x, float4 y) {
  CdfAcc a = {{0.f, 0.f}, {0.f, 0.f}};
  cdf_mac(a, x, y);
  return cdf_fin(a);
}

// Element arithmetic of floquet_start: FP64, or double-float on the FP32 pipe (mixed form).  A
// diagonal element of the work matrix holds K_ii in its real part and E_ii in its imaginary part.
struct FloqF64 {
  static constexpr int kStartMin = 16;  // smallest block that takes floquet_start
  using E = double2;
  using Acc = double2;
  static __device__ __forceinline__ E of(float2 v) { return cmk(v.x, v.y); }
  static __device__ __forceinline__ float2 narrow(E v) { return make_float2(float(v.x), float(v.y)); }
  static __device__ __forceinline__ E conj(E v) { return cconj(v); }
  static __device__ __forceinline__ Acc acc(E v) { return v; }
  static __device__ __forceinline__ void mac(Acc &a, E x, E y) { a = cfma(x, y, a); }
  static __device__ __forceinline__ void macj(Acc &a, E x, E y) { a = cfmaconj(x, y, a); }  // conj(x) y
  static __device__ __forceinline__ E fin(const Acc &a) { return a; }
  static __device__ __forceinline__ E im_of(E d) { return cmk(d.y, 0.0); }  // E_ii of a diagonal element
  static __device__ __forceinline__ void set_im(E &d, E e) { d.y = e.x; }
  static __device__ __forceinline__ E real(E d) { return cmk(d.x, 0.0); }
  static __device__ __forceinline__ float dev_re(E v, float id) { return float(v.x - double(id)); }
  static __device__ __forceinline__ float dev_im(E v) { return float(v.y); }
  static __device__ __forceinline__ E neg_over(E g, E e) {  // -g / e for e = 1 + d, |d| <= 1e-4
    const double d = e.x - 1.0;
    return cscale(g, -fma(-d, fma(-d, fma(-d, fma(-d, 1.0, 1.0), 1.0), 1.0), 1.0));
  }
  static __device__ __forceinline__ E over_sqrt(E v, E e) {
    const double d = e.x - 1.0;
    return cscale(v, fma(-d, fma(-d, fma(-d, 0.3125, 0.375), 0.5), 1.0));
  }
};
struct FloqDf {
  static constexpr int kStartMin = 32;
  using E = float4;
  using Acc = CdfAcc;
  static __device__ __forceinline__ E of(float2 v) { return make_float4(v.x, v.y, 0.f, 0.f); }
  static __device__ __forceinline__ float2 narrow(E v) { return make_float2(v.x + v.z, v.y + v.w); }
  static __device__ __forceinline__ E conj(E v) { return make_float4(v.x, -v.y, v.z, -v.w); }
  static __device__ __forceinline__ Acc acc(E v) { return {{v.x, v.z}, {v.y, v.w}}; }
  static __device__ __forceinline__ void mac(Acc &a, E x, E y) { cdf_mac(a, x, y); }
  static __device__ __forceinline__ void macj(Acc &a, E x, E y) { cdf_mac(a, conj(x), y); }
  static __device__ __forceinline__ E fin(const Acc &a) { return cdf_fin(a); }
  static __device__ __forceinline__ E im_of(E d) { return make_float4(d.y, 0.f, d.w, 0.f); }
  static __device__ __forceinline__ void set_im(E &d, E e) { d.y = e.x, d.w = e.z; }
  static __device__ __forceinline__ E real(E d) { return make_float4(d.x, 0.f, d.z, 0.f); }
  static __device__ __forceinline__ float dev_re(E v, float id) { return (v.x - id) + v.z; }
  static __device__ __forceinline__ float dev_im(E v) { return v.y + v.w; }
  static __device__ __forceinline__ E neg_over(E g, E e) {  // -(g - g d (1 - d)), g of the size of d
    const float d = dev_re(e, 1.f), f = d * (1.f - d);
    const float2 re = dfv_add(make_float2(-g.x, -g.z), make_float2(g.x * f, 0.f)),
                 im = dfv_add(make_float2(-g.y, -g.w), make_float2(g.y * f, 0.f));
    return make_float4(re.x, im.x, re.y, im.y);
  }
  static __device__ __forceinline__ E over_sqrt(E v, E e) {
    const float2 d = dfv_add(make_float2(e.x, e.z), make_float2(-1.f, 0.f));
    const float q = d.x * d.x * (0.375f - 0.3125f * d.x);
    const float2 f = dfv_add(make_float2(1.f, 0.f), dfv_add(make_float2(-0.5f * d.x, -0.5f * d.y), make_float2(q, 0.f)));
    const float2 re = dfv_mul(f, make_float2(v.x, v.z)), im = dfv_mul(f, make_float2(v.y, v.w));
    return make_float4(re.x, im.x, re.y, im.y);
  }
};

// Start of the final sweeps: K = V^H K0 V nearly diagonal (Xk) and its V, orthonormal (Mm), from
// the eigenvectors of K0 (Xk on entry) in single precision.  FP64 issues 2 FMAs per clock and SM
// against 128 in FP32, and a double-float product takes about 30 FP32 operations; all sweeps but
// the last ones only bring the off-diagonal down to where single precision leaves it.  Those run
// in FP32 (K and V in Mm's two halves), V is widened and orthonormalised by the Cholesky factor of
// its Gram matrix (which departs from one by ~1e-6: the reciprocals are short series), and K0 is
// transformed: 11 b^3 multiply-adds against 12 b^3 (FP64; V alone in double-float: 6 b^3) for each
// of the ~5 sweeps that it saves.  Where single precision does not deliver (not finite, or far
// from orthonormal), V = I and the final sweeps do all of the work.
// Blocks below kStartMin stay with the final sweeps alone (sizes measured: FP64, blocks of 10, 320 crystallites:
// 0.66 ms against 0.73; blocks of 20 to 35, 7 spins, 144 crystallites: 8.5 -> 3.0 ms.  Double-float,
// blocks of 20, 677 crystallites: 1.08 ms against 1.62; blocks of 28 to 70, 8 spins, 1154
// crystallites: 74 -> 48 ms, with K's off-diagonal left at 1e-10 of its norm instead of 1e-7).
constexpr int kFloqSweeps32 = 12;
constexpr int kFloqPer = 4;  // elements per thread and group of the in-place products (b <= 4 blockDim.x)

// X <- X V by groups of whole rows, in place
template <class A>
__device__ void mul_in_place(typename A::E *X, const typename A::E *V, int b) {
  constexpr int kPer = kFloqPer;
  const int nt = blockDim.x, tid = threadIdx.x, bb = b * b, group = min(b, kPer * nt / b);
  const float invb = 1.f / float(b);
  for (int r0 = 0; r0 < b; r0 += group) {
    typename A::E out[kPer];
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
      int j;
      const int e = tid + t * nt, r = r0 + fdiv(e, invb, b, j);
      if (e < group * b && r < b) {
        auto a = A::acc(A::of(make_float2(0.f, 0.f)));
        for (int l = 0; l < b; ++l) A::mac(a, X[r * b + l], V[l * b + j]);
        out[t] = A::fin(a);
      }
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
      const int e = tid + t * nt;
      if (e < group * b && r0 * b + e < bb) X[r0 * b + e] = out[t];
    }
  }
  __syncthreads();
}

template <class A>
__device__ void floquet_start(typename A::E *Xk, typename A::E *Mm, int b, const FloqWork &wk) {
  using E = typename A::E;
  const int bb = b * b, nt = blockDim.x, tid = threadIdx.x;
  const float invb = 1.f / float(b), invb1 = 1.f / float(b + 1);
  float2 *K32 = reinterpret_cast<float2 *>(Mm), *V32 = K32 + bb;
  auto one = [&](int e) { return make_float2(e % (b + 1) == 0 ? 1.f : 0.f, 0.f); };
  for (int e = tid; e < bb; e += nt) {
    K32[e] = A::narrow(Xk[e]);
    V32[e] = one(e);
  }
  __syncthreads();
  floquet_sweeps(K32, V32, b, kFloqSweeps32, wk);
  __syncthreads();
  // widen in place, upwards: element e's place ends below element e + 1 of V32
  bool bad = false;
  for (int e0 = 0; e0 < bb; e0 += nt) {
    const int e = e0 + tid;
    float2 v = make_float2(0.f, 0.f);
    if (e < bb) v = V32[e];
    bad = bad || !(fabsf(v.x) <= 2.f && fabsf(v.y) <= 2.f);
    __syncthreads();
    if (e < bb) Mm[e] = A::of(v);
  }
  bad = __syncthreads_or(bad);
  // Gram matrix E of V: E_ij (i < j) in Xk's lower triangle (element j, i), E_ii in the diagonal's
  // imaginary parts; K0 stays in the upper triangle
  const int ntri = b * (b + 1) / 2;
  for (int e = tid; e < ntri && !bad; e += nt) {
    int j;
    const int i = tri_pair(e, b, invb1, j);
    auto a = A::acc(A::of(make_float2(0.f, 0.f)));
    for (int r = 0; r < b; ++r) A::macj(a, Mm[r * b + i], Mm[r * b + j]);
    const E g = A::fin(a);
    if (i == j) A::set_im(Xk[i * b + i], g);
    else Xk[j * b + i] = g;
    bad = !(fabsf(A::dev_re(g, i == j ? 1.f : 0.f)) <= 1e-4f && fabsf(A::dev_im(g)) <= 1e-4f);
  }
  bad = __syncthreads_or(bad);
  // V <- V R^-1 with E = R^H R, right-looking: step k takes column k's part out of the columns
  // above it, in V and in what is left of E; the columns' norms follow at the end
  for (int k = 0; k < b - 1 && !bad; ++k) {
    const E piv = A::im_of(Xk[k * b + k]);
    const int w = b - 1 - k, nv = b * w, ng = w * (w + 1) / 2;
    const float invw = 1.f / float(w), invw1 = 1.f / float(w + 1);
    for (int e = tid; e < nv + ng; e += nt) {
      int j;
      if (e < nv) {
        const int r = fdiv(e, invw, w, j);
        j += k + 1;
        auto a = A::acc(Mm[r * b + j]);
        A::mac(a, Mm[r * b + k], A::neg_over(Xk[j * b + k], piv));
        Mm[r * b + j] = A::fin(a);
      } else {
        const int i = k + 1 + tri_pair(e - nv, w, invw1, j);
        j += k + 1;
        auto a = A::acc(i == j ? A::im_of(Xk[i * b + i]) : Xk[j * b + i]);
        A::macj(a, Xk[i * b + k], A::neg_over(Xk[j * b + k], piv));
        if (i == j) A::set_im(Xk[i * b + i], A::fin(a));
        else Xk[j * b + i] = A::fin(a);
      }
    }
    __syncthreads();
  }
  for (int e = tid; e < bb; e += nt) {
    int q;
    fdiv(e, invb, b, q);
    Mm[e] = bad ? A::of(one(e)) : A::over_sqrt(Mm[e], A::im_of(Xk[q * b + q]));
  }
  __syncthreads();
  auto mirror = [&]() {
    for (int e = tid; e < ntri; e += nt) {
      int j;
      const int i = tri_pair(e, b, invb1, j);
      if (i == j) Xk[i * b + i] = A::real(Xk[i * b + i]);
      else Xk[j * b + i] = A::conj(Xk[i * b + j]);
    }
    __syncthreads();
  };
  mirror();
  if (bad) return;
  // Xk <- K0 V by rows, then V^H (K0 V) by groups of columns, in place
  mul_in_place<A>(Xk, Mm, b);
  constexpr int kPer = kFloqPer;
  const int group = min(b, kPer * nt / b);
  for (int j0 = 0; j0 < b; j0 += group) {
    E out[kPer];
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
      int i;
      const int e = tid + t * nt, j = j0 + fdiv(e, invb, b, i);
      if (e < group * b && j < b && i <= j) {
        auto a = A::acc(A::of(make_float2(0.f, 0.f)));
        for (int l = 0; l < b; ++l) A::macj(a, Mm[l * b + i], Xk[l * b + j]);
        out[t] = A::fin(a);
      }
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
      int i;
      const int e = tid + t * nt, j = j0 + fdiv(e, invb, b, i);
      if (e < group * b && j < b && i <= j) Xk[i * b + j] = out[t];
    }
  }
  __syncthreads();
  mirror();
}

// Columns of V scaled to norm 1, a warp per column.  A rotation by an angle below 2^-26 has c = 1 in
// FP64 and lengthens both of its columns by half the angle's square (the sweeps' angles come from single
// precision, so one more sweep has such angles): b rotations a column add up to 1e-14 at b = 126, which
// the FID carries as an amplitude (9 spins, one crystallite, n = 24, against 80-bit propagation:
// 1.2e-14 without and 1.0e-15 with the scaling).
__device__ __forceinline__ void unit_columns(double2 *V, int b) {
  for (int q = threadIdx.x >> 5; q < b; q += blockDim.x >> 5) {
    double d = 0;
    for (int r = threadIdx.x & 31; r < b; r += 32) {
      const double2 v = V[r * b + q];
      d = fma(v.x, v.x, fma(v.y, v.y, d));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
    const double f = 0.5 * (1.0 - d);  // d^-1/2 - 1 (d - 1 ~ 1e-14)
    for (int r = threadIdx.x & 31; r < b; r += 32) {
      V[r * b + q].x = fma(V[r * b + q].x, f, V[r * b + q].x);
      V[r * b + q].y = fma(V[r * b + q].y, f, V[r * b + q].y);
    }
  }
  __syncthreads();
}

// DFA: A_n is double-float (mixed form); START: the sweeps begin with floquet_start.
template <bool DFA, bool START>
__device__ void floquet_cta(const DevSys &s, int k, int c, FloqWork wk) {
  constexpr bool dfA = DFA;
  __shared__ int piv_s;
  __shared__ double a_s;
  __shared__ int done_s;
  const int b = s.bs[k], bp = s.bpoff[k], bo = s.boff[k], bb = b * b;
  double2 *Mm = wk.Mm, *Xk = wk.Xk, *fv = wk.fv, *lam = wk.lam;
  double *red = wk.red;
  const double2 *U = period_prop(s, b);  // U(r,q) = U[at(bp + r*b + q, c)]
  const float4 *U4 = reinterpret_cast<const float4 *>(U);      // dfA: double-float A (mixed form)
  auto Ug = [&](int r, int q) {
    return dfA ? df_load(U4[big_at(s, b, bp, r * b + q, c)]) : U[big_at(s, b, bp, r * b + q, c)];
  };
  if (threadIdx.x == 0) a_s = 0.5, done_s = 0;
  __syncthreads();
  for (int pass = 0; pass < 2; ++pass) {
    double sa, ca;
    sincos(a_s, &sa, &ca);
    const double2 ea = cmk(ca, sa);
    for (int e = threadIdx.x; e < bb; e += blockDim.x) {
      const double2 w = cmul(ea, Ug(e / b, e % b));
      const double id = (e / b == e % b) ? 1.0 : 0.0;
      Mm[e] = cmk(id + w.x, w.y);
      Xk[e] = cmk(id - w.x, -w.y);
    }
    __syncthreads();
    // Gaussian elimination with partial pivoting: Mm Xk' = Xk
    for (int kc = 0; kc < b; ++kc) {
      if (threadIdx.x == 0) {
        int pv = kc;
        double best = -1;
        for (int r = kc; r < b; ++r) {
          const double2 v = Mm[r * b + kc];
          const double m2 = v.x * v.x + v.y * v.y;
          if (m2 > best) best = m2, pv = r;
        }
        piv_s = pv;
        if (best == 0.0) atomicOr(s.status, kSingularCayley);
      }
      __syncthreads();
      const int pv = piv_s;
      if (pv != kc)
        for (int j = threadIdx.x; j < 2 * b; j += blockDim.x) {
          double2 *Mx = j < b ? Mm : Xk;
          const int jj = j < b ? j : j - b;
          const double2 t = Mx[kc * b + jj];
          Mx[kc * b + jj] = Mx[pv * b + jj];
          Mx[pv * b + jj] = t;
        }
      __syncthreads();
      const double2 inv = cdiv(cmk(1, 0), Mm[kc * b + kc]);
      for (int r = kc + 1 + threadIdx.x; r < b; r += blockDim.x) fv[r] = cmul(Mm[r * b + kc], inv);
      __syncthreads();
      const int rows = b - kc - 1;
      for (int e = threadIdx.x; e < rows * (2 * b); e += blockDim.x) {
        const int r = kc + 1 + e / (2 * b), j = e % (2 * b);
        if (j < b) {
          if (j > kc) Mm[r * b + j] = csub(Mm[r * b + j], cmul(fv[r], Mm[kc * b + j]));
        } else {
          Xk[r * b + (j - b)] = csub(Xk[r * b + (j - b)], cmul(fv[r], Xk[kc * b + (j - b)]));
        }
      }
      __syncthreads();
    }
    for (int kr = b - 1; kr >= 0; --kr) {  // back substitution, all rows above at once
      const double2 inv = cdiv(cmk(1, 0), Mm[kr * b + kr]);
      for (int j = threadIdx.x; j < b; j += blockDim.x) Xk[kr * b + j] = cmul(Xk[kr * b + j], inv);
      __syncthreads();
      for (int e = threadIdx.x; e < kr * b; e += blockDim.x) {
        int j;
        const int r = fdiv(e, 1.f / float(b), b, j);
        Xk[e] = csub(Xk[e], cmul(Mm[r * b + kr], Xk[kr * b + j]));
      }
      __syncthreads();
    }
    // K = Hermitian part of i X, in Xk
    for (int e = threadIdx.x; e < bb; e += blockDim.x) {
      const int r = e / b, q = e % b;
      if (r <= q) {
        const double2 xrq = Xk[r * b + q], xqr = Xk[q * b + r];
        const double2 krq = cmk(-xrq.y, xrq.x), kqr = cmk(-xqr.y, xqr.x);
        const double2 h = cscale(cadd(krq, cconj(kqr)), 0.5);
        Xk[r * b + q] = h;
        Xk[q * b + r] = cconj(h);
      }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < b; e += blockDim.x) Xk[e * b + e].y = 0.0;
    __syncthreads();
    if constexpr (START) {
      floquet_start<FloqF64>(Xk, Mm, b, wk);
    } else {
      for (int e = threadIdx.x; e < bb; e += blockDim.x) Mm[e] = cmk(e / b == e % b ? 1.0 : 0.0, 0.0);
      __syncthreads();
    }
    const bool conv = floquet_sweeps(Xk, Mm, b, kMaxSweeps, wk);
    if (!conv) atomicOr(s.status, kNoConvergeFloquet);
    unit_columns(Mm, b);
    // Rayleigh quotients lam_r = v_r^H (U V)_r, U V in Xk (K is done with)
    for (int e = threadIdx.x; e < bb; e += blockDim.x) Xk[e] = Ug(e / b, e % b);
    __syncthreads();
    mul_in_place<FloqF64>(Xk, Mm, b);
    for (int r = threadIdx.x; r < b; r += blockDim.x) {
      double2 acc = cmk(0, 0);
      for (int kk = 0; kk < b; ++kk) acc = cfmaconj(Mm[kk * b + r], Xk[kk * b + r], acc);
      lam[r] = acc;
    }
    __syncthreads();
    if (pass == 1) break;
    if (threadIdx.x == 0) {
      double mind = 4.0;
      for (int r = 0; r < b; ++r) {
        const double2 w = cmul(ea, lam[r]);
        mind = fmin(mind, (1.0 + w.x) * (1.0 + w.x) + w.y * w.y);
      }
      done_s = conv && mind >= 0.0625;
      if (!done_s) {
        // widest gap of the eigenphases: sort them (insertion sort into red[])
        for (int r = 0; r < b; ++r) {
          const double th = atan2(lam[r].y, lam[r].x);
          int j = r;
          while (j > 0 && red[j - 1] > th) red[j] = red[j - 1], --j;
          red[j] = th;
        }
        double best = -1, mid = 0;
        for (int r = 0; r < b; ++r) {
          const double lo = red[r], hi = (r + 1 < b) ? red[r + 1] : red[0] + kPi2;
          if (hi - lo > best) best = hi - lo, mid = 0.5 * (lo + hi);
        }
        a_s = kPi - mid;
      }
    }
    __syncthreads();
    if (done_s) break;
  }
  for (int e = threadIdx.x; e < bb; e += blockDim.x) s.VF[at(bp + e, c, s.Cpad)] = Mm[e];
  for (int r = threadIdx.x; r < b; r += blockDim.x)
    s.L[at(bo + r, c, s.Cpad)] = cmk(log(hypot(lam[r].x, lam[r].y)), atan2(lam[r].y, lam[r].x));
}

template <bool START>
__device__ void floquet_cta_df(const DevSys &s, int k, int c, FloqWork wk, bool a64 = false);

// One CTA per crystallite: unitary eigen-decomposition of a large block of A_n.  DF: the mixed
// form's double-float path (K in single precision after the two b x b arrays).  The variants are
// kernels of their own: floquet_start's registers would cost the small blocks their occupancy.
template <bool DF, bool DFA, bool START>
__global__ void __launch_bounds__(START ? kBigThreads : 256) k_big_floquet(DevSys s, int k) {
  extern __shared__ double2 bsc[];
  __shared__ double2 rot[(kMaxBigBlock / 2 + 1) * 2];  // (c, 0), (s e^{i ph}) per pair
  __shared__ int rpair[(kMaxBigBlock / 2 + 1) * 2];
  __shared__ double2 fv[kMaxBigBlock];
  __shared__ double2 lam[kMaxBigBlock];
  __shared__ double red[START ? kBigThreads : 256];
  const int b = s.bs[k];
  const FloqWork wk{bsc, bsc + b * b, rot, fv, lam, rpair, red, reinterpret_cast<float2 *>(bsc + 2 * b * b)};
  if constexpr (DF) floquet_cta_df<START>(s, k, blockIdx.x, wk);
  else floquet_cta<DFA, START>(s, k, blockIdx.x, wk);
}

// ------------------------------------------------------------------ mixed form, double-float
// The large-block step and Dyson of the mixed form in double-float on the FP32 pipe (float2 =
// hi, lo; complex elements float4 = re.hi, im.hi, re.lo, im.lo), with the same tiling as the
// FP64 kernels and sums as compensated dot products.

// C = ep(e, A B) for symmetric commuting A, B (upper tiles, mirrored; e the upper element),
// double-float.
template <class EP>
__device__ void cta_mm_sym_df(const float2 *A, const float2 *B, float2 *C, int m, EP ep) {
  const int tm = (m + 1) / 2;
  for (int t = threadIdx.x; t < big_sym_tiles(m); t += blockDim.x) {
    int ti, tj;
    sym_tile(t, tm, ti, tj);
    const int i0 = 2 * ti, j0 = 2 * tj;
    const int i1 = min(i0 + 1, m - 1), j1 = min(j0 + 1, m - 1);
    DfAcc c00 = {0.f, 0.f}, c01 = c00, c10 = c00, c11 = c00;
    for (int l = 0; l < m; ++l) {
      const float2 a0 = A[i0 * m + l], a1 = A[i1 * m + l], b0 = B[l * m + j0], b1 = B[l * m + j1];
      df_dot(c00, a0.x, a0.y, b0.x, b0.y);
      df_dot(c01, a0.x, a0.y, b1.x, b1.y);
      df_dot(c10, a1.x, a1.y, b0.x, b0.y);
      df_dot(c11, a1.x, a1.y, b1.x, b1.y);
    }
    auto put = [&](int i, int j, const DfAcc &v) {
      const float2 x = ep(i * m + j, df_fin(v));
      C[i * m + j] = x;
      if (i != j) C[j * m + i] = x;
    };
    put(i0, j0, c00);
    if (j0 + 1 < m) put(i0, j0 + 1, c01);
    if (i0 + 1 < m) {
      if (ti != tj) put(i0 + 1, j0, c10);
      if (j0 + 1 < m) put(i0 + 1, j0 + 1, c11);
    }
  }
}

// coefficients of cos X = sum c_j Y^j and sin X = X sum s_j Y^j (Y = X^2), double-float
__constant__ float2 kCosDf[8] = {dfv_const(cos_coef(0)), dfv_const(cos_coef(1)), dfv_const(cos_coef(2)),
                                 dfv_const(cos_coef(3)), dfv_const(cos_coef(4)), dfv_const(cos_coef(5)),
                                 dfv_const(cos_coef(6)), dfv_const(cos_coef(7))};
__constant__ float2 kInvDf[8] = {dfv_const(1.0),     dfv_const(1.0),     dfv_const(1.0 / 2), dfv_const(1.0 / 3),
                                 dfv_const(1.0 / 4), dfv_const(1.0 / 5), dfv_const(1.0 / 6), dfv_const(1.0 / 7)};
__constant__ float2 kSinDf[8] = {dfv_const(sin_coef(0)), dfv_const(sin_coef(1)), dfv_const(sin_coef(2)),
                                 dfv_const(sin_coef(3)), dfv_const(sin_coef(4)), dfv_const(sin_coef(5)),
                                 dfv_const(sin_coef(6)), dfv_const(sin_coef(7))};

__host__ __device__ constexpr size_t big_step_df_smem(int b) { return sizeof(float2) * 5 * size_t(b) * size_t(b); }

// One CTA per (crystallite, step): the large block's U_i in double-float: H from the hi/lo
// tables, cos X and sin X to the degree K that taylor_degree gives at 2^-40 by
// Paterson-Stockmeyer in Y^2 (Y = X^2): the degree-2 chunks c_2j + c_2j+1 Y (the highest one with
// c_2j+2 Y^2 where the degree is even) by Horner's rule, so degree 2 of C or S takes no product
// own, 4 one, 6 two; K = 9 takes 5 products where the series term by term takes 8 (8
// spins, 1154 crystallites, n = 200, blocks of 28: all steps 193 -> 180 ms; up to K = 7 the series
// is kept, 6 spins at n = 231 took 7.87 ms by it and 8.12 this way).  The sine comes first, so that X's
// buffer is free for the cosine: five b x b buffers as before.
__global__ void __launch_bounds__(1024) k_big_step_df(DevSys s, int k) {
  extern __shared__ __align__(16) unsigned char bsd[];
  __shared__ float2 fk[kMaxInt];
  __shared__ float red[kMaxBigBlock];
  __shared__ float2 scl;
  __shared__ int nsq, nterms;
  const int c = blockIdx.x % s.C, i = blockIdx.x / s.C;
  const int b = s.bs[k], bp = s.bpoff[k], bb = b * b;
  if (s.fk) {  // k_coef's coefficients: hi/lo pairs after the Taylor step, doubles after eigh
    const float2 *fk2 = reinterpret_cast<const float2 *>(s.fk);
    for (int kk = threadIdx.x; kk < s.nint; kk += blockDim.x) {
      const size_t a = at(i * s.nint + kk, c, s.Cpad);
      fk[kk] = s.fk_df ? fk2[a] : dfv_of(s.fk[a]);
    }
  } else if (threadIdx.x == 0) {
    double t1 = s.t0[c] + double(i) * s.tau, t2 = t1 + s.tau;
    double tmid = (t2 - t1) / 2.0 + t1;
    double sp, cp;
    sincos(tmid * s.wr * kPi2, &sp, &cp);
    double m[3][3];
    orient_rows(s, c, sp, cp, m);
    for (int kk = 0; kk < s.nint; ++kk) fk[kk] = dfv_of(term_coef(s, kk, m));
  }
  __syncthreads();
  float2 *X = reinterpret_cast<float2 *>(bsd), *P = X + bb, *Q = P + bb, *R = Q + bb, *I = R + bb;
  const float2 *Hcb = s.Hc_df + (s.hc_chunks ? size_t(i / s.psub) * s.S2 : 0) + bp;
  for (int x = threadIdx.x; x < bb; x += blockDim.x) {  // each element's own terms, longest first
    const int e = s.tk_order[bp + x];
    float2 h = Hcb[e];
    for (int t = s.tk_ptr[bp + e]; t < s.tk_ptr[bp + e + 1]; ++t)
      h = dfv_add(h, dfv_mul(fk[s.tk_term[t]], s.tk_val[t]));
    X[e] = h;
  }
  __syncthreads();
  for (int p = threadIdx.x; p < b; p += blockDim.x) {
    float rs = 0.f;
    for (int q = 0; q < b; ++q) rs += fabsf(X[p * b + q].x);
    red[p] = rs;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float nrm = 0.f;
    for (int p = 0; p < b; ++p) nrm = fmaxf(nrm, red[p]);
    nrm *= float(s.tau * kPi2) * (1.f + 1e-6f);
    int sq = 0;
    if (nrm > 0.5f) {
      frexpf(nrm / 0.5f, &sq);
      sq = min(sq, 60);
    }
    scl = make_float2(ldexpf(s.tpdf.x, -sq), ldexpf(s.tpdf.y, -sq));
    nsq = sq;
    nterms = taylor_degree(double(ldexpf(nrm, -sq)), true);
  }
  __syncthreads();
  const float2 sc = scl;
  const int sq = nsq, K = nterms;
  const auto keep = [](int, float2 v) { return v; };
  float2 *Y = R, *Y2 = I, *A = P, *B = Q;  // and X
  for (int e = threadIdx.x; e < bb; e += blockDim.x) X[e] = dfv_mul(sc, X[e]);
  __syncthreads();
  float2 *F[3];  // the three buffers that do not hold the result
  if (K <= 7) {  // few terms: the series, one product a term (the chunks' sums would cost one product)
    for (int e = threadIdx.x; e < bb; e += blockDim.x) {
      const float2 x = X[e];
      P[e] = x, R[e] = make_float2((e / b == e % b) ? 1.f : 0.f, 0.f), I[e] = make_float2(-x.x, -x.y);
    }
    __syncthreads();
    for (int kt = 2; kt <= K; ++kt) {
      const float2 ik = kInvDf[kt];
      const int m4 = kt & 3;
      cta_mm_sym_df(P, X, Q, b, [&](int, float2 v) { return dfv_mul(ik, v); });
      __syncthreads();
      for (int e = threadIdx.x; e < bb; e += blockDim.x) {
        const float2 v = Q[e], nv = make_float2(-v.x, -v.y);
        if (m4 == 2) R[e] = dfv_add(R[e], nv);
        else if (m4 == 3) I[e] = dfv_add(I[e], v);
        else if (m4 == 0) R[e] = dfv_add(R[e], v);
        else I[e] = dfv_add(I[e], nv);
      }
      float2 *t = P;
      P = Q, Q = t;
      __syncthreads();
    }
    F[0] = P, F[1] = Q, F[2] = X;
  } else {
  cta_mm_sym_df(X, X, Y, b, keep);
  __syncthreads();
  cta_mm_sym_df(Y, Y, Y2, b, keep);
  __syncthreads();
  // sum_j coef_j Y^j, j <= d, in buffer u or v; returns which
  auto poly = [&](const float2 *coef, int d, float2 *u, float2 *v) -> float2 * {
    const int top = d >= 2 && d % 2 == 0 ? d / 2 - 1 : d / 2;  // chunk that starts the recurrence
    const float2 zero = make_float2(0.f, 0.f);
    const float2 c0 = coef[2 * top], c1 = 2 * top + 1 <= d ? coef[2 * top + 1] : zero,
                 c2 = 2 * top + 2 <= d ? coef[2 * top + 2] : zero;
    for (int e = threadIdx.x; e < bb; e += blockDim.x) {
      float2 x = dfv_mul(c1, Y[e]);
      if (2 * top + 2 <= d) x = dfv_add(x, dfv_mul(c2, Y2[e]));
      u[e] = e / b == e % b ? dfv_add(x, c0) : x;
    }
    __syncthreads();
    for (int t = top - 1; t >= 0; --t) {
      const float2 l0 = coef[2 * t], l1 = coef[2 * t + 1];
      cta_mm_sym_df(Y2, u, v, b, [&](int e, float2 x) {
        x = dfv_add(x, dfv_mul(l1, Y[e]));
        return e / b == e % b ? dfv_add(x, l0) : x;
      });
      __syncthreads();
      float2 *w = u;
      u = v, v = w;
    }
    return u;
  };
  {
    float2 *S = poly(kSinDf, (K - 1) / 2, A, B);
    I = S == A ? B : A;  // -sin X = -X S(Y)
    cta_mm_sym_df(X, S, I, b, [](int, float2 v) { return make_float2(-v.x, -v.y); });
    __syncthreads();
    R = poly(kCosDf, K / 2, X, S);
  }
  F[0] = Y, F[1] = Y2, F[2] = R == X ? (I == A ? B : A) : X;
  }
  // squarings: (R + iI)^2 = (RR - II) + i 2RI, in the three other buffers
  {
    for (int t = 0; t < sq; ++t) {
      cta_mm_sym_df(R, R, F[0], b, keep);
      cta_mm_sym_df(I, I, F[1], b, keep);
      cta_mm_sym_df(R, I, F[2], b, [](int, float2 v) { return make_float2(2.f * v.x, 2.f * v.y); });
      __syncthreads();
      for (int e = threadIdx.x; e < bb; e += blockDim.x) {
        const float2 q = F[1][e];
        R[e] = dfv_add(F[0][e], make_float2(-q.x, -q.y)), I[e] = F[2][e];
      }
      __syncthreads();
    }
  }
  double2 *Ub = s.U + size_t(i) * s.S2 * s.Cpad;
  float4 *U4 = reinterpret_cast<float4 *>(Ub);
  const double2 *fr = frame_of(s, i);
  const int bo = s.boff[k];
  for (int e = threadIdx.x; e < bb; e += blockDim.x) {
    const float2 re = R[e], im = I[e];
    if (fr) {  // rf schedule frames: through FP64
      const double2 u = cmk(double(re.x) + double(re.y), double(im.x) + double(im.y));
      U4[at(bp + e, c, s.Cpad)] = df_store(cmul(cmul(fr[bo + e / b], u), cconj(fr[bo + e % b])));
    } else {
      U4[at(bp + e, c, s.Cpad)] = make_float4(re.x, im.x, re.y, im.y);
    }
  }
}

// The segment's (or prefix) products in double-float, 2 x 2 tiles per thread.
template <int NT>
__global__ void __launch_bounds__(NT == 1 ? 1024 : 768) k_big_dyson_df(DevSys s, int k, bool prefix) {
  extern __shared__ __align__(16) unsigned char bsy[];
  const int c = blockIdx.x % s.C;
  const int b = s.bs[k], bp = s.bpoff[k], bb = b * b;
  float4 *Us = reinterpret_cast<float4 *>(bsy), *As = Us + bb;
  for (int e = threadIdx.x; e < bb; e += blockDim.x) As[e] = make_float4(e / b == e % b ? 1.f : 0.f, 0.f, 0.f, 0.f);
  const int tm = (b + 1) / 2;
  const Chain ch = seg_chain(s, b, blockIdx.x / s.C, prefix);
  for (int i = 0; i < ch.count; ++i) {
    const float4 *Ub = reinterpret_cast<const float4 *>(ch.from(s, i));
    // U lies [item][c]; the segments' products crystallite-major (big_at)
    for (int e = threadIdx.x; e < bb; e += blockDim.x)
      Us[e] = Ub[prefix ? big_at(s, b, bp, e, c) : at(bp + e, c, s.Cpad)];
    __syncthreads();
    float4 out[NT][4];
#pragma unroll
    for (int q = 0; q < NT; ++q) {
      const int t = threadIdx.x + q * blockDim.x;
      if (t >= tm * tm) continue;
      const int i0 = (t / tm) * 2, j0 = (t % tm) * 2;
      const int i1 = min(i0 + 1, b - 1), j1 = min(j0 + 1, b - 1);
      CdfAcc c00 = {{0.f, 0.f}, {0.f, 0.f}}, c01 = c00, c10 = c00, c11 = c00;
      for (int l = 0; l < b; ++l) {
        const float4 a0 = Us[i0 * b + l], a1 = Us[i1 * b + l], b0 = As[l * b + j0], b1 = As[l * b + j1];
        cdf_mac(c00, a0, b0), cdf_mac(c01, a0, b1), cdf_mac(c10, a1, b0), cdf_mac(c11, a1, b1);
      }
      out[q][0] = cdf_fin(c00), out[q][1] = cdf_fin(c01), out[q][2] = cdf_fin(c10), out[q][3] = cdf_fin(c11);
    }
    __syncthreads();
    float4 *Ab = reinterpret_cast<float4 *>(ch.to(s, i));
#pragma unroll
    for (int q = 0; q < NT; ++q) {
      const int t = threadIdx.x + q * blockDim.x;
      if (t >= tm * tm) continue;
      const int i0 = (t / tm) * 2, j0 = (t % tm) * 2;
      for (int d = 0; d < 4; ++d) {
        const int r = i0 + (d >> 1), col = j0 + (d & 1);
        if (r < b && col < b) {
          As[r * b + col] = out[q][d];
          Ab[big_at(s, b, bp, r * b + col, c)] = out[q][d];
        }
      }
    }
    __syncthreads();
  }
}


// ------------------------------------------------------------------ mixed form, Floquet step
// floquet_cta's algorithm for the mixed form's large blocks when the FID spans at most
// kFloq32MaxPeriods periods, with every FP64 part moved to double-float on the FP32 pipe
// (GB300 issues about 2 FP64 FMAs per clock per SM against 128 FP32 FMAs): the Cayley
// transform, by Gauss-Jordan elimination with partial pivoting (the pivot search is a warp
// reduction; every update is parallel, no serial back substitution); V's accumulation of the
// Jacobi rotations, each rotation renormalised in double-float to c^2 + |s|^2 = 1; and the
// Rayleigh quotients lam_r = v_r^H A_n v_r through the CTA-wide product A_n V.  The sweeps over
// K run in FP32 with floquet_sweeps' rules.  Complex double-float elements are float4
// (re.hi, im.hi, re.lo, im.lo) in the 16-byte slots of the FP64 work arrays; the results
// (V, ln lambda) are stored in FP64 as by floquet_cta.

// The sweeps over the FP32 K (Kf) with V (double-float, Vd) accumulating the rotations.
__device__ bool floquet_sweeps_df(float2 *Xk, float4 *Vd, int b, int max_sweeps, const FloqWork &wk) {
  float4 *rot = reinterpret_cast<float4 *>(wk.rot);  // per pair: (c.hi, 0, c.lo, 0), (s as complex df)
  auto rpair = [&](int t, int q) -> int & { return wk.rpair[2 * t + q]; };
  double *red = wk.red;
  const int bb = b * b;
  const float invb = 1.f / float(b);
  const int bq = b + (b & 1);
  const int np = bq / 2;
  bool conv = false, polish = false;
  const int nw = (blockDim.x + 31) / 32, wid = threadIdx.x >> 5, lid = threadIdx.x & 31;
  for (int sweep = 0; sweep < max_sweeps && !conv; ++sweep) {
    // off(K)^2 and diag(K)^2 for the stopping test: FP32 sums per thread (K is FP32), a fixed
    // shuffle tree per warp, the warps' sums added in FP64 by one thread
    float off = 0.f, dg = 0.f;
    for (int e = threadIdx.x; e < bb; e += blockDim.x) {
      int q;
      const int r = fdiv(e, invb, b, q);
      const float2 v = Xk[e];
      if (r < q) off = fmaf(v.x, v.x, fmaf(v.y, v.y, off));
      else if (r == q) dg = fmaf(v.x, v.x, dg);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      off += __shfl_xor_sync(0xffffffffu, off, o);
      dg += __shfl_xor_sync(0xffffffffu, dg, o);
    }
    if (lid == 0) red[2 * wid] = off, red[2 * wid + 1] = dg;
    __syncthreads();
    if (threadIdx.x == 0) {
      double so = 0, sd = 0;
      for (int t = 0; t < nw; ++t) so += red[2 * t], sd += red[2 * t + 1];
      red[2 * nw] = so, red[2 * nw + 1] = sd;
    }
    __syncthreads();
    const double offs = red[2 * nw], dgs = red[2 * nw + 1];
    __syncthreads();
    const bool small = offs <= 1e-10 * dgs || offs == 0.0;
    if (small && (polish || offs == 0.0)) {
      conv = true;
      break;
    }
    polish = polish || small;
    for (int round = 0; round < bq - 1; ++round) {
      for (int t = threadIdx.x; t < np; t += blockDim.x) {
        auto player = [&](int j) { return j == 0 ? 0 : 1 + (j - 1 + round) % (bq - 1); };
        int p = player(t), q = player(bq - 1 - t);
        if (p > q) {
          const int tmp = p;
          p = q, q = tmp;
        }
        rpair(t, 0) = p, rpair(t, 1) = q;
        float4 cr = make_float4(1.f, 0.f, 0.f, 0.f), sr = make_float4(0.f, 0.f, 0.f, 0.f);
        if (q < b) {
          const float2 hpq = Xk[p * b + q];
          const float ab = hypotf(hpq.x, hpq.y);
          if (ab > kSweepTiny) {  // (a denormal element's phase has too few bits to be a rotation's)
            const float phx = hpq.x / ab, phy = hpq.y / ab;
            const float theta = 0.5f * (Xk[q * b + q].x - Xk[p * b + p].x) / ab;
            float tt;
            if (fabsf(theta) > 1e18f) tt = 0.5f / theta;
            else tt = copysignf(1.f, theta) / (fabsf(theta) + sqrtf(fmaf(theta, theta, 1.f)));
            const float cc = rsqrtf(fmaf(tt, tt, 1.f));
            const float sx = phx * (tt * cc), sy = phy * (tt * cc);
            // renormalise: n2 = c^2 + |s|^2 in double-float (exact products), nn = n2^-1/2
            // = 1 - d/2 + 3d^2/8 with d = n2 - 1 (|d| ~ 1e-7)
            DfAcc n2 = {0.f, 0.f};
            df_dot(n2, cc, 0.f, cc, 0.f);
            df_dot(n2, sx, 0.f, sx, 0.f);
            df_dot(n2, sy, 0.f, sy, 0.f);
            const float2 nv = df_fin(n2);
            const float d = __fadd_rn(__fsub_rn(nv.x, 1.f), nv.y);
            const float2 nn = dfv_add(make_float2(1.f, 0.f), make_float2(fmaf(0.375f * d, d, -0.5f * d), 0.f));
            const float2 c2 = dfv_mul(nn, make_float2(cc, 0.f)), s2x = dfv_mul(nn, make_float2(sx, 0.f)),
                         s2y = dfv_mul(nn, make_float2(sy, 0.f));
            cr = make_float4(c2.x, 0.f, c2.y, 0.f);
            sr = make_float4(s2x.x, s2y.x, s2x.y, s2y.y);
          }
        }
        rot[2 * t] = cr, rot[2 * t + 1] = sr;
      }
      __syncthreads();
      // columns p, q of K (FP32) and of V (double-float): X <- X G, G = [[c, sp], [-conj(sp), c]];
      // one (pair, row) per iteration updates both; the pair index runs fastest, so a warp's
      // accesses stay within one row of K and of V
      for (int e = threadIdx.x; e < np * b; e += blockDim.x) {
        const int t = e % np, kk = e / np;
        const int p = rpair(t, 0), q = rpair(t, 1);
        if (q >= b) continue;
        const float4 cr = rot[2 * t], sp = rot[2 * t + 1];
        {
          const float ccr = cr.x + cr.z;
          const float2 spr = make_float2(sp.x + sp.z, sp.y + sp.w), spcr = cconj(spr);
          const float2 xkp = Xk[kk * b + p], xkq = Xk[kk * b + q];
          Xk[kk * b + p] = csub(cscale(xkp, ccr), cmul(spcr, xkq));
          Xk[kk * b + q] = cadd(cmul(spr, xkp), cscale(xkq, ccr));
        }
        {
          const float4 vp = Vd[kk * b + p], vq = Vd[kk * b + q];
          // vp' = c vp - conj(sp) vq,  vq' = sp vp + c vq
          CdfAcc ap = {{0.f, 0.f}, {0.f, 0.f}}, aq = ap;
          cdf_mac(ap, cr, vp);
          cdf_mac(ap, make_float4(-sp.x, sp.y, -sp.z, sp.w), vq);
          cdf_mac(aq, sp, vp);
          cdf_mac(aq, cr, vq);
          Vd[kk * b + p] = cdf_fin(ap);
          Vd[kk * b + q] = cdf_fin(aq);
        }
      }
      __syncthreads();
      // rows p, q of K:  K <- G^H K
      for (int e = threadIdx.x; e < np * b; e += blockDim.x) {
        int kk;
        const int t = fdiv(e, invb, b, kk);
        const int p = rpair(t, 0), q = rpair(t, 1);
        if (q >= b) continue;
        const float4 cr = rot[2 * t], s4 = rot[2 * t + 1];
        const float cc = cr.x + cr.z;
        const float2 sp = make_float2(s4.x + s4.z, s4.y + s4.w), spc = cconj(sp);
        const float2 xpk = Xk[p * b + kk], xqk = Xk[q * b + kk];
        float2 np_ = csub(cscale(xpk, cc), cmul(sp, xqk)), nq_ = cadd(cmul(spc, xpk), cscale(xqk, cc));
        // a non-trivial rotation zeroes K_pq, K_qp and the imaginary parts of K_pp, K_qq
        if ((kk == p || kk == q) && !(s4.x == 0.f && s4.y == 0.f)) {
          if (kk == p) np_.y = 0.f, nq_ = make_float2(0.f, 0.f);
          else np_ = make_float2(0.f, 0.f), nq_.y = 0.f;
        }
        Xk[p * b + kk] = np_;
        Xk[q * b + kk] = nq_;
      }
      __syncthreads();
    }
  }
  return conv;
}

// a64: A_n is FP64 (double2, the huge-block path's storage) instead of double-float
template <bool START>
__device__ void floquet_cta_df(const DevSys &s, int k, int c, FloqWork wk, bool a64) {
  __shared__ int piv_s;
  __shared__ double a_s;
  __shared__ int done_s;
  __shared__ float4 inv_s;
  const int b = s.bs[k], bp = s.bpoff[k], bo = s.boff[k], bb = b * b;
  float4 *M4 = reinterpret_cast<float4 *>(wk.Mm), *X4 = reinterpret_cast<float4 *>(wk.Xk);
  float4 *fv = reinterpret_cast<float4 *>(wk.fv);
  double2 *lam = wk.lam;
  double *red = wk.red;
  float2 *Kf = wk.Kf;
  const double2 *An = period_prop(s, b);
  const float4 *U4 = reinterpret_cast<const float4 *>(An);
  auto Ug = [&](int r, int q) {
    return a64 ? df_store(An[at(bp + r * b + q, c, s.Cpad)]) : U4[big_at(s, b, bp, r * b + q, c)];
  };
  if (threadIdx.x == 0) a_s = 0.5, done_s = 0;
  __syncthreads();
  for (int pass = 0; pass < 2; ++pass) {
    double sa, ca;
    sincos(a_s, &sa, &ca);
    const float4 ea = df_store(cmk(ca, sa));
    // M = I + e^{ia} A_n, X = I - e^{ia} A_n
    for (int e = threadIdx.x; e < bb; e += blockDim.x) {
      const float4 w = cdf_mul(ea, Ug(e / b, e % b));
      const float id = (e / b == e % b) ? 1.f : 0.f;
      const float2 re = dfv_add(make_float2(id, 0.f), make_float2(w.x, w.z));
      const float2 mre = dfv_add(make_float2(id, 0.f), make_float2(-w.x, -w.z));
      M4[e] = make_float4(re.x, w.y, re.y, w.w);
      X4[e] = make_float4(mre.x, -w.y, mre.y, -w.w);
    }
    __syncthreads();
    // Gauss-Jordan with partial pivoting: M X' = X, then X' = diag(M)^-1 X
    for (int kc = 0; kc < b; ++kc) {
      if (threadIdx.x < 32) {
        float best = -1.f;
        int pv = kc;
        for (int r = kc + threadIdx.x; r < b; r += 32) {
          const float4 v = M4[r * b + kc];
          const float m2 = v.x * v.x + v.y * v.y;
          if (m2 > best) best = m2, pv = r;
        }
        for (int o = 16; o; o >>= 1) {
          const float ob = __shfl_xor_sync(0xffffffffu, best, o);
          const int op = __shfl_xor_sync(0xffffffffu, pv, o);
          if (ob > best || (ob == best && op < pv)) best = ob, pv = op;
        }
        if (threadIdx.x == 0) {
          piv_s = pv;
          if (!(best > 0.f)) atomicOr(s.status, kSingularCayley);
        }
      }
      __syncthreads();
      const int pv = piv_s;
      if (pv != kc)
        for (int j = threadIdx.x; j < 2 * b; j += blockDim.x) {
          float4 *Mx = j < b ? M4 : X4;
          const int jj = j < b ? j : j - b;
          const float4 t = Mx[kc * b + jj];
          Mx[kc * b + jj] = Mx[pv * b + jj];
          Mx[pv * b + jj] = t;
        }
      __syncthreads();
      if (threadIdx.x == 0) {
        const double2 piv = df_load(M4[kc * b + kc]);
        inv_s = (piv.x != 0.0 || piv.y != 0.0) ? df_store(cdiv(cmk(1, 0), piv)) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
      __syncthreads();
      const float4 inv = inv_s;
      for (int r = threadIdx.x; r < b; r += blockDim.x) fv[r] = r == kc ? make_float4(0.f, 0.f, 0.f, 0.f) : cdf_mul(M4[r * b + kc], inv);
      __syncthreads();
      const int wM = b - kc - 1, w = wM + b;  // columns kc+1..b-1 of M, all of X
      const float invw = 1.f / float(w);
      for (int e = threadIdx.x; e < (b - 1) * w; e += blockDim.x) {
        int j;
        int r = fdiv(e, invw, w, j);
        r += (r >= kc);
        if (j < wM) M4[r * b + kc + 1 + j] = cdf_fms(M4[r * b + kc + 1 + j], fv[r], M4[kc * b + kc + 1 + j]);
        else X4[r * b + (j - wM)] = cdf_fms(X4[r * b + (j - wM)], fv[r], X4[kc * b + (j - wM)]);
      }
      __syncthreads();
    }
    // X' = diag(M)^-1 X, then K = Hermitian part of i X'
    for (int r = threadIdx.x; r < b; r += blockDim.x) {
      const double2 d = df_load(M4[r * b + r]);
      fv[r] = df_store(cdiv(cmk(1, 0), d));
    }
    __syncthreads();
    for (int e = threadIdx.x; e < bb; e += blockDim.x) X4[e] = cdf_mul(fv[e / b], X4[e]);
    __syncthreads();
    for (int e = threadIdx.x; e < bb; e += blockDim.x) {
      const int r = e / b, q = e % b;
      if (r > q) continue;
      const float4 xrq = X4[r * b + q], xqr = X4[q * b + r];
      // i X_rq = (-Im, Re); conj(i X_qr) = (-Im X_qr, -Re X_qr); halves are exact
      const float2 re = dfv_add(make_float2(-0.5f * xrq.y, -0.5f * xrq.w), make_float2(-0.5f * xqr.y, -0.5f * xqr.w));
      float2 im = dfv_add(make_float2(0.5f * xrq.x, 0.5f * xrq.z), make_float2(-0.5f * xqr.x, -0.5f * xqr.z));
      if (r == q) im = make_float2(0.f, 0.f);
      X4[r * b + q] = make_float4(re.x, im.x, re.y, im.y);
      X4[q * b + r] = make_float4(re.x, -im.x, re.y, -im.y);
    }
    __syncthreads();
    if constexpr (START) {
      floquet_start<FloqDf>(X4, M4, b, wk);
    } else {
      for (int e = threadIdx.x; e < bb; e += blockDim.x)
        M4[e] = make_float4(e / b == e % b ? 1.f : 0.f, 0.f, 0.f, 0.f);
      __syncthreads();
    }
    for (int e = threadIdx.x; e < bb; e += blockDim.x) Kf[e] = FloqDf::narrow(X4[e]);
    __syncthreads();
    const int max_sweeps = kMaxSweeps;
    const bool conv = floquet_sweeps_df(Kf, M4, b, max_sweeps, wk);
    if (!conv) atomicOr(s.status, kNoConvergeFloquet);
    // Rayleigh quotients: Y = A_n V in X's array (A_n converted once: with a64 the conversions run
    // at the FP64 rate), lam_r = sum_k conj(V_kr) Y_kr
    for (int e = threadIdx.x; e < bb; e += blockDim.x) X4[e] = Ug(e / b, e % b);
    __syncthreads();
    mul_in_place<FloqDf>(X4, M4, b);
    for (int r = threadIdx.x; r < b; r += blockDim.x) {
      CdfAcc a = {{0.f, 0.f}, {0.f, 0.f}};
      for (int kk = 0; kk < b; ++kk) {
        const float4 v = M4[kk * b + r];
        cdf_mac(a, make_float4(v.x, -v.y, v.z, -v.w), X4[kk * b + r]);
      }
      lam[r] = df_load(cdf_fin(a));
    }
    __syncthreads();
    if (pass == 1) break;
    if (threadIdx.x == 0) {
      double mind = 4.0;
      const double2 e2 = cmk(ca, sa);
      for (int r = 0; r < b; ++r) {
        const double2 w = cmul(e2, lam[r]);
        mind = fmin(mind, (1.0 + w.x) * (1.0 + w.x) + w.y * w.y);
      }
      done_s = conv && mind >= 0.0625;
      if (!done_s) {
        for (int r = 0; r < b; ++r) {
          const double th = atan2(lam[r].y, lam[r].x);
          int j = r;
          while (j > 0 && red[j - 1] > th) red[j] = red[j - 1], --j;
          red[j] = th;
        }
        double best = -1, mid = 0;
        for (int r = 0; r < b; ++r) {
          const double lo = red[r], hi = (r + 1 < b) ? red[r + 1] : red[0] + kPi2;
          if (hi - lo > best) best = hi - lo, mid = 0.5 * (lo + hi);
        }
        a_s = kPi - mid;
      }
    }
    __syncthreads();
    if (done_s) break;
  }
  for (int e = threadIdx.x; e < bb; e += blockDim.x) s.VF[at(bp + e, c, s.Cpad)] = df_load(M4[e]);
  for (int r = threadIdx.x; r < b; r += blockDim.x)
    s.L[at(bo + r, c, s.Cpad)] = cmk(log(hypot(lam[r].x, lam[r].y)), atan2(lam[r].y, lam[r].x));
}

// ------------------------------------------------------------------ mixed form, 4 x 4 tiles
// The mixed form's single-precision eigenframe and Q/R: 4 x 4 output tiles per thread, operands
// read as 16-byte vectors (two complex elements), 8 shared-memory vectors per 32 complex
// multiply-adds (the 2 x 2 tiles of cta_mm_cplx_regs take 32 8-byte loads for them), one tile per
// thread (blocks up to 74: at most 19 x 19 tiles).  Leading dimensions are multiples of four, so
// that a tile's vectors stay inside its rows; what lies beyond an operand only enters outputs that
// are not stored.  Same operands and the same sum per output element, in the same order, as with
// the 2 x 2 tiles.  Measured on 8 spins, 1154 crystallites, n = 200: eigenframe 59.8 -> 42.9 ms,
// Q/R 71.8 -> 62.6 ms.
__host__ __device__ constexpr int big4_tiles(int m, int n) { return ((m + 3) / 4) * ((n + 3) / 4); }
__host__ __device__ constexpr int big4_threads(int m, int n) { return (big4_tiles(m, n) + 31) / 32 * 32; }
__host__ __device__ constexpr int up4(int x) { return (x + 3) / 4 * 4; }

__device__ __forceinline__ void ld_c2(const float2 *p, float2 &a, float2 &b) {
  const float4 v = *reinterpret_cast<const float4 *>(p);
  a = make_float2(v.x, v.y), b = make_float2(v.z, v.w);
}

// acc (this thread's tile) = A B: A row-major m x k (lda even, column k zero when k is odd), B
// row-major k x n (ldb a multiple of four, row k zero when k is odd)
__device__ __forceinline__ void cta_mm4(const float2 *A, int lda, const float2 *B, int ldb, int m, int n, int k,
                                        float2 (&acc)[4][4]) {
  const int tm = (m + 3) / 4, tn = (n + 3) / 4, t = threadIdx.x;
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = make_float2(0.f, 0.f);
  if (t >= tm * tn) return;
  const int i0 = (t / tn) * 4, j0 = (t % tn) * 4;
  const float2 *ap[4];
#pragma unroll
  for (int a = 0; a < 4; ++a) ap[a] = A + min(i0 + a, m - 1) * lda;
  const float2 *bp = B + j0;
  for (int l = 0; l < k; l += 2, bp += 2 * ldb) {
    float2 av[4][2], bv[2][4];
#pragma unroll
    for (int a = 0; a < 4; ++a) ld_c2(ap[a] + l, av[a][0], av[a][1]);
#pragma unroll
    for (int h = 0; h < 2; ++h) ld_c2(bp + h * ldb, bv[h][0], bv[h][1]), ld_c2(bp + h * ldb + 2, bv[h][2], bv[h][3]);
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = cfma(av[a][h], bv[h][b], acc[a][b]);
  }
}
// acc = A^H B, A row-major k x m (lda a multiple of four)
__device__ __forceinline__ void cta_mm4_h(const float2 *A, int lda, const float2 *B, int ldb, int m, int n, int k,
                                          float2 (&acc)[4][4]) {
  const int tm = (m + 3) / 4, tn = (n + 3) / 4, t = threadIdx.x;
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = make_float2(0.f, 0.f);
  if (t >= tm * tn) return;
  const float2 *ap = A + (t / tn) * 4, *bp = B + (t % tn) * 4;
#pragma unroll 2
  for (int l = 0; l < k; ++l, ap += lda, bp += ldb) {
    float2 av[4], bv[4];
    ld_c2(ap, av[0], av[1]), ld_c2(ap + 2, av[2], av[3]);
    ld_c2(bp, bv[0], bv[1]), ld_c2(bp + 2, bv[2], bv[3]);
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[a][b] = cfmaconj(av[a], bv[b], acc[a][b]);
  }
}
template <class F>
__device__ __forceinline__ void cta_tiles4_store(int m, int n, const float2 (&acc)[4][4], F f) {
  const int tm = (m + 3) / 4, tn = (n + 3) / 4, t = threadIdx.x;
  if (t >= tm * tn) return;
  const int i0 = (t / tn) * 4, j0 = (t % tn) * 4;
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b)
      if (i0 + a < m && j0 + b < n) f(i0 + a, j0 + b, acc[a][b]);
}

// One CTA per (crystallite, kSegLen steps): W_i = A_{i+1} V_F = P_i V_s (mixed form: high parts
// of the double-float A, single-precision V and W).
__host__ __device__ constexpr size_t big_eigframe4_smem(int b) {
  return sizeof(float2) * (size_t(b + 1) * up4(b) + size_t(b) * ((b + 1) / 2 * 2));
}
__global__ void __launch_bounds__(384) k_big_eigframe4(DevSys s, int k) {
  extern __shared__ __align__(16) unsigned char bsr4[];
  const int c = blockIdx.x % s.C, i0 = int(blockIdx.x / s.C) * kSegLen, i1 = min(s.n, i0 + kSegLen);
  const int b = s.bs[k], bp = s.bpoff[k], bb = b * b, lv = up4(b), la = (b + 1) / 2 * 2;
  float2 *Vs = reinterpret_cast<float2 *>(bsr4), *As = Vs + (b + 1) * lv;
  const bool seg = segmented(s, b);
  for (int e = threadIdx.x; e < bb; e += blockDim.x)
    Vs[(e / b) * lv + e % b] = frame_elem<float2>(s, seg, i0, seg ? big_at(s, b, bp, e, c) : at(bp + e, c, s.Cpad));
  for (int e = threadIdx.x; e < lv; e += blockDim.x) Vs[b * lv + e] = make_float2(0.f, 0.f);
  if (la > b)
    for (int r = threadIdx.x; r < b; r += blockDim.x) As[r * la + b] = make_float2(0.f, 0.f);
  float2 acc[4][4];
  for (int i = i0; i < i1; ++i) {
    const float4 *Ab4 = reinterpret_cast<const float4 *>(s.A + size_t(i) * s.S2 * s.Cpad);
    float2 *Wb = s.Wf + size_t(i) * s.S2 * s.Cpad;
    for (int e = threadIdx.x; e < bb; e += blockDim.x) {
      const float4 v = Ab4[big_at(s, b, bp, e, c)];
      As[(e / b) * la + e % b] = make_float2(v.x, v.y);
    }
    __syncthreads();
    cta_mm4(As, la, Vs, lv, b, b, b, acc);
    cta_tiles4_store(b, b, acc, [&](int r, int q, float2 v) { Wb[big_at(s, b, bp, r * b + q, c)] = v; });
    __syncthreads();
  }
}

// k_big_qr in single precision for row blocks from kQr4Min on: W_a, a column chunk of W_b and of X =
// M_ab W_b in shared memory, loaded by asynchronous copies, a warp per row.  Smaller row blocks
// stay with the 2 x 2 tiles: 20 x 20 has 25 tiles of 4 x 4, one warp (6 spins: 2.01 ms by 2 x 2, 2.65
// by 4 x 4; 56 and 70 are faster by 4 x 4, sizes between 20 and 56 were not measured on their own).
constexpr int kQr4Min = 40;
__host__ __device__ constexpr size_t big_qr4_smem(int ba, int bb, int w) {
  return sizeof(float2) * (size_t(ba) * up4(ba) + size_t(bb) * w + size_t(ba) * up4(w));
}
__global__ void __launch_bounds__(384) k_big_qr4(DevSys s, BigPair P) {
  extern __shared__ __align__(16) unsigned char bsr4[];
  const int c = blockIdx.x % s.C, i = blockIdx.x / s.C;
  const int ba = s.bs[P.a], bb = s.bs[P.b], pa = s.bpoff[P.a], pb = s.bpoff[P.b];
  const int w = P.wchunk, la = up4(ba), lx = up4(w);
  const float2 *W = s.Wf + size_t(i) * s.S2 * s.Cpad;
  float2 *Wa = reinterpret_cast<float2 *>(bsr4), *X = Wa + ba * la, *Wb = X + ba * lx;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;  // a warp per row
  for (int r = warp; r < ba; r += nw)
    for (int q = lane; q < ba; q += 32) cp_async8(&Wa[r * la + q], &W[big_at(s, ba, pa, r * ba + q, c)], 8);
  float2 *ob = (P.isq ? s.Qf : s.Rf) + size_t(i) * P.nitems * s.Cpad;
  float2 acc[4][4];
  for (int q0 = 0; q0 < bb; q0 += w) {
    const int wc = min(w, bb - q0);
    for (int r = warp; r < bb; r += nw)
      for (int q = lane; q < wc; q += 32) cp_async8(&Wb[r * w + q], &W[big_at(s, bb, pb, r * bb + q0 + q, c)], 8);
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    for (int l = warp; l < ba; l += nw) {
      const int j0 = __ldg(P.rp + l), j1 = __ldg(P.rp + l + 1);
      for (int q = lane; q < wc; q += 32) {
        float2 x = make_float2(0.f, 0.f);
        for (int j = j0; j < j1; ++j) x = cfma(pair_coef(P, j, x), Wb[__ldg(P.ci + j) * w + q], x);
        X[l * lx + q] = x;
      }
    }
    __syncthreads();
    cta_mm4_h(Wa, la, X, lx, ba, wc, ba, acc);
    cta_tiles4_store(ba, wc, acc, [&](int r, int q, float2 v) { ob[at(P.off + r * bb + q0 + q, c, s.Cpad)] = v; });
    __syncthreads();
  }
}
