// GPU engine: spinning powder FID by gamma-COMPUTE, all arithmetic FP64.
//
// Reference algorithm (paths inside the BlochLib tree):
//   per crystallite  oneFID::singleSpinningFID   src/QMspins/driver/oneFID.h:419-431
//   step loop        compute::calcUFID           src/QMspins/driver/compute.h:257-274
//   H(t)             SolidSys::Hamiltonian       src/QMspins/sys.cc:749-770
//   exp(-i2pi tau H) Mexp (Hermitian)            src/container/matrix/matexp.h:240-252
//   reconstruction   compute::calcFID            src/QMspins/driver/compute.h:308-461
//   powder sum       oneFID::spinningFID         src/QMspins/driver/oneFID.h:339-410
//
// GB300 layout.  Every per-crystallite array is stored with the crystallite index
// fastest ([item][c], stride Cpad = C rounded up to 32) and every kernel maps the 32
// lanes of a warp onto 32 consecutive crystallites, so loads/stores are coalesced and
// all control flow (block sizes, steps, element indices) is warp-uniform.  The
// Hamiltonian of every SolidSys commutes with total Fz, so H, U and the Dyson products
// are block diagonal; the host finds the blocks (connected components of the operator
// pattern) and the kernels work per block.  FP64 issue rate is the bound on GB300
// (~1.2 TFLOP/s DFMA), so the kernels avoid FP64 work rather than memory traffic:
//   k_step_prop  (c, block, step)   H_i block, Jacobi eigh, U_i = V e^{-i2pi tau L} V^T
//   k_dyson      (c, block, column) A_{i+1} = U_i A_i, one column per thread
//   k_floquet    (c, block)         unitary eig of A_n (Cayley transform + Jacobi)
//   k_eigframe   (c, block, step)   W_i = A_{i+1} V_F  (in place)
//   k_qr         (c, step, pair)    Q_i = W^H D W (and R_i = W^H rho W when needed)
//   k_fave       (c, element, p)    G_p = sum_i q_{(i+p)%n} r_i (with the period twist)
//   k_p2p_elems  (c, element)       point-to-point FID terms from Q/R and the Floquet phases
//   k_fid_pair   (c, j pairs, p)    fid[jn+p] = sum_e z_e^j G_p(e); weighted warp sum
//   k_reduce     (k)                compensated sum of warp partials (fixed order)
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <sstream>
#include <stdexcept>
#include <type_traits>

#include "bl_engine.h"

namespace bl {

namespace {

constexpr int kMaxBlock = 8;      // largest Hamiltonian block handled by this engine
constexpr int kMaxSweeps = 40;    // bound on Jacobi sweeps; exceeding it sets a status bit
constexpr int kMaxP2PSteps = 16384;  // steps per rotor period of a point-to-point FID
constexpr int kThreads = 128;
constexpr double kPi = 3.14159265358979323846;
constexpr double kPi2 = 2.0 * kPi;

enum StatusBits { kNoConvergeStep = 1, kNoConvergeFloquet = 2, kSingularCayley = 4 };

#define CUDA_OK(x)                                                                          \
  do {                                                                                      \
    cudaError_t e_ = (x);                                                                   \
    if (e_ != cudaSuccess) throw Error(3, std::string("CUDA: ") + cudaGetErrorString(e_)); \
  } while (0)

// ------------------------------------------------------------------ complex helpers
__device__ __forceinline__ double2 cmk(double r, double i) { return make_double2(r, i); }
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return cmk(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return cmk(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return cmk(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 cconj(double2 a) { return cmk(a.x, -a.y); }
__device__ __forceinline__ double2 cscale(double2 a, double s) { return cmk(a.x * s, a.y * s); }
// acc + a*b
__device__ __forceinline__ double2 cfma(double2 a, double2 b, double2 acc) {
  return cmk(fma(a.x, b.x, fma(-a.y, b.y, acc.x)), fma(a.x, b.y, fma(a.y, b.x, acc.y)));
}
// acc + conj(a)*b
__device__ __forceinline__ double2 cfmaconj(double2 a, double2 b, double2 acc) {
  return cmk(fma(a.x, b.x, fma(a.y, b.y, acc.x)), fma(a.x, b.y, fma(-a.y, b.x, acc.y)));
}
__device__ __forceinline__ double2 cexp(double2 z) {
  double s, c, e = exp(z.x);
  sincos(z.y, &s, &c);
  return cmk(e * c, e * s);
}
__device__ __forceinline__ double2 cdiv(double2 a, double2 b) {
  double d = b.x * b.x + b.y * b.y;
  return cmk((a.x * b.x + a.y * b.y) / d, (a.y * b.x - a.x * b.y) / d);
}
__device__ __forceinline__ double chop1(double v, double eps) { return fabs(v) < eps ? 0.0 : v; }

// v != 0.0 on the integer pipe: an FP64 comparison costs as much as an FP64 FMA, and the skips
// over an operator's structural zeros test every element
__device__ __forceinline__ bool nonzero(double v) {
  return ((unsigned(__double2hiint(v)) << 1) | unsigned(__double2loint(v))) != 0u;
}
__device__ __forceinline__ bool nonzero(double2 v) { return nonzero(v.x) || nonzero(v.y); }

// Single-precision twins for the mixed-precision form (same names, float2 arguments).
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }
__device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
__device__ __forceinline__ float2 cfma(float2 a, float2 b, float2 acc) {
  return make_float2(fmaf(a.x, b.x, fmaf(-a.y, b.y, acc.x)), fmaf(a.x, b.y, fmaf(a.y, b.x, acc.y)));
}
__device__ __forceinline__ float2 cdiv(float2 a, float2 b) {
  float d = b.x * b.x + b.y * b.y;
  return make_float2((a.x * b.x + a.y * b.y) / d, (a.y * b.x - a.x * b.y) / d);
}
__device__ __forceinline__ float2 cfmaconj(float2 a, float2 b, float2 acc) {
  return make_float2(fmaf(a.x, b.x, fmaf(a.y, b.y, acc.x)), fmaf(a.x, b.y, fmaf(-a.y, b.x, acc.y)));
}
template <class C>
__device__ __forceinline__ C mkc(double r, double i);
template <>
__device__ __forceinline__ double2 mkc<double2>(double r, double i) { return make_double2(r, i); }
template <>
__device__ __forceinline__ float2 mkc<float2>(double r, double i) { return make_float2(float(r), float(i)); }
template <class C>
__device__ __forceinline__ C cvt(double2 v) { return mkc<C>(v.x, v.y); }
template <class C>
__device__ __forceinline__ double2 todbl(C v) { return make_double2(double(v.x), double(v.y)); }

// Double-float values (hi + lo, ~2^-48 relative) for the mixed form's Dyson products, where
// GB300's FP32 pipe (about 64 times the FP64 rate) does the work.  A complex element is one
// float4 (re.hi, im.hi, re.lo, im.lo) in the 16-byte slot a double2 would take.  Sums use the
// compensated dot product of Ogita, Rump and Oishi (2005) with the error-free two-sum of Knuth
// and the FMA two-product; the _rn intrinsics keep the compiler from contracting them.
__device__ __forceinline__ float4 df_store(double2 v) {
  const float rh = __double2float_rn(v.x), ih = __double2float_rn(v.y);
  return make_float4(rh, ih, __double2float_rn(v.x - double(rh)), __double2float_rn(v.y - double(ih)));
}
__device__ __forceinline__ double2 df_load(float4 v) {
  return make_double2(double(v.x) + double(v.z), double(v.y) + double(v.w));
}
// running compensated sum of products: s + c
struct DfAcc {
  float s, c;
};
__device__ __forceinline__ void df_dot(DfAcc &a, float xh, float xl, float yh, float yl) {
  const float p = __fmul_rn(xh, yh), pe = __fmaf_rn(xh, yh, -p);       // two-product
  const float s = __fadd_rn(a.s, p), bb = __fsub_rn(s, a.s);           // two-sum
  const float se = __fadd_rn(__fsub_rn(a.s, __fsub_rn(s, bb)), __fsub_rn(p, bb));
  a.s = s;
  a.c = __fadd_rn(a.c, __fadd_rn(__fadd_rn(pe, se), __fmaf_rn(xh, yl, __fmul_rn(xl, yh))));
}
__device__ __forceinline__ float2 df_fin(const DfAcc &a) {  // (hi, lo) of s + c
  const float h = __fadd_rn(a.s, a.c);
  return make_float2(h, __fsub_rn(a.c, __fsub_rn(h, a.s)));
}
// double-float scalars (x = hi, y = lo) for the mixed form's step exponential
__device__ __forceinline__ float2 dfv_of(double d) {
  const float h = __double2float_rn(d);
  return make_float2(h, __double2float_rn(d - double(h)));
}
__host__ __device__ __forceinline__ constexpr float2 dfv_const(double d) {
  return float2{float(d), float(d - double(float(d)))};
}
__device__ __forceinline__ float2 dfv_add(float2 a, float2 b) {
  const float s = __fadd_rn(a.x, b.x), bb = __fsub_rn(s, a.x);
  const float e = __fadd_rn(__fadd_rn(__fsub_rn(a.x, __fsub_rn(s, bb)), __fsub_rn(b.x, bb)), __fadd_rn(a.y, b.y));
  const float h = __fadd_rn(s, e);
  return make_float2(h, __fsub_rn(e, __fsub_rn(h, s)));
}
__device__ __forceinline__ float2 dfv_mul(float2 a, float2 b) {
  const float p = __fmul_rn(a.x, b.x);
  const float e = __fmaf_rn(a.x, b.y, __fmaf_rn(a.y, b.x, __fmaf_rn(a.x, b.x, -p)));
  const float h = __fadd_rn(p, e);
  return make_float2(h, __fsub_rn(e, __fsub_rn(h, p)));
}

// complex double-float elements as float4 (re.hi, im.hi, re.lo, im.lo): compensated sums
struct CdfAcc {
  DfAcc re, im;
};
__device__ __forceinline__ void cdf_mac(CdfAcc &a, float4 x, float4 y) {  // a += x y
  df_dot(a.re, x.x, x.z, y.x, y.z);
  df_dot(a.re, -x.y, -x.w, y.y, y.w);
  df_dot(a.im, x.x, x.z, y.y, y.w);
  df_dot(a.im, x.y, x.w, y.x, y.z);
}
__device__ __forceinline__ float4 cdf_fin(const CdfAcc &a) {
  const float2 r = df_fin(a.re), m = df_fin(a.im);
  return make_float4(r.x, m.x, r.y, m.y);
}

// 8-byte asynchronous copy global -> shared (cp.async); src_bytes 0 writes zeros
__device__ __forceinline__ void cp_async8(void *dst, const void *src, int src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(uint32_t(__cvta_generic_to_shared(dst))), "l"(src),
               "r"(src_bytes)
               : "memory");
}

// ------------------------------------------------------------------ job description
struct DevSys {
  int C, Cpad, n, npts, N, nb, S2, nint, nq, nr, ne, J, rosym, step_method;
  int M, logM, fftq, fave_method;  // FFT length M = fftq 2^logM of the Fave correlation; 0 direct, 1 FFT
  int fave_twist;            // 1: M == n, circular correlation of the twisted sequences
  int is_static;             // static powder FID (oneFID.h:292-336): dt = 1/sw, n = p-period
  int gper;                  // period of the FID split fid[j*gper + p] (n, or the p2p base)
  int p2p, pb, pf, psub;     // point-to-point FID: base, factor, steps per chunk
  // mixed form: 1 when the Floquet sweeps over K may run in FP32, i.e. the FID raises the
  // Floquet eigenvalues to at most kFloq32MaxPeriods periods (phase errors grow with the power)
  int floq32;
  double dt;
  const int *srp, *seo;      // per D pair (a,b): the rho pair (b,a) and first element, or -1
  const double2 *tw;         // exp(-2 pi i k / M), k < M
  double tau, wr, sin_rotb, cos_rotb, scale;
  double wref, wscale;  // mixed form's FID terms: largest |weight|; wref scale / fftq, applied in FP64
  // per block
  const int *bs, *boff, *bpoff;
  // per interaction: crystal tensor (xx xy xz yy yz zz), scale, packed operator
  const double *pas, *iscale, *Tk, *Hc;
  const double *fk;  // per (step, term, crystallite): the term coefficients of k_coef, or null
  // point-to-point rf schedule: hc_chunks > 0 gives one Hc per chunk of the period (step i in
  // chunk i / psub); frames (chunk x N, permuted index) rotate each step's U into the lab frame
  int hc_chunks;
  const double2 *frames;
  // double-float copies for the mixed form's step (hi, lo): term operators, constant parts,
  // and fk_df = 1 when k_coef stores the coefficients as float2 in fk's slots
  const float2 *Tk_df, *Hc_df;
  // the same operators by element for the blocks above kMaxBlock: element e (packed block index)
  // holds entries [tk_ptr[e], tk_ptr[e+1]) of (term, value in FP64 and double-float), terms
  // ascending; tk_order: each block's elements by descending term count
  const int *tk_ptr, *tk_term, *tk_order;
  const float2 *tk_val;
  const double *tk_val64;
  int fk_df;
  float2 tpdf;  // 2 pi tau as double-float
  const int *ikind;  // per term: 0 first order, 1 / 2 second-order quadrupolar (c4 / c2)
  int has2;
  // Q pairs (D blocks) and R pairs (rho blocks)
  int npq, npr;
  const int *qa, *qb, *qoff, *doff;
  const int *ra, *rb, *roff, *rhooff;
  const double2 *Dblk, *Rhoblk;
  // elements of the Fave/FID sums
  const int *eq, *erev, *er, *erg, *esg;
  // per crystallite (this batch): Rp (9 x Cpad), t0, weight
  const double *Rp, *t0, *w;
  // work buffers
  double2 *U, *A, *VF, *L, *Q, *R, *G, *Z, *partial;
  // mixed-precision form: eigenframe, Q/R, Fave and FID arrays in single precision
  int mixed;
  float2 *Wf, *Qf, *Rf, *Gf, *Zf;
  const float2 *twf;
  int warp_base;  // global warp index of this batch's first crystallite
  // k_fid_tiled: thread rows (4 j each), columns (4 p each), element ranges, groups per CTA
  int ft_jt, ft_pt, ft_r, ft_sub;
  int *status;
  unsigned long long *tc_flops;  // [2]: BF16 tensor flops issued by the step and Dyson kernels
  // 1: in the mixed form, A and W of the large blocks (kMaxBlock < b <= kMaxBigBlock) are
  // stored crystallite-major inside each (step, block) region (big_at), so that the
  // one-CTA-per-crystallite kernels move contiguous rows; the other blocks keep [item][c]
  int clay;
  // Segments of the Dyson products: nseg = ceil(n / kSegLen); blocks up to seg_max are segmented
  // (none when nseg == 1).  See seg_E.
  int nseg, seg_max, seg_from;  // (and blocks from seg_from on, the batched-product path's)
};

// Precision-dependent arrays: W (eigenframe; in place over A in FP64), Q, R, G, Z, twiddles.
template <class C> struct Bufs;
template <> struct Bufs<double2> {
  static __device__ double2 *W(const DevSys &s) { return s.A; }
  static __device__ double2 *Q(const DevSys &s) { return s.Q; }
  static __device__ double2 *R(const DevSys &s) { return s.R; }
  static __device__ double2 *G(const DevSys &s) { return s.G; }
  static __device__ double2 *Z(const DevSys &s) { return s.Z; }
  static __device__ const double2 *tw(const DevSys &s) { return s.tw; }
};
template <> struct Bufs<float2> {
  static __device__ float2 *W(const DevSys &s) { return s.Wf; }
  static __device__ float2 *Q(const DevSys &s) { return s.Qf; }
  static __device__ float2 *R(const DevSys &s) { return s.Rf; }
  static __device__ float2 *G(const DevSys &s) { return s.Gf; }
  static __device__ float2 *Z(const DevSys &s) { return s.Zf; }
  static __device__ const float2 *tw(const DevSys &s) { return s.twf; }
};

// ------------------------------------------------------------------ eigen-solvers
// Cyclic Jacobi, real symmetric, B x B in registers.  a becomes diagonal, v the
// eigenvectors (columns).  Returns false if kMaxSweeps was not enough.
template <int B>
__device__ bool jacobi_sym(double (&a)[B][B], double (&v)[B][B]) {
#pragma unroll
  for (int p = 0; p < B; ++p)
#pragma unroll
    for (int q = 0; q < B; ++q) v[p][q] = (p == q) ? 1.0 : 0.0;
  if (B == 1) return true;
  for (int sweep = 0; sweep < kMaxSweeps; ++sweep) {
    double off = 0, dg = 0;
#pragma unroll
    for (int p = 0; p < B; ++p) {
      dg = fma(a[p][p], a[p][p], dg);
#pragma unroll
      for (int q = p + 1; q < B; ++q) off = fma(a[p][q], a[p][q], off);
    }
    if (off <= 1e-34 * dg || off == 0.0) return true;
#pragma unroll
    for (int p = 0; p < B - 1; ++p)
#pragma unroll
      for (int q = p + 1; q < B; ++q) {
        double apq = a[p][q];
        if (apq != 0.0) {
          double theta = (a[q][q] - a[p][p]) / (2.0 * apq);
          double t;
          if (fabs(theta) > 1e100) t = 0.5 / theta;
          else t = copysign(1.0, theta) / (fabs(theta) + sqrt(fma(theta, theta, 1.0)));
          double c = rsqrt(fma(t, t, 1.0));
          double s = t * c, tz = s / (1.0 + c);
          a[p][p] = fma(-t, apq, a[p][p]);
          a[q][q] = fma(t, apq, a[q][q]);
          a[p][q] = 0.0;
          a[q][p] = 0.0;
#pragma unroll
          for (int r = 0; r < B; ++r) {
            if (r != p && r != q) {
              double arp = a[r][p], arq = a[r][q];
              double nrp = arp - s * fma(tz, arp, arq);
              double nrq = arq + s * fma(-tz, arq, arp);
              a[r][p] = nrp, a[p][r] = nrp;
              a[r][q] = nrq, a[q][r] = nrq;
            }
          }
#pragma unroll
          for (int r = 0; r < B; ++r) {
            double vrp = v[r][p], vrq = v[r][q];
            v[r][p] = vrp - s * fma(tz, vrp, vrq);
            v[r][q] = vrq + s * fma(-tz, vrq, vrp);
          }
        }
      }
  }
  return false;
}

// Cyclic Jacobi, complex Hermitian (B x B).  Same rotation as the oracle's.
template <int B>
__device__ bool jacobi_herm(double2 (&h)[B][B], double2 (&v)[B][B]) {
#pragma unroll
  for (int p = 0; p < B; ++p)
#pragma unroll
    for (int q = 0; q < B; ++q) v[p][q] = cmk(p == q ? 1.0 : 0.0, 0.0);
  if (B == 1) return true;
  for (int sweep = 0; sweep < kMaxSweeps; ++sweep) {
    double off = 0, dg = 0;
#pragma unroll
    for (int p = 0; p < B; ++p) {
      dg = fma(h[p][p].x, h[p][p].x, dg);
#pragma unroll
      for (int q = p + 1; q < B; ++q) off += h[p][q].x * h[p][q].x + h[p][q].y * h[p][q].y;
    }
    if (off <= 1e-34 * dg || off == 0.0) return true;
#pragma unroll
    for (int p = 0; p < B - 1; ++p)
#pragma unroll
      for (int q = p + 1; q < B; ++q) {
        double2 hpq = h[p][q];
        double ab = hypot(hpq.x, hpq.y);
        if (ab != 0.0) {
          double2 ph = cmk(hpq.x / ab, hpq.y / ab);
          double theta = 0.5 * (h[q][q].x - h[p][p].x) / ab;
          double t;
          if (fabs(theta) > 1e100) t = 0.5 / theta;
          else t = copysign(1.0, theta) / (fabs(theta) + sqrt(fma(theta, theta, 1.0)));
          double c = rsqrt(fma(t, t, 1.0)), s = t * c;
          double2 sp = cscale(ph, s), spc = cconj(sp);
#pragma unroll
          for (int k = 0; k < B; ++k) {  // columns p, q
            double2 hkp = h[k][p], hkq = h[k][q];
            h[k][p] = csub(cscale(hkp, c), cmul(spc, hkq));
            h[k][q] = cadd(cmul(sp, hkp), cscale(hkq, c));
          }
#pragma unroll
          for (int k = 0; k < B; ++k) {  // rows p, q
            double2 hpk = h[p][k], hqk = h[q][k];
            h[p][k] = csub(cscale(hpk, c), cmul(sp, hqk));
            h[q][k] = cadd(cmul(spc, hpk), cscale(hqk, c));
          }
          h[p][q] = cmk(0, 0);
          h[q][p] = cmk(0, 0);
          h[p][p].y = 0.0;
          h[q][q].y = 0.0;
#pragma unroll
          for (int k = 0; k < B; ++k) {
            double2 vkp = v[k][p], vkq = v[k][q];
            v[k][p] = csub(cscale(vkp, c), cmul(spc, vkq));
            v[k][q] = cadd(cmul(sp, vkp), cscale(vkq, c));
          }
        }
      }
  }
  return false;
}

// Eigen-decomposition of a unitary U = V diag(lam) V^H via the Cayley transform of
// W = e^{ia} U: K = i (I+W)^{-1} (I-W) is Hermitian with U's eigenvectors.  A first
// pass (a = 0.5) locates the spectrum; the second puts -1 in its widest gap.
template <int B>
__device__ int unitary_eig(const double2 (&U)[B][B], double2 (&lam)[B], double2 (&V)[B][B]) {
  int st = 0;
  if (B == 1) {
    lam[0] = U[0][0];
    V[0][0] = cmk(1, 0);
    return 0;
  }
  double a = 0.5;
  for (int pass = 0; pass < 2; ++pass) {
    double sa, ca;
    sincos(a, &sa, &ca);
    double2 ea = cmk(ca, sa);
    double2 M[B][B], X[B][B];
#pragma unroll
    for (int r = 0; r < B; ++r)
#pragma unroll
      for (int c = 0; c < B; ++c) {
        double2 w = cmul(ea, U[r][c]);
        double id = (r == c) ? 1.0 : 0.0;
        M[r][c] = cmk(id + w.x, w.y);
        X[r][c] = cmk(id - w.x, -w.y);
      }
    // Gaussian elimination with partial pivoting: M X' = X
#pragma unroll
    for (int k = 0; k < B; ++k) {
      int piv = k;
      double best = M[k][k].x * M[k][k].x + M[k][k].y * M[k][k].y;
#pragma unroll
      for (int i = k + 1; i < B; ++i) {
        double m2 = M[i][k].x * M[i][k].x + M[i][k].y * M[i][k].y;
        if (m2 > best) best = m2, piv = i;
      }
      if (best == 0.0) {
        st |= kSingularCayley;
        best = 1e-300;
      }
#pragma unroll
      for (int i = k + 1; i < B; ++i) {
        if (i == piv) {
#pragma unroll
          for (int j = 0; j < B; ++j) {
            double2 t = M[k][j];
            M[k][j] = M[i][j];
            M[i][j] = t;
            t = X[k][j];
            X[k][j] = X[i][j];
            X[i][j] = t;
          }
        }
      }
      double2 inv = cdiv(cmk(1, 0), M[k][k]);
#pragma unroll
      for (int i = k + 1; i < B; ++i) {
        double2 f = cmul(M[i][k], inv);
#pragma unroll
        for (int j = k; j < B; ++j) M[i][j] = csub(M[i][j], cmul(f, M[k][j]));
#pragma unroll
        for (int j = 0; j < B; ++j) X[i][j] = csub(X[i][j], cmul(f, X[k][j]));
      }
    }
#pragma unroll
    for (int k = B - 1; k >= 0; --k) {
      double2 inv = cdiv(cmk(1, 0), M[k][k]);
#pragma unroll
      for (int j = 0; j < B; ++j) {
        double2 s = X[k][j];
#pragma unroll
        for (int i = k + 1; i < B; ++i) s = csub(s, cmul(M[k][i], X[i][j]));
        X[k][j] = cmul(s, inv);
      }
    }
    // K = i X, Hermitian part
    double2 K[B][B];
#pragma unroll
    for (int r = 0; r < B; ++r)
#pragma unroll
      for (int c = 0; c < B; ++c) {
        double2 krc = cmk(-X[r][c].y, X[r][c].x);
        double2 kcr = cmk(-X[c][r].y, X[c][r].x);
        K[r][c] = cscale(cadd(krc, cconj(kcr)), 0.5);
      }
    if (!jacobi_herm<B>(K, V)) st |= kNoConvergeFloquet;
    // Rayleigh quotients
#pragma unroll
    for (int r = 0; r < B; ++r) {
      double2 s = cmk(0, 0);
#pragma unroll
      for (int k = 0; k < B; ++k) {
        double2 uv = cmk(0, 0);
#pragma unroll
        for (int l = 0; l < B; ++l) uv = cfma(U[k][l], V[l][r], uv);
        s = cfmaconj(V[k][r], uv, s);
      }
      lam[r] = s;
    }
    if (pass == 0) {
      // well conditioned already (every |1 + e^{ia} lambda| >= 1/4): keep this pass
      double mind = 4.0;
#pragma unroll
      for (int r = 0; r < B; ++r) {
        double2 w = cmul(ea, lam[r]);
        mind = fmin(mind, (1.0 + w.x) * (1.0 + w.x) + w.y * w.y);
      }
      if (mind >= 0.0625) break;
      double th[B];
#pragma unroll
      for (int r = 0; r < B; ++r) th[r] = atan2(lam[r].y, lam[r].x);
      // insertion sort
#pragma unroll
      for (int i = 1; i < B; ++i) {
#pragma unroll
        for (int j = i; j > 0; --j) {
          if (th[j] < th[j - 1]) {
            double t = th[j];
            th[j] = th[j - 1];
            th[j - 1] = t;
          }
        }
      }
      double best = -1, mid = 0;
#pragma unroll
      for (int r = 0; r < B; ++r) {
        double lo = th[r], hi = (r + 1 < B) ? th[r + 1] : th[0] + kPi2;
        if (hi - lo > best) best = hi - lo, mid = 0.5 * (lo + hi);
      }
      a = kPi - mid;
    }
  }
  return st;
}

// ------------------------------------------------------------------ kernels
__device__ __forceinline__ size_t at(int item, int c, int Cpad) { return size_t(item) * Cpad + c; }

// Segmented Dyson products.  The chain A_{i+1} = U_i A_i of n dependent products is cut into
// segments of kSegLen steps that run side by side, each from the identity: A[i] then holds
// P_i = U_i .. U_{first step of its segment}.  A short chain over the segments' last products
// gives E_{s+1} = P_last(s) E_s (E_0 = I, E_nseg = A_n, which the Floquet step decomposes), and
// the eigenframe takes W_i = A_{i+1} V = P_i V_s with V_s = E_s V formed once per segment: the
// full A_i are never needed.  What bounded the chain was the serial steps, not FP64 issue: a
// warp holds 32 crystallites of one (block, column), so 320 crystallites of a 10-block gave
// 320 one-warp CTAs on 608 sub-partitions, each stepping 157 times (1.28 ms per block, FP64
// pipe 32 % busy).  The extra products are 1/kSegLen of the Dyson and eigenframe work; 16 keeps
// that near 6 % of a stage that gets up to nseg times the threads.  The split depends on n
// alone, so a crystallite's result does not depend on how many others run.  Measured (Dyson,
// eigenframe; before -> after): 5 like spins, 320 crystallites, n = 157, FP64 1.73 -> 1.07 and
// 4.76 -> 1.00 ms; 7 spins, 144, n = 120, FP64 23.5 -> 14.6 and 23.3 -> 14.2 ms; 4 spins, 3722,
// n = 128, FP64 1.83 -> 1.33 and 1.14 -> 1.23 ms (the latter FP64-issue bound before too); one
// 3-spin crystallite, n = 64, Dyson 0.151 -> 0.061 ms.
// E_s and V_s live in the U buffer, which is dead once a block's segments are done: E_{s+1} in
// the slots of step s (the same block's items), V_s as float2 (mixed form) from step nseg + s, or
// over E_s in the FP64 form; the batched-product path (bl_huge.cuh) keeps V_s as FP64 from step
// 2 nseg + s (3 nseg <= n).
constexpr int kSegLen = 16;
__device__ __forceinline__ bool segmented(const DevSys &s, int b) { return b <= s.seg_max || b >= s.seg_from; }
__device__ __forceinline__ double2 *seg_E(const DevSys &s, int t) { return s.U + size_t(t) * s.S2 * s.Cpad; }
__device__ __forceinline__ float2 *seg_Vf(const DevSys &s, int t) {
  return reinterpret_cast<float2 *>(s.U + size_t(s.nseg + t) * s.S2 * s.Cpad);
}
// the period propagator A_n of a block of size b
__device__ __forceinline__ const double2 *period_prop(const DevSys &s, int b) {
  return segmented(s, b) ? seg_E(s, s.nseg - 1) : s.A + size_t(s.n - 1) * s.S2 * s.Cpad;
}
// A chain of products x <- M_t x from the identity: the steps of one segment (M = U, results to
// A), or the segments' last products (M = A at each segment's last step, results to E).
struct Chain {
  const double2 *src;
  double2 *dst;
  int first, stride, last, count, dst0;  // M_t = src step min(first + t stride, last); result t to dst step dst0 + t
  __device__ __forceinline__ const double2 *from(const DevSys &s, int t) const {
    return src + size_t(min(first + t * stride, last)) * s.S2 * s.Cpad;
  }
  __device__ __forceinline__ double2 *to(const DevSys &s, int t) const {
    return dst + size_t(dst0 + t) * s.S2 * s.Cpad;
  }
};
__device__ __forceinline__ Chain seg_chain(const DevSys &s, int b, int seg, bool prefix) {
  if (prefix) return Chain{s.A, s.U, kSegLen - 1, kSegLen, s.n - 1, s.nseg, 0};
  if (!segmented(s, b)) return Chain{s.U, s.A, 0, 1, s.n - 1, s.n, 0};
  const int i0 = seg * kSegLen;
  return Chain{s.U, s.A, i0, 1, s.n - 1, min(kSegLen, s.n - i0), i0};
}

// Powers of z = e^{i theta} that k_fid_pair takes (FP64 form): Z row m < pair_rows(J) holds
// z^(m + h), h = 1/2 for an even J and 0 for an odd one; the last row is z^((J-1)/2).
__host__ __device__ __forceinline__ int pair_rows(int J) { return (J + 1) / 2; }
__device__ __forceinline__ double pair_power(int J, int m) { return double(m) + (J % 2 == 0 ? 0.5 : 0.0); }

// Rows of M = R_rotor(phi, beta) R_powder for crystallite c, phi the rotor phase (sin sp,
// cos cp): row 2 always, rows 0 and 1 only when second-order quadrupolar terms need them.
__device__ __forceinline__ void orient_rows(const DevSys &s, int c, double sp, double cp, double (&m)[3][3]) {
  const double rr[3][3] = {{cp, sp, 0.0}, {-s.cos_rotb * sp, cp * s.cos_rotb, s.sin_rotb},
                           {sp * s.sin_rotb, -cp * s.sin_rotb, s.cos_rotb}};
#pragma unroll
  for (int i = 2; i >= 0; --i) {
    if (i < 2 && !s.has2) break;
#pragma unroll
    for (int j = 0; j < 3; ++j)
      m[i][j] = rr[i][0] * s.Rp[at(0 * 3 + j, c, s.Cpad)] + rr[i][1] * s.Rp[at(1 * 3 + j, c, s.Cpad)] +
                rr[i][2] * s.Rp[at(2 * 3 + j, c, s.Cpad)];
  }
}

// u PAS' v for the packed symmetric crystal tensor of term kk
__device__ __forceinline__ double pas_form(const double *P, const double *u, const double *v) {
  return u[0] * (P[0] * v[0] + P[1] * v[1] + P[2] * v[2]) + u[1] * (P[1] * v[0] + P[3] * v[1] + P[4] * v[2]) +
         u[2] * (P[2] * v[0] + P[4] * v[1] + P[5] * v[2]);
}

// Coefficient of term kk: scale (M PAS' M^T)_22 (kind 0); second-order quadrupolar
// scale ((r00-r11)^2/4 + r01^2) (kind 1) and scale (r02^2 + r12^2) (kind 2), r = M PAS' M^T.
__device__ __forceinline__ double term_coef(const DevSys &s, int kk, const double (&m)[3][3]) {
  const double *P = s.pas + 6 * kk;
  const int kind = s.has2 ? s.ikind[kk] : 0;
  double a;
  if (kind == 0) {
    a = pas_form(P, m[2], m[2]);
  } else if (kind == 1) {
    const double r00 = pas_form(P, m[0], m[0]), r11 = pas_form(P, m[1], m[1]), r01 = pas_form(P, m[0], m[1]);
    a = (r00 - r11) * (r00 - r11) / 4.0 + r01 * r01;
  } else {
    const double r02 = pas_form(P, m[0], m[2]), r12 = pas_form(P, m[1], m[2]);
    a = r02 * r02 + r12 * r12;
  }
  return s.iscale[kk] * a;
}

// Constant part of H and rf frame of step i: one per chunk under a point-to-point rf
// schedule (chunk i / psub), else the single Hc and no frame.
__device__ __forceinline__ const double *hc_of(const DevSys &s, int i) {
  return s.hc_chunks ? s.Hc + size_t(i / s.psub) * s.S2 : s.Hc;
}
__device__ __forceinline__ const double2 *frame_of(const DevSys &s, int i) {
  return s.frames ? s.frames + size_t(i / s.psub) * s.N : nullptr;
}

// Stores u = U'(p,q) = U'(q,p) of a step's real-symmetric-H block; with a frame r the lab-frame
// U = R U' R^H takes r_p u conj(r_q) at (p,q) and r_q u conj(r_p) at (q,p).
__device__ __forceinline__ void store_u_pair(double2 *Ub, int c, int Cpad, int bp, int bo, int B, int p, int q,
                                             double2 u, const double2 *fr, bool dfl) {
  double2 upq = u, uqp = u;
  if (fr) {
    const double2 rp = fr[bo + p], rq = fr[bo + q];
    upq = cmul(cmul(rp, u), cconj(rq));
    uqp = cmul(cmul(rq, u), cconj(rp));
  }
  if (dfl) {  // mixed form: double-float for k_dyson_df
    float4 *U4 = reinterpret_cast<float4 *>(Ub);
    U4[at(bp + p * B + q, c, Cpad)] = df_store(upq);
    if (q != p) U4[at(bp + q * B + p, c, Cpad)] = df_store(uqp);
    return;
  }
  Ub[at(bp + p * B + q, c, Cpad)] = upq;
  if (q != p) Ub[at(bp + q * B + p, c, Cpad)] = uqp;
}

// H_i block at the midpoint of step i (sys.cc:749-770): rotor phase 2 pi wr t_mid,
// a = (M PAS M^T)_22 with M = R_rotor R_powder, H = Hc + sum_k scale_k a_k T_k.
template <int B>
__device__ __forceinline__ void build_h_at(const DevSys &s, int c, double sp, double cp, const double *Hcb,
                                           int bp, double (&h)[B][B]) {
  double m[3][3];
  orient_rows(s, c, sp, cp, m);
#pragma unroll
  for (int p = 0; p < B; ++p)
#pragma unroll
    for (int q = 0; q < B; ++q) h[p][q] = Hcb[p * B + q];
  for (int kk = 0; kk < s.nint; ++kk) {
    const double f = term_coef(s, kk, m);
    const double *T = s.Tk + size_t(kk) * s.S2 + bp;
#pragma unroll
    for (int p = 0; p < B; ++p)
#pragma unroll
      for (int q = 0; q < B; ++q) {
        const double t = T[p * B + q];  // same for every lane: the skip is warp-uniform
        if (nonzero(t)) h[p][q] = fma(f, t, h[p][q]);
      }
  }
}

// Fourier coefficients of the first-order terms over the rotor phase, one thread per (term,
// crystallite): with the rows R_0, R_1, R_2 of R_powder and A_ij = R_i PAS' R_j, the rotor row
// (sin phi sin b, -cos phi sin b, cos b) gives
//   a(phi) = f0 + f1 cos phi + f2 sin phi + f3 cos 2 phi + f4 sin 2 phi.
__global__ void __launch_bounds__(kThreads) k_term_series(DevSys s, double *series) {
  const long tid = long(blockIdx.x) * blockDim.x + threadIdx.x;
  const int c = int(tid % s.Cpad), kk = int(tid / s.Cpad);
  if (kk >= s.nint || c >= s.C) return;
  double R[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) R[i][j] = s.Rp[at(3 * i + j, c, s.Cpad)];
  const double *P = s.pas + 6 * kk;
  const double a00 = pas_form(P, R[0], R[0]), a01 = pas_form(P, R[0], R[1]), a02 = pas_form(P, R[0], R[2]),
               a11 = pas_form(P, R[1], R[1]), a12 = pas_form(P, R[1], R[2]), a22 = pas_form(P, R[2], R[2]);
  const double sc = s.iscale[kk], ss = s.sin_rotb * s.sin_rotb * sc, s2 = 2.0 * s.sin_rotb * s.cos_rotb * sc;
  double *f = series + at(5 * kk, c, s.Cpad);
  f[0] = fma(0.5 * ss, a00 + a11, s.cos_rotb * s.cos_rotb * sc * a22);
  f[size_t(1) * s.Cpad] = -s2 * a12;
  f[size_t(2) * s.Cpad] = s2 * a02;
  f[size_t(3) * s.Cpad] = 0.5 * ss * (a11 - a00);
  f[size_t(4) * s.Cpad] = -ss * a01;
}

// Term coefficients for every crystallite and step, once for all blocks.  Where every term is
// first order and the crystallites start together (phase: cos, sin of phi and 2 phi per step,
// from the host), a thread takes one term of one crystallite over kCoefRun steps: four FMAs a
// coefficient from its Fourier series, against a sincos per step and about 20 FP64 operations per
// coefficient otherwise (4 spins, 3722 crystallites, n = 128: the step stage 1.19 -> 1.08 ms).
constexpr int kCoefRun = 16;
__global__ void __launch_bounds__(kThreads) k_coef_series(DevSys s, const double *__restrict__ series,
                                                         const double *__restrict__ phase, double *fk) {
  const long tid = long(blockIdx.x) * blockDim.x + threadIdx.x;
  const int c = int(tid % s.Cpad), kk = int(tid / s.Cpad % s.nint), i0 = int(tid / s.Cpad / s.nint) * kCoefRun;
  if (i0 >= s.n || c >= s.C) return;
  double f[5];
#pragma unroll
  for (int t = 0; t < 5; ++t) f[t] = series[at(5 * kk + t, c, s.Cpad)];
  float2 *fk2 = reinterpret_cast<float2 *>(fk);
  const int i1 = min(s.n, i0 + kCoefRun);
  for (int i = i0; i < i1; ++i) {
    const double2 p1 = *reinterpret_cast<const double2 *>(phase + 4 * i), p2 = *reinterpret_cast<const double2 *>(phase + 4 * i + 2);
    const double v = fma(f[4], p2.y, fma(f[3], p2.x, fma(f[2], p1.y, fma(f[1], p1.x, f[0]))));
    if (s.fk_df) fk2[at(i * s.nint + kk, c, s.Cpad)] = dfv_of(v);
    else fk[at(i * s.nint + kk, c, s.Cpad)] = v;
  }
}

// The same, step by step, for second-order terms or crystallites that start apart.
__global__ void __launch_bounds__(kThreads) k_coef(DevSys s, double *fk) {
  long tid = long(blockIdx.x) * blockDim.x + threadIdx.x;
  const int c = int(tid % s.Cpad), i = int(tid / s.Cpad);
  if (i >= s.n || c >= s.C) return;
  double t1 = s.t0[c] + double(i) * s.tau, t2 = t1 + s.tau;
  double tmid = (t2 - t1) / 2.0 + t1;
  double sp, cp;
  sincos(tmid * s.wr * kPi2, &sp, &cp);
  double m[3][3];
  orient_rows(s, c, sp, cp, m);
  float2 *fk2 = reinterpret_cast<float2 *>(fk);
  for (int kk = 0; kk < s.nint; ++kk) {
    const double f = term_coef(s, kk, m);
    if (s.fk_df) fk2[at(i * s.nint + kk, c, s.Cpad)] = dfv_of(f);
    else fk[at(i * s.nint + kk, c, s.Cpad)] = f;
  }
}

template <int B>
__device__ __forceinline__ void build_h(const DevSys &s, int c, int i, int bp, double (&h)[B][B]) {
  const double *Hcb = hc_of(s, i) + bp;
  if (s.fk) {  // coefficients from k_coef
#pragma unroll
    for (int p = 0; p < B; ++p)
#pragma unroll
      for (int q = 0; q < B; ++q) h[p][q] = Hcb[p * B + q];
    for (int kk = 0; kk < s.nint; ++kk) {
      const double f = s.fk[at(i * s.nint + kk, c, s.Cpad)];
      const double *T = s.Tk + size_t(kk) * s.S2 + bp;
#pragma unroll
      for (int p = 0; p < B; ++p)
#pragma unroll
        for (int q = 0; q < B; ++q) {
          const double t = T[p * B + q];
          if (nonzero(t)) h[p][q] = fma(f, t, h[p][q]);
        }
    }
    return;
  }
  double t1 = s.t0[c] + double(i) * s.tau, t2 = t1 + s.tau;
  double tmid = (t2 - t1) / 2.0 + t1;
  double sp, cp;
  sincos(tmid * s.wr * kPi2, &sp, &cp);
  build_h_at<B>(s, c, sp, cp, Hcb, bp, h);
}

// Static powder FID, step 1 (oneFID.h:301-311): one thread per (crystallite, block): H at
// rotor phase 0 (Hamiltonian(0, dt), wr = 0), Jacobi eigen-decomposition; V (real) goes to
// VF, the eigenvalues to L.x.
template <int B>
__global__ void __launch_bounds__(kThreads) k_static_eig(DevSys s, const int *__restrict__ blist, int nblist) {
  long tid = long(blockIdx.x) * blockDim.x + threadIdx.x;
  int c = int(tid % s.Cpad);
  long rest = tid / s.Cpad;
  if (rest >= nblist) return;
  int k = blist[rest];
  if (c >= s.C) return;
  const int bp = s.bpoff[k], bo = s.boff[k];
  double h[B][B], v[B][B];
  build_h_at<B>(s, c, 0.0, 1.0, s.Hc + bp, bp, h);
  if (!jacobi_sym<B>(h, v)) atomicOr(s.status, kNoConvergeStep);
#pragma unroll
  for (int r = 0; r < B; ++r) {
#pragma unroll
    for (int q = 0; q < B; ++q) s.VF[at(bp + r * B + q, c, s.Cpad)] = cmk(v[r][q], 0.0);
    s.L[at(bo + r, c, s.Cpad)] = cmk(h[r][r], 0.0);
  }
}

// Static powder FID, step 2 (oneFID.h:312-334): one thread per (crystallite, element (i, j) of
// D's block pairs (a,b) with rho_ba != 0, chunk of kStaticRun values of p).  Do = V_a^T D_ab V_b,
// sig0 = V_b^T rho_ba V_a, A_ij = Do(i,j) sig0(j,i) (dropped when |A|^2 <= 1e-10, as the
// reference does), B_ij = e^{i th}, th = 2 pi dt (lambda_i - lambda_j).  fid[k] = sum A B^k is
// written for the reconstruction kernel as G_p = A B^p (p < n, by products within a chunk) and,
// by one further thread per element, the powers of B^n that k_fid_pair takes.  A thread per
// element and chunk instead of one per block pair: 113 -> 26 us for three spins, 1154
// crystallites (65 of 152 SMs had a CTA).
constexpr int kStaticRun = 32;
__global__ void __launch_bounds__(kThreads) k_static_elems(DevSys s) {
  const long tid = long(blockIdx.x) * blockDim.x + threadIdx.x;
  const int c = int(tid % s.Cpad), nch = (s.n + kStaticRun - 1) / kStaticRun;
  const long rest = tid / s.Cpad;
  if (rest >= long(s.ne) * (nch + 1) || c >= s.C) return;
  const int e = int(rest % s.ne), ch = int(rest / s.ne);
  const double th = s.dt * kPi2 * (s.L[at(s.erg[e], c, s.Cpad)].x - s.L[at(s.esg[e], c, s.Cpad)].x);
  if (ch == nch) {  // the powers of B^n: by products, each restarted from sincos every 16
    double2 z1, zm = cmk(1, 0);
    sincos(double(s.n) * th, &z1.y, &z1.x);
    for (int m = 0; m < pair_rows(s.J); ++m) {
      if (m % 16 == 0) sincos(pair_power(s.J, m) * double(s.n) * th, &zm.y, &zm.x);
      s.Z[at(m * s.ne + e, c, s.Cpad)] = zm;
      zm = cmul(zm, z1);
    }
    return;
  }
  int pq = 0;  // the element's block pair: the last one that starts at or before e
  for (int t = 0; t < s.npq; ++t)
    if (s.seo[t] >= 0 && s.seo[t] <= e) pq = t;
  const int a = s.qa[pq], b = s.qb[pq];
  const int ba = s.bs[a], bb = s.bs[b], pa = s.bpoff[a], pb = s.bpoff[b];
  const int i = (e - s.seo[pq]) / bb, j = (e - s.seo[pq]) % bb;
  const double2 *D = s.Dblk + s.doff[pq], *Rh = s.Rhoblk + s.rhooff[s.srp[pq]];  // D_ab (ba x bb), rho_ba (bb x ba)
  double2 dij = cmk(0, 0), sji = cmk(0, 0);
  for (int l = 0; l < ba; ++l) {
    const double va = s.VF[at(pa + l * ba + i, c, s.Cpad)].x;
    double2 x = cmk(0, 0), y = cmk(0, 0);
    for (int m = 0; m < bb; ++m) {
      const double2 d = D[l * bb + m], r = Rh[m * ba + l];
      if (!nonzero(d) && !nonzero(r)) continue;
      const double vb = s.VF[at(pb + m * bb + j, c, s.Cpad)].x;
      x.x = fma(d.x, vb, x.x), x.y = fma(d.y, vb, x.y);
      y.x = fma(r.x, vb, y.x), y.y = fma(r.y, vb, y.y);
    }
    dij.x = fma(va, x.x, dij.x), dij.y = fma(va, x.y, dij.y);
    sji.x = fma(va, y.x, sji.x), sji.y = fma(va, y.y, sji.y);
  }
  double2 A = cmul(dij, sji);
  if (A.x * A.x + A.y * A.y <= 1.0e-10) A = cmk(0, 0);
  double2 B, g = cmk(1, 0);
  sincos(th, &B.y, &B.x);
  const int p0 = ch * kStaticRun, p1 = min(s.n, p0 + kStaticRun);
  if (p0) sincos(double(p0) * th, &g.y, &g.x);
  g = cmul(A, g);
  for (int p = p0; p < p1; ++p) {
    s.G[at(p * s.ne + e, c, s.Cpad)] = g;
    g = cmul(g, B);
  }
}

// One thread per (crystallite, block k, step i): U_i = V diag(chop(e^{-i 2pi tau L})) V^T
// from a cyclic Jacobi eigen-decomposition of the real symmetric H_i block (the
// reference's method, matexp.h:240-252).
template <int B>
__global__ void __launch_bounds__(kThreads) k_step_prop(DevSys s, const int *__restrict__ blist, int nblist) {
  long tid = long(blockIdx.x) * blockDim.x + threadIdx.x;
  int c = int(tid % s.Cpad);
  long rest = tid / s.Cpad;
  if (rest >= long(nblist) * s.n) return;
  int i = int(rest % s.n);
  int k = blist[rest / s.n];
  if (c >= s.C) return;
  const int bp = s.bpoff[k];
  double h[B][B];
  build_h<B>(s, c, i, bp, h);
  double v[B][B];
  if (!jacobi_sym<B>(h, v)) atomicOr(s.status, kNoConvergeStep);
  double2 e[B];
  const double tp = s.tau * kPi2;
#pragma unroll
  for (int j = 0; j < B; ++j) {
    double sn, cs;
    sincos(tp * h[j][j], &sn, &cs);
    e[j] = cmk(chop1(cs, 1e-12), chop1(-sn, 1e-12));
  }
  double2 *Ub = s.U + size_t(i) * s.S2 * s.Cpad;
  const double2 *fr = frame_of(s, i);
  const int bo = s.boff[k];
#pragma unroll
  for (int p = 0; p < B; ++p)
#pragma unroll
    for (int q = p; q < B; ++q) {
      double2 u = cmk(0, 0);
#pragma unroll
      for (int j = 0; j < B; ++j) {
        double vv = v[p][j] * v[q][j];
        u.x = fma(vv, e[j].x, u.x);
        u.y = fma(vv, e[j].y, u.y);
      }
      store_u_pair(Ub, c, s.Cpad, bp, bo, B, p, q, u, fr, s.mixed != 0);
    }
}

// Largest power of the period propagator (periods the FID spans: npts/n for the gamma-COMPUTE
// FID, npts*factor/base for the point-to-point one) for which the mixed form sweeps over the
// Floquet K in FP32: the residual ~1e-7 off-diagonal of V's basis grows into the eigenphases
// with the power; the benchmark FIDs (2048-4096 points, 100-200 steps a period) span at most 21.
constexpr long kFloq32MaxPeriods = 64;
constexpr int kTaylorTerms = 15;  // ||x|| <= 1/2: remainder 0.5^16/16! < 1e-18

// Taylor degree for exp(-iX) with ||X||_inf = x <= 1/2: the smallest K whose first omitted
// term bound x^(K+1)/(K+1)! is at most 2^-56, i.e. x <= ((K+1)! 2^-56)^(1/(K+1)) (table for
// K = 1..14; K = 15 covers x <= 0.601).  The mixed form, whose target is 1e-6 relative and
// whose eigenframe onwards is single precision, takes 2^-40 instead (<= 1e-12 per step,
// <= 1e-10 over a period of 128 steps): two to four fewer terms.
__device__ __forceinline__ int taylor_degree(double x, bool loose) {
  constexpr double thr[14] = {5.268356063861754e-09, 4.3667382909901915e-06, 0.00013509300777591815,
                              0.0011073892359697527, 0.004640970307744106,   0.013203184215395692,
                              0.029408989058618194,  0.05554895835340547,    0.09337020827678472,
                              0.14404487618659187,   0.2082354986608797,     0.2861946964536857,
                              0.3778659482136564,    0.4829712994609099};
  constexpr double thr40[14] = {1.3486991523486091e-06, 0.00017605585575041613, 0.0021614881244146904,
                                0.010176449549599028,   0.029468324594664686,   0.06437944735017741,
                                0.11763595623447277,    0.19047604120885106,    0.2830455430072978,
                                0.39478407585236897,    0.524720576196396,      0.671676320302853,
                                0.8343956619942197,     1.0116260068329037};
  int K = kTaylorTerms;
#pragma unroll
  for (int j = 13; j >= 0; --j)
    if (x <= (loose ? thr40[j] : thr[j])) K = j + 1;
  return K;
}

// Upper-triangle index of a symmetric B x B matrix stored packed.
template <int B>
__device__ __forceinline__ constexpr int sx(int p, int q) {
  return p <= q ? p * B - p * (p - 1) / 2 + (q - p) : q * B - q * (q - 1) / 2 + (p - q);
}

// C = X Y for commuting real symmetric X, Y (the product is symmetric): upper triangle.
template <int B>
__device__ __forceinline__ void sym_mul(const double *X, const double *Y, double *C, double scale) {
#pragma unroll
  for (int p = 0; p < B; ++p)
#pragma unroll
    for (int q = p; q < B; ++q) {
      double acc = 0;
#pragma unroll
      for (int l = 0; l < B; ++l) acc = fma(X[sx<B>(p, l)], Y[sx<B>(l, q)], acc);
      C[sx<B>(p, q)] = acc * scale;
    }
}

// cos X = sum_j c_j Y^j, sin X = X sum_j s_j Y^j (Y = X^2): c_j = (-1)^j/(2j)!, s_j = (-1)^j/(2j+1)!
__device__ __forceinline__ constexpr double cos_coef(int j) {
  return j == 0 ? 1.0 : j == 1 ? -1.0 / 2 : j == 2 ? 1.0 / 24 : j == 3 ? -1.0 / 720 : j == 4 ? 1.0 / 40320
       : j == 5 ? -1.0 / 3628800 : j == 6 ? 1.0 / 479001600 : -1.0 / 87178291200.0;
}
__device__ __forceinline__ constexpr double sin_coef(int j) {
  return j == 0 ? 1.0 : j == 1 ? -1.0 / 6 : j == 2 ? 1.0 / 120 : j == 3 ? -1.0 / 5040 : j == 4 ? 1.0 / 362880
       : j == 5 ? -1.0 / 39916800 : j == 6 ? 1.0 / 6227020800.0 : -1.0 / 1307674368000.0;
}

// acc = sum_{j <= d} coef_j Y^j (d <= 7) for this thread's d: pairs L_m = coef_2m I +
// coef_2m+1 Y (zero beyond d); acc = L_top, then acc = acc Y2 + L_m for m = top-1 .. 0
// (Paterson-Stockmeyer with Y2 = Y^2: d/2 symmetric products).
template <int B, bool SIN>
__device__ __forceinline__ void ps_poly(int d, const double *Y, const double *Y2, double *acc, double *tmp) {
  constexpr int NP = B * (B + 1) / 2;
  const int top = d / 2;
#pragma unroll
  for (int m = 3; m >= 0; --m) {
    if (m > top) continue;
    const double a0 = SIN ? sin_coef(2 * m) : cos_coef(2 * m);
    const double a1 = (2 * m + 1 <= d) ? (SIN ? sin_coef(2 * m + 1) : cos_coef(2 * m + 1)) : 0.0;
    if (m < top) sym_mul<B>(acc, Y2, tmp, 1.0);
#pragma unroll
    for (int p = 0; p < B; ++p)
#pragma unroll
      for (int q = p; q < B; ++q) {
        const int j = sx<B>(p, q);
        const double l = fma(a1, Y[j], p == q ? a0 : 0.0);
        acc[j] = (m < top) ? tmp[j] + l : l;
      }
  }
  (void)NP;
}

// The same in double-float (float2 = hi, lo): compensated dot products over l.
template <int B>
__device__ __forceinline__ void sym_mul_df(const float2 *X, const float2 *Y, float2 *C, float scale) {
#pragma unroll
  for (int p = 0; p < B; ++p)
#pragma unroll
    for (int q = p; q < B; ++q) {
      DfAcc acc = {0.f, 0.f};
#pragma unroll
      for (int l = 0; l < B; ++l) {
        const float2 x = X[sx<B>(p, l)], y = Y[sx<B>(l, q)];
        df_dot(acc, x.x, x.y, y.x, y.y);
      }
      const float2 v = df_fin(acc);
      C[sx<B>(p, q)] = make_float2(v.x * scale, v.y * scale);  // scale is +-1 or 2: exact
    }
}
template <int B, bool SIN>
__device__ __forceinline__ void ps_poly_df(int d, const float2 *Y, const float2 *Y2, float2 *acc, float2 *tmp) {
  const int top = d / 2;
#pragma unroll
  for (int m = 3; m >= 0; --m) {
    if (m > top) continue;
    const float2 a0 = dfv_const(SIN ? sin_coef(2 * m) : cos_coef(2 * m));
    const float2 a1 = (2 * m + 1 <= d) ? dfv_const(SIN ? sin_coef(2 * m + 1) : cos_coef(2 * m + 1)) : float2{0.f, 0.f};
    if (m < top) sym_mul_df<B>(acc, Y2, tmp, 1.f);
#pragma unroll
    for (int p = 0; p < B; ++p)
#pragma unroll
      for (int q = p; q < B; ++q) {
        const int j = sx<B>(p, q);
        float2 l = dfv_mul(a1, Y[j]);
        if (p == q) l = dfv_add(l, a0);
        acc[j] = (m < top) ? dfv_add(tmp[j], l) : l;
      }
  }
}

// H of step i in double-float from the double-float copies of Hc, the operators and k_coef's
// coefficients.
template <int B>
__device__ __forceinline__ void build_h_df(const DevSys &s, int c, int i, int bp, float2 (&h)[B][B]) {
  const float2 *Hcb = s.Hc_df + (s.hc_chunks ? size_t(i / s.psub) * s.S2 : 0) + bp;
#pragma unroll
  for (int p = 0; p < B; ++p)
#pragma unroll
    for (int q = 0; q < B; ++q) h[p][q] = Hcb[p * B + q];
  const float2 *fk2 = reinterpret_cast<const float2 *>(s.fk);
  for (int kk = 0; kk < s.nint; ++kk) {
    const float2 f = fk2[at(i * s.nint + kk, c, s.Cpad)];
    const float2 *T = s.Tk_df + size_t(kk) * s.S2 + bp;
#pragma unroll
    for (int p = 0; p < B; ++p)
#pragma unroll
      for (int q = 0; q < B; ++q) {
        const float2 t = T[p * B + q];  // same for every lane: the skip is warp-uniform
        if (t.x != 0.f) h[p][q] = dfv_add(h[p][q], dfv_mul(f, t));
      }
  }
}

// The mixed form's step exponential in double-float on the FP32 pipe (~2^-48, against the
// form's 2^-40 truncation): H from build_h_df, its norm from the high parts (it only picks the
// scaling and the degree), the polynomial and the squarings; U stored as double-float for
// k_dyson_df.
template <int B>
__global__ void __launch_bounds__(kThreads) k_step_taylor_df(DevSys s, const int *__restrict__ blist, int nblist) {
  long tid = long(blockIdx.x) * blockDim.x + threadIdx.x;
  int c = int(tid % s.Cpad);
  long rest = tid / s.Cpad;
  if (rest >= long(nblist) * s.n) return;
  int i = int(rest % s.n);
  int k = blist[rest / s.n];
  if (c >= s.C) return;
  const int bp = s.bpoff[k];
  constexpr int NP = B * (B + 1) / 2;
  float2 h[B][B];
  build_h_df<B>(s, c, i, bp, h);
  const float tpf = float(s.tau * kPi2);
  float nrm = 0.f;
#pragma unroll
  for (int p = 0; p < B; ++p) {
    float rs = 0.f;
#pragma unroll
    for (int q = 0; q < B; ++q) rs += fabsf(h[p][q].x);
    nrm = fmaxf(nrm, rs);
  }
  nrm *= tpf * (1.f + 1e-6f);  // margin over the rounding of the high parts
  int sq = 0;
  if (nrm > 0.5f) {
    frexpf(nrm / 0.5f, &sq);
    sq = min(sq, 60);
  }
  float2 sc = make_float2(ldexpf(s.tpdf.x, -sq), ldexpf(s.tpdf.y, -sq));  // 2 pi tau 2^-sq, exact scaling
  const int K = taylor_degree(double(ldexpf(nrm, -sq)), true);
  __shared__ float2 Xs[NP * kThreads];
  float2 Y[NP], Y2[NP], R[NP], S[NP], T[NP];
#pragma unroll
  for (int p = 0; p < B; ++p)
#pragma unroll
    for (int q = p; q < B; ++q) T[sx<B>(p, q)] = dfv_mul(sc, h[p][q]);
#pragma unroll
  for (int j = 0; j < NP; ++j) Xs[j * blockDim.x + threadIdx.x] = T[j];
  sym_mul_df<B>(T, T, Y, 1.f);
  sym_mul_df<B>(Y, Y, Y2, 1.f);
  ps_poly_df<B, false>(K / 2, Y, Y2, R, T);
  ps_poly_df<B, true>((K - 1) / 2, Y, Y2, S, T);
#pragma unroll
  for (int j = 0; j < NP; ++j) T[j] = Xs[j * blockDim.x + threadIdx.x];
  float2 *I = Y2;
  sym_mul_df<B>(T, S, I, -1.f);
  for (int t = 0; t < sq; ++t) {
    sym_mul_df<B>(R, R, Y, 1.f);
    sym_mul_df<B>(I, I, S, 1.f);
    sym_mul_df<B>(R, I, T, 2.f);
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      R[j] = dfv_add(Y[j], make_float2(-S[j].x, -S[j].y));
      I[j] = T[j];
    }
  }
  double2 *Ub = s.U + size_t(i) * s.S2 * s.Cpad;
  float4 *U4 = reinterpret_cast<float4 *>(Ub);
  const double2 *fr = frame_of(s, i);
  const int bo = s.boff[k];
#pragma unroll
  for (int p = 0; p < B; ++p)
#pragma unroll
    for (int q = p; q < B; ++q) {
      const float2 re = R[sx<B>(p, q)], im = I[sx<B>(p, q)];
      if (fr) {  // rf schedule frames: through FP64
        const double2 u = cmk(double(re.x) + double(re.y), double(im.x) + double(im.y));
        store_u_pair(Ub, c, s.Cpad, bp, bo, B, p, q, u, fr, true);
      } else {
        const float4 v = make_float4(re.x, im.x, re.y, im.y);
        U4[at(bp + p * B + q, c, s.Cpad)] = v;
        if (q != p) U4[at(bp + q * B + p, c, s.Cpad)] = v;
      }
    }
}

// One thread per (crystallite, block k, step i): U_i = exp(-i 2pi tau H_i) by a Taylor
// series of the scaled real symmetric block plus repeated squaring.  Real and imaginary
// parts of U are polynomials in H, hence symmetric and commuting, so every product is a
// real symmetric one (B^2(B+1)/2 FMA) and no division or square root is needed.
template <int B>
__global__ void __launch_bounds__(kThreads) k_step_taylor(DevSys s, const int *__restrict__ blist, int nblist) {
  long tid = long(blockIdx.x) * blockDim.x + threadIdx.x;
  int c = int(tid % s.Cpad);
  long rest = tid / s.Cpad;
  if (rest >= long(nblist) * s.n) return;
  int i = int(rest % s.n);
  int k = blist[rest / s.n];
  if (c >= s.C) return;
  const int bp = s.bpoff[k];
  constexpr int NP = B * (B + 1) / 2;
  double h[B][B];
  build_h<B>(s, c, i, bp, h);
  const double tp = s.tau * kPi2;
  double nrm = 0;
#pragma unroll
  for (int p = 0; p < B; ++p) {
    double rs = 0;
#pragma unroll
    for (int q = 0; q < B; ++q) rs += fabs(h[p][q]);
    nrm = fmax(nrm, rs);
  }
  nrm *= tp;
  int sq = 0;
  if (nrm > 0.5) {
    frexp(nrm / 0.5, &sq);  // nrm / 0.5 < 2^sq
    sq = min(sq, 60);
  }
  const double sc = ldexp(tp, -sq);
  const int K = taylor_degree(ldexp(nrm, -sq), s.mixed != 0);
  // The degree-K Taylor polynomial of exp(-iX) as cos X - i sin X with cos X = C(Y) of degree
  // K/2 and sin X = X S(Y) of degree (K-1)/2 in Y = X^2, each by Paterson-Stockmeyer in Y^2
  // (K = 11: 7 symmetric products instead of 10).  X waits in this thread's slice of shared
  // memory, so that five packed arrays are live in registers.
  __shared__ double Xs[NP * kThreads];
  double Y[NP], Y2[NP], R[NP], S[NP], T[NP];
#pragma unroll
  for (int p = 0; p < B; ++p)
#pragma unroll
    for (int q = p; q < B; ++q) T[sx<B>(p, q)] = sc * h[p][q];
#pragma unroll
  for (int j = 0; j < NP; ++j) Xs[j * blockDim.x + threadIdx.x] = T[j];
  sym_mul<B>(T, T, Y, 1.0);
  sym_mul<B>(Y, Y, Y2, 1.0);
  ps_poly<B, false>(K / 2, Y, Y2, R, T);        // R = cos X
  ps_poly<B, true>((K - 1) / 2, Y, Y2, S, T);   // S(Y)
#pragma unroll
  for (int j = 0; j < NP; ++j) T[j] = Xs[j * blockDim.x + threadIdx.x];
  double *I = Y2;
  sym_mul<B>(T, S, I, -1.0);  // I = -sin X = -X S(Y)
  // (R + iI)^2 = (R R - I I) + i 2 R I
  for (int t = 0; t < sq; ++t) {
    sym_mul<B>(R, R, Y, 1.0);
    sym_mul<B>(I, I, S, 1.0);
    sym_mul<B>(R, I, T, 2.0);
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      R[j] = Y[j] - S[j];
      I[j] = T[j];
    }
  }
  double2 *Ub = s.U + size_t(i) * s.S2 * s.Cpad;
  const double2 *fr = frame_of(s, i);
  const int bo = s.boff[k];
#pragma unroll
  for (int p = 0; p < B; ++p)
#pragma unroll
    for (int q = p; q < B; ++q) {
      double2 u = cmk(R[sx<B>(p, q)], I[sx<B>(p, q)]);
      store_u_pair(Ub, c, s.Cpad, bp, bo, B, p, q, u, fr, s.mixed != 0);
    }
}

// One thread per (crystallite, block, segment, column j): column j of the segment's products
// P_i = U_i P_{i-1}, or (prefix) of the chain over the segments' last products (seg_chain).
template <int B>
__global__ void __launch_bounds__(kThreads) k_dyson(DevSys s, const int *__restrict__ blist, int nblist, int nseg,
                                                    bool prefix) {
  long tid = long(blockIdx.x) * blockDim.x + threadIdx.x;
  int c = int(tid % s.Cpad);
  long rest = tid / s.Cpad;
  if (rest >= long(nblist) * B * nseg) return;
  int j = int(rest % B);
  const int seg = int(rest / B % nseg);
  int k = blist[rest / B / nseg];
  if (c >= s.C) return;
  const int bp = s.bpoff[k];
  const Chain ch = seg_chain(s, B, seg, prefix);
  double2 x[B];
#pragma unroll
  for (int r = 0; r < B; ++r) x[r] = cmk(r == j ? 1.0 : 0.0, 0.0);
  for (int i = 0; i < ch.count; ++i) {
    const double2 *Ub = ch.from(s, i);
    double2 y[B];
#pragma unroll
    for (int r = 0; r < B; ++r) {
      double2 acc = cmk(0, 0);
#pragma unroll
      for (int l = 0; l < B; ++l) acc = cfma(Ub[at(bp + r * B + l, c, s.Cpad)], x[l], acc);
      y[r] = acc;
    }
    double2 *Ab = ch.to(s, i);
#pragma unroll
    for (int r = 0; r < B; ++r) {
      x[r] = y[r];
      Ab[at(bp + r * B + j, c, s.Cpad)] = y[r];
    }
  }
}

// The mixed form's Dyson product in double-float: one lane per (crystallite, block, segment,
// column, row), U_i and A_{i+1} as float4 double-float elements; each element of U_i x is four
// compensated dot products (re and im, each of a U-hi/lo x-hi/lo expansion).
template <int B>
__global__ void __launch_bounds__(kThreads) k_dyson_df(DevSys s, const int *__restrict__ blist, int nblist, int nseg,
                                                       bool prefix) {
  // G lanes per (crystallite, column j): lane r < B owns row r of the column; a warp holds
  // 32/G consecutive crystallites of one (block, column), so the U rows it loads are whole
  // 16-byte runs of consecutive crystallites.  y_r = sum_l U_rl x_l, l ascending, each x_l
  // broadcast from lane l of the group: the same sums in the same order as one thread per
  // column, with B times the threads on the chain of n dependent steps.  The next step's U
  // row is loaded while this step is summed.
  constexpr int G = B <= 1 ? 1 : B <= 2 ? 2 : B <= 4 ? 4 : 8;
  static_assert(B <= 8, "k_dyson_df takes blocks of at most 8");
  const long tid = long(blockIdx.x) * blockDim.x + threadIdx.x;
  const int r = int(tid % G);
  const long rest = tid / G;
  const int c = int(rest % s.Cpad);
  const long rest2 = rest / s.Cpad;
  if (rest2 >= long(nblist) * B * nseg) return;  // warp-uniform (G Cpad is a multiple of 32)
  const int j = int(rest2 % B), seg = int(rest2 / B % nseg), k = blist[rest2 / B / nseg];
  const int bp = s.bpoff[k];
  const Chain ch = seg_chain(s, B, seg, prefix);
  const bool own = r < B;
  const int lane0 = int(threadIdx.x & 31) & ~(G - 1);
  float4 u[B], un[B];
  auto load_row = [&](int i, float4(&d)[B]) {
    const float4 *Ub = reinterpret_cast<const float4 *>(ch.from(s, i));
#pragma unroll
    for (int l = 0; l < B; ++l) d[l] = own ? Ub[at(bp + r * B + l, c, s.Cpad)] : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  load_row(0, u);
  float4 x = make_float4(r == j ? 1.f : 0.f, 0.f, 0.f, 0.f);
  for (int i = 0; i < ch.count; ++i) {
    if (i + 1 < ch.count) load_row(i + 1, un);
    DfAcc re = {0.f, 0.f}, im = {0.f, 0.f};
#pragma unroll
    for (int l = 0; l < B; ++l) {
      float4 xl;
      xl.x = __shfl_sync(0xffffffffu, x.x, lane0 + l);
      xl.y = __shfl_sync(0xffffffffu, x.y, lane0 + l);
      xl.z = __shfl_sync(0xffffffffu, x.z, lane0 + l);
      xl.w = __shfl_sync(0xffffffffu, x.w, lane0 + l);
      const float4 uu = u[l];
      df_dot(re, uu.x, uu.z, xl.x, xl.z);    // ur xr
      df_dot(re, -uu.y, -uu.w, xl.y, xl.w);  // - ui xi
      df_dot(im, uu.x, uu.z, xl.y, xl.w);    // ur xi
      df_dot(im, uu.y, uu.w, xl.x, xl.z);    // ui xr
    }
    const float2 a = df_fin(re), b = df_fin(im);
    x = make_float4(a.x, b.x, a.y, b.y);
    if (own && c < s.C) {
      float4 *Ab = reinterpret_cast<float4 *>(ch.to(s, i));
      Ab[at(bp + r * B + j, c, s.Cpad)] = x;
    }
#pragma unroll
    for (int l = 0; l < B; ++l) u[l] = un[l];
  }
}

// One thread per (crystallite, block): Floquet eigen-decomposition of A_n.
template <int B>
__global__ void __launch_bounds__(kThreads) k_floquet(DevSys s, const int *__restrict__ blist, int nblist) {
  long tid = long(blockIdx.x) * blockDim.x + threadIdx.x;
  int c = int(tid % s.Cpad);
  long rest = tid / s.Cpad;
  if (rest >= nblist) return;
  int k = blist[rest];
  if (c >= s.C) return;
  const int bp = s.bpoff[k], bo = s.boff[k];
  const double2 *An = period_prop(s, B);
  const float4 *An4 = reinterpret_cast<const float4 *>(An);  // mixed form: double-float A
  double2 U[B][B], lam[B], V[B][B];
#pragma unroll
  for (int r = 0; r < B; ++r)
#pragma unroll
    for (int q = 0; q < B; ++q)
      U[r][q] = s.mixed ? df_load(An4[at(bp + r * B + q, c, s.Cpad)]) : An[at(bp + r * B + q, c, s.Cpad)];
  int st = unitary_eig<B>(U, lam, V);
  if (st) atomicOr(s.status, st);
#pragma unroll
  for (int r = 0; r < B; ++r) {
#pragma unroll
    for (int q = 0; q < B; ++q) s.VF[at(bp + r * B + q, c, s.Cpad)] = V[r][q];
    // principal-branch log: (ln|lam|, atan2)   (complex.h:1058-1061)
    s.L[at(bo + r, c, s.Cpad)] = cmk(log(hypot(lam[r].x, lam[r].y)), atan2(lam[r].y, lam[r].x));
  }
}


// ------------------------------------------------------------------ Floquet, lanes per matrix
// The FP64 pipe costs a warp instruction whatever its active lanes, so one thread per
// (crystallite, block) leaves most SM sub-partitions idle when there are few blocks.  Here B
// lanes work on one matrix (lane r owns row r), 32/B matrices per warp: the same Cayley
// transform with partial pivoting and back substitution as unitary_eig, then a parallel
// (round-robin) complex Jacobi on K as in floquet_cta, and the Rayleigh quotients.  Every
// index into a lane's row is a compile-time constant (the rounds and pairs are unrolled);
// rows move between lanes by shuffles within the group.
template <int B>
struct LaneGroup {
  unsigned mask;
  int base;
  __device__ __forceinline__ double shfl(double v, int src) const { return __shfl_sync(mask, v, base + src); }
  __device__ __forceinline__ double2 shfl(double2 v, int src) const { return cmk(shfl(v.x, src), shfl(v.y, src)); }
  __device__ __forceinline__ int shfl(int v, int src) const { return __shfl_sync(mask, v, base + src); }
  __device__ __forceinline__ float shfl(float v, int src) const { return __shfl_sync(mask, v, base + src); }
  __device__ __forceinline__ float2 shfl(float2 v, int src) const {
    return make_float2(shfl(v.x, src), shfl(v.y, src));
  }
};
template <class T> struct LaneCx;
template <> struct LaneCx<double> { using type = double2; };
template <> struct LaneCx<float> { using type = float2; };
__device__ __forceinline__ double2 cxm(double r, double i) { return make_double2(r, i); }
__device__ __forceinline__ float2 cxm(float r, float i) { return make_float2(r, i); }

// K = Hermitian part of i (I+W)^{-1} (I-W), W = ea U, for the group's matrix (lane r holds row r):
// Gaussian elimination with partial pivoting (first largest |M[i][k]|, i >= k) and back
// substitution in T.  Returns kSingularCayley for a zero pivot; soft: such pivots (and those
// below 1e-7, which single precision cannot tell from zero) are replaced by 1e-7 instead.
template <int B, class T>
__device__ __forceinline__ int lanes_cayley(const LaneGroup<B> &g, int r, const double2 (&U)[B], double2 ea,
                                            typename LaneCx<T>::type (&K)[B], bool soft) {
  using CT = typename LaneCx<T>::type;
  int st = 0;
  CT M[B], X[B];
#pragma unroll
  for (int q = 0; q < B; ++q) {
    const double id = (q == r) ? 1.0 : 0.0;
    // I + W and I - W rounded once: W rounded on its own would add 2^-24 where they are small
    const double2 w = soft ? todbl(cmul(cvt<float2>(ea), cvt<float2>(U[q]))) : cmul(ea, U[q]);
    M[q] = cxm(T(id + w.x), T(w.y)), X[q] = cxm(T(id - w.x), T(-w.y));
  }
#pragma unroll
  for (int kc = 0; kc < B; ++kc) {
    const T m2 = (r >= kc) ? M[kc].x * M[kc].x + M[kc].y * M[kc].y : T(-1);
    int piv = kc;
    T best = g.shfl(m2, kc);
#pragma unroll
    for (int i = kc + 1; i < B; ++i) {
      const T v = g.shfl(m2, i);
      if (v > best) best = v, piv = i;
    }
    if (best == T(0) && !soft) st |= kSingularCayley;
    const int src = (r == kc) ? piv : (r == piv ? kc : r);
#pragma unroll
    for (int q = 0; q < B; ++q) M[q] = g.shfl(M[q], src), X[q] = g.shfl(X[q], src);
    if (soft && best < T(1e-14) && r == kc) M[kc] = cxm(T(1e-7), T(0));
    CT Mk[B], Xk[B];
#pragma unroll
    for (int q = 0; q < B; ++q) Mk[q] = g.shfl(M[q], kc), Xk[q] = g.shfl(X[q], kc);
    if (r > kc) {
      const CT f = cmul(M[kc], cdiv(cxm(T(1), T(0)), Mk[kc]));
#pragma unroll
      for (int q = kc; q < B; ++q) M[q] = csub(M[q], cmul(f, Mk[q]));
#pragma unroll
      for (int q = 0; q < B; ++q) X[q] = csub(X[q], cmul(f, Xk[q]));
    }
  }
  // back substitution, row kc on lane kc from the final rows below it
#pragma unroll
  for (int kc = B - 1; kc >= 0; --kc) {
    CT acc[B];
#pragma unroll
    for (int q = 0; q < B; ++q) acc[q] = X[q];
#pragma unroll
    for (int i = kc + 1; i < B; ++i) {
      const CT mki = M[i];  // M[kc][i] on lane kc
#pragma unroll
      for (int q = 0; q < B; ++q) {
        const CT xiq = g.shfl(X[q], i);
        acc[q] = csub(acc[q], cmul(mki, xiq));
      }
    }
    if (r == kc) {
      const CT inv = cdiv(cxm(T(1), T(0)), M[kc]);
#pragma unroll
      for (int q = 0; q < B; ++q) X[q] = cmul(acc[q], inv);
    }
  }
  // Hermitian part of i X (row r needs column r of X: X[q][r] from lane q)
#pragma unroll
  for (int q = 0; q < B; ++q) {
    CT xqr = cxm(T(0), T(0));
#pragma unroll
    for (int t = 0; t < B; ++t) {
      const CT v = g.shfl(X[t], q);
      if (t == r) xqr = v;
    }
    const CT krq = cxm(-X[q].y, X[q].x), kqr = cxm(-xqr.y, xqr.x);
    K[q] = cscale(cadd(krq, cconj(kqr)), T(0.5));
    if (q == r) K[q].y = T(0);
  }
  return st;
}

// FP64 sweeps: a rotated element is set to zero when it was at most kSweepZero of the pair's larger
// diagonal element (an angle from single precision leaves under 2^-21 of it), and neither rotated nor
// kept at kSweepRound of it.  Either form: no rotation for an element of at most kSweepTiny (off(K)^2
// is below 1e-60 then; 1 / |K_pq| overflows from 2^-128 down, and equal diagonal elements make that
// factor count).
constexpr float kSweepZero = 0x1p-32f, kSweepRound = 0x1p-52f, kSweepTiny = 1e-30f;
// Parallel (round-robin) complex Jacobi sweeps over K, at most `sweeps`; with VEC, V (FP64)
// accumulates the rotations from the identity.  The rotation angles come from single precision
// in both forms (an FP64 hypot, three divisions and two square roots per rotation were more than
// half of the kernel's FP64 instructions): a rotation that misses its angle by 1e-7 of it leaves
// 1e-7 of the element, which the next sweep removes.  Where that is below the rounding of the
// diagonal (kSweepZero), the element is set to zero after its rotation, and one at the rounding
// itself (kSweepRound) without a rotation: between equal eigenvalues (equivalent spins, spins
// without couplings) the angle is of order one, and what such a rotation leaves is fresh rounding of
// the diagonal, sweep after sweep.  Sweeps of matrices with two to b distinct eigenvalues, b = 2 to
// 35, in this arithmetic on the host: 5.5 on average and at most 17 (with FP64 angles and every rotated
// element set to zero 5.4 and at most 30); of generic ones 5.6 (5.1).  In single precision the angle
// has all of K's bits and every rotated element is set to zero: turning what its rounding leaves once
// more would put that into V.  Each rotation is scaled to c^2 + |s|^2 = 1 in FP64 (n^-1/2 = 1 - d/2 + 3 d^2/8 for n = 1 + d, d ~ 1e-7), so V
// stays unitary to FP64 rounding; K takes the scaled rotation in FP64 and the single-precision
// one otherwise.  T = double stops at off(K)^2 <= 1e-34 diag(K)^2 (or 1e-60: K = tan(phase / 2), so
// what is left is far below any phase); T = float one sweep after 1e-10 diag(K)^2 (quadratic
// convergence takes that to the float floor).
template <int B, class T, bool VEC>
__device__ __forceinline__ bool lanes_sweeps(const LaneGroup<B> &g, int r, typename LaneCx<T>::type (&K)[B],
                                             double2 (&V)[B], int sweeps) {
  using CT = typename LaneCx<T>::type;
  constexpr bool F32 = sizeof(T) == sizeof(float);
  constexpr int BQ = B + (B & 1), NP = BQ / 2;  // round-robin players (one dummy when B is odd)
  if (VEC) {
#pragma unroll
    for (int q = 0; q < B; ++q) V[q] = cmk(q == r ? 1.0 : 0.0, 0.0);
  }
  bool polish = false;
  for (int sweep = 0; sweep < sweeps; ++sweep) {
    T off = 0, dg = 0;
#pragma unroll
    for (int q = 0; q < B; ++q) {
      if (q > r) off += K[q].x * K[q].x + K[q].y * K[q].y;
      if (q == r) dg += K[q].x * K[q].x;
    }
    T offs = 0, dgs = 0;
#pragma unroll
    for (int t = 0; t < B; ++t) offs += g.shfl(off, t), dgs += g.shfl(dg, t);
    if (F32) {
      const bool small = offs <= T(1e-10) * dgs || offs == T(0);
      if (small && (polish || offs == T(0))) return true;
      polish = polish || small;
    } else if (offs <= T(1e-34) * dgs || offs <= T(1e-60)) {
      return true;
    }
#pragma unroll
    for (int round = 0; round < BQ - 1; ++round) {
      // this lane's pair (mp, mq) of the round, or none
      int mp = r, mq = r;
      bool paired = false;
#pragma unroll
      for (int t = 0; t < NP; ++t) {
        const int j1 = t, j2 = BQ - 1 - t;
        int p = j1 == 0 ? 0 : 1 + (j1 - 1 + round) % (BQ - 1);
        int q = j2 == 0 ? 0 : 1 + (j2 - 1 + round) % (BQ - 1);
        if (p > q) { const int x = p; p = q; q = x; }
        if (q < B && (r == p || r == q)) mp = p, mq = q, paired = true;
      }
      // the pair's rotation, computed identically by both of its lanes from K[p][q]
      // (lane p's entry q), K[p][p] and K[q][q]
      CT own_q = cxm(T(0), T(0)), own_d = cxm(T(0), T(0));
#pragma unroll
      for (int q2 = 0; q2 < B; ++q2) {
        if (q2 == mq) own_q = K[q2];
        if (q2 == r) own_d = K[q2];
      }
      const CT hpq = g.shfl(own_q, mp);
      const T kpp = g.shfl(own_d.x, mp), kqq = g.shfl(own_d.x, mq);
      float cf = 1.f, sx = 0.f, sy = 0.f;
      bool zero = false;
      if (paired) {
        const float hx = float(hpq.x), hy = float(hpq.y);
        const float ab = hypotf(hx, hy), dmax = F32 ? 0.f : fmaxf(fabsf(float(kpp)), fabsf(float(kqq)));
        zero = !F32 && ab <= fmaxf(kSweepZero * dmax, kSweepTiny);
        if (ab > fmaxf(kSweepRound * dmax, kSweepTiny)) {
          const float theta = 0.5f * float(kqq - kpp) / ab;
          float tt;
          if (fabsf(theta) > 1e18f) tt = 0.5f / theta;  // theta^2 stays finite
          else tt = copysignf(1.f, theta) / (fabsf(theta) + sqrtf(fmaf(theta, theta, 1.f)));
          cf = rsqrtf(fmaf(tt, tt, 1.f));
          const float ts = tt * cf / ab;
          sx = hx * ts, sy = hy * ts;
          zero = zero || F32;
        }
      }
      double cd = cf;
      double2 sd = cmk(sx, sy);
      if (VEC || !F32) {
        const double d = fma(cd, cd, fma(sd.x, sd.x, fma(sd.y, sd.y, -1.0)));
        const double nn = fma(fma(0.375, d, -0.5), d, 1.0);
        cd *= nn, sd = cscale(sd, nn);
      }
      T cs;
      CT sp;
      if constexpr (F32) cs = cf, sp = cxm(sx, sy);
      else cs = cd, sp = sd;
      // columns p, q of K and V for every pair: K <- K G, V <- V G, G = [[c, sp], [-conj(sp), c]]
#pragma unroll
      for (int t = 0; t < NP; ++t) {
        const int j1 = t, j2 = BQ - 1 - t;
        int p = j1 == 0 ? 0 : 1 + (j1 - 1 + round) % (BQ - 1);
        int q = j2 == 0 ? 0 : 1 + (j2 - 1 + round) % (BQ - 1);
        if (p > q) { const int x = p; p = q; q = x; }
        if (q >= B) continue;
        const T cst = g.shfl(cs, p);
        const CT spt = g.shfl(sp, p), spc = cconj(spt);
        const CT kp = K[p], kq = K[q];
        K[p] = csub(cscale(kp, cst), cmul(spc, kq));
        K[q] = cadd(cmul(spt, kp), cscale(kq, cst));
        if (VEC) {
          double ct;
          double2 st;
          if constexpr (F32) ct = g.shfl(cd, p), st = g.shfl(sd, p);
          else ct = cst, st = spt;
          const double2 vp = V[p], vq = V[q];
          V[p] = csub(cscale(vp, ct), cmul(cconj(st), vq));
          V[q] = cadd(cmul(st, vp), cscale(vq, ct));
        }
      }
      // rows p, q of K: K <- G^H K, as row = alpha row_p + beta row_q in every lane
      // (lane p: cs, -sp; lane q: conj(sp), cs; a lane without a pair keeps its row)
      const bool isp = paired && r == mp;
      const CT al = isp ? cxm(cs, T(0)) : cconj(sp), be = isp ? cxm(-sp.x, -sp.y) : cxm(cs, T(0));
#pragma unroll
      for (int q2 = 0; q2 < B; ++q2) {
        const CT kpk = g.shfl(K[q2], mp), kqk = g.shfl(K[q2], mq);
        if (paired) {
          // one of alpha, beta is real: the products differ between the lanes of a pair
          const CT u = isp ? kpk : kqk, v = isp ? kqk : kpk, sg = isp ? be : al;
          K[q2] = cadd(cscale(u, cs), cmul(sg, v));
          if (q2 == r) K[q2].y = T(0);
          if (zero && q2 == (isp ? mq : mp)) K[q2] = cxm(T(0), T(0));
        }
      }
    }
  }
  return false;
}

// T = double: the FP64 form.  T = float (mixed form): the Cayley transform and the sweeps over K
// in single precision, V in FP64 (the FID's reconstruction takes V^-1 = V^H, which a
// single-precision V, unitary to ~1e-7 per rotation, breaks by more than 1e-6).  The eigenvalues
// are FP64 Rayleigh quotients in both: their error is quadratic in V's, so the phases that the
// FID carries over npts points keep FP64 accuracy.
// The shift a has to keep every |1 + e^{ia} lambda| well above zero.  Phases near 0 (A_n near I, as
// under fast spinning) take a = 1/2; otherwise -1 goes into the widest gap of the spectrum, found
// by a single-precision pass without vectors (K's eigenvalues are tan((theta + a) / 2)) where a
// full first pass found it before.  A second pass follows only if the first turns out badly
// conditioned after all.  Measured, with the single-precision angles: a 4-block under rf, 677
// crystallites, FP64 215 -> 100 us; 4 spins, 3722 crystallites, FP64 0.78 -> 0.58 ms, mixed 0.34 ->
// 0.20 ms; one 3-spin crystallite 89 -> 63 us.
template <int B, class T>
__global__ void __launch_bounds__(kThreads) k_floquet_lanes(DevSys s, const int *__restrict__ blist, int nblist) {
  using CT = typename LaneCx<T>::type;
  constexpr int GPW = 32 / B;             // matrices per warp
  const int lane = threadIdx.x & 31;
  const long warp = (long(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int gi = lane / B, r = lane % B;
  if (gi >= GPW) return;
  const long item = warp * GPW + gi;
  if (item >= long(nblist) * s.Cpad) return;
  const int c = int(item % s.Cpad), k = blist[item / s.Cpad];
  if (c >= s.C) return;  // the whole group leaves together
  const LaneGroup<B> g{((1u << B) - 1u) << (gi * B), gi * B};
  const int bp = s.bpoff[k], bo = s.boff[k];
  const double2 *An = period_prop(s, B);
  const float4 *An4 = reinterpret_cast<const float4 *>(An);  // mixed form: double-float A
  double2 U[B], lam[B], V[B];  // V accumulates in FP64 in both forms
#pragma unroll
  for (int q = 0; q < B; ++q)
    U[q] = s.mixed ? df_load(An4[at(bp + r * B + q, c, s.Cpad)]) : An[at(bp + r * B + q, c, s.Cpad)];
  int st = 0;
  double a = 0.5;
  float dev = 0.f;  // |A_n - I|_F^2
#pragma unroll
  for (int q = 0; q < B; ++q) {
    const float2 u = cvt<float2>(U[q]);
    dev = fmaf(u.y, u.y, fmaf(u.x - (q == r ? 1.f : 0.f), u.x - (q == r ? 1.f : 0.f), dev));
  }
  float devs = 0.f;
#pragma unroll
  for (int t = 0; t < B; ++t) devs += g.shfl(dev, t);
  if (devs > 1.44f) {  // some phase may exceed 1.3: where to put -1, in single precision
    float2 Kf[B];
    lanes_cayley<B, float>(g, r, U, cmk(0.87758256189037271612, 0.47942553860420300027), Kf, true);  // e^{i/2}
    lanes_sweeps<B, float, false>(g, r, Kf, V, 12);
    float own = 0.f;
#pragma unroll
    for (int q = 0; q < B; ++q)
      if (q == r) own = 2.f * atanf(Kf[q].x) - 0.5f;
    if (own < -3.14159265f) own += 6.28318531f;
    float th[B];
#pragma unroll
    for (int q = 0; q < B; ++q) th[q] = g.shfl(own, q);
#pragma unroll
    for (int i = 1; i < B; ++i)
#pragma unroll
      for (int j = i; j > 0; --j)
        if (th[j - 1] > th[j]) { const float x = th[j]; th[j] = th[j - 1]; th[j - 1] = x; }
    float best = -1.f, mid = 0.f;
#pragma unroll
    for (int q = 0; q < B; ++q) {
      const float lo = th[q], hi = (q + 1 < B) ? th[q + 1] : th[0] + 6.28318531f;
      if (hi - lo > best) best = hi - lo, mid = 0.5f * (lo + hi);
    }
    if (best > 0.f) a = kPi - double(mid);  // (not a number: the first shift stays)
  }
  for (int pass = 0; pass < 2; ++pass) {
    double sa, ca;
    sincos(a, &sa, &ca);
    const double2 ea = cmk(ca, sa);
    CT K[B];
    st |= lanes_cayley<B, T>(g, r, U, ea, K, false);
    if (!lanes_sweeps<B, T, true>(g, r, K, V, kMaxSweeps)) st |= kNoConvergeFloquet;
    // Rayleigh quotients lam_r = v_r^H U v_r (columns of V), in every lane
    double2 uv[B];
#pragma unroll
    for (int q = 0; q < B; ++q) uv[q] = cmk(0, 0);
#pragma unroll
    for (int l = 0; l < B; ++l)
#pragma unroll
      for (int q = 0; q < B; ++q) uv[q] = cfma(U[l], todbl(g.shfl(V[q], l)), uv[q]);  // (U V)[r][q], l ascending
#pragma unroll
    for (int q = 0; q < B; ++q) lam[q] = cmk(0, 0);
#pragma unroll
    for (int kk = 0; kk < B; ++kk)
#pragma unroll
      for (int q = 0; q < B; ++q) lam[q] = cfmaconj(todbl(g.shfl(V[q], kk)), g.shfl(uv[q], kk), lam[q]);
    if (pass == 1) break;
    double mind = 4.0;
#pragma unroll
    for (int q = 0; q < B; ++q) {
      const double2 w = cmul(ea, lam[q]);
      mind = fmin(mind, (1.0 + w.x) * (1.0 + w.x) + w.y * w.y);
    }
    if (mind >= 0.0625) break;
    // widest gap of the eigenphases (every lane, same values): -1 into its middle
    double th[B];
#pragma unroll
    for (int q = 0; q < B; ++q) th[q] = atan2(lam[q].y, lam[q].x);
#pragma unroll
    for (int i = 1; i < B; ++i)
#pragma unroll
      for (int j = i; j > 0; --j)
        if (th[j - 1] > th[j]) { const double x = th[j]; th[j] = th[j - 1]; th[j - 1] = x; }
    double best = -1, mid = 0;
#pragma unroll
    for (int q = 0; q < B; ++q) {
      const double lo = th[q], hi = (q + 1 < B) ? th[q + 1] : th[0] + kPi2;
      if (hi - lo > best) best = hi - lo, mid = 0.5 * (lo + hi);
    }
    a = kPi - mid;
  }
  if (st && r == 0) atomicOr(s.status, st);
#pragma unroll
  for (int q = 0; q < B; ++q) s.VF[at(bp + r * B + q, c, s.Cpad)] = todbl(V[q]);
  double2 lr = cmk(0, 0);
#pragma unroll
  for (int q = 0; q < B; ++q)
    if (q == r) lr = lam[q];
  // principal-branch log: (ln|lam|, atan2)   (complex.h:1058-1061)
  s.L[at(bo + r, c, s.Cpad)] = cmk(log(hypot(lr.x, lr.y)), atan2(lr.y, lr.x));
}

// One thread per (crystallite, block, segment s): V_s = E_s V_F, s = 1 .. nseg - 1, in FP64 over
// E_s; in the mixed form (s = 0 included, where it is V_F) in double-float, rounded to float2.
template <int B, bool MIX>
__global__ void __launch_bounds__(kThreads) k_seg_frame(DevSys s, const int *__restrict__ blist, int nblist) {
  const long tid = long(blockIdx.x) * blockDim.x + threadIdx.x;
  const int c = int(tid % s.Cpad), ns = MIX ? s.nseg : s.nseg - 1;
  const long rest = tid / s.Cpad;
  if (rest >= long(nblist) * ns) return;
  const int t = int(rest % ns) + (MIX ? 0 : 1), k = blist[rest / ns];
  if (c >= s.C) return;
  const int bp = s.bpoff[k];
  if constexpr (MIX) {
    float2 *Vo = seg_Vf(s, t);
    if (t == 0) {
#pragma unroll
      for (int e = 0; e < B * B; ++e) Vo[at(bp + e, c, s.Cpad)] = cvt<float2>(s.VF[at(bp + e, c, s.Cpad)]);
      return;
    }
    const float4 *E = reinterpret_cast<const float4 *>(seg_E(s, t - 1));
#pragma unroll 1
    for (int q = 0; q < B; ++q) {  // a column of V at a time
      float4 v[B];
#pragma unroll
      for (int l = 0; l < B; ++l) v[l] = df_store(s.VF[at(bp + l * B + q, c, s.Cpad)]);
#pragma unroll
      for (int r = 0; r < B; ++r) {
        CdfAcc a = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll
        for (int l = 0; l < B; ++l) cdf_mac(a, E[at(bp + r * B + l, c, s.Cpad)], v[l]);
        const float4 w = cdf_fin(a);
        Vo[at(bp + r * B + q, c, s.Cpad)] = make_float2(w.x, w.y);
      }
    }
  } else {
    double2 *E = seg_E(s, t - 1);
    double2 V[B][B];
#pragma unroll
    for (int r = 0; r < B; ++r)
#pragma unroll
      for (int q = 0; q < B; ++q) V[r][q] = s.VF[at(bp + r * B + q, c, s.Cpad)];
#pragma unroll
    for (int r = 0; r < B; ++r) {
      double2 e[B];
#pragma unroll
      for (int l = 0; l < B; ++l) e[l] = E[at(bp + r * B + l, c, s.Cpad)];
#pragma unroll
      for (int q = 0; q < B; ++q) {
        double2 acc = cmk(0, 0);
#pragma unroll
        for (int l = 0; l < B; ++l) acc = cfma(e[l], V[l][q], acc);
        E[at(bp + r * B + q, c, s.Cpad)] = acc;
      }
    }
  }
}

// V of step i in the precision of C: V_F, or the V_s of the step's segment.
template <class C>
__device__ __forceinline__ C frame_elem(const DevSys &s, bool seg, int i, size_t x) {
  if constexpr (std::is_same<C, float2>::value)
    return seg ? seg_Vf(s, i / kSegLen)[x] : cvt<C>(s.VF[x]);
  else
    return seg && i >= kSegLen ? seg_E(s, i / kSegLen - 1)[x] : s.VF[x];
}

// One thread per (crystallite, block, step): W_i = A_{i+1} V_F = P_i V_s (in place over A in
// FP64; into the single-precision W array in the mixed form).
template <int B, class C>
__global__ void __launch_bounds__(kThreads) k_eigframe(DevSys s, const int *__restrict__ blist, int nblist) {
  long tid = long(blockIdx.x) * blockDim.x + threadIdx.x;
  int c = int(tid % s.Cpad);
  long rest = tid / s.Cpad;
  if (rest >= long(nblist) * s.n) return;
  int i = int(rest % s.n);
  int k = blist[rest / s.n];
  if (c >= s.C) return;
  const int bp = s.bpoff[k];
  C V[B][B];
#pragma unroll
  for (int r = 0; r < B; ++r)
#pragma unroll
    for (int q = 0; q < B; ++q) V[r][q] = frame_elem<C>(s, segmented(s, B), i, at(bp + r * B + q, c, s.Cpad));
  const double2 *Ab = s.A + size_t(i) * s.S2 * s.Cpad;
  const float4 *Ab4 = reinterpret_cast<const float4 *>(Ab);  // mixed form: double-float A
  C *Wb = Bufs<C>::W(s) + size_t(i) * s.S2 * s.Cpad;
#pragma unroll
  for (int r = 0; r < B; ++r) {
    C a[B];
#pragma unroll
    for (int l = 0; l < B; ++l) {
      if (s.mixed) {  // single precision from here on: the high parts
        const float4 v = Ab4[at(bp + r * B + l, c, s.Cpad)];
        a[l] = mkc<C>(v.x, v.y);
      } else {
        a[l] = cvt<C>(Ab[at(bp + r * B + l, c, s.Cpad)]);
      }
    }
#pragma unroll
    for (int q = 0; q < B; ++q) {
      C acc = mkc<C>(0, 0);
#pragma unroll
      for (int l = 0; l < B; ++l) acc = cfma(a[l], V[l][q], acc);
      Wb[at(bp + r * B + q, c, s.Cpad)] = acc;
    }
  }
}

// One thread per (crystallite, step, pair): Q^{ab} = W_a^H D_ab W_b  (and R pairs).
// compute.h:378-383: Qs[i] = adjprop(evect, adjprop(As[i+1], det)).
template <class C>
__global__ void __launch_bounds__(kThreads) k_qr(DevSys s) {
  long tid = long(blockIdx.x) * blockDim.x + threadIdx.x;
  int c = int(tid % s.Cpad);
  long rest = tid / s.Cpad;
  int npair = s.npq + s.npr;
  if (rest >= long(npair) * s.n) return;
  int i = int(rest % s.n);
  int pr = int(rest / s.n);
  if (c >= s.C) return;
  bool isq = pr < s.npq;
  int a, b, off, moff;
  const double2 *M;
  C *out;
  int nitems;
  if (isq) {
    a = s.qa[pr], b = s.qb[pr], off = s.qoff[pr], moff = s.doff[pr], M = s.Dblk, out = Bufs<C>::Q(s), nitems = s.nq;
  } else {
    int p2 = pr - s.npq;
    a = s.ra[p2], b = s.rb[p2], off = s.roff[p2], moff = s.rhooff[p2], M = s.Rhoblk, out = Bufs<C>::R(s);
    nitems = s.nr;
  }
  const int ba = s.bs[a], bb = s.bs[b], pa = s.bpoff[a], pb = s.bpoff[b];
  if (ba > kMaxBlock || bb > kMaxBlock) return;  // k_big_qr handles pairs with a large block
  const C *W = Bufs<C>::W(s) + size_t(i) * s.S2 * s.Cpad;
  C X[kMaxBlock * kMaxBlock];
  // X = M_ab W_b  (ba x bb)
  for (int l = 0; l < ba; ++l)
    for (int q = 0; q < bb; ++q) X[l * bb + q] = mkc<C>(0, 0);
  for (int l = 0; l < ba; ++l)
    for (int m = 0; m < bb; ++m) {
      double2 d2 = M[moff + l * bb + m];
      if (!nonzero(d2)) continue;
      const C d = cvt<C>(d2);
      for (int q = 0; q < bb; ++q) X[l * bb + q] = cfma(d, W[at(pb + m * bb + q, c, s.Cpad)], X[l * bb + q]);
    }
  C *ob = out + size_t(i) * nitems * s.Cpad;
  for (int r = 0; r < ba; ++r)
    for (int q = 0; q < bb; ++q) {
      C acc = mkc<C>(0, 0);
      for (int l = 0; l < ba; ++l) acc = cfmaconj(W[at(pa + l * ba + r, c, s.Cpad)], X[l * bb + q], acc);
      ob[at(off + r * bb + q, c, s.Cpad)] = acc;
    }
}

constexpr int kFavePT = 8;

// One thread per (crystallite, element, tile of kFavePT values of p).
// G_p = sum_{i<n-p} q_{i+p} r_i + z sum_{i>=n-p} q_{i+p-n} r_i with z = e^{i n tau w}.
// Equals compute.h:406-427's Fave_p(r,s) times e^{i p tau w_rs}, so that
// fid[jn+p] = sum_e z_e^j G_p(e) reproduces compute.h:440-459.
__global__ void __launch_bounds__(kThreads) k_fave(DevSys s) {
  long tid = long(blockIdx.x) * blockDim.x + threadIdx.x;
  int c = int(tid % s.Cpad);
  long rest = tid / s.Cpad;
  int ntile = (s.n + kFavePT - 1) / kFavePT;
  if (rest >= long(s.ne) * ntile) return;
  int tile = int(rest % ntile);
  int e = int(rest / ntile);
  if (c >= s.C) return;
  const int eq = s.eq[e], erev = s.erev[e], er = s.er[e];
  // w_rs = chop((l_r - l_s)/(i n tau), 1e-10)   (compute.h:327-335)
  double2 lr = s.L[at(s.erg[e], c, s.Cpad)], ls = s.L[at(s.esg[e], c, s.Cpad)];
  double2 d = csub(lr, ls);
  double nt = double(s.n) * s.tau;
  double2 w = cmk(chop1(d.y / nt, 1e-10), chop1(-d.x / nt, 1e-10));
  // z = exp(i n tau w)
  double2 z = cexp(cmk(-nt * w.y, nt * w.x));
  if (tile == 0) {
    for (int m = 0; m < pair_rows(s.J); ++m) {
      const double pw = pair_power(s.J, m);
      s.Z[at(m * s.ne + e, c, s.Cpad)] = cexp(cmk(-pw * nt * w.y, pw * nt * w.x));
    }
  }
  // Three phases over i for the tile p0..p0+PT-1: all j = i+p < n (no wrap), the mixed
  // band of at most PT-1 steps, and all wrapped.  Only the band tests j < n per p, so
  // the bulk issues exactly one complex FMA per (i, p).  q_{(i+p) mod n} for the tile
  // sits in a register window that shifts by one element per step.
  const int n = s.n, p0 = tile * kFavePT;
  const size_t qstride = size_t(s.nq) * s.Cpad, rstride = size_t(s.nr) * s.Cpad;
  const double2 *qb = s.Q + at(eq, c, s.Cpad);
  const double2 *qr = s.Q + at(erev >= 0 ? erev : 0, c, s.Cpad);
  const double2 *rb = s.R + at(er >= 0 ? er : 0, c, s.Cpad);
  const bool rosym = s.rosym != 0, has_rev = erev >= 0;
  double2 s1[kFavePT], s2[kFavePT], win[kFavePT];
#pragma unroll
  for (int t = 0; t < kFavePT; ++t) {
    s1[t] = s2[t] = cmk(0, 0);
    win[t] = qb[size_t((p0 + t) % n) * qstride];
  }
  int jl = (p0 + kFavePT) % n;  // next window element to load
  auto rho_at = [&](int i) -> double2 {
    if (rosym) {
      double2 r = cconj(qb[size_t(i) * qstride]);
      if (has_rev) r = cadd(r, qr[size_t(i) * qstride]);
      return r;
    }
    return rb[size_t(i) * rstride];
  };
  auto shift = [&]() {
#pragma unroll
    for (int t = 0; t < kFavePT - 1; ++t) win[t] = win[t + 1];
    win[kFavePT - 1] = qb[size_t(jl) * qstride];
    jl = (jl + 1 == n) ? 0 : jl + 1;
  };
  int iA = n - p0 - (kFavePT - 1);
  if (iA < 0) iA = 0;
  const int iC = n - p0;
  int i = 0;
  for (; i < iA; ++i) {
    double2 rho = rho_at(i);
#pragma unroll
    for (int t = 0; t < kFavePT; ++t) s1[t] = cfma(win[t], rho, s1[t]);
    shift();
  }
  for (; i < iC; ++i) {
    double2 rho = rho_at(i);
#pragma unroll
    for (int t = 0; t < kFavePT; ++t) {
      if (i + p0 + t < n) s1[t] = cfma(win[t], rho, s1[t]);
      else s2[t] = cfma(win[t], rho, s2[t]);
    }
    shift();
  }
  for (; i < n; ++i) {
    double2 rho = rho_at(i);
#pragma unroll
    for (int t = 0; t < kFavePT; ++t) s2[t] = cfma(win[t], rho, s2[t]);
    shift();
  }
#pragma unroll
  for (int t = 0; t < kFavePT; ++t) {
    int p = p0 + t;
    if (p < n) s.G[at(p * s.ne + e, c, s.Cpad)] = cfma(z, s2[t], s1[t]);
  }
}

// Decimation-in-time FFT (negative exponent) of CG interleaved sequences of length M = q 2^a,
// q = 1, 3 or 5, held in shared memory as X[i * CG + cc]: q transforms of length 2^a (radix 2,
// segment r holding the points q m + r in bit-reversed order of m), then one combining pass of
// radix q; output in natural order.  tw[k] = exp(-2 pi i k / (M twm)), k < M twm (twm = 2: a
// half-length transform on the table of the full length).  The radix-2 stages run in passes of up
// to three: a thread holds the 2^LR points of one group in registers and applies LR stages to
// them, so a pass costs one shared-memory round trip and one barrier, and every point sees the
// same butterflies in the same order as stage by stage (the result does not depend on the
// grouping).  In FP64 the butterflies bound the kernel: a +- t d takes six FMAs (a + t d by four,
// a - t d = 2a - (a + t d) by two) instead of four multiplies or FMAs and four additions.

// a + w d and a - w d
__device__ __forceinline__ void butterfly(double2 &a, double2 &d, double2 w) {
  const double2 u = cmk(fma(w.x, d.x, fma(-w.y, d.y, a.x)), fma(w.x, d.y, fma(w.y, d.x, a.y)));
  d = cmk(fma(2.0, a.x, -u.x), fma(2.0, a.y, -u.y));
  a = u;
}
__device__ __forceinline__ void butterfly(float2 &a, float2 &d, float2 w) {
  const float2 t = cmul(w, d), a0 = a;
  a = cadd(a0, t), d = csub(a0, t);
}

// Stages st .. st+LR-1 on x[k] = point (group base) + pos + k 2^st, pos < 2^st.  HALF: the odd
// points are zero before stage 0.
template <class C, int LR, bool HALF = false>
__device__ __forceinline__ void fft_regs(C (&x)[1 << LR], int st, int pos, int M, const C *__restrict__ tw,
                                         int twm) {
#pragma unroll
  for (int l = 0; l < LR; ++l) {
    const int sl = st + l, tstride = M >> (sl + 1);
#pragma unroll
    for (int k = 0; k < (1 << LR); ++k) {
      if ((k >> l) & 1) continue;
      const int k1 = k + (1 << l);
      const int p = pos + ((k & ((1 << l) - 1)) << st);  // position within the half block
      if (HALF && l == 0) {
        x[k1] = x[k];
      } else if (sl <= 1) {
        const C a = x[k], d = x[k1];
        C t = d;
        if (sl == 1 && p) t.x = d.y, t.y = -d.x;
        x[k] = cadd(a, t), x[k1] = csub(a, t);
      } else {
        butterfly(x[k], x[k1], tw[p * tstride * twm]);
      }
    }
  }
}

// One pass of LR stages from st over the q 2^a points of X (and Y), in place; ends with a
// barrier.  M2 = 2^a; the twiddles of its transforms are every (q twm)-th of the table.
template <int CG, class C, int LR>
__device__ void fft_pass(C *X, C *Y, int M2, int q, int st, const C *__restrict__ tw, int twm) {
  constexpr int R = 1 << LR;
  const int h = 1 << st, items = (M2 >> LR) * q * CG;
  for (int idx = threadIdx.x; idx < items; idx += blockDim.x) {
    const int cc = idx % CG, b = idx / CG;
    const int pos = b & (h - 1), grp = b >> st;
    const int base = ((grp << (st + LR)) + pos) * CG + cc;
    for (int w = 0; w < (Y ? 2 : 1); ++w) {
      C *V = w ? Y : X;
      C x[R];
#pragma unroll
      for (int k = 0; k < R; ++k) x[k] = V[base + k * h * CG];
      fft_regs<C, LR>(x, st, pos, M2, tw, q * twm);
#pragma unroll
      for (int k = 0; k < R; ++k) V[base + k * h * CG] = x[k];
    }
  }
  __syncthreads();
}

// q-point DFT in place, q odd: the pairs x_r +- x_(q-r) against cos and sin
template <int Q, class C>
__device__ __forceinline__ void dft_odd(C (&x)[Q]) {
  using R = decltype(C::x);
  constexpr int H = (Q - 1) / 2;
  // cos and sin of 2 pi j / Q
  constexpr double c3[2] = {1.0, -0.5}, s3[2] = {0.0, 0.86602540378443864676};
  constexpr double c5[3] = {1.0, 0.30901699437494742410, -0.80901699437494742410};
  constexpr double s5[3] = {0.0, 0.95105651629515357212, 0.58778525229247312917};
  C p[H + 1], m[H + 1], y[Q];
#pragma unroll
  for (int r = 1; r <= H; ++r) p[r] = cadd(x[r], x[Q - r]), m[r] = csub(x[r], x[Q - r]);
  y[0] = x[0];
#pragma unroll
  for (int r = 1; r <= H; ++r) y[0] = cadd(y[0], p[r]);
#pragma unroll
  for (int s = 1; s <= H; ++s) {
    C a = x[0], b = mkc<C>(0, 0);  // X_s = a - i b, X_(Q-s) = a + i b
#pragma unroll
    for (int r = 1; r <= H; ++r) {
      const int j = (r * s) % Q, f = j <= H ? j : Q - j;
      const R c = R(Q == 3 ? c3[f % 2] : c5[f % 3]), sn = R((j <= H ? 1.0 : -1.0) * (Q == 3 ? s3[f % 2] : s5[f % 3]));
      a.x = fma(c, p[r].x, a.x), a.y = fma(c, p[r].y, a.y);
      b.x = fma(sn, m[r].x, b.x), b.y = fma(sn, m[r].y, b.y);
    }
    y[s].x = a.x + b.y, y[s].y = a.y - b.x;
    y[Q - s].x = a.x - b.y, y[Q - s].y = a.y + b.x;
  }
#pragma unroll
  for (int s = 0; s < Q; ++s) x[s] = y[s];
}

// The combining pass: X[k + 2^a s] = sum_r W^(rk) e^(-2 pi i rs / Q) (segment r)[k].
template <int CG, int Q, class C>
__device__ void fft_combine(C *X, C *Y, int M2, const C *__restrict__ tw, int twm) {
  for (int idx = threadIdx.x; idx < M2 * CG; idx += blockDim.x) {
    const int k = idx / CG;
    for (int w = 0; w < (Y ? 2 : 1); ++w) {
      C *V = w ? Y : X;
      C x[Q];
      x[0] = V[idx];
#pragma unroll
      for (int r = 1; r < Q; ++r) x[r] = cmul(tw[r * k * twm], V[r * M2 * CG + idx]);
      dft_odd<Q>(x);
#pragma unroll
      for (int t = 0; t < Q; ++t) V[t * M2 * CG + idx] = x[t];
    }
  }
  __syncthreads();
}

// Stages st0 .. a-1 in passes of three (the last pass two or one), then the combining pass.
template <int CG, class C>
__device__ void fft_dit(C *X, C *Y, int a, int q, const C *__restrict__ tw, int twm = 1, int st0 = 0) {
  const int M2 = 1 << a;
  int st = st0;
  for (; st + 3 <= a; st += 3) fft_pass<CG, C, 3>(X, Y, M2, q, st, tw, twm);
  if (a - st == 2) fft_pass<CG, C, 2>(X, Y, M2, q, st, tw, twm);
  else if (a - st == 1) fft_pass<CG, C, 1>(X, Y, M2, q, st, tw, twm);
  if (q == 3) fft_combine<CG, 3>(X, Y, M2, tw, twm);
  else if (q == 5) fft_combine<CG, 5>(X, Y, M2, tw, twm);
}

// natural index of the point stored at position x: segment x >> a, bit-reversed within it
__device__ __forceinline__ int fft_index(int x, int a, int q) {
  const int m = a ? int(__brev(unsigned(x & ((1 << a) - 1))) >> (32 - a)) : 0;
  return q * m + (x >> a);
}

// The first pass (stages 0..2, a >= 3) fused with the load: position j of column cc is
// load(natural index, cc, x, y); the transformed groups go to X (and Y when it is given).  HALF:
// the upper half of the sequence is zero (the odd points of every group).  Ends with a barrier;
// fft_dit(..., st0 = 3) continues.
template <int CG, bool HALF, class C, class F>
__device__ void fft_first_pass(C *X, C *Y, int a, int q, const C *__restrict__ tw, int twm, F &&load) {
  const int items = ((1 << a) >> 3) * q * CG;
  for (int idx = threadIdx.x; idx < items; idx += blockDim.x) {
    const int cc = idx % CG, grp = idx / CG;
    C x[8], y[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (!HALF || !(k & 1)) load(fft_index(grp * 8 + k, a, q), cc, x[k], y[k]);
    fft_regs<C, 3, HALF>(x, 0, 0, 1 << a, tw, q * twm);
#pragma unroll
    for (int k = 0; k < 8; ++k) X[(grp * 8 + k) * CG + cc] = x[k];
    if (Y) {
      fft_regs<C, 3, HALF>(y, 0, 0, 1 << a, tw, q * twm);
#pragma unroll
      for (int k = 0; k < 8; ++k) Y[(grp * 8 + k) * CG + cc] = y[k];
    }
  }
  __syncthreads();
}
// The first pass where a < 3: plain loads into position.
template <int CG, class C, class F>
__device__ void fft_load(C *X, C *Y, int a, int q, F &&load) {
  for (int idx = threadIdx.x; idx < (q << a) * CG; idx += blockDim.x) {
    const int cc = idx % CG, x = idx / CG;
    C u, v;
    load(fft_index(x, a, q), cc, u, v);
    X[idx] = u;
    if (Y) Y[idx] = v;
  }
  __syncthreads();
}

// z^j in float for z = e^{a + i b}, from e = (a, b_hi, b_lo): b = b_hi + b_lo with |b| < 2 pi
// (a difference of two principal-branch arguments).  The phase j b is j b_hi (with its exact
// rounding error, by fma) plus j b_lo, reduced modulo 2 pi against a three-term float 2 pi
// (Cody-Waite: 6.28125 has 8 significant bits, so k 6.28125 is exact); then float sincos
// with the small remainder added to the argument and a float exp of j a.  All float
// arithmetic; error a few float ulp.
__device__ __forceinline__ float2 z_pow_f(float4 e, int j) {
  constexpr float kInv2Pi = 0.15915494f, kP1 = 6.28125f, kP2 = 0.0019353071693331003f, kP3 = 1.0253131677018246e-11f;
  const float jf = float(j);
  const float p = jf * e.y, pe = __fmaf_rn(jf, e.y, -p), corr = __fmaf_rn(jf, e.z, pe);
  const float k = rintf(p * kInv2Pi);
  float r = __fmaf_rn(-k, kP1, p);
  r = __fmaf_rn(-k, kP2, r);
  r = __fmaf_rn(-k, kP3, r) + corr;
  float sn, cs;
  sincosf(r, &sn, &cs);
  const float m = expf(jf * e.x);
  return make_float2(m * cs, m * sn);
}

// Fave by FFT.  One CTA per (element e, group of CG crystallites).  With q zero outside
// [0, n), Lin_d = sum_i q_{i+d} r_i for |d| < n is the linear cross-correlation, obtained
// from zero-padded transforms of length M = 2^a, 3 2^a or 5 2^a >= 2n:  Lin = IFFT(FFT(q) . conj(FFT(conj r))).
// Then G_p = Lin_p + z Lin_{p-n} (the same G as k_fave).  When r = conj(q) (rho = (D+D^H)/2
// and D has no block pair (b,a) for this element) the product is |FFT(q)|^2 and the second
// forward transform is skipped.
// Twisted form (fave_twist, n a power of two, M = n): with zeta^n = z, u_i = zeta^-i q_i and
// v_i = zeta^i r_i, the circular correlation C_p = sum_i v_i u_{(i+p) mod n} equals
// zeta^-p G_p (the wrapped terms carry zeta^n = z), so G_p = zeta^p C_p from transforms of
// length n instead of 2n.  zeta = e^{i tau w}; in the autocorrelation case r = conj(q) needs
// |zeta| = 1, and zeta = e^{i tau Re w} is used there: exact when the chop has zeroed Im w,
// otherwise G_p carries z e^{-n tau Im w} in place of z on its wrapped part (relative error
// at most n tau |Im w|).
// POW2: M is a power of two (fftq = 1).
template <int CG, class C, bool POW2>
__global__ void __launch_bounds__(128) k_fave_fft(DevSys s) {
  extern __shared__ __align__(16) unsigned char fsm_raw[];
  const int M = s.M, la = s.logM, q5 = POW2 ? 1 : s.fftq, n = s.n;  // M = q5 2^la
  C *X = reinterpret_cast<C *>(fsm_raw), *Y = X + size_t(M) * CG;
  // twist tables per column: zeta^b (b < 8), zeta^8a (a < M/8), and those of zeta^-1
  double2 *tp1 = reinterpret_cast<double2 *>(Y + size_t(M) * CG), *tp8 = tp1 + 8 * CG;
  double2 *tm1 = tp8 + (M / 8) * CG, *tm8 = tm1 + 8 * CG;
  __shared__ C zc[CG];
  const int groups = s.Cpad / CG;
  const int e = blockIdx.x / groups;
  const int c0 = (blockIdx.x % groups) * CG;
  const int eq = s.eq[e], erev = s.erev[e], er = s.er[e];
  const bool autoc = s.rosym && erev < 0;
  const size_t qstride = size_t(s.nq) * s.Cpad, rstride = size_t(s.nr) * s.Cpad;
  const C *Qb = Bufs<C>::Q(s), *Rb = Bufs<C>::R(s);
  const double nt = double(n) * s.tau;
  // per crystallite of the group: w_rs = chop((l_r - l_s)/(i n tau), 1e-10), z = e^{i n tau w},
  // and the powers of the FID reconstruction (FP64 form: pair_power's; mixed form: z^j).  FP64
  // form: four powers per thread, one cexp and three products (error a few ulp).  Single-precision form (the powers are stored
  // as float): the exponent of z^j in FP64, then z_pow_f per power (after the first pass).
  constexpr bool kF = std::is_same<C, float2>::value;
  __shared__ float4 zexp[CG];
  if constexpr (kF) {  // z = e^{n tau (i w)} = e^{d} with d = l_r - l_s, chopped as w is
    for (int cc = threadIdx.x; cc < CG; cc += blockDim.x) {
      const int c = c0 + cc;
      float4 ze = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c < s.C) {
        const double2 d = csub(s.L[at(s.erg[e], c, s.Cpad)], s.L[at(s.esg[e], c, s.Cpad)]);
        const double thr = 1e-10 * nt;
        const double dx = fabs(d.x) < thr ? 0.0 : d.x, dy = fabs(d.y) < thr ? 0.0 : d.y;
        const float yh = float(dy);
        ze = make_float4(float(dx), yh, float(dy - double(yh)), 0.f);
      }
      zexp[cc] = ze;
    }
  } else {
    constexpr int kZrun = 4;
    const int mr = pair_rows(s.J), nzr = (mr + kZrun - 1) / kZrun;
    for (int idx = threadIdx.x; idx < CG * nzr; idx += blockDim.x) {
      const int cc = idx % CG, m0 = (idx / CG) * kZrun, c = c0 + cc;
      if (c >= s.C) continue;
      double2 d = csub(s.L[at(s.erg[e], c, s.Cpad)], s.L[at(s.esg[e], c, s.Cpad)]);
      double2 w = cmk(chop1(d.y / nt, 1e-10), chop1(-d.x / nt, 1e-10));
      const double2 z1 = cexp(cmk(-nt * w.y, nt * w.x));
      const double pw = pair_power(s.J, m0);
      double2 zm = cexp(cmk(-pw * nt * w.y, pw * nt * w.x));
      if (m0 == 0) zc[cc] = cvt<C>(z1);
      for (int m = m0; m < min(m0 + kZrun, mr); ++m) {
        Bufs<C>::Z(s)[at(m * s.ne + e, c, s.Cpad)] = cvt<C>(zm);
        zm = cmul(zm, z1);
      }
    }
  }
  const bool twist = s.fave_twist;
  if (twist) {
    // one thread per column: zeta^b by products, zeta^8a by products restarted from cexp
    // every 16 entries; zeta^-k the same from -log zeta (the conjugate when |zeta| = 1)
    for (int cc = threadIdx.x; cc < CG; cc += blockDim.x) {
      const int c = c0 + cc;
      double2 zl = cmk(0, 0);
      if (c < s.C) {
        double2 d = csub(s.L[at(s.erg[e], c, s.Cpad)], s.L[at(s.esg[e], c, s.Cpad)]);
        double2 w = cmk(chop1(d.y / nt, 1e-10), chop1(-d.x / nt, 1e-10));
        zl = autoc ? cmk(0.0, s.tau * w.x) : cmk(-s.tau * w.y, s.tau * w.x);
      }
      // |zeta| = 1 in the autocorrelation case: zeta^-k is conj(zeta^k) (bit for bit, as the
      // products of conjugates are the conjugated products)
      for (int sgn = 0; sgn < 2; ++sgn) {
        const double2 l = sgn ? cmk(-zl.x, -zl.y) : zl;
        double2 *t1 = sgn ? tm1 : tp1, *t8 = sgn ? tm8 : tp8;
        if (sgn && autoc) {
          for (int b = 0; b < 8; ++b) t1[b * CG + cc] = cconj(tp1[b * CG + cc]);
          for (int a = 0; a < M / 8; ++a) t8[a * CG + cc] = cconj(tp8[a * CG + cc]);
          continue;
        }
        const double2 z1 = cexp(l);
        t1[cc] = cmk(1, 0);
        for (int b = 1; b < 8; ++b) t1[b * CG + cc] = cmul(t1[(b - 1) * CG + cc], z1);
        const double2 z8 = cmul(t1[7 * CG + cc], z1);
        t8[cc] = cmk(1, 0);
        for (int a = 1; a < M / 8; ++a)
          t8[a * CG + cc] = (a % 16 == 0) ? cexp(cmk(8.0 * a * l.x, 8.0 * a * l.y)) : cmul(t8[(a - 1) * CG + cc], z8);
      }
    }
    __syncthreads();
  }
  // q (and conj r) at natural index i, zero-padded
  auto load = [&](int i, int cc, C &qo, C &yo) {
    const int c = c0 + cc;
    C q = mkc<C>(0, 0), y = mkc<C>(0, 0);
    if (i < n && c < s.C) {
      q = Qb[i * qstride + at(eq, c, s.Cpad)];
      C r;
      if (!autoc) {
        if (s.rosym) r = cadd(cconj(q), Qb[i * qstride + at(erev, c, s.Cpad)]);
        else r = Rb[i * rstride + at(er, c, s.Cpad)];
        y = cconj(r);
      }
      if (twist) {  // u_i = zeta^-i q_i, conj(v_i) = conj(zeta^i r_i)
        const int a = i >> 3, b = i & 7;
        q = cvt<C>(cmul(cmul(tm8[a * CG + cc], tm1[b * CG + cc]), todbl(q)));
        if (!autoc) y = cconj(cvt<C>(cmul(cmul(tp8[a * CG + cc], tp1[b * CG + cc]), todbl(r))));
      }
    }
    qo = q, yo = y;
  };
  const C *tw = Bufs<C>::tw(s);
  C *Yf = autoc ? nullptr : Y;
  if (la < 3) fft_load<CG>(X, Yf, la, q5, load);
  else if (twist || (kF && CG < 8)) fft_first_pass<CG, false>(X, Yf, la, q5, tw, 1, load);
  else fft_first_pass<CG, true>(X, Yf, la, q5, tw, 1, load);  // q is zero from n <= M/2 on
  if constexpr (kF) {  // z^j, j < J, and z itself (the exponents were written before the first pass's barrier)
    for (int idx = threadIdx.x; idx < CG * (s.J + 1); idx += blockDim.x) {
      const int cc = idx % CG, j = idx / CG, c = c0 + cc;
      if (c >= s.C) continue;
      if (j == s.J) zc[cc] = z_pow_f(zexp[cc], 1);
      else Bufs<C>::Z(s)[at(j * s.ne + e, c, s.Cpad)] = z_pow_f(zexp[cc], j);
    }
  }
  fft_dit<CG, C>(X, Yf, la, q5, tw, 1, la >= 3 ? 3 : 0);
  // Inverse transform by a forward one: conj(FFT(x))/M.  Autocorrelation: the spectrum
  // S = |FFT q|^2 is real, so its transform takes one of half length on z_k = S_2k + i S_2k+1
  // (each column on its own, so a crystallite's result does not depend on its neighbours):
  // with Z = FFT_{M/2}(z), E_p = (Z_p + conj Z_-p)/2, O_p = (Z_p - conj Z_-p)/(2i),
  // FFT(S)_p = E_p + w^p O_p and FFT(S)_{p+M/2} = E_p - w^p O_p, w = exp(-2 pi i / M).
  const int Mh = M / 2;
  const bool half = autoc && la >= 2;
  const C *twb = tw;
  if (half) {
    auto spow = [&](int k, int cc, C &zo, C &) {
      const C xe = X[(2 * k) * CG + cc], xo = X[(2 * k + 1) * CG + cc];
      zo = mkc<C>(xe.x * xe.x + xe.y * xe.y, xo.x * xo.x + xo.y * xo.y);
    };
    if (la - 1 >= 3) fft_first_pass<CG, false>(Y, (C *)nullptr, la - 1, q5, twb, 2, spow);
    else fft_load<CG>(Y, (C *)nullptr, la - 1, q5, spow);
    fft_dit<CG, C>(Y, nullptr, la - 1, q5, twb, 2, la - 1 >= 3 ? 3 : 0);
  } else {
    // conj of the cross spectrum, in place in X (same index read and written)
    for (int idx = threadIdx.x; idx < M * CG; idx += blockDim.x) {
      C x = X[idx];
      if (autoc) X[idx] = mkc<C>(x.x * x.x + x.y * x.y, 0.0);
      else X[idx] = cconj(cmul(x, cconj(Y[idx])));
    }
    __syncthreads();
    auto fromX = [&](int f, int cc, C &xo, C &) { xo = X[f * CG + cc]; };
    if (la >= 3) fft_first_pass<CG, false>(Y, (C *)nullptr, la, q5, tw, 1, fromX);
    else fft_load<CG>(Y, (C *)nullptr, la, q5, fromX);
    fft_dit<CG, C>(Y, nullptr, la, q5, tw, 1, la >= 3 ? 3 : 0);
  }
  // transform of column cc at frequency p
  auto spec = [&](int p, int cc) -> C {
    if (!half) return Y[p * CG + cc];
    const int q = p < Mh ? p : p - Mh;
    const C zp = Y[q * CG + cc], zm = cconj(Y[(q ? Mh - q : 0) * CG + cc]);
    const C ev = cscale(cadd(zp, zm), 0.5), d = csub(zp, zm);
    const C wo = cmul(twb[q], mkc<C>(0.5 * d.y, -0.5 * d.x));
    return p < Mh ? cadd(ev, wo) : csub(ev, wo);
  };
  // 1/M; in single precision its power of two only (exact), 1/q follows with the weights (wscale)
  const double invM = 1.0 / double(kF ? M / q5 : M);
  C *Gb = Bufs<C>::G(s);
  if (half && twist) {  // n == M: frequencies q and q + M/2 share E_q and w^q O_q
    for (int idx = threadIdx.x; idx < Mh * CG; idx += blockDim.x) {
      const int cc = idx % CG, q = idx / CG, c = c0 + cc;
      if (c >= s.C) continue;
      const C zp = Y[q * CG + cc], zm = cconj(Y[(q ? Mh - q : 0) * CG + cc]);
      const C ev = cscale(cadd(zp, zm), 0.5), d = csub(zp, zm);
      const C wo = cmul(twb[q], mkc<C>(0.5 * d.y, -0.5 * d.x));
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const int p = q + hh * Mh;
        const C lp = cscale(cconj(hh ? csub(ev, wo) : cadd(ev, wo)), invM);
        const C g = cvt<C>(cmul(cmul(tp8[(p >> 3) * CG + cc], tp1[(p & 7) * CG + cc]), todbl(lp)));
        Gb[at(p * s.ne + e, c, s.Cpad)] = g;
      }
    }
    return;
  }
  for (int idx = threadIdx.x; idx < n * CG; idx += blockDim.x) {
    const int cc = idx % CG, p = idx / CG, c = c0 + cc;
    if (c >= s.C) continue;
    C lp = cscale(cconj(spec(p, cc)), invM);
    C g = lp;
    if (twist) {  // G_p = zeta^p C_p
      g = cvt<C>(cmul(cmul(tp8[(p >> 3) * CG + cc], tp1[(p & 7) * CG + cc]), todbl(lp)));
    } else if (p > 0) {
      C lm = cscale(cconj(spec(M + p - n, cc)), invM);
      g = cfma(zc[cc], lm, lp);
    }
    Gb[at(p * s.ne + e, c, s.Cpad)] = g;
  }
}

// Shared memory of k_fave_fft's twist tables (four per column, 8 or M/8 entries).
static size_t fave_twist_bytes(const DevSys &s, int cg) {
  return s.fave_twist ? sizeof(double2) * size_t(cg) * 2 * (8 + s.M / 8) : 0;
}

#include "bl_big.cuh"
#include "bl_huge.cuh"
#include "bl_tc.cuh"
#include "bl_xs.cuh"

// FID terms of the FP64 form: fid[j gper + p] = sum_c w_c sum_e z_e^j G_p(e).  The FP64 pipe
// bounds it, so the j's are taken in pairs about the middle of their range: with G' = w z^((J-1)/2) G
// and z^m = cos + i sin (|z| = 1), the four real sums of cos G'x, sin G'y, cos G'y and sin G'x give
// both z^m G' and z^-m G' (sum and difference, formed once at the end): four FMAs for two
// complex terms instead of eight, plus one product by the middle power per (element, p, row
// tile).  A warp takes 32 consecutive crystallites and a JT x PT tile of (m, p); W warps share
// a tile's elements (W from the element count alone) and add up in shared memory.  The warp's
// 4 JT PT sums over its lanes go by halving exchanges (each lane ends with two of them: 62 adds
// instead of 5 per sum).  A crystallite's terms are summed in the same order alone and in a
// batch.  Measured, before (4 x 4 tiles of plain complex products, all lanes reducing every
// sum) -> after: 4 spins, 3722 crystallites, 2048 points 3.07 -> 1.80 ms; 7 spins, 144
// crystallites (113 CTAs) 11.3 -> 3.55 ms; a pair, 1154 crystallites, 0.070 -> 0.033 ms.
template <int JT, int PT>
__global__ void __launch_bounds__(256) k_fid_pair(DevSys s, int W) {
  constexpr int V = (4 * JT * PT + 31) / 32 * 32;
  extern __shared__ double fps[];  // [warp][V]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, er = warp % W;
  const int mr = pair_rows(s.J), nmt = (mr + JT - 1) / JT, npt = (s.gper + PT - 1) / PT;
  const long tile = long(blockIdx.x) * (blockDim.x / 32 / W) + warp / W;
  const bool valid = tile < long(s.Cpad / 32) * npt * nmt;
  const int m0 = int(tile % nmt) * JT, p0 = int(tile / nmt % npt) * PT, g = int(tile / nmt / npt);
  const int c = g * 32 + lane;
  double acc[V];
#pragma unroll
  for (int x = 0; x < V; ++x) acc[x] = 0.0;
  if (valid && c < s.C) {
    const double wc = s.w[c] * s.scale;
    const int e1 = int(long(s.ne) * (er + 1) / W);
    for (int e = int(long(s.ne) * er / W); e < e1; ++e) {
      double2 zm[JT], gp[PT];
      const double2 zc = cscale(s.Z[at((mr - 1) * s.ne + e, c, s.Cpad)], wc);
#pragma unroll
      for (int a = 0; a < JT; ++a) zm[a] = m0 + a < mr ? s.Z[at((m0 + a) * s.ne + e, c, s.Cpad)] : cmk(0, 0);
#pragma unroll
      for (int b = 0; b < PT; ++b) gp[b] = p0 + b < s.gper ? s.G[at((p0 + b) * s.ne + e, c, s.Cpad)] : cmk(0, 0);
#pragma unroll
      for (int b = 0; b < PT; ++b) {
        const double2 q = cmul(zc, gp[b]);
#pragma unroll
        for (int a = 0; a < JT; ++a) {
          double *v = acc + 4 * (a * PT + b);
          v[0] = fma(zm[a].x, q.x, v[0]);
          v[1] = fma(zm[a].y, q.y, v[1]);
          v[2] = fma(zm[a].x, q.y, v[2]);
          v[3] = fma(zm[a].y, q.x, v[3]);
        }
      }
    }
  }
  // sum x of the tile over the warp's lanes ends in lane x / (V / 32)
#pragma unroll
  for (int o = 16, half = V / 2; o > 0; o >>= 1, half >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int x = 0; x < half; ++x) {
      const double send = up ? acc[x] : acc[x + half], keep = up ? acc[x + half] : acc[x];
      acc[x] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
#pragma unroll
  for (int r = 0; r < V / 32; ++r) fps[warp * V + lane * (V / 32) + r] = acc[r];
  __syncthreads();
  if (!valid) return;
  const double *t0 = fps + (warp - er) * V;  // the tile's sums, one row per warp
  for (int x = er * 32 + lane; x < JT * PT; x += 32 * W) {
    const int m = m0 + x / PT, p = p0 + x % PT;
    if (m >= mr || p >= s.gper) continue;
    double v[4] = {0, 0, 0, 0};
    for (int w = 0; w < W; ++w)
      for (int q = 0; q < 4; ++q) v[q] += t0[w * V + 4 * x + q];
    const int jp = (s.J % 2 ? (s.J - 1) / 2 : s.J / 2) + m, jm = s.J - 1 - jp;
    double2 *row = s.partial + size_t(s.warp_base + g) * s.npts;
    const long kp = long(jp) * s.gper + p, km = long(jm) * s.gper + p;
    if (kp < s.npts) row[kp] = cmk(v[0] - v[1], v[2] + v[3]);
    if (jm != jp && km < s.npts) row[km] = cmk(v[0] + v[1], v[2] - v[3]);
  }
}

// Point-to-point FID terms, one thread per (crystallite, element (r,s)).
// With W_i = A_{i+1} V (A_n = Omega = V diag(lam) V^H), Q_i = W_i^H D W_i and R_{n-1} =
// W_{n-1}^H rho W_{n-1} = diag(lam)^H (V^H rho V) diag(lam), the density matrix after
// m_tot chunks, G = A_{j'} Omega^{q'} with m_tot = q' b + j' (1 <= j' <= b), gives
//   Tr(D G rho G^H) = sum_rs Q_i(r,s) R_{n-1}(s,r) e^{i m (th_s - th_r)},
//   i = j' sub - 1, m = q' + 1   (m_tot = 0: i = n - 1, m = 0).
// Point p = j b + k has m_tot = p f: its i depends on k only and m grows by f per j, so
// G[k] = Q_{i_k}(r,s) R(s,r) e^{i m_k d} and Z[j] = e^{i j f d} (d = th_s - th_r) feed
// the FID terms' fid[j b + k] = sum_e Z[j] G[k].  The chunk products are never formed: the
// reference's PropReduce (examples/qmsims/MMMQMAS/propreduce.cc:455-521) builds every
// dwell propagator from shared sub-products; here the Floquet powers replace them.  (FP64
// form: Z holds the powers that k_fid_pair takes instead.)
template <class C>
__global__ void __launch_bounds__(kThreads) k_p2p_elems(DevSys s) {
  long tid = long(blockIdx.x) * blockDim.x + threadIdx.x;
  int c = int(tid % s.Cpad);
  long rest = tid / s.Cpad;
  if (rest >= s.ne) return;
  const int e = int(rest);
  if (c >= s.C) return;
  const C *Q = Bufs<C>::Q(s), *R = Bufs<C>::R(s);
  const int qlast = (s.n - 1) * s.nq;
  double2 rsr;  // R_{n-1}(s,r)
  if (s.rosym) {  // rho = (D + D^H)/2: R = (Q(s,r) + conj(Q(r,s)))/2
    double2 v = cconj(todbl(Q[at(qlast + s.eq[e], c, s.Cpad)]));
    if (s.erev[e] >= 0) v = cadd(v, todbl(Q[at(qlast + s.erev[e], c, s.Cpad)]));
    rsr = cscale(v, 0.5);
  } else {
    rsr = todbl(R[at((s.n - 1) * s.nr + s.er[e], c, s.Cpad)]);
  }
  const double d = s.L[at(s.esg[e], c, s.Cpad)].y - s.L[at(s.erg[e], c, s.Cpad)].y;
  for (int k = 0; k < s.pb; ++k) {
    const long mt = long(k) * s.pf;
    int i = s.n - 1;
    long m = 0;
    if (mt > 0) {
      const long jp = (mt - 1) % s.pb + 1, qp = (mt - jp) / s.pb;
      i = int(jp) * s.psub - 1;
      m = qp + 1;
    }
    double sn, cs;
    sincos(double(m) * d, &sn, &cs);
    const double2 g = cmul(cmul(todbl(Q[at(i * s.nq + s.eq[e], c, s.Cpad)]), rsr), cmk(cs, sn));
    Bufs<C>::G(s)[at(k * s.ne + e, c, s.Cpad)] = cvt<C>(g);
  }
  // Z[j] = e^{i j f d}: a running product, re-anchored by an exact sincos every 64 powers
  // (its rounding then stays near 64 eps; arguments reach ~10^4 rad)
  double2 z1;
  sincos(double(s.pf) * d, &z1.y, &z1.x);
  double2 zj = cmk(1, 0);
  constexpr bool kPair = std::is_same<C, double2>::value;  // k_fid_pair's powers in the FP64 form
  const int nz = kPair ? pair_rows(s.J) : s.J;
  for (int j = 0; j < nz; ++j) {
    const double pw = kPair ? pair_power(s.J, j) : double(j);
    if ((j & 63) == 0 && pw != 0.0) sincos(pw * double(s.pf) * d, &zj.y, &zj.x);
    Bufs<C>::Z(s)[at(j * s.ne + e, c, s.Cpad)] = cvt<C>(zj);
    zj = cmul(zj, z1);
  }
}

// Mixed form: the FID terms as a tiled product.  fid[j gper + p] = sum_c w_c sum_e
// z_e^j(c) G_p(e, c) is a product with K = (crystallite, element); one CTA takes a group of
// 32 crystallites (one warp of the batch layout), a range of the elements (ft_r ranges, a
// function of the element count only) and a (j, p) tile of ft_jt x ft_pt threads, each
// thread a 4 x 4 register tile (the tile shape follows J and gper, so little is padded).
// Per element it stages z_e^j and G_p(e) of its 32 crystallites in shared memory by
// asynchronous copies (coalesced: crystallites are fastest in HBM; double-buffered, so the
// next element's copies are in flight while this one is summed), and each thread updates its
// tile with (w_c / wref) z, accumulating one element in FP32 and folding it into double-float
// (hi + lo) sums.  ft_sub groups of 64 threads each take a part of the
// range and add up their double-float sums in order (one or two 64-thread CTAs an SM before where
// there are few elements or crystallites: 4 spins, 3722 crystallites 0.315 -> 0.274 ms; 9 spins, 32
// crystallites 11.5 -> 4.1 ms; 8 spins, 1154 crystallites 26.6 -> 22.7 ms).  The CTA writes its tile to partial row (warp * ft_r + range); k_reduce
// sums the rows of the populated warps in a fixed order.  Each output's summation order
// (crystallites 0..31 per element, elements in order within a sub-range, sub-ranges in order) follows
// from the element count and the tile shape (ft_sub does), that is from the job's points and steps,
// and not from the batch, so a crystallite's contribution does not depend on its neighbours.
constexpr int kFtThreads = 64, kFtR = 16, kFtJmax = 32;
// Dynamic shared memory of k_fid_tiled: two buffers of 32 crystallites x (4 jt + 4 pt).
// Groups per CTA: as many as leave their buffers within 200 KB.
static int fid_tiled_sub(int jt, int pt) { return jt + pt <= 24 ? 4 : jt + pt <= 48 ? 2 : 1; }
static size_t fid_tiled_smem(int jt, int pt) {  // (at least the sums handed over at the end)
  const int sub = fid_tiled_sub(jt, pt);
  return std::max(sizeof(float2) * 2 * 32 * 4 * size_t(jt + pt) * sub, sizeof(float4) * 16 * kFtThreads * size_t(sub - 1));
}
__global__ void __launch_bounds__(kFtThreads * 4) k_fid_tiled(DevSys s) {
  extern __shared__ __align__(16) float2 ftsm[];
  const int JT = 4 * s.ft_jt, PT = 4 * s.ft_pt;
  const int sub = threadIdx.x / kFtThreads;
  float2 *zs = ftsm + size_t(sub) * 2 * 32 * (JT + PT), *gs = zs + 2 * 32 * JT;  // [buffer][c][j], [buffer][c][p]
  __shared__ float ws[32];
  const int tid = threadIdx.x % kFtThreads;
  const int g = blockIdx.x;  // group of 32 crystallites in this batch
  const int npr = (s.gper + PT - 1) / PT;
  const int pr = blockIdx.y % npr, jr = blockIdx.y / npr, er = blockIdx.z;
  const int p0 = pr * PT, j0 = jr * JT;
  const int parts = s.ft_r * s.ft_sub, part = er * s.ft_sub + sub;
  const int e_lo = int((long(s.ne) * part) / parts), e_hi = int((long(s.ne) * (part + 1)) / parts);
  const int c0 = g * 32;
  if (threadIdx.x < 32) {
    const int c = c0 + tid;
    ws[tid] = c < s.C ? float(s.w[c] / s.wref) : 0.f;
  }
  __syncthreads();
  auto sub_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(sub + 1), "n"(kFtThreads) : "memory"); };
  const bool active = tid < s.ft_jt * s.ft_pt;
  const int jt = active ? tid / s.ft_pt : 0, pt = active ? tid % s.ft_pt : 0;  // j0 + 4 jt + a, p0 + 4 pt + b
  float2 acc[4][4];
  float2 hi[4][4], lo[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) hi[a][b] = lo[a][b] = make_float2(0.f, 0.f);
  const float2 *Zb = s.Zf, *Gb = s.Gf;
  // z (JT x 32) and G (PT x 32) of element e into buffer buf, zeros outside J, gper and C
  auto stage = [&](int e, int buf) {
    for (int t = tid; t < JT * 32; t += kFtThreads) {
      const int jj = t / 32, c = t % 32, j = j0 + jj;
      const bool ok = j < s.J && c0 + c < s.C;
      cp_async8(&zs[(buf * 32 + c) * JT + jj], ok ? &Zb[at(j * s.ne + e, c0 + c, s.Cpad)] : Zb, ok ? 8 : 0);
    }
    for (int t = tid; t < PT * 32; t += kFtThreads) {
      const int pp = t / 32, c = t % 32, p = p0 + pp;
      const bool ok = p < s.gper && c0 + c < s.C;
      cp_async8(&gs[(buf * 32 + c) * PT + pp], ok ? &Gb[at(p * s.ne + e, c0 + c, s.Cpad)] : Gb, ok ? 8 : 0);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (e_lo < e_hi) stage(e_lo, 0);
  int buf = 0;
  for (int e = e_lo; e < e_hi; ++e) {
    if (e + 1 < e_hi) {
      stage(e + 1, buf ^ 1);  // in flight while this element is summed
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    sub_sync();
    if (active) {
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = make_float2(0.f, 0.f);
      const float2 *zrow = zs + buf * 32 * JT + 4 * jt, *grow = gs + buf * 32 * PT + 4 * pt;
#pragma unroll 2
      for (int c = 0; c < 32; ++c) {
        const float w = ws[c];
        const float4 z01 = *reinterpret_cast<const float4 *>(zrow + c * JT);
        const float4 z23 = *reinterpret_cast<const float4 *>(zrow + c * JT + 2);
        const float4 g01 = *reinterpret_cast<const float4 *>(grow + c * PT);
        const float4 g23 = *reinterpret_cast<const float4 *>(grow + c * PT + 2);
        const float2 zz[4] = {make_float2(w * z01.x, w * z01.y), make_float2(w * z01.z, w * z01.w),
                              make_float2(w * z23.x, w * z23.y), make_float2(w * z23.z, w * z23.w)};
        const float2 gg[4] = {make_float2(g01.x, g01.y), make_float2(g01.z, g01.w), make_float2(g23.x, g23.y),
                              make_float2(g23.z, g23.w)};
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b) acc[a][b] = cfma(zz[a], gg[b], acc[a][b]);
      }
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const float2 x = dfv_add(make_float2(hi[a][b].x, lo[a][b].x), make_float2(acc[a][b].x, 0.f));
          const float2 y = dfv_add(make_float2(hi[a][b].y, lo[a][b].y), make_float2(acc[a][b].y, 0.f));
          hi[a][b] = make_float2(x.x, y.x), lo[a][b] = make_float2(x.y, y.y);
        }
    }
    sub_sync();  // the next stage() overwrites this buffer
    buf ^= 1;
  }
  // the sub-ranges' sums, added in order by the first group
  __syncthreads();
  float4 *hand = reinterpret_cast<float4 *>(ftsm);
  if (sub > 0) {
#pragma unroll
    for (int x = 0; x < 16; ++x)
      hand[((sub - 1) * 16 + x) * kFtThreads + tid] =
          make_float4(hi[x / 4][x % 4].x, hi[x / 4][x % 4].y, lo[x / 4][x % 4].x, lo[x / 4][x % 4].y);
  }
  __syncthreads();
  if (sub > 0) return;
  for (int u = 0; u < s.ft_sub - 1; ++u)
#pragma unroll
    for (int x = 0; x < 16; ++x) {
      const float4 v = hand[(u * 16 + x) * kFtThreads + tid];
      const int a = x / 4, b = x % 4;
      const float2 re = dfv_add(make_float2(hi[a][b].x, lo[a][b].x), make_float2(v.x, v.z));
      const float2 im = dfv_add(make_float2(hi[a][b].y, lo[a][b].y), make_float2(v.y, v.w));
      hi[a][b] = make_float2(re.x, im.x), lo[a][b] = make_float2(re.y, im.y);
    }
  if (!active) return;
  const long row = long(s.warp_base + g) * s.ft_r + er;
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int j = j0 + 4 * jt + a, p = p0 + 4 * pt + b;
      const long k = long(j) * s.gper + p;
      if (j < s.J && p < s.gper && k < s.npts)
        s.partial[row * s.npts + k] = make_double2((double(hi[a][b].x) + double(lo[a][b].x)) * s.wscale,
                                                   (double(hi[a][b].y) + double(lo[a][b].y)) * s.wscale);
    }
}

// Compensated (Kahan) sum of the warp partials in a fixed order: warp g of a block sums rows g,
// g + G, ... of 32 points (G groups of at least four rows); the first warp adds the groups' sums
// and compensations in order.  One thread per point over every row was a serial chain of loads (37 rows, 1024
// points: 27 us on 4 CTAs; now 16 us; 1872 rows, 2048 points 75 -> 22 us).
constexpr int kRedGroups = 16;
__global__ void __launch_bounds__(32 * kRedGroups) k_reduce(const double2 *__restrict__ partial, int nw, int npts,
                                                           double2 *__restrict__ fid) {
  __shared__ double2 sum[kRedGroups][32], comp[kRedGroups][32];
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5, k = blockIdx.x * 32 + lane;
  double sx = 0, sy = 0, cx = 0, cy = 0;
  auto add = [&](double2 v) {
    double yx = v.x - cx, tx = sx + yx;
    cx = (tx - sx) - yx, sx = tx;
    double yy = v.y - cy, ty = sy + yy;
    cy = (ty - sy) - yy, sy = ty;
  };
  const int G = min(kRedGroups, (nw + 3) / 4);
  if (k < npts && g < G) {
#pragma unroll 4
    for (int w = g; w < nw; w += G) add(partial[size_t(w) * npts + k]);
  }
  sum[g][lane] = make_double2(sx, sy), comp[g][lane] = make_double2(-cx, -cy);
  __syncthreads();
  if (g != 0 || k >= npts) return;
  double2 cs = make_double2(0, 0);  // the other groups' compensations: below an ulp of the sums
  for (int t = 1; t < G; ++t) add(sum[t][lane]), cs = cadd(cs, comp[t][lane]);
  add(cs);
  fid[k] = make_double2(sx, sy);
}

// A non-zero of the packed term operators: element idx of the (term, packed block index) table.
struct TermEntry {
  int idx, pad;
  double v;
};
// The dense term tables (zeroed before) from their non-zeros; Tdf may be null.
__global__ void __launch_bounds__(kThreads) k_scatter_terms(const TermEntry *__restrict__ t, int n, double *T, float2 *Tdf) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= n) return;
  T[t[x].idx] = t[x].v;
  if (Tdf) Tdf[t[x].idx] = dfv_of(t[x].v);
}
// R_powder(phi, theta, gamma) (the 3-angle Cartesian rotation, space_ten.cc:578-618) of every
// crystallite, batch-major [batch][element][c], from the angles [phi | theta | gamma].
__global__ void __launch_bounds__(kThreads) k_orient(const double *__restrict__ ang, int all, int Cb, double *Rp) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= all) return;
  double sa, ca, sb, cb, sg, cg;
  sincos(ang[x], &sa, &ca), sincos(ang[all + x], &sb, &cb), sincos(ang[2 * all + x], &sg, &cg);
  double *R = Rp + size_t(x / Cb) * 9 * Cb + x % Cb;
  const double m[9] = {ca * cb * cg - sa * sg, sa * cb * cg + ca * sg, -sb * cg,
                       -ca * cb * sg - sa * cg, -sa * cb * sg + ca * cg, sb * sg,
                       ca * sb, sa * sb, cb};
#pragma unroll
  for (int e = 0; e < 9; ++e) R[size_t(e) * Cb] = m[e];
}

inline unsigned grid_for(long threads) { return unsigned((threads + kThreads - 1) / kThreads); }

}  // namespace

// ------------------------------------------------------------------ host side
Context::~Context() {
  for (auto e : join_ev) cudaEventDestroy(e);
  for (auto a : aux) cudaStreamDestroy(a);
  if (fork_ev) cudaEventDestroy(fork_ev);
  if (stage_ev) cudaEventDestroy(stage_ev);
  if (stage) cudaFreeHost(stage);
  if (stream) cudaStreamDestroy(stream);
}

// Bump allocator over a caller-provided device region.  The allocation-free entry point
// (powder_fid_noalloc) and job_in_region install one while they build a Job.
struct ScratchArena {
  char *base = nullptr;
  size_t cap = 0, used = 0;
  const char *label = "static device scratch of the allocation-free entry point";
  bool aux_streams = false;  // the Job may create its own streams (not on the allocation-free path)
};
static thread_local ScratchArena *g_arena = nullptr;
// Set by job_in_asked_region: the constructor asks it for the region once the job is planned.
static thread_local const RegionFn *g_region = nullptr;
// Set by job_bytes: the Job constructor records its memory plan here and returns before
// touching the device.
struct JobSizing {
  size_t per_c = 0;
  long cpad = 0;
  size_t extra = 0;   // bytes independent of the batch size (huge-block workspace)
  size_t tables = 0;  // the system's operator tables on the device (and their double-float copies)
};
static thread_local JobSizing *g_sizing = nullptr;

template <class T>
struct DevBuf {
  T *p = nullptr;
  size_t n = 0;
  bool owned = true;  // false: carved from a ScratchArena, never freed here
  void alloc(size_t count) {
    n = count;
    if (!count) return;
    if (g_arena) {
      size_t off = (g_arena->used + 255) & ~size_t(255);
      size_t bytes = count * sizeof(T);
      if (off + bytes > g_arena->cap)
        throw Error(4, "job needs more than the " + std::to_string(g_arena->cap >> 20) + " MiB " + g_arena->label);
      p = reinterpret_cast<T *>(g_arena->base + off);
      g_arena->used = off + bytes;
      owned = false;
      return;
    }
    CUDA_OK(cudaMalloc(&p, count * sizeof(T)));
  }
  DevBuf() {}
  DevBuf(const DevBuf &) = delete;
  DevBuf &operator=(const DevBuf &) = delete;
  DevBuf(DevBuf &&o) noexcept : p(o.p), n(o.n), owned(o.owned) { o.p = nullptr, o.n = 0; }
  ~DevBuf() {
    if (p && owned) cudaFree(p);
  }
};

// The job's inputs and tables: gathered on the host at 256-byte offsets, then one device
// buffer and one copy (forty copies of a few hundred bytes each took most of a small call).
class Uploads {
 public:
  template <class T>
  void add(DevBuf<T> &buf, const std::vector<T> &v) {
    const size_t off = (host_.size() + 255) & ~size_t(255), bytes = v.size() * sizeof(T);
    buf.n = v.size();
    if (v.empty()) return;
    host_.resize(off + bytes);
    std::memcpy(host_.data() + off, v.data(), bytes);
    total_ += bytes;
    DevBuf<T> *b = &buf;
    set_.push_back([b, off](unsigned char *base) { b->p = reinterpret_cast<T *>(base + off), b->owned = false; });
  }
  // enqueues the copy on the context's stream and sets every added buffer's address in `dev`;
  // the pinned buffer is used unless the job may not allocate (pinned == false)
  void flush(Context &ctx, DevBuf<unsigned char> &dev, bool pinned) {
    if (host_.empty()) return;
    dev.alloc(host_.size());
    std::lock_guard<std::mutex> lock(ctx.mu);
    const void *src = host_.data();
    if (pinned && host_.size() <= Context::kMaxStage) {
      if (ctx.stage_ev) CUDA_OK(cudaEventSynchronize(ctx.stage_ev));  // the last copy out of it has ended
      else CUDA_OK(cudaEventCreateWithFlags(&ctx.stage_ev, cudaEventDisableTiming));
      if (ctx.stage_bytes < host_.size()) {
        if (ctx.stage) CUDA_OK(cudaFreeHost(ctx.stage));
        ctx.stage = nullptr, ctx.stage_bytes = 0;
        size_t want = size_t(256) << 10;
        while (want < host_.size()) want *= 2;
        CUDA_OK(cudaMallocHost(&ctx.stage, want));
        ctx.stage_bytes = want;
      }
      std::memcpy(ctx.stage, host_.data(), host_.size());
      src = ctx.stage;
    }
    // (a pageable copy returns once its source has been read)
    CUDA_OK(cudaMemcpyAsync(dev.p, src, host_.size(), cudaMemcpyHostToDevice, ctx.stream));
    if (src == ctx.stage) CUDA_OK(cudaEventRecord(ctx.stage_ev, ctx.stream));
    for (auto &f : set_) f(dev.p);
  }
  size_t bytes() const { return total_; }

 private:
  std::vector<unsigned char> host_;
  std::vector<std::function<void(unsigned char *)>> set_;
  size_t total_ = 0;
};

struct JobImpl {
  Context *ctx;
  FidParams P;
  int C = 0, n = 0, gammaloop = 1, J = 0, rosym = 0, is_static = 0;
  double tau = 0, sw_out = 0, dt = 0;
  BlockLayout L;
  int nint = 0, nq = 0, nr = 0, ne = 0, npq = 0, npr = 0;
  int Cb = 0, nbatch = 0, nwarps_total = 0;
  int ft_jt = 1, ft_pt = 1, ft_r = 1;  // k_fid_tiled tile shape and element ranges
  std::vector<std::vector<int>> blocks_by_size;  // size -> list of block indices (size <= kMaxBlock)
  std::vector<int> big_blocks;                   // blocks kMaxBlock < b <= kMaxBigBlock
  std::vector<BigPair> big_pairs;                // Q/R pairs whose largest block is one of those
  // blocks on the batched products (bl_huge.cuh, bl_xs.cuh): those above kMaxBigBlock, and in the
  // FP64 form those from kXsMin64 on (xs_from: the smallest)
  std::vector<int> huge_blocks;
  int xs_from = 0;
  bool side = false;  // some blocks run on the auxiliary streams
  std::vector<int> huge_sq;                      // per huge block: squarings that bound every step's
  std::vector<BigPair> huge_pairs;               // Q/R pairs with a huge block
  size_t huge_ws_bytes = 0;                      // workspace of the huge-block products
  int huge_items = 0;                            // largest chunk of exponential items
  DevBuf<double2> huge_ws;
  DevBuf<double> hfk;
  DevBuf<int> hsq;
  std::vector<size_t> big_rp_off, huge_rp_off;   // each pair's row pointers in big_rp
  DevBuf<int> big_rp, big_ci;                    // non-zeros of M_ab by row, all big pairs
  DevBuf<double2> big_cv;
  DevBuf<float2> big_cvf;
  DevBuf<int> bs, boff, bpoff, qa, qb, qoff, doff, ra, rb, roff, rhooff, eq, erev, er, erg, esg, status, srp, seo;
  std::vector<DevBuf<int>> blist;
  DevBuf<unsigned char> tables;  // the one buffer behind the uploaded inputs and tables
  DevBuf<double> pas, iscale, Tk, Hc, angles, Rp_all, t0_all, w_all;
  DevBuf<TermEntry> tk_entries;  // large systems: the term operators' non-zeros, scattered into Tk
  DevBuf<int> ikind;
  int has2 = 0;  // second-order quadrupolar terms present
  int p2p = 0, pb = 1, pf = 1, psub = 1;  // point-to-point FID: base, factor, steps per chunk
  DevBuf<double> fkc;                      // the term coefficients of every step
  DevBuf<double> phase;                    // per step: cos, sin of the rotor phase and of twice it
  DevBuf<double2> frames;                  // rf schedule: per chunk frame (permuted index)
  DevBuf<float2> Tk_df, Hc_df;             // mixed form: double-float operators and constant parts
  DevBuf<int> hl_elem;                    // tensor-core blocks: the elements k_tc_hamil assembles
  std::vector<int> hl_off, hl_n;
  DevBuf<int> tk_ptr, tk_term, tk_order;  // blocks above kMaxBlock: the operators' non-zeros by element
  DevBuf<float2> tk_val;
  DevBuf<double> tk_val64;
  DevBuf<double2> Dblk, Rhoblk;
  DevBuf<double2> U, A, VF, Lb, Q, R, G, Z, partial, fid, tw;
  DevBuf<float2> Wf, Qf, Rf, Gf, Zf, twf;  // mixed-precision form
  // mixed form on the tensor cores (large blocks): the step writes each (crystallite, step)'s
  // U slices to a slab the Dyson product reads; one region per large block
  bool tc = false;
  DevBuf<unsigned char> usl;
  DevBuf<unsigned long long> tcf;  // the two tensor-flop counters
  std::vector<size_t> usl_off;  // per block index: byte offset of its region (large blocks)
  int mixed = 0;
  int Ceff = 0;
  double flops = 0;
  int launches = 0;
  size_t h2d = 0;
  bool profiling = false;
  double stage_ms[Job::kStages] = {0};
  int stage_launch[Job::kStages] = {0};
  double stage_fl[Job::kStages] = {0};
  std::vector<cudaEvent_t> evpool;  // stage-boundary events (created when profiling)
  struct Mark {
    int stage, b, e, nlaunch;
  };
  std::vector<Mark> marks;
  int evnext = 0;
  // the context's streams on which the large blocks of one stage run side by side (fork/join
  // on the context stream), so that their one-CTA-per-crystallite launches fill the SMs together
  std::vector<cudaStream_t> aux;
  cudaEvent_t fork_ev = nullptr;
  std::vector<cudaEvent_t> join_ev;
  ~JobImpl() {
    for (auto &e : evpool) cudaEventDestroy(e);
  }
  double cos_rotb = 1, sin_rotb = 0;
  DevSys base{};
};

// Device bytes outside the batch-sized work buffers: tables, per-crystallite inputs (11
// doubles each, padded by up to one batch), warp partials and the FID.
static size_t fixed_bytes(const Powder &pw, const FidParams &p) {
  long n = p.wr != 0.0 ? long(std::floor(p.sw / p.wr + 0.5)) : 1;
  long g = (n >= 1 && n <= 10) ? std::max(1L, 10 / n) : 1;
  size_t ceff = size_t(pw.size()) * size_t(g) + 32;
  // warp partials: up to kFtR rows per warp in the mixed form (k_fid_tiled's element ranges)
  return (size_t(8) << 20) + 2 * ceff * 11 * sizeof(double) +
         (ceff / 32 + 1) * size_t(p.precision == 1 ? kFtR : 1) * size_t(std::max(p.npts, 0)) * sizeof(double2);
}

// Bytes of a planned job with one warp (32) of crystallites per batch and with all of them in one.
static void planned_bytes(const JobSizing &plan, const Powder &pw, const FidParams &p, size_t *min_bytes,
                          size_t *full_bytes) {
  // work buffers are carved with 256-byte alignment: allow for it on each of ~40 buffers
  const size_t fixed = fixed_bytes(pw, p) + 40 * 256 + plan.extra + plan.tables;
  if (min_bytes) *min_bytes = fixed + plan.per_c * 32;
  if (full_bytes) *full_bytes = fixed + plan.per_c * size_t(plan.cpad);
}

// Length q 2^a of Fave's transforms: n itself when twisted (n a power of two), else the length
// >= 2n of least work, per point 3 FP64 operations a radix-2 stage, about 7 for a radix-3 and 10 for
// a radix-5 combining pass (n = 157: 320 points instead of 512).  Lengths of at most 4096 stay
// there: a power of two is always tried.
static void fave_length(int n, bool twist, int &q, int &a) {
  q = 1, a = 1;
  while ((1 << a) < (twist ? n : 2 * n)) ++a;
  if (twist) return;
  double best = double(1 << a) * 3.0 * a;
  for (int t : {3, 5}) {
    int b = 2;
    while ((t << b) < 2 * n) ++b;
    const double cost = double(t << b) * (3.0 * b + (t == 3 ? 7.0 : 10.0));
    if (cost < best && (t << b) < (1 << a)) best = cost, q = t, a = b;
  }
}

static float2 df_split(double v) {
  const float h = float(v);
  return make_float2(h, float(v - double(h)));
}
// term operators of up to this many elements in all go up dense
constexpr size_t kDenseTerms = size_t(1) << 15;

// Smallest block on the batched products in the FP64 form: 7 spins (blocks 21 and 35), 144
// crystallites, n = 120: Dyson 14.6 -> 7.3 ms, eigenframe 14.3 -> 8.7, Q/R 13.3 -> 9.1 against the
// FP64 tiles of k_big_*; below 20 a block fills less than a third of the 64-row tile.  The step stays
// in k_big_step (18.5 ms there, 42 ms as batched products: seven matrices per item through HBM).
constexpr int kXsMin64 = 20;
// Which block pairs (a, b) of M hold a non-zero: one pass over M.
static std::vector<char> nonzero_blocks(const CMatrix &M, const BlockLayout &L) {
  const size_t nb = L.size.size();
  std::vector<char> f(nb * nb, 0);
  for (int r = 0; r < M.n; ++r)
    for (int c = 0; c < M.n; ++c)
      if (M(r, c) != cplx(0, 0)) f[size_t(L.block_of[L.inv[r]]) * nb + size_t(L.block_of[L.inv[c]])] = 1;
  return f;
}

// Every kernel with dynamic shared memory may take all that its static part leaves (once per
// context: the limit is the same for every job, whatever runs beside it).
static void ready_kernels(Context &ctx) {
  std::lock_guard<std::mutex> lock(ctx.mu);
  if (ctx.kernels_ready) return;
  int most = 0;
  CUDA_OK(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx.device));
  auto all = [&](const void *f) {
    cudaFuncAttributes a;
    CUDA_OK(cudaFuncGetAttributes(&a, f));
    CUDA_OK(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, most - int(a.sharedSizeBytes)));
  };
  for (const void *f :
       {(const void *)k_big_step, (const void *)k_big_step_df, (const void *)k_big_dyson<1>,
        (const void *)k_big_dyson<2>, (const void *)k_big_dyson_df<1>, (const void *)k_big_dyson_df<2>,
        (const void *)k_tc_step, (const void *)k_tc_step_stk, (const void *)k_tc_dyson, (const void *)k_tc_dyson_stk,
        (const void *)k_big_seg_frame<false>, (const void *)k_big_seg_frame<true>,
        (const void *)k_big_eigframe<1, double2>, (const void *)k_big_eigframe<2, double2>,
        (const void *)k_big_eigframe4, (const void *)k_big_floquet<true, true, true>, (const void *)k_big_floquet<true, true, false>,
        (const void *)k_big_floquet<false, true, true>, (const void *)k_big_floquet<false, true, false>,
        (const void *)k_big_floquet<false, false, true>, (const void *)k_big_floquet<false, false, false>,
        (const void *)k_huge_floquet,
        (const void *)k_big_qr4, (const void *)k_big_qr<1, float2>, (const void *)k_big_qr<1, double2>,
        (const void *)k_big_qr<2, double2>,
        (const void *)k_fave_fft<8, double2, true>, (const void *)k_fave_fft<8, double2, false>,
        (const void *)k_fave_fft<8, float2, true>, (const void *)k_fave_fft<8, float2, false>,
        (const void *)k_fave_fft<4, double2, true>, (const void *)k_fave_fft<4, double2, false>,
        (const void *)k_fave_fft<4, float2, true>, (const void *)k_fave_fft<4, float2, false>,
        (const void *)k_fave_fft<2, double2, true>, (const void *)k_fave_fft<2, double2, false>,
        (const void *)k_fave_fft<2, float2, true>, (const void *)k_fave_fft<2, float2, false>,
        (const void *)k_fave_fft<1, double2, true>, (const void *)k_fave_fft<1, double2, false>,
        (const void *)k_fave_fft<1, float2, true>, (const void *)k_fave_fft<1, float2, false>,
        (const void *)k_fid_tiled, (const void *)k_xs_gemm<true, 6, false, double2>,
        (const void *)k_xs_gemm<true, 7, false, double2>, (const void *)k_xs_gemm<true, 7, true, double2>,
        (const void *)k_xs_gemm<false, 6, false, double>, (const void *)k_xs_gemm<false, 7, false, double>})
    all(f);
  ctx.kernels_ready = true;
}

Job::Job(Context &ctx, const SpinSystem &sys, const Powder &pw, const CMatrix &ro_in, const CMatrix &det_in,
         const FidParams &p)
    : d_(new JobImpl) {
  JobImpl &J = *d_;
  J.ctx = &ctx;
  J.P = p;
  if (!g_sizing) CUDA_OK(cudaSetDevice(ctx.device));
  if (p.precision != 0 && p.precision != 1) throw Error(1, "precision must be 0 (FP64) or 1 (mixed)");
  if (p.step_method != 0 && p.step_method != 1) throw Error(1, "step_method must be 0 (eigh) or 1 (Taylor)");
  if (p.fave_method < 0 || p.fave_method > 2) throw Error(1, "fave_method must be 0 (auto), 1 (direct) or 2 (FFT)");
  if (p.npts <= 0) throw Error(1, "npts must be positive");
  if (pw.size() <= 0) throw Error(1, "empty powder");
  const int N = sys.dim();
  if (ro_in.n != N || det_in.n != N) throw Error(1, "rho/detect dimension does not match the spin system");
  // oneFID::FID dispatch (oneFID.h:206): no spinning or rotor angle 0 -> static powder FID
  J.is_static = (p.wr == 0.0 || p.rotb_deg == 0.0) ? 1 : 0;
  double tmin = p.start_t;
  J.p2p = p.p2p_base > 0 ? 1 : 0;
  if (J.p2p) {
    if (p.p2p_factor <= 0) throw Error(1, "the point-to-point factor must be positive");
    // PropReduce::setParams (examples/qmsims/MMMQMAS/propreduce.cc:16-33): base and factor
    // divided by their greatest common divisor
    int u = p.p2p_base, v = p.p2p_factor;
    while (v) {
      const int t = u % v;
      u = v, v = t;
    }
    J.pb = p.p2p_base / u, J.pf = p.p2p_factor / u;
    if (!p.rf_chunks.empty()) {  // the schedule is given on the caller's chunks
      if (J.is_static) throw Error(1, "an rf schedule within the rotor period needs spinning (wr > 0, rotor angle != 0)");
      J.pb = p.p2p_base, J.pf = p.p2p_factor;
      for (const auto &rc : p.rf_chunks)
        if (rc.chunk < 0 || rc.chunk >= J.pb) throw Error(1, "rf schedule: chunk outside 0 .. base-1");
    }
    J.gammaloop = 1;
    if (J.is_static) {  // time-independent H: one step of 1/sw per point
      if (!(p.sw > 0)) throw Error(1, "sw must be positive");
      J.pb = J.pf = J.psub = J.n = 1;
      J.tau = 1.0 / p.sw;
      J.sw_out = p.sw;
    } else {
      // chunk of 1/(wr base); steps of at most maxtstep in it, as Propogation::propogator
      // splits a pulse (examples/solid-2.0/src/propogation.cc:246-253)
      const double chunk = 1.0 / (p.wr * J.pb);
      double sub = p.maxtstep > 0 ? std::ceil(chunk / p.maxtstep) : 1.0;
      if (!(sub >= 1.0)) sub = 1.0;
      if (double(J.pb) * sub > double(kMaxP2PSteps))
        throw Error(5, "point-to-point FID needs more than " + std::to_string(kMaxP2PSteps) +
                           " steps per rotor period (base x ceil(chunk/maxtstep))");
      J.psub = int(sub);
      J.n = J.pb * J.psub;
      J.tau = chunk / J.psub;
      J.sw_out = p.wr * J.pb / J.pf;
    }
    J.is_static = 0;  // spinning machinery: steps, Dyson, Floquet, Q/R, then the p2p terms
  } else if (!p.rf_chunks.empty()) {
    throw Error(1, "an rf schedule within the rotor period needs the point-to-point form");
  } else if (J.is_static) {
    // oneFID::singleStaticFID (oneFID.h:292-336): dt = 1/sw as given; the FID index k is
    // split as k = j*ns + p for the reconstruction kernel
    if (!(p.sw > 0)) throw Error(1, "sw must be positive");
    J.n = std::min(64, p.npts);
    J.gammaloop = 1;
    J.sw_out = p.sw;
    J.tau = 0.0;
    J.dt = 1.0 / p.sw;
  } else {
    // compute::CalcComputeStep and the constructor (compute.h:86-97, 213-235)
    J.n = int(std::floor(p.sw / p.wr + 0.5));
    if (J.n < 1) throw Error(1, "sw/wr gives fewer than one step per rotor period");
    int gamma_step = 10;
    J.gammaloop = gamma_step >= J.n ? gamma_step / J.n : 1;
    if (J.gammaloop < 1) J.gammaloop = 1;
    J.sw_out = double(J.n * p.wr);
    double tmax = p.start_t + 1.0 / p.wr;
    J.tau = (tmax - tmin) / J.n;
    if (!(J.tau > 0)) throw Error(1, "the propagator time step is not positive");
  }
  // rf schedule: one system per chunk (the system's own rf plus the chunk's fields) for its
  // constant H and rf frame; the block layout of a system with every scheduled isotope
  // irradiated holds all of them
  const bool sched = !p.rf_chunks.empty();
  std::vector<SpinSystem> chunk_sys;
  if (sched) {
    SpinSystem su = sys;
    std::vector<std::string> isos;
    for (const auto &rc : p.rf_chunks)
      if (rc.field.amp != 0.0 && std::find(isos.begin(), isos.end(), rc.field.iso) == isos.end())
        isos.push_back(rc.field.iso);
    for (const auto &iso : isos) su.add_rf(RfField{iso, 1.2345, 0.0, 0.0});
    J.L = su.layout();
    for (int kc = 0; kc < J.pb; ++kc) {
      chunk_sys.push_back(sys);
      for (const auto &rc : p.rf_chunks)
        if (rc.chunk == kc) chunk_sys.back().add_rf(rc.field);
    }
  } else {
    J.L = sys.layout();
  }
  const BlockLayout &L = J.L;
  if (L.max_block > kMaxHugeBlock)
    throw Error(5, "Hamiltonian block of size " + std::to_string(L.max_block) + " exceeds this engine's limit of " +
                       std::to_string(kMaxHugeBlock));
  if (J.is_static && L.max_block > kMaxBlock)
    throw Error(5, "static powder FIDs support Hamiltonian blocks up to " + std::to_string(kMaxBlock));
  const int nb = int(L.size.size());
  // rosym: exact test ro == 0.5*(det + det^H) on the caller's matrices   (compute.h:75-83)
  J.rosym = 1;
  for (int r = 0; r < N && J.rosym; ++r)
    for (int s = 0; s < N; ++s)
      if (ro_in(r, s) != 0.5 * (det_in(r, s) + std::conj(det_in(s, r)))) {
        J.rosym = 0;
        break;
      }
  // rf phases: the engine propagates the real H' = R^H H R, so rho and det enter as R^H X R
  // (under an rf schedule each step's U is turned back into the lab frame instead)
  const bool turned = !sched && !sys.frame().empty();
  CMatrix ro_t, det_t;
  if (turned) ro_t = sys.to_frame(ro_in), det_t = sys.to_frame(det_in);
  const CMatrix &ro = turned ? ro_t : ro_in, &det = turned ? det_t : det_in;
  if (J.is_static) J.rosym = 0;  // the static FID always transforms rho itself
  // Hamiltonian terms, packed per block
  const int nhc = sched ? J.pb : 1;
  std::vector<double> pas, isc, Hc(size_t(L.S2) * nhc, 0.0);
  std::vector<TermEntry> Tnz;  // non-zeros of the packed operators, term by term
  size_t nnz = 0;              // their number (counted also where only the plan is wanted)
  auto pack = [&](const std::vector<double> &M, double *dst) {
    for (int k = 0; k < nb; ++k)
      for (int r = 0; r < L.size[k]; ++r)
        for (int q = 0; q < L.size[k]; ++q)
          dst[L.poff[k] + r * L.size[k] + q] = M[size_t(L.perm[L.off[k] + r]) * N + L.perm[L.off[k] + q]];
  };
  if (!g_sizing) {  // planning needs only the counts
    if (sched)
      for (int kc = 0; kc < J.pb; ++kc) pack(chunk_sys[kc].h_const(), Hc.data() + size_t(kc) * L.S2);
    else
      pack(sys.h_const(), Hc.data());
  }
  // orientation-dependent terms: kind 0 = scale (M PAS' M^T)_22 T; a quadrupole in a field
  // adds kind 1 = s2 ((r00-r11)^2/4 + r01^2) c4 and kind 2 = -s2 (r02^2 + r12^2) c2 with
  // s2 = Qp^2/(B nu_rel), r = M PAS' M^T (qua.cc:219-267: order 1 or |B| <= 1e-12 first order
  // only, order 2 second order only, otherwise both)
  const auto &ints = sys.interactions();
  const double Bf = sys.bfield();
  std::vector<int> ikind;
  auto entry = [&](int r, int c, double v) {
    const int pr = L.inv[r], pc = L.inv[c], k = L.block_of[pr];
    Tnz.push_back({J.nint * L.S2 + L.poff[k] + (pr - L.off[k]) * L.size[k] + (pc - L.off[k]), 0, v});
  };
  auto add_term = [&](const Interaction &I, int kind, double scale, size_t kk) {
    pas.insert(pas.end(), {I.pas[0][0], I.pas[0][1], I.pas[0][2], I.pas[1][1], I.pas[1][2], I.pas[2][2]});
    isc.push_back(scale);
    ikind.push_back(kind);
    nnz += kind == 0 ? sys.h_nonzeros()[kk].size() : size_t(N);
    if (!g_sizing) {
      if (kind == 0) {
        for (const auto &e : sys.h_nonzeros()[kk]) entry(e.r, e.c, e.v);
      } else {  // the second-order operators are diagonal
        const auto &op = kind == 1 ? sys.h_ops_q4()[kk] : sys.h_ops_q2()[kk];
        for (int r = 0; r < N; ++r)
          if (op[size_t(r) * N + r] != 0.0) entry(r, r, op[size_t(r) * N + r]);
      }
    }
    ++J.nint;
  };
  for (size_t kk = 0; kk < ints.size(); ++kk) {
    const auto &I = ints[kk];
    if (I.kind == 'J') continue;
    const bool quad = I.kind == 'Q';
    const bool first_only = !quad || I.order == 1 || std::fabs(Bf) <= 1e-12;
    const bool second_only = !first_only && I.order == 2;
    if (!second_only) add_term(I, 0, I.op_scale, kk);
    if (!first_only) {
      const double s2 = I.op_scale * I.op_scale / (Bf * isotope_rel_freq(sys.isotopes()[I.s1]));
      add_term(I, 1, s2, kk);
      add_term(I, 2, -s2, kk);
    }
  }
  J.has2 = std::any_of(ikind.begin(), ikind.end(), [](int k) { return k != 0; }) ? 1 : 0;
  // Q pairs (blocks of D) and R pairs (blocks of rho when rho != (D + D^H)/2)
  std::vector<int> qa, qb, qoff, doff, ra, rb, roff, rhooff;
  std::vector<double2> Dblk, Rhoblk;
  std::vector<std::vector<int>> qpair(nb, std::vector<int>(nb, -1)), rpair(nb, std::vector<int>(nb, -1));
  const std::vector<char> det_nz = nonzero_blocks(det, L),
                          ro_nz = J.rosym ? std::vector<char>() : nonzero_blocks(ro, L);
  for (int a = 0; a < nb; ++a)
    for (int b = 0; b < nb; ++b) {
      if (det_nz[size_t(a) * nb + b]) {
        qpair[a][b] = int(qa.size());
        qa.push_back(a), qb.push_back(b), qoff.push_back(J.nq), doff.push_back(int(Dblk.size()));
        for (int r = 0; r < L.size[a]; ++r)
          for (int s = 0; s < L.size[b]; ++s) {
            cplx v = det(L.perm[L.off[a] + r], L.perm[L.off[b] + s]);
            Dblk.push_back(make_double2(v.real(), v.imag()));
          }
        J.nq += L.size[a] * L.size[b];
      }
      if (!J.rosym && ro_nz[size_t(a) * nb + b]) {
        rpair[a][b] = int(ra.size());
        ra.push_back(a), rb.push_back(b), roff.push_back(J.nr), rhooff.push_back(int(Rhoblk.size()));
        for (int r = 0; r < L.size[a]; ++r)
          for (int s = 0; s < L.size[b]; ++s) {
            cplx v = ro(L.perm[L.off[a] + r], L.perm[L.off[b] + s]);
            Rhoblk.push_back(make_double2(v.real(), v.imag()));
          }
        J.nr += L.size[a] * L.size[b];
      }
    }
  J.npq = int(qa.size());
  J.npr = int(ra.size());
  // elements (r,s): Q(r,s) structurally non-zero and R(s,r) structurally non-zero
  std::vector<int> eq, erev, er, erg, esg, srp(J.npq, -1), seo(J.npq, -1);
  for (int pq = 0; pq < J.npq; ++pq) {
    int a = qa[pq], b = qb[pq];
    if (!J.rosym && rpair[b][a] >= 0) srp[pq] = rpair[b][a], seo[pq] = int(eq.size());
    for (int r = 0; r < L.size[a]; ++r)
      for (int s = 0; s < L.size[b]; ++s) {
        int rv = -1, ri = -1;
        if (J.rosym) {
          if (qpair[b][a] >= 0) rv = qoff[qpair[b][a]] + s * L.size[a] + r;
        } else {
          if (rpair[b][a] < 0) continue;
          ri = roff[rpair[b][a]] + s * L.size[a] + r;
        }
        eq.push_back(qoff[pq] + r * L.size[b] + s);
        erev.push_back(rv);
        er.push_back(ri);
        erg.push_back(L.off[a] + r);
        esg.push_back(L.off[b] + s);
      }
  }
  J.ne = int(eq.size());
  J.J = (p.npts + (J.p2p ? J.pb : J.n) - 1) / (J.p2p ? J.pb : J.n);
  {  // k_fid_tiled: up to kFtJmax j's per tile, then as few p tiles as fit 64 threads, each
     // as narrow as it can be; element ranges of at least 64 elements (a function of ne only)
    const int gp = J.p2p ? J.pb : J.n;
    J.ft_jt = std::max(1, std::min(kFtJmax / 4, (J.J + 3) / 4));
    const int pt_max = std::max(1, kFtThreads / J.ft_jt);
    const int ntile = (gp + 4 * pt_max - 1) / (4 * pt_max);
    J.ft_pt = std::max(1, (gp + 4 * ntile - 1) / (4 * ntile));
    J.ft_r = std::max(1, std::min(kFtR, J.ne / 64));
  }
  // crystallites, expanded by the gamma loop (compute.h:294-306: fid summed over q)
  J.C = pw.size();
  J.Ceff = J.C * J.gammaloop;
  const double d2r = kPi / 180.0;
  J.cos_rotb = std::cos(p.rotb_deg * d2r);
  J.sin_rotb = std::sin(p.rotb_deg * d2r);
  // batch size from the memory budget
  const size_t nsteps = J.is_static ? 0 : size_t(J.n);  // U, A, Q, R exist only when spinning
  // mixed form (spinning only): eigenframe W, Q/R, Fave G and z powers Z in single precision
  J.mixed = (p.precision == 1 && !J.is_static) ? 1 : 0;
  const size_t wide = nsteps * (J.nq + J.nr) + size_t(J.n) * J.ne + size_t(J.J) * J.ne;
  size_t per_c = J.mixed ? sizeof(double2) * (nsteps * L.S2 * 2 + L.S2 + N) + sizeof(float2) * (nsteps * L.S2 + wide)
                         : sizeof(double2) * (nsteps * L.S2 * 2 + L.S2 + N + wide);
  per_c += sizeof(double) * 11;
  // term coefficients per (step, term), computed once for all small blocks (k_coef)
  const bool use_fk = !J.is_static && J.nint > 0;
  if (use_fk) per_c += sizeof(double) * size_t(J.n) * size_t(J.nint);
  // tensor-core step and Dyson of the mixed form's large blocks (double-float coefficients
  // from k_coef, no rf schedule): the U slab of every (step, large block)
  J.tc = J.mixed && use_fk && p.step_method == 1 && !sched;
  size_t usl_per_c = 0;
  // FP64 form: blocks from kXsMin64 on take the batched products too (Dyson, eigenframe, Q/R),
  // with the buffer of the FID terms G, idle until Fave, as their workspace; where 32 crystallites'
  // G would not hold two items of each use they stay with k_big_* (a rule on the job's shape, not
  // on its crystallites)
  int xs_from = kMaxBigBlock + 1;
  if (!J.mixed && !J.is_static) {
    size_t need = 0;
    for (int k = 0; k < nb; ++k)
      if (L.size[k] >= kXsMin64 && L.size[k] <= kMaxBigBlock)
        need = std::max(need, sizeof(double2) * size_t(L.size[k]) * L.size[k]);
    for (int pr = 0; pr < J.npq + J.npr; ++pr) {
      const bool isq = pr < J.npq;
      const int ba = L.size[isq ? qa[pr] : ra[pr - J.npq]], bb = L.size[isq ? qb[pr] : rb[pr - J.npq]];
      need = std::max(need, sizeof(double2) * size_t(ba) * bb);
    }
    if (L.max_block <= kMaxBigBlock && size_t(J.n) * J.ne * sizeof(double2) * 32 >= 2 * need + 4096) xs_from = kXsMin64;
  }
  J.xs_from = xs_from;
  if (J.tc) {
    J.usl_off.assign(nb, 0);
    for (int k = 0; k < nb; ++k)
      if (L.size[k] >= tc::kMinB && L.size[k] <= tc::kMaxB) usl_per_c += nsteps * tc::slab_bytes(L.size[k]);
    per_c += usl_per_c;
  }
  long cpad_all = ((long(J.Ceff) + 31) / 32) * 32;
  // huge blocks: one workspace for their batched products, at least one item of each use
  // (exponential: 7 real b x b; Floquet: 2 complex b x b, 3 in the mixed form; eigenframe, Q/R: one complex
  // matrix), else 1 GiB
  size_t huge_fixed = 0;
  {
    size_t need = 0;
    int bmin = 0;
    for (int k = 0; k < nb; ++k) {
      const size_t b = size_t(L.size[k]);
      if (L.size[k] <= kMaxBigBlock) continue;
      need = std::max(need, std::max(sizeof(double) * kHugeSlots * b * b,
                                     (p.precision == 1 ? 3 : 2) * sizeof(double2) * b * b));
      bmin = bmin ? std::min(bmin, L.size[k]) : L.size[k];
    }
    for (int pr = 0; pr < J.npq + J.npr; ++pr) {
      const bool isq = pr < J.npq;
      const int ba = L.size[isq ? qa[pr] : ra[pr - J.npq]], bb = L.size[isq ? qb[pr] : rb[pr - J.npq]];
      if (std::max(ba, bb) > kMaxBigBlock) need = std::max(need, sizeof(double2) * size_t(ba) * bb);
    }
    if (need && !J.is_static) {
      J.huge_ws_bytes = (std::max(need, size_t(1) << 30) + 255) / 256 * 256;
      J.huge_items = int(std::min<size_t>(kHugeMaxItems, J.huge_ws_bytes / (sizeof(double) * kHugeSlots *
                                                                            size_t(bmin) * size_t(bmin))));
      huge_fixed = J.huge_ws_bytes + size_t(J.huge_items) * (sizeof(double) * (J.nint + 1) + sizeof(int)) + 4096;
    }
  }
  JobSizing plan;
  plan.per_c = per_c;
  plan.cpad = cpad_all;
  plan.extra = huge_fixed;
  {  // Tk and Hc (per chunk), their double-float copies in the mixed form, the D and rho
     // blocks, the rf frames, and 256-byte alignment per buffer
    const size_t tk = size_t(J.nint) * L.S2, hc = size_t(L.S2) * (sched ? J.pb : 1);
    plan.tables = (tk + hc) * sizeof(double) * ((p.precision == 1 && !J.is_static) ? 2 : 1) +
                  (Dblk.size() + Rhoblk.size()) * sizeof(double2) + size_t(N) * J.pb * sizeof(double2) + 64 * 256;
    // the tables in index form: FID elements, pairs, M_ab by row, operators by term and by element.  Up
    // to 9 spins they fit the allowance of fixed_bytes; what goes beyond it is counted here (11 spins:
    // 24 MB)
    auto nonzeros = [](const std::vector<double2> &v) {
      return size_t(std::count_if(v.begin(), v.end(), [](double2 z) { return z.x != 0.0 || z.y != 0.0; }));
    };
    size_t rows = 0;
    for (int pr = 0; pr < J.npq + J.npr; ++pr) rows += size_t(L.size[pr < J.npq ? qa[pr] : ra[pr - J.npq]]) + 1;
    const size_t index = size_t(J.ne) * 5 * sizeof(int) + size_t(J.npq + J.npr) * 6 * sizeof(int) + rows * sizeof(int) +
                         (nonzeros(Dblk) + nonzeros(Rhoblk)) * (sizeof(int) + sizeof(double2) + sizeof(float2)) +
                         nnz * (sizeof(TermEntry) + sizeof(int) + sizeof(double) + sizeof(float2)) +
                         size_t(L.S2) * 3 * sizeof(int) + size_t(J.n) * 4 * sizeof(double) + 4096 * sizeof(double2);
    constexpr size_t kAllowance = size_t(7) << 20;  // of fixed_bytes' 8 MiB
    if (index > kAllowance) plan.tables += index - kAllowance;
  }
  if (g_sizing) {
    *g_sizing = plan;
    return;
  }
  size_t budget = ctx.hbm_budget;
  ScratchArena asked;
  struct ArenaScope {
    bool on = false;
    ScratchArena *prev = nullptr;
    ~ArenaScope() {
      if (on) g_arena = prev;
    }
  } arena_scope;
  if (g_region) {
    size_t lo = 0, full = 0, bytes = 0;
    planned_bytes(plan, pw, p, &lo, &full);
    asked.base = static_cast<char *>((*g_region)(lo, full, &bytes));
    const size_t fixed = fixed_bytes(pw, p);
    if (!asked.base || fixed >= bytes) throw Error(4, "job does not fit its device region");
    asked.cap = bytes, asked.label = "device region given to the job", asked.aux_streams = true;
    arena_scope.prev = g_arena, arena_scope.on = true;
    g_arena = &asked;
    budget = bytes - fixed;
  }
  if (!budget) {  // default: 60% of the device memory free when the job is created
    size_t fr = 0, tot = 0;
    CUDA_OK(cudaMemGetInfo(&fr, &tot));
    budget = size_t(0.6 * double(fr));
  }
  if (g_arena && g_arena->aux_streams) {  // a region holds the tables too
    const size_t tables = plan.tables + 40 * 256;
    budget = budget > tables ? budget - tables : 0;
  }
  budget = budget > huge_fixed ? budget - huge_fixed : 0;
  long cb = long(budget / std::max<size_t>(per_c, 1));
  cb = (cb / 32) * 32;
  if (cb < 32) throw Error(4, "job does not fit the device memory budget (one warp of crystallites)");
  // as few batches as the budget allows, of equal size (no small remainder batch)
  const long nb_min = (cpad_all + cb - 1) / cb;
  J.Cb = int(((long(J.Ceff) + nb_min - 1) / nb_min + 31) / 32 * 32);
  J.nbatch = int((cpad_all + J.Cb - 1) / J.Cb);
  J.nwarps_total = J.nbatch * (J.Cb / 32);
  // block lists by size
  J.blocks_by_size.assign(kMaxBlock + 1, {});
  for (int k = 0; k < nb; ++k) {
    if (L.size[k] <= kMaxBlock) J.blocks_by_size[L.size[k]].push_back(k);
    else if (L.size[k] < xs_from) J.big_blocks.push_back(k);
    else J.huge_blocks.push_back(k);
  }
  // per huge block: squarings enough for every step, from a rotation-free bound on
  // ||2 pi tau H||_inf (|a_k| <= ||PAS'_k||_F); the kernels skip items that need fewer
  std::vector<double> row_bound;  // per permuted row: largest constant part plus the terms' bounds
  if (!J.huge_blocks.empty()) {
    row_bound.assign(N, 0.0);
    for (int k : J.huge_blocks)
      for (int r = 0; r < L.size[k]; ++r)
        for (int q = 0; q < L.size[k]; ++q) {
          double v = 0;  // the largest over the chunks of an rf schedule
          for (int kc = 0; kc < nhc; ++kc)
            v = std::max(v, std::fabs(Hc[size_t(kc) * L.S2 + L.poff[k] + r * L.size[k] + q]));
          row_bound[L.off[k] + r] += v;
        }
    std::vector<int> row_of(L.S2);
    for (int k = 0; k < nb; ++k)
      for (int e = 0; e < L.size[k] * L.size[k]; ++e) row_of[L.poff[k] + e] = L.off[k] + e / L.size[k];
    for (const TermEntry &e : Tnz) {
      const int kk = e.idx / L.S2;
      const double *Pa = pas.data() + 6 * kk;
      const double fro = std::sqrt(Pa[0] * Pa[0] + Pa[3] * Pa[3] + Pa[5] * Pa[5] +
                                   2 * (Pa[1] * Pa[1] + Pa[2] * Pa[2] + Pa[4] * Pa[4]));
      // |r_ij| <= ||PAS'||_F: first order |a| <= fro, second order |a| <= 2 fro^2
      const double amax = ikind[kk] == 0 ? fro : 2.0 * fro * fro;
      row_bound[row_of[e.idx % L.S2]] += std::fabs(isc[kk]) * amax * std::fabs(e.v);
    }
  }
  for (int k : J.huge_blocks) {
    double nrm = 0;
    for (int r = 0; r < L.size[k]; ++r) nrm = std::max(nrm, row_bound[L.off[k] + r]);
    nrm *= J.tau * kPi2 * (1.0 + 1e-10);  // margin over the rounding of either side's sums
    int q = 0;
    if (nrm > 0.5) {
      std::frexp(nrm / 0.5, &q);
      q = std::min(q, 60);
    }
    J.huge_sq.push_back(q);
  }
  std::vector<int> big_rp_h, big_ci_h;
  std::vector<double2> big_cv_h;
  if (!J.big_blocks.empty() || !J.huge_blocks.empty()) {
    if (std::any_of(L.size.begin(), L.size.end(), [](int b) { return b > kMaxBlock && b <= kMaxBigBlock; }) &&
        J.nint > kMaxInt)
      throw Error(5, "more than " + std::to_string(kMaxInt) + " anisotropic interactions");
    // Q/R pairs with a big block: M_ab's non-zeros by row, and the W_b column chunk that
    // keeps W_a, W_b and X within half the shared memory (two CTAs per SM) where it can
    for (int pr = 0; pr < J.npq + J.npr; ++pr) {
      const bool isq = pr < J.npq;
      const int a = isq ? qa[pr] : ra[pr - J.npq], b = isq ? qb[pr] : rb[pr - J.npq];
      const int ba = L.size[a], bb = L.size[b];
      if (ba <= kMaxBlock && bb <= kMaxBlock) continue;
      const double2 *M = isq ? Dblk.data() + doff[pr] : Rhoblk.data() + rhooff[pr - J.npq];
      const size_t rp_off = big_rp_h.size();
      for (int l = 0; l < ba; ++l) {
        big_rp_h.push_back(int(big_ci_h.size()));
        for (int m = 0; m < bb; ++m) {
          const double2 v = M[l * bb + m];
          if (v.x != 0.0 || v.y != 0.0) big_ci_h.push_back(m), big_cv_h.push_back(v);
        }
      }
      big_rp_h.push_back(int(big_ci_h.size()));
      int nch = 1, w = bb;
      for (;;) {
        w = (bb + nch - 1) / nch;
        if ((J.mixed ? big_qr4_smem(ba, bb, w) : big_qr_smem<double2>(ba, bb, w)) <= (size_t(113) << 10) || w <= 8) break;
        ++nch;
      }
      double most = 1e-300;  // largest row or column sum of |M_ab|
      std::vector<double> col(bb, 0.0);
      for (int l = 0; l < ba; ++l) {
        double row = 0;
        for (int m = 0; m < bb; ++m) {
          const double v = std::hypot(M[l * bb + m].x, M[l * bb + m].y);
          row += v, col[m] += v;
        }
        most = std::max(most, row);
      }
      for (double v : col) most = std::max(most, v);
      int e2 = 0;
      std::frexp(most, &e2);  // most < 2^e2
      BigPair P{a, b, isq ? qoff[pr] : roff[pr - J.npq], isq ? J.nq : J.nr, isq ? 1 : 0, w, e2, nullptr, nullptr, nullptr, nullptr};
      if (std::max(ba, bb) >= xs_from) {  // k_huge_mx + a product
        J.huge_pairs.push_back(P);
        J.huge_rp_off.push_back(rp_off);
        continue;
      }
      J.big_pairs.push_back(P);
      J.big_rp_off.push_back(rp_off);
    }
  }
  ready_kernels(ctx);
  J.side = !J.big_blocks.empty() || (xs_from <= kMaxBigBlock && !J.huge_blocks.empty());
  if (J.side && (!g_arena || g_arena->aux_streams)) {
    const size_t naux = std::min<size_t>(4, std::max({J.big_blocks.size(), J.big_pairs.size(), J.huge_blocks.size()}));
    std::lock_guard<std::mutex> lock(ctx.mu);
    if (!ctx.fork_ev) CUDA_OK(cudaEventCreateWithFlags(&ctx.fork_ev, cudaEventDisableTiming));
    while (ctx.join_ev.size() < naux) {
      cudaStream_t x;
      cudaEvent_t e;
      if (ctx.aux.size() == ctx.join_ev.size()) {
        CUDA_OK(cudaStreamCreateWithFlags(&x, cudaStreamNonBlocking));
        ctx.aux.push_back(x);
      }
      CUDA_OK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
      ctx.join_ev.push_back(e);
    }
    J.aux.assign(ctx.aux.begin(), ctx.aux.begin() + std::ptrdiff_t(naux));
    J.join_ev.assign(ctx.join_ev.begin(), ctx.join_ev.begin() + std::ptrdiff_t(naux));
    J.fork_ev = ctx.fork_ev;
  }
  J.blist.resize(kMaxBlock + 1);
  cudaStream_t st = ctx.stream;
  Uploads up;
  for (int b = 1; b <= kMaxBlock; ++b) up.add(J.blist[b], J.blocks_by_size[b]);
  up.add(J.bs, L.size), up.add(J.boff, L.off), up.add(J.bpoff, L.poff);
  up.add(J.qa, qa), up.add(J.qb, qb), up.add(J.qoff, qoff), up.add(J.doff, doff);
  up.add(J.ra, ra), up.add(J.rb, rb), up.add(J.roff, roff), up.add(J.rhooff, rhooff);
  up.add(J.eq, eq), up.add(J.erev, erev), up.add(J.er, er), up.add(J.erg, erg), up.add(J.esg, esg);
  up.add(J.srp, srp), up.add(J.seo, seo);
  up.add(J.big_rp, big_rp_h), up.add(J.big_ci, big_ci_h), up.add(J.big_cv, big_cv_h);
  if (J.mixed) {
    std::vector<float2> f(big_cv_h.size());
    for (size_t x = 0; x < f.size(); ++x) f[x] = make_float2(float(big_cv_h[x].x), float(big_cv_h[x].y));
    up.add(J.big_cvf, f);
  }
  up.add(J.pas, pas), up.add(J.iscale, isc), up.add(J.Hc, Hc);
  // the packed operators: dense from the host while they are small, else their non-zeros go up
  // and k_scatter_terms fills the (zeroed) dense tables (9 spins: 17.5 MB in each precision, 45
  // terms of 768 non-zeros)
  const bool df_tables = p.precision == 1 && !J.is_static;
  const size_t tk_n = size_t(J.nint) * L.S2;
  const bool scatter = tk_n > kDenseTerms;
  if (scatter) {
    up.add(J.tk_entries, Tnz);
  } else {
    std::vector<double> Tk(tk_n, 0.0);
    for (const TermEntry &e : Tnz) Tk[size_t(e.idx)] = e.v;
    up.add(J.Tk, Tk);
    if (df_tables) {
      std::vector<float2> t(tk_n);
      for (size_t x = 0; x < tk_n; ++x) t[x] = df_split(Tk[x]);
      up.add(J.Tk_df, t);
    }
  }
  if (p.precision == 1 && !J.is_static) {  // hi, lo splits for the mixed form's double-float step
    std::vector<float2> h(Hc.size());
    for (size_t x = 0; x < Hc.size(); ++x) h[x] = df_split(Hc[x]);
    up.add(J.Hc_df, h);
  }
  if (L.max_block > kMaxBlock) {
    // by element, terms ascending: a counting pass, then the entries in term order
    std::vector<int> ptr(size_t(L.S2) + 1, 0), term(Tnz.size());
    std::vector<float2> val(df_tables ? Tnz.size() : 0);
    std::vector<double> val64(Tnz.size());
    for (const TermEntry &e : Tnz) ++ptr[size_t(e.idx % L.S2) + 1];
    for (int e = 0; e < L.S2; ++e) ptr[size_t(e) + 1] += ptr[e];
    {
      std::vector<int> at(ptr.begin(), ptr.end() - 1);
      for (const TermEntry &e : Tnz) {
        const int x = at[e.idx % L.S2]++;
        term[x] = e.idx / L.S2, val64[x] = e.v;
        if (df_tables) val[x] = df_split(e.v);
      }
    }
    // per block, its elements by descending term count (ties in element order): the
    // step's H build visits them in this order, so a warp's lanes walk similar lengths
    std::vector<int> order(size_t(L.S2), 0);
    for (size_t kb = 0; kb < L.size.size(); ++kb) {
      const int b = L.size[kb], bp = L.poff[kb];
      int *o = order.data() + bp;
      std::vector<int> first(size_t(J.nint) + 2, 0);  // by term count, the largest first
      auto bucket = [&](int e) { return size_t(J.nint - (ptr[bp + e + 1] - ptr[bp + e])); };
      for (int e = 0; e < b * b; ++e) ++first[bucket(e) + 1];
      for (int t = 0; t <= J.nint; ++t) first[size_t(t) + 1] += first[size_t(t)];
      for (int e = 0; e < b * b; ++e) o[first[bucket(e)]++] = e;
    }
    up.add(J.tk_ptr, ptr), up.add(J.tk_term, term), up.add(J.tk_val, val), up.add(J.tk_val64, val64);
    up.add(J.tk_order, order);
    if (J.tc) {
      std::vector<int> elem;
      J.hl_off.assign(L.size.size(), 0), J.hl_n.assign(L.size.size(), 0);
      for (size_t kb = 0; kb < L.size.size(); ++kb) {
        const int b = L.size[kb], bp = L.poff[kb];
        if (b < tc::kMinB || b > tc::kMaxB) continue;
        J.hl_off[kb] = int(elem.size());
        for (int x = 0; x < b * b; ++x) {
          const int e = order[size_t(bp) + x];
          if (e / b <= e % b && (ptr[size_t(bp) + e + 1] > ptr[size_t(bp) + e] || Hc[size_t(bp) + e] != 0.0))
            elem.push_back(e);
        }
        J.hl_n[kb] = int(elem.size()) - J.hl_off[kb];
      }
      up.add(J.hl_elem, elem);
    }
  }
  if (sched) {  // per chunk: the rf frame of each permuted index (1 where a chunk has none)
    bool any = false;
    for (const auto &cs : chunk_sys) any = any || !cs.frame().empty();
    if (any) {
      std::vector<double2> fr(size_t(J.pb) * N, make_double2(1.0, 0.0));
      for (int kc = 0; kc < J.pb; ++kc) {
        const auto &f = chunk_sys[kc].frame();
        if (f.empty()) continue;
        for (int x = 0; x < N; ++x) fr[size_t(kc) * N + x] = make_double2(f[L.perm[x]].real(), f[L.perm[x]].imag());
      }
      up.add(J.frames, fr);
    }
  }
  up.add(J.ikind, ikind);
  up.add(J.Dblk, Dblk), up.add(J.Rhoblk, Rhoblk);
  // per-crystallite inputs, batch-major and crystallite-fastest: the powder angles (k_orient
  // forms the rotations), start times and weights, expanded by the gamma loop
  // (compute.h:294-306: fid summed over q)
  {
    const size_t all = size_t(J.nbatch) * J.Cb;
    std::vector<double> ang(3 * all, 0.0), t0(all, 0.0), w(all, 0.0);
    for (int c = 0; c < J.C; ++c)
      for (int q = 0; q < J.gammaloop; ++q) {
        const size_t cg = size_t(c) * J.gammaloop + q;  // batches are Cb apart: its own place too
        ang[cg] = pw.phi[c], ang[all + cg] = pw.theta[c], ang[2 * all + cg] = pw.gamma[c];
        t0[cg] = q == 0 ? tmin : tmin + kPi2 * double(q) / double(J.gammaloop * J.n) / p.wr;
        w[cg] = pw.weight[c];
      }
    up.add(J.angles, ang), up.add(J.t0_all, t0), up.add(J.w_all, w);
  }
  // FFT length of the Fave correlation: n itself when it is a power of two (twisted circular
  // correlation; FP64 form only, its twist factors are FP64 work), else the cheapest of 2^a, 3 2^a and
  // 5 2^a from 2n on (zero-padded linear correlation; fave_length)
  DevSys &s = J.base;
  if (!J.p2p) {
    s.fave_twist = (!J.mixed && J.n >= 8 && (J.n & (J.n - 1)) == 0) ? 1 : 0;
    fave_length(J.n, s.fave_twist != 0, s.fftq, s.logM);
    s.M = s.fftq << s.logM;
    // FFT correlation up to M = 4096 (its shared-memory tile is M * max(1, 2048/M) * 32 B)
    if (p.fave_method == 2 && s.M > 4096) throw Error(5, "FFT Fave supports at most 2048 steps per period");
    s.fave_method = (p.fave_method != 1 && s.M <= 4096) ? 1 : 0;
    if (J.mixed && !s.fave_method) throw Error(5, "the mixed form needs the FFT correlation (at most 2048 steps)");
    if (s.fave_method) {
      std::vector<double2> tw(s.M);
      for (int k = 0; k < s.M; ++k) {
        double a = kPi2 * double(k) / double(s.M);
        tw[k] = make_double2(std::cos(a), -std::sin(a));
      }
      if (J.mixed) {
        std::vector<float2> twf(tw.size());
        for (size_t k = 0; k < tw.size(); ++k) twf[k] = make_float2(float(tw[k].x), float(tw[k].y));
        up.add(J.twf, twf);
      } else {
        up.add(J.tw, tw);
      }
    }
  } else {  // no Fave: the point-to-point terms come from Q/R and the Floquet phases
    s.fave_twist = 0, s.logM = 0, s.M = 0, s.fftq = 1, s.fave_method = 0;
  }
  // (the series' 5 nint doubles per crystallite have to fit A: n S2 complex)
  if (use_fk && !J.has2 && J.gammaloop == 1 && size_t(5) * J.nint <= 2 * nsteps * L.S2) {
    std::vector<double> ph(size_t(4) * J.n);
    for (int i = 0; i < J.n; ++i) {
      const double t1 = tmin + double(i) * J.tau, t2 = t1 + J.tau, a = ((t2 - t1) / 2.0 + t1) * p.wr * kPi2;
      ph[4 * i] = std::cos(a), ph[4 * i + 1] = std::sin(a), ph[4 * i + 2] = std::cos(2 * a), ph[4 * i + 3] = std::sin(2 * a);
    }
    up.add(J.phase, ph);
  }
  up.flush(ctx, J.tables, !g_arena || g_arena->aux_streams);
  J.h2d = up.bytes();
  s.tw = J.tw.p, s.twf = J.twf.p;
  for (size_t t = 0; t < J.big_pairs.size(); ++t)
    J.big_pairs[t].rp = J.big_rp.p + J.big_rp_off[t], J.big_pairs[t].ci = J.big_ci.p, J.big_pairs[t].cv = J.big_cv.p,
    J.big_pairs[t].cvf = J.big_cvf.p;
  for (size_t t = 0; t < J.huge_pairs.size(); ++t)
    J.huge_pairs[t].rp = J.big_rp.p + J.huge_rp_off[t], J.huge_pairs[t].ci = J.big_ci.p,
    J.huge_pairs[t].cv = J.big_cv.p, J.huge_pairs[t].cvf = J.big_cvf.p;
  if (scatter) {
    J.Tk.alloc(tk_n);
    CUDA_OK(cudaMemsetAsync(J.Tk.p, 0, tk_n * sizeof(double), st));
    if (df_tables) {
      J.Tk_df.alloc(tk_n);
      CUDA_OK(cudaMemsetAsync(J.Tk_df.p, 0, tk_n * sizeof(float2), st));
    }
    k_scatter_terms<<<grid_for(long(Tnz.size())), kThreads, 0, st>>>(J.tk_entries.p, int(Tnz.size()), J.Tk.p, J.Tk_df.p);
  }
  J.Rp_all.alloc(size_t(J.nbatch) * 9 * J.Cb);
  k_orient<<<grid_for(long(J.nbatch) * J.Cb), kThreads, 0, st>>>(J.angles.p, J.nbatch * J.Cb, J.Cb, J.Rp_all.p);
  CUDA_OK(cudaGetLastError());
  size_t Cb = J.Cb;
  J.U.alloc(std::max<size_t>(1, nsteps * L.S2 * Cb));
  J.A.alloc(std::max<size_t>(1, nsteps * L.S2 * Cb));
  J.VF.alloc(size_t(L.S2) * Cb);
  J.Lb.alloc(size_t(N) * Cb);
  const size_t nQ = std::max<size_t>(1, nsteps * J.nq * Cb), nR = std::max<size_t>(1, nsteps * J.nr * Cb);
  const size_t nG = std::max<size_t>(1, size_t(J.n) * J.ne * Cb), nZ = std::max<size_t>(1, size_t(J.J) * J.ne * Cb);
  if (J.mixed) {
    J.Wf.alloc(std::max<size_t>(1, nsteps * L.S2 * Cb));
    J.Qf.alloc(nQ), J.Rf.alloc(nR), J.Gf.alloc(nG), J.Zf.alloc(nZ);
    J.Q.alloc(1), J.R.alloc(1), J.G.alloc(1), J.Z.alloc(1);
  } else {
    J.Q.alloc(nQ), J.R.alloc(nR), J.G.alloc(nG), J.Z.alloc(nZ);
  }
  J.partial.alloc(size_t(J.nwarps_total) * (J.mixed ? J.ft_r : 1) * p.npts);
  if (!J.huge_blocks.empty() && xs_from <= kMaxBigBlock) {  // the workspace lies in G
    J.huge_ws_bytes = J.G.n * sizeof(double2);
    J.huge_ws.p = J.G.p, J.huge_ws.n = J.G.n, J.huge_ws.owned = false;
  } else if (J.huge_ws_bytes) {
    J.huge_ws.alloc(J.huge_ws_bytes / sizeof(double2));
    J.hfk.alloc(size_t(J.huge_items) * std::max(J.nint, 1));
    J.hsq.alloc(size_t(J.huge_items));
  }
  // the FID, then the status word and the two tensor-flop counters: one read brings them all
  J.fid.alloc(size_t(p.npts) + 2);
  J.status.p = reinterpret_cast<int *>(J.fid.p + p.npts), J.status.n = 1, J.status.owned = false;
  J.tcf.p = reinterpret_cast<unsigned long long *>(J.fid.p + p.npts + 1), J.tcf.n = 2, J.tcf.owned = false;
  if (use_fk) J.fkc.alloc(size_t(J.n) * J.nint * Cb);
  if (J.tc && usl_per_c) {
    J.usl.alloc(usl_per_c * Cb);
    size_t off = 0;
    for (int k = 0; k < nb; ++k)
      if (L.size[k] >= tc::kMinB && L.size[k] <= tc::kMaxB) {
        J.usl_off[k] = off;
        off += nsteps * tc::slab_bytes(L.size[k]) * Cb;
      }
  }
  // algorithmic flop count (one complex MAC = 8 flop; eigh counted as 32 b^3, the
  // Floquet eig as 100 b^3)
  double S3 = 0;
  for (int k = 0; k < nb; ++k) S3 += double(L.size[k]) * L.size[k] * L.size[k];
  double pairs = 0;
  for (int pq = 0; pq < J.npq + J.npr; ++pq) {
    int a = pq < J.npq ? qa[pq] : ra[pq - J.npq], b = pq < J.npq ? qb[pq] : rb[pq - J.npq];
    pairs += double(L.size[a]) * L.size[b] * (L.size[a] + L.size[b]);
  }
  double S2H = 0;  // H build: one FMA per operator entry per interaction
  for (int k = 0; k < nb; ++k) S2H += double(L.size[k]) * L.size[k];
  double Ce = J.Ceff;
  J.stage_fl[0] = Ce * (J.is_static ? 1 : J.n) * (11.0 * S3 + 2.0 * J.nint * S2H);  // eigh + U + H build
  const double spin_steps = J.is_static ? 0.0 : double(J.n);
  J.stage_fl[1] = Ce * spin_steps * 8.0 * S3;                   // Dyson
  J.stage_fl[2] = J.is_static ? 0.0 : Ce * 100.0 * S3;          // Floquet eig
  J.stage_fl[3] = Ce * spin_steps * 8.0 * S3;                   // W = A V_F
  J.stage_fl[4] = Ce * spin_steps * 8.0 * pairs;               // Q, R transforms
  {
    // Fave correlation: direct 8 n^2 per element; FFT: 5 M log2 M per length-M transform
    // (two when r = conj(q), three otherwise), 8 M for the spectrum product, 8 n for G
    // (length n with 6 flop per twisted point when n is a power of two, else length >= 2n)
    const bool twist = !J.mixed && J.n >= 8 && (J.n & (J.n - 1)) == 0;
    int fq = 1, lm = 1;
    fave_length(J.n, twist, fq, lm);
    double M = double(fq << lm), fftf = 5.0 * M * std::log2(M);
    bool fft = p.fave_method != 1 && M <= 4096;
    double per = 0;
    for (int e = 0; e < J.ne; ++e) {
      bool autoc = J.rosym && erev[e] < 0;
      per += fft ? (autoc ? 2 : 3) * fftf + 8.0 * M + 8.0 * J.n + (twist ? (autoc ? 12.0 : 18.0) * J.n : 0.0)
                 : 8.0 * J.n * J.n;
    }
    J.stage_fl[5] = J.is_static ? Ce * (16.0 * pairs + 8.0 * J.n * J.ne) : Ce * per;
    if (J.p2p) J.stage_fl[5] = Ce * 16.0 * J.pb * J.ne;  // two complex products per (k, element)
  }
  J.stage_fl[6] = Ce * 8.0 * p.npts * J.ne;                     // FID reconstruction
  J.stage_fl[7] = 4.0 * p.npts * J.nwarps_total * (J.mixed ? J.ft_r : 1);  // compensated powder sum
  J.flops = 0;
  for (double f : J.stage_fl) J.flops += f;
  // static part of the device description
  s.n = J.n, s.npts = p.npts, s.N = N, s.nb = nb, s.S2 = L.S2, s.nint = J.nint, s.nq = J.nq, s.nr = J.nr;
  s.ne = J.ne, s.J = J.J, s.rosym = J.rosym, s.step_method = p.step_method;
  s.tau = J.tau, s.wr = p.wr, s.sin_rotb = J.sin_rotb, s.cos_rotb = J.cos_rotb;
  s.is_static = J.is_static, s.dt = J.dt, s.srp = J.srp.p, s.seo = J.seo.p;
  s.scale = J.is_static ? 1.0 : double(1. / double(J.n / (J.rosym ? 2 : 1)));
  s.gper = J.n, s.p2p = J.p2p, s.pb = J.pb, s.pf = J.pf, s.psub = J.psub;
  s.ft_jt = J.ft_jt, s.ft_pt = J.ft_pt, s.ft_r = J.ft_r;
  s.ft_sub = fid_tiled_sub(J.ft_jt, J.ft_pt);
  if (J.p2p) {  // fid = sum_c w_c Tr(rho_c det) / Tr(det det^H)  (sequencerun_funcs.cc:624-645)
    double dd = 0;
    for (const auto &v : det.a) dd += std::norm(v);
    if (!(dd > 0)) throw Error(1, "the detection operator is zero");
    s.scale = 1.0 / dd;
    s.gper = J.pb;
  }
  // A factor that every term shares (1/M, the scale, equal weights) is no single-precision number in
  // general, and its rounding, up to 2^-24, would shift the whole FID: 6e-8 at 48 steps.
  s.wref = 0.0;
  for (int c = 0; c < J.C; ++c) s.wref = std::max(s.wref, std::fabs(pw.weight[c]));
  if (!(s.wref > 0.0 && std::isfinite(s.wref))) s.wref = 1.0;
  s.wscale = s.wref * s.scale / double(s.fftq);
  s.bs = J.bs.p, s.boff = J.boff.p, s.bpoff = J.bpoff.p;
  s.pas = J.pas.p, s.iscale = J.iscale.p, s.Tk = J.Tk.p, s.Hc = J.Hc.p;
  s.fk = use_fk ? J.fkc.p : nullptr;
  s.hc_chunks = sched ? J.pb : 0;
  s.frames = J.frames.n ? J.frames.p : nullptr;
  s.Tk_df = J.Tk_df.p, s.Hc_df = J.Hc_df.p;
  s.tk_ptr = J.tk_ptr.p, s.tk_term = J.tk_term.p, s.tk_val = J.tk_val.p, s.tk_val64 = J.tk_val64.p, s.tk_order = J.tk_order.p;
  s.fk_df = (J.mixed && p.step_method == 1 && use_fk) ? 1 : 0;
  {
    const double tp = J.tau * kPi2;
    const float h = float(tp);
    s.tpdf = make_float2(h, float(tp - double(h)));
  }
  s.ikind = J.ikind.p, s.has2 = J.has2;
  s.npq = J.npq, s.npr = J.npr;
  s.qa = J.qa.p, s.qb = J.qb.p, s.qoff = J.qoff.p, s.doff = J.doff.p;
  s.ra = J.ra.p, s.rb = J.rb.p, s.roff = J.roff.p, s.rhooff = J.rhooff.p;
  s.Dblk = J.Dblk.p, s.Rhoblk = J.Rhoblk.p;
  s.mixed = J.mixed;
  s.floq32 = 0;
  if (J.mixed && J.n > 0 && J.pb > 0) {  // the mixed form spins (never static)
    const long periods = J.p2p ? (long(p.npts) - 1) * J.pf / J.pb + 1 : (long(p.npts) - 1) / J.n + 1;
    s.floq32 = periods <= kFloq32MaxPeriods ? 1 : 0;
  }
  s.Wf = J.Wf.p, s.Qf = J.Qf.p, s.Rf = J.Rf.p, s.Gf = J.Gf.p, s.Zf = J.Zf.p;
  s.eq = J.eq.p, s.erev = J.erev.p, s.er = J.er.p, s.erg = J.erg.p, s.esg = J.esg.p;
  s.U = J.U.p, s.A = J.A.p, s.VF = J.VF.p, s.L = J.Lb.p, s.Q = J.Q.p, s.R = J.R.p, s.G = J.G.p, s.Z = J.Z.p;
  s.partial = J.partial.p;
  s.status = J.status.p;
  s.tc_flops = J.tcf.p;
  s.clay = (J.mixed && J.huge_blocks.empty()) ? 1 : 0;
  s.Cpad = J.Cb;
  // the tensor-core blocks (mixed form) keep one chain per crystallite
  s.nseg = J.is_static ? 1 : (J.n + kSegLen - 1) / kSegLen;
  s.seg_max = s.nseg > 1 ? (J.tc ? tc::kMinB - 1 : kMaxBigBlock) : 0;
  s.seg_from = s.nseg > 1 ? kMaxBigBlock + 1 : 1 << 30;
}

Job::~Job() {}

template <int B>
static void launch_block_kernels(JobImpl &J, DevSys &s, int stage) {
  const auto &lst = J.blocks_by_size[B];
  if (lst.empty()) return;
  int nl = int(lst.size());
  const int *bl = J.blist[B].p;
  cudaStream_t st = J.ctx->stream;
  long Cp = s.Cpad;
  if (s.is_static) {
    if (stage == 0) k_static_eig<B><<<grid_for(Cp * nl), kThreads, 0, st>>>(s, bl, nl);
    else return;
    ++J.launches;
    return;
  }
  switch (stage) {
    case 0:
      if (s.step_method == 1 && s.mixed) k_step_taylor_df<B><<<grid_for(Cp * nl * s.n), kThreads, 0, st>>>(s, bl, nl);
      else if (s.step_method == 1) k_step_taylor<B><<<grid_for(Cp * nl * s.n), kThreads, 0, st>>>(s, bl, nl);
      else k_step_prop<B><<<grid_for(Cp * nl * s.n), kThreads, 0, st>>>(s, bl, nl);
      break;
    case 1:
      if (s.mixed) {
        constexpr int G = B <= 1 ? 1 : B <= 2 ? 2 : B <= 4 ? 4 : 8;
        k_dyson_df<B><<<grid_for(Cp * nl * s.nseg * B * G), kThreads, 0, st>>>(s, bl, nl, s.nseg, false);
        if (s.nseg > 1) k_dyson_df<B><<<grid_for(Cp * nl * B * G), kThreads, 0, st>>>(s, bl, nl, 1, true);
      } else {
        k_dyson<B><<<grid_for(Cp * nl * s.nseg * B), kThreads, 0, st>>>(s, bl, nl, s.nseg, false);
        if (s.nseg > 1) k_dyson<B><<<grid_for(Cp * nl * B), kThreads, 0, st>>>(s, bl, nl, 1, true);
      }
      if (s.nseg > 1) ++J.launches;
      break;
    case 2:
      if constexpr (B == 1) {
        k_floquet<B><<<grid_for(Cp * nl), kThreads, 0, st>>>(s, bl, nl);
      } else {  // B lanes per matrix, 32/B matrices per warp
        const long warps = (Cp * nl + (32 / B) - 1) / (32 / B);
        if (s.floq32) k_floquet_lanes<B, float><<<grid_for(warps * 32), kThreads, 0, st>>>(s, bl, nl);
        else k_floquet_lanes<B, double><<<grid_for(warps * 32), kThreads, 0, st>>>(s, bl, nl);
      }
      break;
    case 3:
      if (s.nseg > 1) {
        if (s.mixed) k_seg_frame<B, true><<<grid_for(Cp * nl * s.nseg), kThreads, 0, st>>>(s, bl, nl);
        else k_seg_frame<B, false><<<grid_for(Cp * nl * (s.nseg - 1)), kThreads, 0, st>>>(s, bl, nl);
        ++J.launches;
      }
      if (s.mixed) k_eigframe<B, float2><<<grid_for(Cp * nl * s.n), kThreads, 0, st>>>(s, bl, nl);
      else k_eigframe<B, double2><<<grid_for(Cp * nl * s.n), kThreads, 0, st>>>(s, bl, nl);
      break;
  }
  ++J.launches;
}

// Work enqueued on the auxiliary streams after fork() waits for everything before it on
// the context stream; join() makes the context stream wait for all of it.
static void fork(JobImpl &J) {
  if (J.aux.empty()) return;
  CUDA_OK(cudaEventRecord(J.fork_ev, J.ctx->stream));
  for (auto a : J.aux) CUDA_OK(cudaStreamWaitEvent(a, J.fork_ev, 0));
}
static void join(JobImpl &J) {
  for (size_t a = 0; a < J.aux.size(); ++a) {
    CUDA_OK(cudaEventRecord(J.join_ev[a], J.aux[a]));
    CUDA_OK(cudaStreamWaitEvent(J.ctx->stream, J.join_ev[a], 0));
  }
}
static cudaStream_t aux_stream(JobImpl &J, size_t idx) {
  return J.aux.empty() ? J.ctx->stream : J.aux[idx % J.aux.size()];
}


// ------------------------------------------------------------------ huge blocks (bl_huge.cuh)
// All on the context stream; every launch covers at most kHugeMaxItems items and the
// workspace holds one launch's items.
template <class T>
static HMat<T> item_mat(T *p, long off, long sstr, int ld, int Cpad) {
  return HMat<T>{p, off, sstr, long(ld), long(Cpad), 1};
}
template <class T>
static HMat<T> ws_mat(T *p, long j0, long mat, int C, int ld) {
  return HMat<T>{p, -j0 * mat, long(C) * mat, long(ld), 1, mat};
}
static unsigned tiles(int m, int n) { return unsigned(((m + kHT - 1) / kHT) * ((n + kHT - 1) / kHT)); }

// Products O = op(A) B of `items` items from j0 on: exact digit slices on the tensor cores
// (bl_xs.cuh) up to K' = 2k = 512 digits (its comment on exactness; the mixed form, which needs
// 2^-44, always) and the result's exponents stay within FP64 (the slices' joining has no denormals),
// else FP64 tiles.  |A| <= 2^ea, |B| <= 2^eb.
static void huge_mm(JobImpl &J, const DevSys &s, cudaStream_t st, bool conjA, HMat<const double2> A,
                    HMat<const double2> B, HMat<double2> O, int m, int n, int k, int Cb, long j0, int items, int ea,
                    int eb) {
  const unsigned tx = unsigned(((m + 63) / 64) * ((n + xs::kN - 1) / xs::kN));
  const XsReal none{};
  for (; items > 0; j0 += kHugeMaxItems, items -= kHugeMaxItems) {  // grid y is limited
    const unsigned gy = unsigned(std::min(items, kHugeMaxItems));
    if (s.mixed) {
      k_xs_gemm<true, 6, false, double2><<<dim3(tx, gy), xs::kThreadsXs, xs::smem<6>(), st>>>(
          A, B, O, m, n, k, Cb, j0, ea, eb, none, s.status);
    } else if (2 * k <= 512 && std::abs(ea + eb) <= 900) {
      if (conjA)
        k_xs_gemm<true, 7, true, double2><<<dim3(tx, gy), xs::kThreadsXs, xs::smem<7>(), st>>>(
            A, B, O, m, n, k, Cb, j0, ea, eb, none, s.status);
      else
        k_xs_gemm<true, 7, false, double2><<<dim3(tx, gy), xs::kThreadsXs, xs::smem<7>(), st>>>(
            A, B, O, m, n, k, Cb, j0, ea, eb, none, s.status);
    } else if (conjA) {
      k_huge_zgemm<double2, true, double2, double2, double2>
          <<<dim3(tiles(m, n), gy), kHThreads, 0, st>>>(A, B, O, m, n, k, Cb, j0, 1.0);
    } else {
      k_huge_zgemm<double2, false, double2, double2, double2>
          <<<dim3(tiles(m, n), gy), kHThreads, 0, st>>>(A, B, O, m, n, k, Cb, j0, 1.0);
    }
    ++J.launches;
  }
}

// U_i of huge block k for every (crystallite, step): symmetric Paterson-Stockmeyer.
static void huge_step(JobImpl &J, DevSys &s, size_t kh) {
  const int k = J.huge_blocks[kh], b = J.L.size[k], bp = J.L.poff[k];
  const long bb = long(b) * b, total = long(s.C) * J.n;
  const long per = std::min<long>(J.huge_items, long(J.huge_ws_bytes / (sizeof(double) * kHugeSlots * bb)));
  cudaStream_t st = J.ctx->stream;
  double *ws = reinterpret_cast<double *>(J.huge_ws.p);
  const unsigned ge = unsigned((bb + 255) / 256), tm = unsigned((b + kHT - 1) / kHT), gs = tm * (tm + 1) / 2;
  const unsigned gx = unsigned(((b + 127) / 128) * ((b + xs::kN - 1) / xs::kN));
  for (long j0 = 0; j0 < total; j0 += per) {
    const int items = int(std::min(per, total - j0));
    auto sym = [&](int a, int bsl, int o, double alpha, int round, bool low, double c0, double c1, double c2,
                   double c3) {
      if (s.mixed || b <= 512) {
        const long cs = kHugeSlots * bb;
        const HMat<const double> A{ws + a * bb, 0, 0, b, 1, cs}, B{ws + bsl * bb, 0, 0, b, 1, cs};
        const HMat<double> O{ws + o * bb, 0, 0, b, 1, cs};
        const XsReal ep{low ? 1 : 0, alpha, c0, c1, c2, c3, ws + bb, ws + 2 * bb, ws + 3 * bb,
                        round >= 0 ? J.hsq.p : nullptr, round};
        if (s.mixed)
          k_xs_gemm<false, 6, false, double><<<dim3(gx, unsigned(items)), xs::kThreadsXs, xs::smem<6>(), st>>>(
              A, B, O, b, b, b, 1 << 30, 0, 0, 0, ep, s.status);
        else
          k_xs_gemm<false, 7, false, double><<<dim3(gx, unsigned(items)), xs::kThreadsXs, xs::smem<7>(), st>>>(
              A, B, O, b, b, b, 1 << 30, 0, 0, 0, ep, s.status);
      } else {
        SymArgs g{ws, J.hsq.p, bb, b, a, bsl, o, alpha, round, low ? 1 : 0, c0, c1, c2, c3};
        k_huge_sym<<<dim3(gs, unsigned(items)), kHThreads, 0, st>>>(g);
      }
      ++J.launches;
    };
    const bool own_fk = !s.fk || s.fk_df;  // k_coef's coefficients are absent or split into floats
    if (own_fk) k_huge_fk<<<unsigned((items + 127) / 128), 128, 0, st>>>(s, j0, items, J.hfk.p);
    k_huge_hbuild<<<dim3(ge, unsigned(items)), 256, 0, st>>>(s, bp, b, own_fk ? J.hfk.p : nullptr, ws, j0);
    k_huge_norm<<<unsigned(items), 256, 0, st>>>(ws, b, s.tau * kPi2, J.hsq.p);
    J.launches += 3;
    sym(0, 0, 1, 1.0, -1, false, 0, 0, 0, 0);  // Y = X X
    sym(1, 1, 2, 1.0, -1, false, 0, 0, 0, 0);  // Y^2
    sym(2, 1, 3, 1.0, -1, false, 0, 0, 0, 0);  // Y^3
    sym(2, 2, 4, 1.0, -1, false, 0, 0, 0, 0);  // Y^4
    // cos X = C(Y), coefficients (-1)^j/(2j)!;  sin X = X S(Y), (-1)^j/(2j+1)!
    k_huge_low<<<dim3(ge, unsigned(items)), 256, 0, st>>>(ws, b, 1.0 / 40320, -1.0 / 3628800, 1.0 / 479001600,
                                                          -1.0 / 87178291200.0);
    sym(4, 5, 6, 1.0, -1, true, 1.0, -1.0 / 2, 1.0 / 24, -1.0 / 720);  // R = cos X
    k_huge_low<<<dim3(ge, unsigned(items)), 256, 0, st>>>(ws, b, 1.0 / 362880, -1.0 / 39916800,
                                                          1.0 / 6227020800.0, -1.0 / 1307674368000.0);
    sym(4, 5, 3, 1.0, -1, true, 1.0, -1.0 / 6, 1.0 / 120, -1.0 / 5040);  // S(Y) over Y^3
    sym(0, 3, 1, -1.0, -1, false, 0, 0, 0, 0);                           // I = -X S
    J.launches += 2;
    // squarings: the host bound for the block; each item skips the rounds it does not need
    for (int t = 0; t < J.huge_sq[kh]; ++t) {
      sym(6, 6, 2, 1.0, t, false, 0, 0, 0, 0);
      sym(1, 1, 4, 1.0, t, false, 0, 0, 0, 0);
      sym(6, 1, 5, 2.0, t, false, 0, 0, 0, 0);
      k_huge_sqcomb<<<dim3(ge, unsigned(items)), 256, 0, st>>>(ws, b, J.hsq.p, t);
      ++J.launches;
    }
    k_huge_store_u<<<dim3(ge, unsigned(items)), 256, 0, st>>>(s, ws, bp, J.L.off[k], b, j0);
    ++J.launches;
  }
}

// The segments' products P_i = U_i P_{i-1} of huge block k (step t of every segment in one
// launch), then the chain E_{s+1} = P_last(s) E_s; without segments the one chain of all steps.
static void huge_dyson(JobImpl &J, DevSys &s, size_t kh, cudaStream_t st) {
  const int k = J.huge_blocks[kh], b = J.L.size[k], bp = J.L.poff[k], n = J.n;
  const unsigned ge = unsigned((long(b) * b + 255) / 256);
  const int len = s.nseg > 1 ? kSegLen : n;
  const size_t step = size_t(s.S2) * s.Cpad;
  auto copy = [&](const double2 *src, double2 *dst, int src0, int dst0, int stride, int segs) {
    const long items = long(segs) * s.C;
    for (long g0 = 0; g0 < items; g0 += kHugeMaxItems) {
      k_huge_copy<<<dim3(ge, unsigned(std::min<long>(kHugeMaxItems, items - g0))), 256, 0, st>>>(s, src, dst, src0, dst0,
                                                                                              stride, bp, b, g0);
      ++J.launches;
    }
  };
  copy(s.U, s.A, 0, 0, len, s.nseg);
  for (int t = 1; t < len; ++t) {
    const int segs = (n - t + len - 1) / len;  // segments that have a step t
    const auto U = item_mat<const double2>(s.U + t * step, bp, long(len) * s.S2, b, s.Cpad);
    const auto Ain = item_mat<const double2>(s.A + (t - 1) * step, bp, long(len) * s.S2, b, s.Cpad);
    const auto Aout = item_mat<double2>(s.A + t * step, bp, long(len) * s.S2, b, s.Cpad);
    huge_mm(J, s, st, false, U, Ain, Aout, b, b, b, s.C, 0, segs * s.C, 0, 0);
  }
  if (s.nseg <= 1) return;
  copy(s.A, s.U, std::min(len, n) - 1, 0, 0, 1);
  for (int t = 1; t < s.nseg; ++t) {
    const auto P = item_mat<const double2>(s.A + (std::min((t + 1) * len, n) - 1) * step, bp, 0, b, s.Cpad);
    const auto Ein = item_mat<const double2>(s.U + (t - 1) * step, bp, 0, b, s.Cpad);
    const auto Eout = item_mat<double2>(s.U + t * step, bp, 0, b, s.Cpad);
    huge_mm(J, s, st, false, P, Ein, Eout, b, b, b, s.C, 0, s.C, 0, 0);
  }
}

// Floquet of all huge blocks: one launch per group of kMaxHugeLaunch blocks and chunk of
// crystallites, each (crystallite, block) with its own part of the workspace.
static void huge_floquet_all(JobImpl &J, DevSys &s) {
  const size_t nh = J.huge_blocks.size();
  for (size_t g0 = 0; g0 < nh; g0 += kMaxHugeLaunch) {
    HugeFloq hf{};
    hf.n = int(std::min<size_t>(kMaxHugeLaunch, nh - g0));
    hf.mats = s.floq32 ? 3 : 2;  // the mixed form's FP32 K takes half a third matrix
    size_t per_c = 0, smem = 0;
    for (int t = 0; t < hf.n; ++t) {
      const size_t b = size_t(J.L.size[J.huge_blocks[g0 + t]]);
      per_c += size_t(hf.mats) * b * b;
      smem = std::max(smem, huge_floquet_smem(int(b)));
    }
    const int per = int(std::min<size_t>(size_t(s.C), J.huge_ws_bytes / (sizeof(double2) * per_c)));
    if (per < 1) throw Error(3, "the huge-block workspace holds no crystallite's Floquet matrices");
    long off = 0;
    for (int t = 0; t < hf.n; ++t) {
      const long b = J.L.size[J.huge_blocks[g0 + t]];
      hf.k[t] = J.huge_blocks[g0 + t];
      hf.ws[t] = off;
      off += long(per) * hf.mats * b * b;
    }
    for (int c0 = 0; c0 < s.C; c0 += per) {
      k_huge_floquet<<<dim3(unsigned(std::min(per, s.C - c0)), unsigned(hf.n)), kHugeFloqThreads, smem,
                       J.ctx->stream>>>(s, hf, J.huge_ws.p, c0);
      ++J.launches;
    }
  }
}

// W_i = A_{i+1} V_F = P_i V_s for huge block k, segment by segment (V_s = E_s V_F first):
// straight into W in the mixed form; through the workspace and back over A in FP64 (a product
// may not overwrite its own operand).
static void huge_eigframe(JobImpl &J, DevSys &s, size_t kh) {
  const int k = J.huge_blocks[kh], b = J.L.size[k], bp = J.L.poff[k];
  const long bb = long(b) * b;
  cudaStream_t st = J.ctx->stream;
  const size_t step = size_t(s.S2) * s.Cpad;
  double2 *Vseg = s.U + size_t(2 * s.nseg) * step;  // V_s at step slot 2 nseg + s
  if (s.nseg > 1) {
    const auto E = item_mat<const double2>(s.U, bp, s.S2, b, s.Cpad);  // E_{sl+1}
    const auto V = item_mat<const double2>(s.VF, bp, 0, b, s.Cpad);
    const auto O = item_mat<double2>(Vseg + step, bp, s.S2, b, s.Cpad);
    huge_mm(J, s, st, false, E, V, O, b, b, b, s.C, 0, s.C * (s.nseg - 1), 0, 0);
  }
  const int len = s.nseg > 1 ? kSegLen : J.n;
  for (int seg = 0; seg < s.nseg; ++seg) {
    const int i0 = seg * len, i1 = std::min(J.n, i0 + len);
    const auto V = item_mat<const double2>(seg ? Vseg + seg * step : s.VF, bp, 0, b, s.Cpad);
    const auto A = item_mat<const double2>(s.A, bp, s.S2, b, s.Cpad);
    const long total = long(s.C) * i1;
    if (s.mixed) {
      const auto W = item_mat<float2>(s.Wf, bp, s.S2, b, s.Cpad);
      for (long j0 = long(s.C) * i0; j0 < total; j0 += kHugeMaxItems) {
        const int items = int(std::min<long>(kHugeMaxItems, total - j0));
        k_huge_zgemm<float2, false, double2, double2, float2>
            <<<dim3(tiles(b, b), unsigned(items)), kHThreads, 0, st>>>(A, V, W, b, b, b, s.C, j0, 1.0);
        ++J.launches;
      }
      continue;
    }
    const long per = std::min<long>(kHugeMaxItems, long(J.huge_ws_bytes / (sizeof(double2) * bb)));
    for (long j0 = long(s.C) * i0; j0 < total; j0 += per) {
      const int items = int(std::min(per, total - j0));
      const auto O = ws_mat<double2>(J.huge_ws.p, j0, bb, s.C, b);
      huge_mm(J, s, st, false, A, V, O, b, b, b, s.C, j0, items, 0, 0);
      k_huge_copy_back<<<dim3(unsigned((bb + 255) / 256), unsigned(items)), 256, 0, st>>>(s, J.huge_ws.p, bp, b, j0);
      ++J.launches;
    }
  }
}

// Q^{ab} (or R) = W_a^H (M_ab W_b) for a pair with a huge block, every (crystallite, step).
template <class C>
static void huge_qr(JobImpl &J, DevSys &s, const BigPair &P, C *Wbuf, C *out) {
  const int ba = J.L.size[P.a], bb = J.L.size[P.b], pa = J.L.poff[P.a];
  const long ne = long(ba) * bb, total = long(s.C) * J.n;
  const long per = std::min<long>(kHugeMaxItems, long(J.huge_ws_bytes / (sizeof(C) * ne)));
  cudaStream_t st = J.ctx->stream;
  C *ws = reinterpret_cast<C *>(J.huge_ws.p);
  const auto Wa = item_mat<const C>(Wbuf, pa, s.S2, ba, s.Cpad);
  const auto O = item_mat<C>(out, P.off, P.nitems, bb, s.Cpad);
  for (long j0 = 0; j0 < total; j0 += per) {
    const int items = int(std::min(per, total - j0));
    k_huge_mx<C><<<dim3(unsigned((ne + 255) / 256), unsigned(items)), 256, 0, st>>>(s, P, j0, ws);
    const auto X = ws_mat<const C>(ws, j0, ne, s.C, bb);
    ++J.launches;
    if constexpr (std::is_same<C, double2>::value) {
      huge_mm(J, s, st, true, Wa, X, O, ba, bb, ba, s.C, j0, items, 0, P.e2);
    } else {
      k_huge_zgemm<C, true, C, C, C><<<dim3(tiles(ba, bb), unsigned(items)), kHThreads, 0, st>>>(Wa, X, O, ba, bb, ba,
                                                                                               s.C, j0, 1.0);
      ++J.launches;
    }
  }
}

static void launch_stage(JobImpl &J, DevSys &s, int stage) {
  if (stage == 0 && s.fk) {  // the small blocks' term coefficients, before the streams fork
    if (J.phase.n) {
      // the series' few values per crystallite wait in A, which the Dyson stage writes later
      k_term_series<<<grid_for(long(s.Cpad) * s.nint), kThreads, 0, J.ctx->stream>>>(s, reinterpret_cast<double *>(s.A));
      k_coef_series<<<grid_for(long(s.Cpad) * s.nint * ((s.n + kCoefRun - 1) / kCoefRun)), kThreads, 0, J.ctx->stream>>>(
          s, reinterpret_cast<const double *>(s.A), J.phase.p, J.fkc.p);
      ++J.launches;
    } else {
      k_coef<<<grid_for(long(s.Cpad) * s.n), kThreads, 0, J.ctx->stream>>>(s, J.fkc.p);
    }
    ++J.launches;
  }
  if (J.side) fork(J);
  launch_block_kernels<1>(J, s, stage);
  launch_block_kernels<2>(J, s, stage);
  launch_block_kernels<3>(J, s, stage);
  launch_block_kernels<4>(J, s, stage);
  launch_block_kernels<5>(J, s, stage);
  launch_block_kernels<6>(J, s, stage);
  launch_block_kernels<7>(J, s, stage);
  launch_block_kernels<8>(J, s, stage);
  // blocks larger than kMaxBlock: one CTA per crystallite (per step for the exponential),
  // each block on its own auxiliary stream
  for (size_t kb = 0; kb < J.big_blocks.size(); ++kb) {
    const int k = J.big_blocks[kb];
    const int b = J.L.size[k];
    cudaStream_t st = aux_stream(J, kb);
    const size_t smat = sizeof(double2) * 2 * size_t(b) * b;
    const size_t sw = (s.mixed ? sizeof(float2) : sizeof(double2)) * 2 * size_t(b) * b;
    const unsigned th = big_threads(b, b), th_step = unsigned((big_sym_tiles(b) + 31) / 32 * 32);
    const bool nt1 = big_nt(b, b) == 1;
    switch (stage) {
      case 0:
        if (J.tc && b >= tc::kMinB) {
          k_tc_hamil<<<unsigned(s.Cpad / 32) * unsigned(s.n), 256, sizeof(float2) * 32 * size_t(s.nint), st>>>(
              s, k, J.hl_elem.p + J.hl_off[k], J.hl_n[k]);
          ++J.launches;
        }
        if (J.tc && b >= tc::kMinB && tc::up16(b) <= 64)  // the two Horner chains stacked in one M = 128 tile
          k_tc_step_stk<<<unsigned(s.C) * unsigned(s.n), tc::kTcThreads, tc_step_stk_smem(b), st>>>(
              s, k, J.hl_elem.p + J.hl_off[k], J.hl_n[k], J.usl.p + J.usl_off[k]);
        else if (J.tc && b >= tc::kMinB)
          k_tc_step<<<unsigned(s.C) * unsigned(s.n), tc::kTcThreads, tc_step_smem(b), st>>>(
              s, k, J.hl_elem.p + J.hl_off[k], J.hl_n[k], J.usl.p + J.usl_off[k]);
        else if (s.mixed) k_big_step_df<<<unsigned(s.C) * unsigned(s.n), th_step, big_step_df_smem(b), st>>>(s, k);
        else k_big_step<<<unsigned(s.C) * unsigned(s.n), th_step, big_step_smem(b), st>>>(s, k);
        break;
      case 1:
        if (J.tc && b >= tc::kMinB) {  // exact-slice BF16 products on the tensor cores
          if (tc::up16(b) <= 64)  // re and im stacked in one M = 128 tile
            k_tc_dyson_stk<<<unsigned(s.C), tc::kTcThreads, tc_dyson_stk_smem(b), st>>>(s, k, J.usl.p + J.usl_off[k]);
          else
            k_tc_dyson<<<unsigned(s.C), tc::kTcThreads, tc_dyson_smem(b), st>>>(s, k, J.usl.p + J.usl_off[k]);
        } else {
          for (int prefix = 0; prefix < (s.nseg > 1 ? 2 : 1); ++prefix) {
            const unsigned grid = unsigned(s.C) * unsigned(prefix ? 1 : s.nseg);
            if (s.mixed) {
              if (nt1) k_big_dyson_df<1><<<grid, th, smat, st>>>(s, k, prefix != 0);
              else k_big_dyson_df<2><<<grid, th, smat, st>>>(s, k, prefix != 0);
            } else {
              if (nt1) k_big_dyson<1><<<grid, th, smat, st>>>(s, k, prefix != 0);
              else k_big_dyson<2><<<grid, th, smat, st>>>(s, k, prefix != 0);
            }
            J.launches += prefix;
          }
        }
        break;
      case 2:  // the mixed form's single-precision K follows the two b x b double2 arrays
        if (s.floq32 && b >= FloqDf::kStartMin)
          k_big_floquet<true, true, true><<<unsigned(s.C), floquet_threads(b), smat + sizeof(float2) * size_t(b) * b, st>>>(s, k);
        else if (s.floq32)
          k_big_floquet<true, true, false><<<unsigned(s.C), 256, smat + sizeof(float2) * size_t(b) * b, st>>>(s, k);
        else if (s.mixed && b >= FloqF64::kStartMin)
          k_big_floquet<false, true, true><<<unsigned(s.C), floquet_threads(b), smat, st>>>(s, k);
        else if (s.mixed)
          k_big_floquet<false, true, false><<<unsigned(s.C), 256, smat, st>>>(s, k);
        else if (b >= FloqF64::kStartMin)
          k_big_floquet<false, false, true><<<unsigned(s.C), floquet_threads(b), smat, st>>>(s, k);
        else
          k_big_floquet<false, false, false><<<unsigned(s.C), 256, smat, st>>>(s, k);
        break;
      case 3:
        if (b <= s.seg_max) {
          if (s.mixed) k_big_seg_frame<true><<<unsigned(s.C) * unsigned(s.nseg), th, smat, st>>>(s, k);
          else k_big_seg_frame<false><<<unsigned(s.C) * unsigned(s.nseg - 1), th, smat, st>>>(s, k);
          ++J.launches;
        }
        if (s.mixed) {
          k_big_eigframe4<<<unsigned(s.C) * unsigned(s.nseg), unsigned(big4_threads(b, b)), big_eigframe4_smem(b), st>>>(s, k);
        } else {
          if (nt1) k_big_eigframe<1, double2><<<unsigned(s.C) * unsigned(s.nseg), th, sw, st>>>(s, k);
          else k_big_eigframe<2, double2><<<unsigned(s.C) * unsigned(s.nseg), th, sw, st>>>(s, k);
        }
        break;
    }
    ++J.launches;
  }
  // blocks larger than kMaxBigBlock: batched products on the context stream, alongside the
  // large blocks on the auxiliary streams
  for (size_t kh = 0; kh < J.huge_blocks.size(); ++kh) {
    switch (stage) {
      case 0:
        if (J.xs_from <= kMaxBigBlock) {  // one fused kernel keeps its seven matrices in shared memory
          const int k = J.huge_blocks[kh], b = J.L.size[k];
          k_big_step<<<unsigned(s.C) * unsigned(s.n), unsigned((big_sym_tiles(b) + 31) / 32 * 32), big_step_smem(b),
                       aux_stream(J, J.big_blocks.size() + kh)>>>(s, k);
          ++J.launches;
        } else {
          huge_step(J, s, kh);
        }
        break;
      case 1:  // (no workspace: the blocks run side by side)
        huge_dyson(J, s, kh, J.xs_from <= kMaxBigBlock ? aux_stream(J, J.big_blocks.size() + kh) : J.ctx->stream);
        break;
      case 2:
        if (J.xs_from <= kMaxBigBlock) {  // fits shared memory
          const int k = J.huge_blocks[kh], b = J.L.size[k];
          k_big_floquet<false, false, true><<<unsigned(s.C), floquet_threads(b), sizeof(double2) * 2 * size_t(b) * b,
                                             aux_stream(J, J.big_blocks.size() + kh)>>>(s, k);
          ++J.launches;
        } else if (kh == 0) {
          huge_floquet_all(J, s);
        }
        break;
      case 3: huge_eigframe(J, s, kh); break;
    }
  }
  if (J.side) join(J);
}

static void mark_begin(JobImpl &J, int stage);
static void mark_end(JobImpl &J, int stage, int nlaunch);

// k_fid_pair with the (m, p) tile that needs the fewest FP64 operations over the padded range.
template <int JT, int PT>
static void launch_fid_tile(const DevSys &s, long groups, int W, cudaStream_t st) {
  const long tiles = groups * ((pair_rows(s.J) + JT - 1) / JT) * ((s.gper + PT - 1) / PT);
  const int warps = std::max(4, W), per = warps / W;
  constexpr int V = (4 * JT * PT + 31) / 32 * 32;
  k_fid_pair<JT, PT><<<unsigned((tiles + per - 1) / per), 32 * warps, sizeof(double) * V * warps, st>>>(s, W);
}
static void launch_fid(const DevSys &s, long Cp, cudaStream_t st) {
  // warps per tile: about 8 elements each, at most 8 (a function of the element count alone)
  const int W = s.ne < 16 ? 1 : s.ne < 32 ? 2 : s.ne < 256 ? 4 : 8;
  static const int shape[][2] = {{8, 2}, {7, 2}, {6, 2}, {5, 3}, {4, 4}, {3, 5}, {2, 8}, {1, 8}};
  int best = 0;
  double cost = 1e300;
  for (int t = 0; t < 8; ++t) {
    const int JT = shape[t][0], PT = shape[t][1];
    const double n = double((pair_rows(s.J) + JT - 1) / JT) * double((s.gper + PT - 1) / PT);
    const double x = n * ((4.0 * JT * PT + 4.0 * PT + 2.0) * (double(s.ne) / W + 1.0) + 4.0 * JT * PT);
    if (x < cost) cost = x, best = t;
  }
  const long groups = Cp / 32;
  switch (best) {
    case 0: launch_fid_tile<8, 2>(s, groups, W, st); break;
    case 1: launch_fid_tile<7, 2>(s, groups, W, st); break;
    case 2: launch_fid_tile<6, 2>(s, groups, W, st); break;
    case 3: launch_fid_tile<5, 3>(s, groups, W, st); break;
    case 4: launch_fid_tile<4, 4>(s, groups, W, st); break;
    case 5: launch_fid_tile<3, 5>(s, groups, W, st); break;
    case 6: launch_fid_tile<2, 8>(s, groups, W, st); break;
    default: launch_fid_tile<1, 8>(s, groups, W, st); break;
  }
}

template <int CG>
static void launch_fave(const DevSys &s, unsigned grid, size_t smem, cudaStream_t st) {
  if (s.mixed) {
    if (s.fftq == 1) k_fave_fft<CG, float2, true><<<grid, 128, smem, st>>>(s);
    else k_fave_fft<CG, float2, false><<<grid, 128, smem, st>>>(s);
  } else {
    if (s.fftq == 1) k_fave_fft<CG, double2, true><<<grid, 128, smem, st>>>(s);
    else k_fave_fft<CG, double2, false><<<grid, 128, smem, st>>>(s);
  }
}

void Job::run() {
  JobImpl &J = *d_;
  CUDA_OK(cudaSetDevice(J.ctx->device));
  cudaStream_t st = J.ctx->stream;
  J.launches = 0;
  J.marks.clear();
  J.evnext = 0;
  if (J.profiling && J.evpool.empty()) {
    J.evpool.resize(size_t(2) * Job::kStages * (J.nbatch + 1));
    for (auto &e : J.evpool) CUDA_OK(cudaEventCreate(&e));
  }
  CUDA_OK(cudaMemsetAsync(J.status.p, 0, 2 * sizeof(double2), st));  // the status word and the tensor-flop counters
  for (int bi = 0; bi < J.nbatch; ++bi) {
    DevSys s = J.base;
    int c0 = bi * J.Cb;
    s.C = std::min(J.Cb, J.Ceff - c0);
    s.Cpad = J.Cb;
    s.Rp = J.Rp_all.p + size_t(bi) * 9 * J.Cb;
    s.t0 = J.t0_all.p + size_t(bi) * J.Cb;
    s.w = J.w_all.p + size_t(bi) * J.Cb;
    s.warp_base = c0 / 32;
    for (int stage = 0; stage < 4; ++stage) {
      mark_begin(J, stage);
      int before = J.launches;
      launch_stage(J, s, stage);
      mark_end(J, stage, J.launches - before);
    }
    long Cp = s.Cpad;
    mark_begin(J, 4);
    const int qr_before = J.launches;
    if (!J.is_static && J.npq + J.npr > 0) {
      if (!J.big_pairs.empty()) fork(J);
      if (s.mixed) k_qr<float2><<<grid_for(Cp * (J.npq + J.npr) * J.n), kThreads, 0, st>>>(s);
      else k_qr<double2><<<grid_for(Cp * (J.npq + J.npr) * J.n), kThreads, 0, st>>>(s);
      ++J.launches;
      for (size_t t = 0; t < J.big_pairs.size(); ++t) {
        const BigPair &P = J.big_pairs[t];
        cudaStream_t st = aux_stream(J, t);
        const int ba = J.L.size[P.a], bb = J.L.size[P.b];
        const unsigned grid = unsigned(s.C) * unsigned(J.n), th = big_threads(ba, P.wchunk);
        const bool nt1 = big_nt(ba, P.wchunk) == 1;
        if (s.mixed) {
          if (ba >= kQr4Min)
            k_big_qr4<<<grid, unsigned(big4_threads(ba, P.wchunk)), big_qr4_smem(ba, bb, P.wchunk), st>>>(s, P);
          else  // at most 20 x 37 tiles
            k_big_qr<1, float2><<<grid, th, big_qr_smem<float2>(ba, bb, P.wchunk), st>>>(s, P);
        } else {
          const size_t sm = big_qr_smem<double2>(ba, bb, P.wchunk);
          if (nt1) k_big_qr<1, double2><<<grid, th, sm, st>>>(s, P);
          else k_big_qr<2, double2><<<grid, th, sm, st>>>(s, P);
        }
        ++J.launches;
      }
      for (const BigPair &P : J.huge_pairs) {
        if (s.mixed) huge_qr<float2>(J, s, P, s.Wf, P.isq ? s.Qf : s.Rf);
        else huge_qr<double2>(J, s, P, s.A, P.isq ? s.Q : s.R);
      }
      if (!J.big_pairs.empty()) join(J);
    }
    mark_end(J, 4, J.launches - qr_before);
    mark_begin(J, 5);
    if (J.is_static && J.ne > 0) {
      k_static_elems<<<grid_for(Cp * J.ne * ((J.n + kStaticRun - 1) / kStaticRun + 1)), kThreads, 0, st>>>(s);
      ++J.launches;
    } else if (J.p2p && J.ne > 0) {
      if (s.mixed) k_p2p_elems<float2><<<grid_for(Cp * J.ne), kThreads, 0, st>>>(s);
      else k_p2p_elems<double2><<<grid_for(Cp * J.ne), kThreads, 0, st>>>(s);
      ++J.launches;
    } else if (J.ne > 0) {
      if (s.fave_method == 1) {
        int cg = s.M <= 256 ? 8 : s.M <= 512 ? 4 : s.M <= 1024 ? 2 : 1;
        const size_t shm = sizeof(double2) * size_t(s.M) * cg * 2 + fave_twist_bytes(s, cg);
        const size_t shmf = sizeof(float2) * size_t(s.M) * cg * 2 + fave_twist_bytes(s, cg);
        unsigned grid = unsigned(J.ne) * unsigned(Cp / cg);
        switch (cg) {
          case 8: launch_fave<8>(s, grid, s.mixed ? shmf : shm, st); break;
          case 4: launch_fave<4>(s, grid, s.mixed ? shmf : shm, st); break;
          case 2: launch_fave<2>(s, grid, s.mixed ? shmf : shm, st); break;
          default: launch_fave<1>(s, grid, s.mixed ? shmf : shm, st); break;
        }
      } else {
        int ntile = (J.n + kFavePT - 1) / kFavePT;
        k_fave<<<grid_for(Cp * J.ne * ntile), kThreads, 0, st>>>(s);
      }
      ++J.launches;
    }
    mark_end(J, 5, J.ne > 0 ? 1 : 0);
    // every (row, k) of this batch is written, so partials need no clearing
    mark_begin(J, 6);
    if (s.mixed) {
      const unsigned npr = unsigned((s.gper + 4 * s.ft_pt - 1) / (4 * s.ft_pt));
      const unsigned njr = unsigned((J.J + 4 * s.ft_jt - 1) / (4 * s.ft_jt));
      k_fid_tiled<<<dim3(unsigned(Cp / 32), npr * njr, unsigned(s.ft_r)), kFtThreads * unsigned(s.ft_sub),
                    fid_tiled_smem(s.ft_jt, s.ft_pt), st>>>(s);
    } else {
      launch_fid(s, Cp, st);
    }
    ++J.launches;
    mark_end(J, 6, 1);
  }
  mark_begin(J, 7);
  // only warps that hold crystallites: the sum is then independent of the batch size
  k_reduce<<<(J.P.npts + 31) / 32, 32 * kRedGroups, 0, st>>>(J.partial.p, (J.Ceff + 31) / 32 * (J.mixed ? J.ft_r : 1),
                                                    J.P.npts, J.fid.p);
  ++J.launches;
  mark_end(J, 7, 1);
  CUDA_OK(cudaGetLastError());
  if (J.profiling && !J.marks.empty()) {
    CUDA_OK(cudaEventSynchronize(J.evpool[J.marks.back().e]));
    for (const auto &m : J.marks) {
      float ms = 0;
      CUDA_OK(cudaEventElapsedTime(&ms, J.evpool[m.b], J.evpool[m.e]));
      J.stage_ms[m.stage] += ms;
      J.stage_launch[m.stage] += m.nlaunch;
    }
  }
}

// Stage markers: with profiling on, an event pair on the launching stream brackets each
// stage; run() folds the elapsed times into the per-stage totals once its last event
// has completed (one synchronisation per run, none between stages).
static void mark_begin(JobImpl &J, int stage) {
  if (!J.profiling) return;
  CUDA_OK(cudaEventRecord(J.evpool[J.evnext], J.ctx->stream));
  J.marks.push_back({stage, J.evnext, -1, 0});
  ++J.evnext;
}

static void mark_end(JobImpl &J, int stage, int nlaunch) {
  if (!J.profiling) return;
  CUDA_OK(cudaEventRecord(J.evpool[J.evnext], J.ctx->stream));
  J.marks.back().e = J.evnext;
  J.marks.back().nlaunch = nlaunch;
  (void)stage;
  ++J.evnext;
}

void Job::read(double *fid_out) {
  JobImpl &J = *d_;
  std::vector<double2> host(size_t(J.P.npts) + 1);  // the FID and the status word behind it
  CUDA_OK(cudaMemcpyAsync(host.data(), J.fid.p, sizeof(double2) * host.size(), cudaMemcpyDeviceToHost, J.ctx->stream));
  CUDA_OK(cudaStreamSynchronize(J.ctx->stream));
  std::memcpy(fid_out, host.data(), sizeof(double2) * J.P.npts);
  int status = 0;
  std::memcpy(&status, host.data() + J.P.npts, sizeof(int));
  if (status & (kNoConvergeStep | kNoConvergeFloquet))
    throw Error(7, "an eigen-decomposition did not converge within its sweep limit");
  if (status & kSingularCayley) throw Error(7, "singular Cayley transform in the Floquet eigen-decomposition");
  if (status & kTcTimeout) throw Error(7, "a tensor-core product did not complete within its wait limit");
}

const char *Job::stage_name(int s) {
  static const char *names[kStages] = {"k_step_prop", "k_dyson",  "k_floquet", "k_eigframe",
                                       "k_qr",        "k_fave",   "k_fid",     "k_reduce"};
  return (s >= 0 && s < kStages) ? names[s] : "";
}
void Job::set_profiling(bool on) { d_->profiling = on; }
void Job::stage_times(double *ms, int *launches) const {
  for (int i = 0; i < kStages; ++i) {
    if (ms) ms[i] = d_->stage_ms[i];
    if (launches) launches[i] = d_->stage_launch[i];
  }
}
void Job::stage_flops(double *f) const {
  for (int i = 0; i < kStages; ++i) f[i] = d_->stage_fl[i];
}
void Job::reset_stage_times() {
  for (int i = 0; i < kStages; ++i) d_->stage_ms[i] = 0, d_->stage_launch[i] = 0;
}
size_t Job::h2d_bytes() const { return d_->h2d; }
size_t Job::d2h_bytes() const { return sizeof(double2) * d_->P.npts; }
double Job::run_timed(int iters) {
  JobImpl &J = *d_;
  cudaEvent_t a, b;
  CUDA_OK(cudaEventCreate(&a));
  CUDA_OK(cudaEventCreate(&b));
  CUDA_OK(cudaEventRecord(a, J.ctx->stream));
  for (int i = 0; i < iters; ++i) run();
  CUDA_OK(cudaEventRecord(b, J.ctx->stream));
  CUDA_OK(cudaEventSynchronize(b));
  float ms = 0;
  CUDA_OK(cudaEventElapsedTime(&ms, a, b));
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  return ms;
}

namespace {
// 8 independent DFMA chains per thread; 2*8*iters flop per thread.
__global__ void k_dfma_probe(double *out, int iters, double a, double b) {
  double x[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) x[c] = threadIdx.x + c;
  for (int it = 0; it < iters; ++it)
#pragma unroll
    for (int c = 0; c < 8; ++c) x[c] = fma(x[c], a, b);
  double s = 0;
#pragma unroll
  for (int c = 0; c < 8; ++c) s += x[c];
  out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}
// The same with FP32 FMA chains: the FP32 pipe that the mixed form's double-float stages use.
__global__ void k_ffma_probe(float *out, int iters, float a, float b) {
  float x[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) x[c] = threadIdx.x + c;
  for (int it = 0; it < iters; ++it)
#pragma unroll
    for (int c = 0; c < 8; ++c) x[c] = fmaf(x[c], a, b);
  float s = 0;
#pragma unroll
  for (int c = 0; c < 8; ++c) s += x[c];
  out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}
}  // namespace

double error_statement(Context &ctx, const SpinSystem &sys, const Powder &pw, const CMatrix &ro, const CMatrix &det,
                       const FidParams &p, int sample) {
  const int C = pw.size();
  const int m = std::min(std::max(sample, 1), C);
  Powder sub;
  for (int k = 0; k < m; ++k) {
    const int c = int((2L * k + 1) * C / (2L * m));
    sub.theta.push_back(pw.theta[c]), sub.phi.push_back(pw.phi[c]), sub.gamma.push_back(pw.gamma[c]);
    sub.weight.push_back(pw.weight[c]);
  }
  FidParams p1 = p, p0 = p;
  p1.precision = 1, p0.precision = 0;
  p1.error_sample = p0.error_sample = 0;
  std::vector<double> f1(2 * size_t(p.npts)), f0(2 * size_t(p.npts));
  {
    Job j(ctx, sys, sub, ro, det, p1);
    j.run();
    j.read(f1.data());
  }
  {
    Job j(ctx, sys, sub, ro, det, p0);
    j.run();
    j.read(f0.data());
  }
  double num = 0, den = 0;
  for (size_t x = 0; x < f0.size(); ++x) num += (f1[x] - f0[x]) * (f1[x] - f0[x]), den += f0[x] * f0[x];
  return den > 0 ? std::sqrt(num / den) : 0.0;
}

double probe_fp32_tflops(Context &ctx) {
  CUDA_OK(cudaSetDevice(ctx.device));
  int sms = 0;
  CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx.device));
  int blocks = sms * 8, threads = 256, iters = 40000;
  DevBuf<float> out;
  out.alloc(size_t(blocks) * threads);
  cudaEvent_t a, b;
  CUDA_OK(cudaEventCreate(&a));
  CUDA_OK(cudaEventCreate(&b));
  k_ffma_probe<<<blocks, threads, 0, ctx.stream>>>(out.p, 10, 0.999f, 0.001f);
  double best = 0;
  for (int rep = 0; rep < 3; ++rep) {
    CUDA_OK(cudaEventRecord(a, ctx.stream));
    k_ffma_probe<<<blocks, threads, 0, ctx.stream>>>(out.p, iters, 0.999f, 0.001f);
    CUDA_OK(cudaEventRecord(b, ctx.stream));
    CUDA_OK(cudaEventSynchronize(b));
    float ms = 0;
    CUDA_OK(cudaEventElapsedTime(&ms, a, b));
    best = std::max(best, 2.0 * 8 * double(iters) * blocks * threads / (ms * 1e-3) / 1e12);
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  return best;
}

double probe_fp64_tflops(Context &ctx) {
  CUDA_OK(cudaSetDevice(ctx.device));
  int sms = 0;
  CUDA_OK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx.device));
  int blocks = sms * 4, threads = 256, iters = 4000;
  DevBuf<double> out;
  out.alloc(size_t(blocks) * threads);
  cudaEvent_t a, b;
  CUDA_OK(cudaEventCreate(&a));
  CUDA_OK(cudaEventCreate(&b));
  k_dfma_probe<<<blocks, threads, 0, ctx.stream>>>(out.p, 10, 0.999, 0.001);
  double best = 0;
  for (int rep = 0; rep < 3; ++rep) {
    CUDA_OK(cudaEventRecord(a, ctx.stream));
    k_dfma_probe<<<blocks, threads, 0, ctx.stream>>>(out.p, iters, 0.999, 0.001);
    CUDA_OK(cudaEventRecord(b, ctx.stream));
    CUDA_OK(cudaEventSynchronize(b));
    float ms = 0;
    CUDA_OK(cudaEventElapsedTime(&ms, a, b));
    best = std::max(best, 2.0 * 8 * double(iters) * blocks * threads / (ms * 1e-3) / 1e12);
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  return best;
}

double Job::sw_out() const { return d_->sw_out; }
int Job::npts() const { return d_->P.npts; }
int Job::kernels_per_run() const { return d_->launches; }
const double *Job::device_fid() const { return reinterpret_cast<const double *>(d_->fid.p); }
double Job::flops() const { return d_->flops; }
void Job::tensor_flops(double *step, double *dyson) const {
  unsigned long long v[2] = {0, 0};
  CUDA_OK(cudaMemcpyAsync(v, d_->tcf.p, sizeof(v), cudaMemcpyDeviceToHost, d_->ctx->stream));
  CUDA_OK(cudaStreamSynchronize(d_->ctx->stream));
  if (step) *step = double(v[0]);
  if (dyson) *dyson = double(v[1]);
}

std::string Job::describe() const {
  const JobImpl &J = *d_;
  std::ostringstream o;
  o << "{\"N\": " << J.L.N << ", \"blocks\": [";
  for (size_t k = 0; k < J.L.size.size(); ++k) o << (k ? ", " : "") << J.L.size[k];
  o << "], \"S2\": " << J.L.S2 << ", \"n\": " << J.n << ", \"gammaloop\": " << J.gammaloop
    << ", \"crystallites\": " << J.C << ", \"rosym\": " << J.rosym << ", \"q_pairs\": " << J.npq
    << ", \"r_pairs\": " << J.npr << ", \"elements\": " << J.ne << ", \"batch\": " << J.Cb
    << ", \"batches\": " << J.nbatch << ", \"flops\": " << J.flops << "}";
  return o.str();
}

// ------------------------------------------------------------------ allocation-free entry
// Some callers may not allocate device memory at all: a host program that reserves the
// GPU's memory for itself up front and forbids other allocators, or a timing-critical loop
// in which cudaMalloc/cudaFree (which synchronise the device) are not allowed.  For them
// powder_fid_noalloc runs the same pipeline with every device buffer (inputs, tables, work
// buffers, warp partials, FID, status word) carved from one static device array of
// kNoAllocScratch bytes; larger jobs are processed in crystallite batches that fit it, and
// a job whose smallest batch does not fit is rejected with BL_ERR_NOMEM.  Every GPU that
// loads this library holds the array until the process exits.  All calls share it and it
// keeps the previous call's contents: each call zeroes what must start at zero (the status word,
// the counters, scattered operator tables) and writes every warp partial that it sums, and calls
// that overlap on the GPU race on it.
namespace {
constexpr size_t kNoAllocScratch = size_t(64) << 20;
__device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratch];
}  // namespace

size_t noalloc_scratch_bytes() { return kNoAllocScratch; }

// Device address of the static array in the current device's context.  Host code may not
// use the symbol itself as a device pointer, so every call asks the runtime (a host-side
// lookup that allocates nothing); an address kept from an earlier call would dangle once the
// host program resets the device or its primary context is rebuilt.  The first lookup on a
// device loads this library's device code, and with it the array, so the first call should
// come before any stream capture and before the host program claims the device's memory.
static char *noalloc_base() {
  void *ptr = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
  if (e != cudaSuccess || !ptr) throw Error(3, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
  return static_cast<char *>(ptr);
}

void job_bytes(int device, const SpinSystem &sys, const Powder &pw, const CMatrix &ro, const CMatrix &det,
               const FidParams &p, size_t *min_bytes, size_t *full_bytes) {
  Context ctx;
  ctx.device = device;
  JobSizing plan;
  struct Scope {
    JobSizing *prev;
    explicit Scope(JobSizing *z) : prev(g_sizing) { g_sizing = z; }
    ~Scope() { g_sizing = prev; }
  } scope(&plan);
  Job job(ctx, sys, pw, ro, det, p);
  planned_bytes(plan, pw, p, min_bytes, full_bytes);
}

void powder_fid_noalloc(Context &ctx, const SpinSystem &sys, const Powder &pw, const CMatrix &ro, const CMatrix &det,
                        const FidParams &p, double *fid_out, double *sw_out) {
  CUDA_OK(cudaSetDevice(ctx.device));
  // the host-side plan (no device memory is touched): the batch-independent bytes as the
  // arena will carve them, and the bytes each crystallite of a batch adds
  JobSizing plan;
  {
    struct Scope {
      JobSizing *prev;
      explicit Scope(JobSizing *z) : prev(g_sizing) { g_sizing = z; }
      ~Scope() { g_sizing = prev; }
    } scope(&plan);
    Context probe;
    probe.device = ctx.device;
    Job sizing(probe, sys, pw, ro, det, p);
  }
  // work buffers are carved with 256-byte alignment: allow for it on each of ~40 buffers
  const size_t fixed = fixed_bytes(pw, p) + 40 * 256 + plan.extra + plan.tables;
  const size_t smallest = fixed + plan.per_c * 32;  // with one 32-crystallite batch
  if (smallest > kNoAllocScratch)
    throw Error(4, "job needs " + std::to_string((smallest + (size_t(1) << 20) - 1) >> 20) +
                       " MiB for its smallest batch, more than the " + std::to_string(kNoAllocScratch >> 20) +
                       " MiB static device scratch of the allocation-free entry point");
  ScratchArena arena;
  arena.base = noalloc_base();
  arena.cap = kNoAllocScratch;
  Context view;  // same device and stream; budget = what the scratch leaves for work buffers
  ready_kernels(ctx);
  view.device = ctx.device;
  view.stream = ctx.stream;
  view.kernels_ready = true;
  view.hbm_budget = kNoAllocScratch - (fixed - plan.extra);  // the Job sets the workspace (extra) aside itself
  struct Release {
    Context &c;
    ~Release() { c.stream = nullptr; }  // the stream belongs to the caller's context
  } release{view};
  struct Scope {
    ScratchArena *prev;
    explicit Scope(ScratchArena *a) : prev(g_arena) { g_arena = a; }
    ~Scope() { g_arena = prev; }
  } scope(&arena);
  try {
    Job job(view, sys, pw, ro, det, p);
    job.run();
    job.read(fid_out);
    if (sw_out) *sw_out = job.sw_out();
  } catch (const Error &e) {
    if (e.code == 4 && std::string(e.what()).find("static device scratch") == std::string::npos)
      throw Error(4, std::string("job does not fit the ") + std::to_string(kNoAllocScratch >> 20) +
                         " MiB static device scratch of the allocation-free entry point: " + e.what());
    throw;
  }
}

std::unique_ptr<Job> job_in_asked_region(Context &ctx, const RegionFn &region, const SpinSystem &sys, const Powder &pw,
                                         const CMatrix &ro, const CMatrix &det, const FidParams &p) {
  CUDA_OK(cudaSetDevice(ctx.device));
  struct Scope {
    const RegionFn *prev;
    explicit Scope(const RegionFn *r) : prev(g_region) { g_region = r; }
    ~Scope() { g_region = prev; }
  } scope(&region);
  return std::unique_ptr<Job>(new Job(ctx, sys, pw, ro, det, p));
}

// A resident Job whose every device buffer lives in [base, base + bytes): the serving loop
// gives each slot such a region, so admitting a request allocates nothing.  The caller's
// Context (device, stream) must outlive the Job; its hbm_budget is set here.
std::unique_ptr<Job> job_in_region(Context &ctx, void *base, size_t bytes, const SpinSystem &sys, const Powder &pw,
                                   const CMatrix &ro, const CMatrix &det, const FidParams &p) {
  CUDA_OK(cudaSetDevice(ctx.device));
  ScratchArena arena;
  arena.base = static_cast<char *>(base);
  arena.cap = bytes;
  arena.label = "device region given to the job";
  arena.aux_streams = true;
  size_t fixed = fixed_bytes(pw, p);
  if (fixed >= bytes) throw Error(4, "job does not fit a device region of " + std::to_string(bytes >> 20) + " MiB");
  ctx.hbm_budget = bytes - fixed;
  struct Scope {
    ScratchArena *prev;
    explicit Scope(ScratchArena *a) : prev(g_arena) { g_arena = a; }
    ~Scope() { g_arena = prev; }
  } scope(&arena);
  return std::unique_ptr<Job>(new Job(ctx, sys, pw, ro, det, p));
}

}  // namespace bl
