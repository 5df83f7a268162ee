// Batched exact-slice products on the tensor cores for matrices that live in HBM, included by
// bl_engine.cu after bl_huge.cuh and bl_tc.cuh: O = A B for FP64 operands, real or complex, of
// any size, one 128-row output tile per CTA.
//
// An operand (|x| <= 2^e, e given per operand) becomes a fixed-point integer x 2^(8S-1-e),
// written as S balanced base-256 digits q_j (exact in BF16), and the product takes the digit
// pairs with i + j <= top level into one FP32 accumulator per level in tensor memory; the epilogue
// joins the levels in 64-bit integers and rounds once to FP64, without touching the FP64 pipe.
// A level's sums are integers, accumulated exactly below 2^24.  Norms (rows and columns of length
// ~1) bound the leading digit only; the others reach 128, so exactness is certain where (l - 1) K'
// <= 992 at level l: every level up to K' = 165 digits, levels 0 to 4 at 252 (blocks of 126).
// Digits beyond the first are close to uniform and of either sign: on propagators of 9 and 10 spins
// (K' = 252 and 504) the largest sum was 0.05 and 0.08 of 2^24, which the dispatch's limit of K' <=
// 512 rests on.  With all entries of both operands equal, K' = 504, it reaches 1.5 from level 4 on; a
// sum in [2^24, 2^25) is rounded to 2 units, of 2^-46 at level 4.
//   S = 7 (FP64 form): levels 0..7, the last two in one accumulator (rounded at 2^-24 of its sum,
//     2^-68): 34 pairs, operand rounding 2^-56 and dropped levels below 2^-60 for |O| ~ 1.  9 spins,
//     one crystallite, n = 24: 1.0e-15 from 80-bit propagation, 1.4e-15 with FP64 step products;
//   S = 6 (mixed form): levels 0..5, 21 pairs, dropped levels ~2^-44, the size of the compensated
//     double-float sums they take the place of.
// Why: GB300 issues 2 FP64 FMAs per clock and SM (a 126 x 126 complex product: 3.9 M clocks on
// one SM; ~0.9 M in double-float on the FP32 pipe), while the 34 BF16 products of a 64 x 64 x 16
// complex chunk take ~2200 clocks of the tensor pipe and the digit conversions of its operands
// about 1100 of the integer and FP32 pipes, which run beside it.
//
// Complex operands are interleaved in place: complex row r is rows 2r (re) and 2r+1 (im) of the
// M = 128 tile, complex k is K entries 2k, 2k+1: A(r, l) = a + ib fills [[a, -b], [b, a]] and
// B(l, n) = c + id the pair (c, d), so one real product per tile gives re and im in adjacent
// tensor-memory lanes, and four complex elements are one 16-byte core-matrix row.
// Pipeline: 31 warps convert K chunks of 32 entries into two shared-memory buffers (K-major, no
// swizzle, 8-row groups padded by 16 bytes), one warp issues the products of a full buffer;
// every wait is bounded (tc::wait_parity).
namespace xs {

constexpr int kConv = 992;           // converting threads (31 warps), then the issuing warp: 32
constexpr int kThreadsXs = kConv + 32;  // resident warps hide the integer chains' latency
                                        // (with 544 threads the issue slots were 43 % busy)
constexpr int kN = 64;               // output columns per tile
constexpr int kK = 32;               // K entries (16 complex) per chunk
constexpr int kGroup = kK * 16 + 16; // bytes of an 8-row group (tc::sbo_bytes(kK))
constexpr int kPlaneA = 16 * kGroup, kPlaneB = 8 * kGroup;
template <int S>
__host__ __device__ constexpr int buf_bytes() { return S * (kPlaneA + kPlaneB); }
template <int S>
__host__ __device__ constexpr size_t smem() { return 2 * size_t(buf_bytes<S>()) + 1024; }
// rows of the output per tile
__host__ __device__ constexpr int tile_rows(bool cplx) { return cplx ? 64 : 128; }

__device__ __forceinline__ void arrive(uint64_t *mbar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::saddr(mbar)) : "memory");
}
__device__ __forceinline__ void init(uint64_t *mbar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(tc::saddr(mbar)), "r"(count));
}

// round(x 2^(8S-1-e)) plus the digit bias (128 in every digit but the first), on the integer
// pipe: the mantissa with its leading bit at 63, shifted right once.  bad: set when x is not
// finite or |x| >= 2^(e+1).
template <int S>
__device__ __forceinline__ long long fixed(double x, int e, bool &bad) {
  constexpr unsigned long long kBias = 0x0080808080808080ull & ((1ull << (8 * (S - 1))) - 1);
  const unsigned hi = unsigned(__double2hiint(x)), lo = unsigned(__double2loint(x));
  const int ex = int(hi >> 20) & 0x7ff;
  bad = bad || ex > 1023 + e;
  // |x| = m 2^(ex - 1086) with m's leading bit at 63 (zeros and denormals: too small to matter)
  const unsigned mh = 0x80000000u | (hi << 11) | (lo >> 21), ml = lo << 11;
  const int sh = max(1086 - (8 * S - 1) + e - ex - 1, 0);  // one less than the whole shift
  const unsigned long long m = sh < 64 ? ((unsigned long long)mh << 32) | ml : 0ull;
  const unsigned long long v = ((m >> (sh & 63)) + 1) >> 1;
  return (long long)kBias + ((int)hi < 0 ? -(long long)v : (long long)v);
}
// digit j of a biased fixed-point value, times 2^-8j, as a float (exact)
template <int S>
__device__ __forceinline__ float digit(long long w, int j) {
  const float sc = __uint_as_float(uint32_t(127 - 8 * j) << 23);
  if (j == 0)  // -256 .. 256
    return __fadd_rn(__int_as_float(0x4B000200 + int(w >> (8 * (S - 1)))), -8389120.f);
  const int byte = S - 1 - j;
  const uint32_t word = byte < 4 ? uint32_t(w) : uint32_t((unsigned long long)w >> 32);
  const float f = __uint_as_float(__byte_perm(word, 0x4B000000u, 0x7540u + uint32_t(byte & 3)));  // 2^23 + byte
  return __fmaf_rn(f, sc, -8388736.f * sc);
}
// warp-wide: 4 consecutive 32-bit columns of this thread's tensor-memory lane
__device__ __forceinline__ void ld4(uint32_t taddr, float (&v)[4]) {
  uint32_t r[4];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
#pragma unroll
  for (int j = 0; j < 4; ++j) v[j] = __uint_as_float(r[j]);
}
// two floats that are exact in BF16, packed (a in the low half)
__device__ __forceinline__ uint32_t pack(float a, float b) {
  return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632u);
}

// v 2^(e - 61) rounded to FP64, on the integer pipe
__device__ __forceinline__ double join(long long v, int e) {
  const unsigned sign = unsigned((unsigned long long)v >> 32) & 0x80000000u;
  const unsigned long long u = v < 0 ? (unsigned long long)-v : (unsigned long long)v;
  const int lz = __clzll((long long)u);
  // leading bit at 62, rounded to 53 bits; a carry out of the rounding moves into the exponent
  const unsigned long long m = ((u << lz) >> 1) + (1ull << 9);
  const unsigned long long r = ((unsigned long long)(unsigned)(1023 + 2 - lz + e - 1) << 52) + (m >> 10);
  return u ? __hiloint2double(int(unsigned(r >> 32) | sign), int(unsigned(r))) : 0.0;
}

}  // namespace xs

// Epilogue of a real product (the step exponential): adds c0 I + c1 Y + c2 Y2 + c3 Y3 of the item
// when low != 0; items whose squarings are done (sq[item] <= round) are skipped.
struct XsReal {
  int low;
  double alpha, c0, c1, c2, c3;
  const double *Y, *Y2, *Y3;  // item 0's matrices; item stride is the output's
  const int *sq;
  int round;
};

// O = op(A) B for items g = j0 + blockIdx.y (op(A) = A^H when CONJ_A, A then stored k x m; a real
// A is symmetric and read down its columns, as B is).
// |A| <= 2^ea, |B| <= 2^eb.  A non-finite or larger operand makes the tile NaN.
template <bool CPLX, int S, bool CONJ_A, class T>
__global__ void __launch_bounds__(xs::kThreadsXs, 1)
    k_xs_gemm(HMat<const T> A, HMat<const T> B, HMat<T> O, int m, int n, int k, int Cb, long j0, int ea, int eb,
              XsReal ep, int *status) {
  using namespace xs;
  constexpr int kLev = S == 7 ? 7 : 6;   // accumulators
  constexpr int kTop = S == 7 ? 7 : 5;   // highest digit level taken
  constexpr int TM = tile_rows(CPLX);
  extern __shared__ __align__(1024) unsigned char xsm[];
  __shared__ uint32_t tbase;
  __shared__ __align__(8) uint64_t full[2], empty[2], done;
  __shared__ int failed, bad_s;
  if (!CPLX && ep.sq && ep.sq[blockIdx.y] <= ep.round) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long g = j0 + blockIdx.y;
  const int c = int(g % Cb), sl = int(g / Cb);
  const int tn = (n + kN - 1) / kN;
  const int r0 = int(blockIdx.x / tn) * TM, q0 = int(blockIdx.x % tn) * kN;
  const int rows = min(TM, m - r0), cols = min(kN, n - q0);
  const int kc = CPLX ? kK / 2 : kK;  // source k per chunk
  const int nch = (k + kc - 1) / kc;
  unsigned char *base = xsm + ((1024 - (tc::saddr(xsm) & 1023)) & 1023);
  if (warp == 0) tc::tmem_alloc(&tbase, 512);
  if (tid == 0) {
    init(&full[0], kConv), init(&full[1], kConv), init(&empty[0], 1), init(&empty[1], 1), init(&done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;");
    failed = 0, bad_s = 0;
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tbase;
  bool ok = true;
  if (warp < kConv / 32) {
    bool bad = false;
    constexpr int U = 8;  // K entries per unit: one 16-byte core-matrix row (4 complex)
    // units of a chunk: A rows x 4 k groups, then B columns x 4 k groups; rows (columns) fastest
    const int nA = rows * 4, nU = nA + cols * 4;
    // the products that read chunk ch's buffer two chunks ago have ended
    auto released = [&](int ch) -> bool {
      if (ch < 2 || tc::wait_parity(&empty[ch & 1], uint32_t((ch / 2 - 1) & 1))) return true;
      failed = 1;
      return false;
    };
    for (int ch = 0; ch < nch; ++ch) {
      const int buf = ch & 1;
      unsigned char *sa = base + buf * buf_bytes<S>(), *sb = sa + S * kPlaneA;
      bool waited = false;
      for (int u = tid; u < nU; u += kConv) {
        const bool isA = u < nA;
        const int x = isA ? u % rows : (u - nA) % cols, kg = isA ? u / rows : (u - nA) / cols;
        const int l0 = ch * kc + kg * (kc / 4);
        double v[U];
        // source entry t of the unit at p + t d (A runs along its rows, or down its columns when
        // it is conjugate-transposed or symmetric; B down its columns)
        const bool down = !isA || CONJ_A || !CPLX;
        const T *p = isA ? (down ? &A(c, sl, l0, r0 + x) : &A(c, sl, r0 + x, l0)) : &B(c, sl, l0, q0 + x);
        const long d = isA ? (down ? A.ld * A.es : A.es) : B.ld * B.es;
#pragma unroll
        for (int t = 0; t < (CPLX ? 4 : 8); ++t) {
          if constexpr (CPLX) {
            double2 z = make_double2(0.0, 0.0);
            if (l0 + t < k) z = p[t * d];
            v[2 * t] = z.x, v[2 * t + 1] = CONJ_A && isA ? -z.y : z.y;
          } else {
            v[t] = l0 + t < k ? p[t * d] : 0.0;
          }
        }
        long long w[U];
#pragma unroll
        for (int t = 0; t < U; ++t) w[t] = fixed<S>(v[t], isA ? ea : eb, bad);
        if (!waited) {
          waited = true;
          if (!(ok = released(ch))) break;
        }
        const int row = isA ? (CPLX ? 2 * x : x) : x;
        unsigned char *dst = (isA ? sa : sb) + (row >> 3) * kGroup + kg * 128 + (row & 7) * 16;
        const int plane = isA ? kPlaneA : kPlaneB;
#pragma unroll
        for (int j = 0; j < S; ++j) {
          float f[U];
#pragma unroll
          for (int t = 0; t < U; ++t) f[t] = digit<S>(w[t], j);
          uint4 p = make_uint4(pack(f[0], f[1]), pack(f[2], f[3]), pack(f[4], f[5]), pack(f[6], f[7]));
          if (CPLX && isA) {  // row 2x: (a, -b); row 2x + 1: (b, a)
            const uint4 q = make_uint4(pack(f[1], f[0]), pack(f[3], f[2]), pack(f[5], f[4]), pack(f[7], f[6]));
            *reinterpret_cast<uint4 *>(dst + j * plane + 16) = q;
            p.x ^= 0x80000000u, p.y ^= 0x80000000u, p.z ^= 0x80000000u, p.w ^= 0x80000000u;
          }
          *reinterpret_cast<uint4 *>(dst + j * plane) = p;
        }
      }
      // a thread without units waits too: it must not arrive for this chunk before the last one
      // of the same buffer is through
      if (!waited) ok = released(ch);
      if (!ok) break;
      tc::fence_smem_async();
      arrive(&full[buf]);
    }
    if (bad) bad_s = 1;
    if (ok && !tc::wait_parity(&done, 0)) failed = 1;
  } else if (lane == 0) {
    for (int ch = 0; ch < nch; ++ch) {
      const int buf = ch & 1;
      if (!tc::wait_parity(&full[buf], uint32_t((ch / 2) & 1))) {
        failed = 1;
        break;
      }
      tc::fence_after();
      const uint32_t a = tc::sdesc_lo(tc::saddr(base + buf * buf_bytes<S>())), b = a + S * kPlaneA / 16;
      // the last chunk's K entries beyond k are zeros; a whole 16-entry half of them is skipped
      const int ks = (ch == nch - 1 && (k - ch * kc) * (CPLX ? 2 : 1) <= 16) ? 1 : 2;
      // A's digit i with B's digits j, j + 1, ..: the digit planes of B follow one another in whole
      // row groups as the levels' accumulators do in columns, so up to four pairs are one MMA
      // (N <= 256; columns beyond the tile's are not read).  Unrolled, a descriptor costs one
      // addition: 16 MMAs a K step for 34 pairs (S = 7), 8 for 21 (S = 6).
      auto pairs = [&](int i, int j, int w, int lev) {
#pragma unroll
        for (int kk = 0; kk < 2; ++kk)
          if (kk < ks)
            tc::mma(tmem + uint32_t(lev * kN), a + uint32_t(i * kPlaneA / 16 + kk * 16),
                    b + uint32_t(j * kPlaneB / 16 + kk * 16), tc::sdesc_hi(kK), tc::idesc_bf16(w * kN, false),
                    i == 0 && lev < kLev && kk == 0 && j == lev ? uint32_t(ch != 0) : 1u);
      };
#pragma unroll
      for (int i = 0; i < S; ++i) {
#pragma unroll
        for (int j = 0; j < kLev - i; j += 4) pairs(i, j, min(4, kLev - i - j), i + j);
      }
      if (kTop >= kLev) {  // the last level shares an accumulator with the one before
#pragma unroll
        for (int i = kTop - (S - 1); i < S; ++i) pairs(i, kTop - i, 1, kLev - 1);
      }
      tc::commit(&empty[buf]);
    }
    tc::commit(&done);
  }
  __syncwarp();
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const bool fine = failed == 0;
  if (fine) {
    const bool nan = bad_s != 0;
    const int q4 = warp & 3, L = 32 * q4 + lane;  // tensor-memory lane: tile row
    const int live = CPLX ? 2 * rows : rows, c8 = 8 * (warp >> 2);
    if (32 * q4 < live && c8 < cols) {  // warp-uniform
#pragma unroll 1
      for (int c0 = c8; c0 < c8 + 8; c0 += 4) {
        float a[kLev][4];
        const uint32_t ta = tmem + (uint32_t(32 * q4) << 16) + uint32_t(c0);
#pragma unroll
        for (int l = 0; l < kLev; ++l) ld4(ta + uint32_t(l * kN), a[l]);
        double add[4] = {0, 0, 0, 0};
        if constexpr (!CPLX) {  // the low terms, loaded together before anything is stored
          if (ep.low && L < live) {
            double y[3][4];
            const int r = r0 + L;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              const long e = long(c) * O.cs + long(r) * O.ld + min(q0 + c0 + t, n - 1);
              y[0][t] = ep.Y[e], y[1][t] = ep.Y2[e], y[2][t] = ep.Y3[e];
            }
#pragma unroll
            for (int t = 0; t < 4; ++t)
              add[t] = fma(ep.c3, y[2][t], fma(ep.c2, y[1][t], fma(ep.c1, y[0][t], r == q0 + c0 + t ? ep.c0 : 0.0)));
          }
        }
        tc::wait_ld();
        double d[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          int I[7];
#pragma unroll
          for (int l = 0; l < kLev; ++l) I[l] = __float2int_rn(a[l][t] * __uint_as_float(uint32_t(127 + 8 * l) << 23));
          // sum of I_l 2^(-14-8l) in units of 2^-61 (|sum| < 2: level 0 to 2 fit 32 bits)
          long long v = (long long)((I[0] << 16) + (I[1] << 8) + I[2]) << 31;
          v += (long long)I[3] * (1 << 23);
          v += (long long)I[4] * (1 << 15);
          v += (long long)I[5] * (1 << 7);
          if constexpr (kLev == 7) v += I[6] >> 1;
          d[t] = nan ? __longlong_as_double(0x7FF8000000000000ll) : join(v, ea + eb);
        }
        if constexpr (CPLX) {
          const bool odd = L & 1;
          const int r = r0 + (L >> 1);
#pragma unroll
          for (int t = 0; t < 4; t += 2) {
            const double send = odd ? d[t] : d[t + 1];
            const double got = __shfl_xor_sync(0xffffffffu, send, 1);
            const int q = q0 + c0 + t + (odd ? 1 : 0);
            if (L < live && q < n) O(c, sl, r, q) = odd ? make_double2(got, d[t + 1]) : make_double2(d[t], got);
          }
        } else if (L < live) {
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const int q = q0 + c0 + t;
            double v = ep.alpha == 1.0 ? d[t] : ep.alpha * d[t];
            if (ep.low) v += add[t];
            if (q < n) O(c, sl, r0 + L, q) = v;
          }
        }
      }
    }
  } else {
    if (tid == 0) atomicOr(status, kTcTimeout);
    tc::wait_parity(&done, 0);  // bounded: let products in flight drain before TMEM is freed
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  if (warp == 0) tc::tmem_free(tmem, 512);
}
