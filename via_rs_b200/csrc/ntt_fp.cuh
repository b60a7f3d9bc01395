// The register-resident negacyclic transform of ntt.cuh in double precision,
// for primes q < 2^44. Residues are integer-valued doubles in a signed
// range, and every product is exact:
//
//   fp_mulmod(a, b): ph = fl(a b), pl = a b - ph (one FMA: the error-free
//   product), qt = round(ph / q) (an FMA against a rounded 1/q plus the
//   1.5 * 2^52 rounding constant), r = (ph - qt q) + pl.
//
// For integers |a| < 2^48 and |b| < q, |qt - a b / q| <= 1/2 + 2^-4, so
// ph - qt q and r are integers far below 2^53 and both steps are exact:
// r = a b (mod q) with |r| <= 0.5625 q (checked against 128-bit integer
// products over these ranges). This is the floating-point reduction of
// modular products used by Shoup's NTL (a quotient estimate in floating point,
// an exact integer correction), with the FMA two-product making the product
// itself exact. Explicit _rn intrinsics keep the compiler from contracting or
// reassociating any step.
//
// Bounds: forward butterflies (a, c) -> (a + t, a - t), t = fp_mulmod(c, w), grow by at
// most 0.5625 q per stage; inverse butterflies (a, c) -> (a + c, fp_mulmod(a - c, w)) at
// most double per stage, so inputs below 2 q of a prime up to 2^35 stay below 2^48 through
// twelve stages. Larger primes bring the values back within q / 2 on the way
// (fp_inverse_w). The inverse ends with an fp_mulmod by n^-1.
#pragma once
#include "ntt.cuh"

namespace via {

constexpr double FP_ROUND = 6755399441055744.0;  // 1.5 * 2^52: x + FP_ROUND - FP_ROUND rounds x to an integer

__device__ __forceinline__ double fp_mulmod(double a, double b, double q, double qinv) {
  const double ph = __dmul_rn(a, b);
  const double pl = __fma_rn(a, b, -ph);
  const double qt = __dadd_rn(__fma_rn(ph, qinv, FP_ROUND), -FP_ROUND);
  return __dadd_rn(__fma_rn(-qt, q, ph), pl);
}

// Signed residue x (|x| < 2^50) -> canonical residue in [0, q).
__device__ __forceinline__ double fp_canonical(double x, double q, double qinv) {
  const double qt = __dadd_rn(__fma_rn(x, qinv, FP_ROUND), -FP_ROUND);
  double r = __fma_rn(-qt, q, x);  // exact, |r| <= q / 2 + 1
  if (r < 0) r = __dadd_rn(r, q);
  if (r >= q) r = __dadd_rn(r, -q);
  return r;
}

// A product's residue (|r| <= 0.5625 q) -> canonical residue.
__device__ __forceinline__ double fp_wrap(double r, double q) { return r < 0 ? __dadd_rn(r, q) : r; }

// Integers below 2^52 to and from doubles, exactly, without the conversion unit: the
// double 2^52 + x has the bit pattern 0x4330000000000000 | x.
__device__ __forceinline__ double fp_from_u64(u64 x) {
  return __dadd_rn(__longlong_as_double((long long)(x | 0x4330000000000000ull)), -4503599627370496.0);
}
__device__ __forceinline__ u64 fp_to_u64(double x) {
  return (u64)__double_as_longlong(__dadd_rn(x, 4503599627370496.0)) & 0xFFFFFFFFFFFFFull;
}
// x brought back within q / 2 + 1 (|x| < 2^53).
__device__ __forceinline__ double fp_reduce(double x, double q, double qinv) {
  return __fma_rn(-__dadd_rn(__fma_rn(x, qinv, FP_ROUND), -FP_ROUND), q, x);
}

// Eight consecutive words of a thread, as two 32-byte accesses. Keys (ld8_nc) stay in L1
// before anything else.
__device__ __forceinline__ void ld8(const u64* p, u64 (&x)[8]) {
#pragma unroll
  for (int h = 0; h < 2; ++h)
    asm volatile("ld.global.v4.u64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(x[4 * h]), "=l"(x[4 * h + 1]), "=l"(x[4 * h + 2]), "=l"(x[4 * h + 3])
                 : "l"(p + 4 * h));
}
// Read (or written) once: not worth a line of L1 where keys want it.
__device__ __forceinline__ void ld8_stream(const u64* p, u64 (&x)[8]) {
#pragma unroll
  for (int h = 0; h < 2; ++h)
    asm volatile("ld.global.L1::no_allocate.v4.u64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(x[4 * h]), "=l"(x[4 * h + 1]), "=l"(x[4 * h + 2]), "=l"(x[4 * h + 3])
                 : "l"(p + 4 * h));
}
__device__ __forceinline__ void ld8_nc(const u64* p, u64 (&x)[8]) {
#pragma unroll
  for (int h = 0; h < 2; ++h)
    asm("ld.global.nc.L1::evict_last.v4.u64 {%0, %1, %2, %3}, [%4];"
        : "=l"(x[4 * h]), "=l"(x[4 * h + 1]), "=l"(x[4 * h + 2]), "=l"(x[4 * h + 3])
        : "l"(p + 4 * h));
}
__device__ __forceinline__ void st8(u64* p, const u64 (&x)[8]) {
#pragma unroll
  for (int h = 0; h < 2; ++h)
    asm volatile("st.global.v4.u64 [%0], {%1, %2, %3, %4};" ::"l"(p + 4 * h), "l"(x[4 * h]), "l"(x[4 * h + 1]),
                 "l"(x[4 * h + 2]), "l"(x[4 * h + 3])
                 : "memory");
}

__device__ __forceinline__ void st8_stream(u64* p, const u64 (&x)[8]) {
#pragma unroll
  for (int h = 0; h < 2; ++h)
    asm volatile("st.global.L1::no_allocate.v4.u64 [%0], {%1, %2, %3, %4};" ::"l"(p + 4 * h), "l"(x[4 * h]), "l"(x[4 * h + 1]),
                 "l"(x[4 * h + 2]), "l"(x[4 * h + 3])
                 : "memory");
}

// One phase (up to three butterfly stages) on doubles, with the forward layouts of
// NttPhase<LOGN, false, P>. Phase P works within aligned blocks of SPAN elements. The
// inverse undoes the forward phases last to first in the same layouts: it starts on
// eight consecutive elements a thread and ends in the layout the forward starts in.
//
// 32 threads hold the same aligned 256 elements in every layout with SPAN <= 256, so an
// exchange between two such layouts stays within a warp (fp_sync); at n = 2048 one
// exchange of three needs the whole CTA.
template <int LOGN, int P>
struct FpPhase {
  using Ix = NttPhase<LOGN, false, P>;
  static constexpr int n = Ix::n, S0 = Ix::S0, R = Ix::R, NSUB = Ix::NSUB, STRIDE = Ix::STRIDE, SPAN = n >> S0;

  // Twiddles of level lvl: consecutive, aligned to their number.
  __device__ __forceinline__ static void twiddles(const double* t, int at, int count, double (&w)[4]) {
    if (count == 1) {
      w[0] = __ldg(t + at);
    } else {
#pragma unroll
      for (int j = 0; j < 4; j += 2)
        if (j < count) {
          const double2 v = __ldg(reinterpret_cast<const double2*>(t + at + j));
          w[j] = v.x;
          w[j + 1] = v.y;
        }
    }
  }

  // W polynomials at once: one load of each twiddle, W independent butterflies of it.
  template <int W>
  __device__ __forceinline__ static void forward(double (&e)[W][8], int tid, const NttTable& T) {
    const double q = T.qd, qinv = T.qinv;
#pragma unroll
    for (int sub = 0; sub < NSUB; ++sub) {
      const int b0 = (tid * NSUB + sub) / STRIDE;
#pragma unroll
      for (int lvl = 0; lvl < R; ++lvl) {
        const int hk = 1 << (R - 1 - lvl);
        double w[4];
        twiddles(T.psi_d, n / (2 * STRIDE * hk) + (b0 << lvl), 1 << lvl, w);
#pragma unroll
        for (int k = 0; k < (1 << R); ++k) {
          if (k & hk) continue;
#pragma unroll
          for (int x = 0; x < W; ++x) {
            double& a = e[x][sub * (1 << R) + k];
            double& c = e[x][sub * (1 << R) + k + hk];
            const double t = fp_mulmod(c, w[k >> (R - lvl)], q, qinv), av = a;
            a = __dadd_rn(av, t);
            c = __dadd_rn(av, -t);
          }
        }
      }
    }
  }

  template <int W>
  __device__ __forceinline__ static void inverse(double (&e)[W][8], int tid, const NttTable& T) {
    const double q = T.qd, qinv = T.qinv;
#pragma unroll
    for (int sub = 0; sub < NSUB; ++sub) {
      const int b0 = (tid * NSUB + sub) / STRIDE;
#pragma unroll
      for (int lvl = R - 1; lvl >= 0; --lvl) {
        const int hk = 1 << (R - 1 - lvl);
        double w[4];
        twiddles(T.ipsi_d, n / (2 * STRIDE * hk) + (b0 << lvl), 1 << lvl, w);
#pragma unroll
        for (int k = 0; k < (1 << R); ++k) {
          if (k & hk) continue;
#pragma unroll
          for (int x = 0; x < W; ++x) {
            double& a = e[x][sub * (1 << R) + k];
            double& c = e[x][sub * (1 << R) + k + hk];
            const double av = a, cv = c;
            a = __dadd_rn(av, cv);
            c = fp_mulmod(__dadd_rn(av, -cv), w[k >> (R - lvl)], q, qinv);
          }
        }
      }
    }
  }
};

// The first three forward stages on small integers (digits): the eight outputs are sums
// of the inputs times products of the seven twiddles, 34 exact multiply-adds instead of
// twelve butterflies of eight operations. Sums stay below 8 |e| q: 2^48 for |e| <= 127 and
// q <= 2^38.
constexpr double FP_DIGIT_Q = 274877906944.0;  // 2^38
__device__ __forceinline__ void fp_digit_phase(double (&e)[8], const NttTable& T) {
  const double* c = T.d8;
  const double s = __fma_rn(c[0], e[4], e[0]), d = __fma_rn(-c[0], e[4], e[0]);
  const double t = __fma_rn(c[2], e[6], __dmul_rn(c[1], e[2])), u = __fma_rn(-c[4], e[6], __dmul_rn(c[3], e[2]));
  const double ev[4] = {__dadd_rn(s, t), __dadd_rn(s, -t), __dadd_rn(d, u), __dadd_rn(d, -u)};
  const double x1 = e[1], x5 = e[5], x3 = e[3], x7 = e[7];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const double* k = c + 5 + 4 * i;
    const double o = __fma_rn(k[3], x7, __fma_rn(k[2], x3, __fma_rn(k[1], x5, __dmul_rn(k[0], x1))));
    e[2 * i] = __dadd_rn(ev[i], o);
    e[2 * i + 1] = __dadd_rn(ev[i], -o);
  }
}

// Both twiddle tables of degree 2^LOGN into L1, a line a thread of 2^LOGN / 8: kernels of one
// or two transforms would otherwise wait for L2 in every phase.
template <int LOGN>
__device__ __forceinline__ void fp_prefetch_twiddles(int tid, const NttTable& T) {
  const double* t = tid < (1 << LOGN) / 16 ? T.psi_d + 16 * tid : T.ipsi_d + 16 * (tid - (1 << LOGN) / 16);
  asm volatile("prefetch.global.L1 [%0];" ::"l"(t));
}
__device__ __forceinline__ void fp_prefetch(const u64* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

template <int SPAN>
__device__ __forceinline__ void fp_sync() {
  if constexpr (SPAN <= 256)
    __syncwarp();
  else
    __syncthreads();
}

// Forward transform of W segments held in the phase-0 layout (tid + k n / 8); leaves each as
// eight consecutive elements a thread, signed residues below |input| + 0.5625 LOGN q.
// Phases before P have run. `ssm`: W exchange areas of n elements each (addressed through
// swz from `sbase`; W = 1 where several segments share a CTA). On entry no other warp may
// still read them. A transform is a chain of about 90 dependent FP64 operations and a few
// exchanges, 4 to 5 us however many run beside it: two at once (W = 2) take little longer
// than one.
template <int LOGN, int P = 0, int W = 1>
__device__ __forceinline__ void fp_forward_w(double (&e)[W][8], int tid, const NttTable& T, double* ssm, int sbase = 0) {
  constexpr int NPH = (LOGN + 2) / 3, n = 1 << LOGN;
  if constexpr (P > 0) {
    using Pv = FpPhase<LOGN, P - 1>;
    using Ph = FpPhase<LOGN, P>;
    if constexpr (P > 1) fp_sync<Pv::SPAN>();  // the previous exchange's reads
#pragma unroll
    for (int x = 0; x < W; ++x)
#pragma unroll
      for (int v = 0; v < 8; ++v) ssm[x * n + swz(sbase + Pv::Ix::index(v, tid))] = e[x][v];
    fp_sync<Pv::SPAN>();
#pragma unroll
    for (int x = 0; x < W; ++x)
#pragma unroll
      for (int v = 0; v < 8; ++v) e[x][v] = ssm[x * n + swz(sbase + Ph::Ix::index(v, tid))];
  }
  FpPhase<LOGN, P>::template forward<W>(e, tid, T);
  if constexpr (P + 1 < NPH) fp_forward_w<LOGN, P + 1, W>(e, tid, T, ssm, sbase);
}

// The same from digits, with the dense first phase where the caller finds its sums below
// 2^48 (uniform in the CTA).
template <int LOGN, int W>
__device__ __forceinline__ void fp_forward_digits_w(double (&e)[W][8], int tid, const NttTable& T, double* ssm, int sbase,
                                                    bool dense) {
  if (dense) {
#pragma unroll
    for (int x = 0; x < W; ++x) fp_digit_phase(e[x], T);
  } else {
    FpPhase<LOGN, 0>::template forward<W>(e, tid, T);
  }
  if constexpr (LOGN > 3) fp_forward_w<LOGN, 1, W>(e, tid, T, ssm, sbase);
}

// Inverse transforms, without the n^-1 scaling, of W segments held as eight consecutive
// elements a thread, inputs below 2 q in magnitude; leaves signed values in the phase-0
// layout, at most 2^48: every stage may double them, so 2 q * 2^12 for q <= 2^35. Primes above
// 2^35 return to q / 2 after the second phase (six stages at most before it: 2 q * 2^6 <= 2^47
// for q < 2^40), above 2^40 after every phase (2 q * 2^3 < 2^48 for q < 2^44). On entry no other
// warp may still read the exchange areas.
template <int LOGN, int P, int W>
__device__ __forceinline__ void fp_inverse_w(double (&e)[W][8], int tid, const NttTable& T, double* ssm, int sbase = 0) {
  constexpr int LAST = (LOGN + 2) / 3 - 1, n = 1 << LOGN;
  FpPhase<LOGN, P>::template inverse<W>(e, tid, T);
  if constexpr (P > 0) {
    using Ph = FpPhase<LOGN, P>;
    using Nx = FpPhase<LOGN, P - 1>;
    if (T.qd > 34359738368.0 && (P == LAST - 1 || T.qd > 1099511627776.0)) {
#pragma unroll
      for (int x = 0; x < W; ++x)
#pragma unroll
        for (int v = 0; v < 8; ++v) e[x][v] = fp_reduce(e[x][v], T.qd, T.qinv);
    }
    if constexpr (P < LAST) fp_sync<Ph::SPAN>();  // the previous exchange's reads
#pragma unroll
    for (int x = 0; x < W; ++x)
#pragma unroll
      for (int v = 0; v < 8; ++v) ssm[x * n + swz(sbase + Ph::Ix::index(v, tid))] = e[x][v];
    fp_sync<Nx::SPAN>();
#pragma unroll
    for (int x = 0; x < W; ++x)
#pragma unroll
      for (int v = 0; v < 8; ++v) e[x][v] = ssm[x * n + swz(sbase + Nx::Ix::index(v, tid))];
    fp_inverse_w<LOGN, P - 1, W>(e, tid, T, ssm, sbase);
  }
}

// One segment.
template <int LOGN>
__device__ __forceinline__ void fp_forward(double (&e)[8], int tid, const NttTable& T, double* ssm, int sbase = 0) {
  fp_forward_w<LOGN, 0, 1>(reinterpret_cast<double(&)[1][8]>(e), tid, T, ssm, sbase);
}
template <int LOGN>
__device__ __forceinline__ void fp_forward_digits(double (&e)[8], int tid, const NttTable& T, double* ssm, int sbase,
                                                  bool dense) {
  fp_forward_digits_w<LOGN, 1>(reinterpret_cast<double(&)[1][8]>(e), tid, T, ssm, sbase, dense);
}
template <int LOGN>
__device__ __forceinline__ void fp_inverse(double (&e)[8], int tid, const NttTable& T, double* ssm, int sbase = 0) {
  fp_inverse_w<LOGN, (LOGN + 2) / 3 - 1, 1>(reinterpret_cast<double(&)[1][8]>(e), tid, T, ssm, sbase);
}
// Two at once; `ssm` holds 2 n elements.
template <int LOGN>
__device__ __forceinline__ void fp_forward2(double (&e)[2][8], int tid, const NttTable& T, double* ssm) {
  fp_forward_w<LOGN, 0, 2>(e, tid, T, ssm);
}
template <int LOGN>
__device__ __forceinline__ void fp_forward_digits2(double (&e)[2][8], int tid, const NttTable& T, double* ssm, bool dense) {
  fp_forward_digits_w<LOGN, 2>(e, tid, T, ssm, 0, dense);
}
template <int LOGN>
__device__ __forceinline__ void fp_inverse2(double (&e)[2][8], int tid, const NttTable& T, double* ssm) {
  fp_inverse_w<LOGN, (LOGN + 2) / 3 - 1, 2>(e, tid, T, ssm);
}

}  // namespace via
