// The VIA-C answer pipeline on the device (crates/via-server/src/answer.rs:83-354):
//
//   1 QueryDecomp   LWE -> RLWE cascade (prim/conversion/cascade.rs) + RLWE -> RGSW
//   2 DMux tree     trivial RLWE(delta) -> I RLWEs at q1      (prim/gates/mux.rs:222)
//   3 ModSwitch     q1 -> q2                                   (prim/switching/mod_switch.rs:57)
//   4 FirstDim      I x J database scan                        (srv/first_dim.rs:94)
//   5 CMux tree     J -> 1 at q2                               (prim/gates/mux.rs:167)
//   6 CRot          slot extraction                            (prim/gates/rotate.rs:128)
//   7 RespComp      q2 -> q3, ring switch n1 -> n2, body -> q4 (srv/resp_comp.rs:46)
//
// Every gadget product is: exact decomposition into balanced digits (kernel
// k_decompose) -> forward NTT of the digit polys -> one pointwise
// multiply-accumulate against the eval-form key (k_mac) -> inverse NTT. Linear
// steps between products are done in whichever domain saves transforms; since
// the NTT is exact, the coefficient-form results equal the reference's.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "cascade_tc.cuh"
#include "first_dim.cuh"
#include "gadget.cuh"
#include "gadget_fp.cuh"
#include "server.cuh"

namespace via {

// Grid size below which k_cascade_mac splits its output masks over more blocks.
constexpr long CASCADE_SPLIT_BLOCKS = 4 * 148;

// in: npolys polys [p][nl][n_in]; out: digit polys [p][L][nl][n_out] in sample
// order (slot s = L-1-k holds digit k). n_out = n_in * stride: the input is
// first embedded at slot 0 (reshape.rs:58), so other positions get digit 0.
__global__ void k_decompose(const u64* __restrict__ in, int n_in, int stride, long npolys, DevRing R, Gadget g,
                            u64* __restrict__ out) {
  long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= npolys * n_in) return;
  long p = gid / n_in;
  int i = (int)(gid % n_in);
  const int nl = R.nl;
  const u64* src = in + p * nl * n_in;
  u64 a0 = src[i], a1 = nl == 2 ? src[n_in + i] : 0;
  if (a0 >= R.m[0].q) a0 = reduce64(a0, R.m[0]);  // a caller's word may be any 64 bits
  if (a1 >= R.m[1].q) a1 = reduce64(a1, R.m[1]);
  const int n_out = n_in * stride;
  const long step = (long)nl * n_out;
  // Digit k goes to sample slot L - 1 - k.
  u64* o = out + p * (long)g.L * step + (long)(g.L - 1) * step + (long)i * stride;
  if (g.fp && R.ntt && stride == 1) {
    double v = nl == 2 ? fp_scaled2(fp_from_u64(a0), fp_from_u64(a1), g, R)
                       : fp_scaled(fp_reduce(fp_from_u64(a0), (double)R.m[0].q, R.t[0].qinv), g.dS, R.t[0].qinv);
    for (int k = 0; k < g.L; ++k, o -= step) {
      const double d = fp_next_digit(v, g);
      for (int l = 0; l < nl; ++l) {
        const double q = (double)R.m[l].q;
        o[(long)l * n_out] = fp_to_u64(d < 0.0 ? __dadd_rn(d, q) : d);
      }
    }
    return;
  }
  for_each_digit(gadget_scaled(a0, a1, R, g), g, [&](int, i64 d) {
    for (int l = 0; l < nl; ++l) {
      u64* ol = o + (long)l * n_out;
      ol[0] = lift_i64(d, R.m[l]);
      for (int z = 1; z < stride; ++z) ol[z] = 0;
    }
    o -= step;
  });
}

// The same digits as signed bytes for gadgets with B <= 255 (|digit| <= 127),
// limb-free: out [p][L][n_in] in sample order; the 8-bit transforms lift them
// per limb. A sixteenth of the bytes of the u64 digits of a two-limb ring.
__global__ void k_decompose_i8(const u64* __restrict__ in, int n_in, long npolys, DevRing R, Gadget g,
                               int8_t* __restrict__ out) {
  const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= npolys * n_in) return;
  const long p = gid / n_in;
  const int i = (int)(gid % n_in);
  const int nl = R.nl;
  const u64* src = in + p * nl * n_in;
  const u64 a0 = src[i], a1 = nl == 2 ? src[n_in + i] : 0;
  int8_t* o = out + p * (long)g.L * n_in + (long)(g.L - 1) * n_in + i;
  for_each_digit(gadget_scaled(a0, a1, R, g), g, [&](int, i64 d) {
    *o = (int8_t)d;
    o -= n_in;
  });
}

// The same for the gadgets of ct_digits_ok, by exact steps on doubles (cascade_tc.cuh).
// Thread = four consecutive coefficients, four digits a store. About 64 FP64 and 100 integer
// operations a coefficient, where the 128-bit divisions of k_decompose_i8 take about 500: the
// four late splits of 2688 LWEs 1034 -> 217 us.
__global__ void __launch_bounds__(128) k_ct_decompose(const u64* __restrict__ in, int n_in, long npolys, CtDigits D,
                                                      int8_t* __restrict__ out) {
  const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid * 4 >= npolys * n_in) return;
  const long p = gid * 4 / n_in;
  const int i = (int)(gid * 4 % n_in);
  const u64* src = in + p * 2 * n_in + i;
  u32 f[4][3];
  {
    const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(src), a1 = *reinterpret_cast<const ulonglong2*>(src + 2);
    const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(src + n_in),
                     b1 = *reinterpret_cast<const ulonglong2*>(src + n_in + 2);
    const u64 a[4] = {a0.x, a0.y, a1.x, a1.y}, b[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
    for (int r = 0; r < 4; ++r)
      ct_pieces(fp_mulmod(fp_from_u64(a[r]), D.yscale[0], D.q[0], D.qinv[0]),
                fp_mulmod(fp_from_u64(b[r]), D.yscale[1], D.q[1], D.qinv[1]), D, f[r]);
  }
  int8_t* o = out + p * (long)CT_L * n_in + i;
#pragma unroll
  for (int x = 0; x < 3; ++x)
#pragma unroll
    for (int k = 0; k < CT_LP; ++k, o += n_in) {
      const u32 d = ct_digit(f[0][x], D.base) | ct_digit(f[1][x], D.base) << 8 | ct_digit(f[2][x], D.base) << 16 |
                    ct_digit(f[3][x], D.base) << 24;
      *reinterpret_cast<u32*>(o) = ct_signed(d, D.o);
    }
}

// Which eval-form key samples output o multiplies: K_o = base + ((o / div) % mod) * stride.
// stride = 0 means "consecutive keys" (T*2*nl*n residues apart, T = samples per key).
struct KeySel {
  const u64* base;
  long div, mod, stride;
};
static inline KeySel keys_shared(const u64* base) { return KeySel{base, 1, 1, 0}; }
static inline KeySel keys_cyclic(const u64* base, long mod) { return KeySel{base, 1, mod, 0}; }

// ---------------------------------------------------------------------------
// Multiply-accumulate against eval-form keys.
//   out[o].{mask,body} = sum_{s<T} D[o*T + s] (*) K_o[s].{mask,body}
// K_o selected by a KeySel (T samples per key).
// ---------------------------------------------------------------------------
__global__ void k_mac_ntt(const u64* __restrict__ D, KeySel ks, u64* __restrict__ out, int T, int n, int nl, long nout,
                          DevRing R) {
  long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  long per = (long)nl * n;
  if (gid >= nout * per) return;
  long o = gid / per;
  int rem = (int)(gid % per);
  int l = rem / n;
  const u64* Ko = ks.base + ((o / ks.div) % ks.mod) * (ks.stride ? ks.stride : (long)T * 2 * per);
  const u64* Do = D + o * (long)T * per;
  Acc128 am{0, 0}, ab{0, 0};
#pragma unroll 6
  for (int s = 0; s < T; ++s) {
    u64 dv = Do[s * per + rem];
    mac128(am, dv, Ko[(2 * s) * per + rem]);
    mac128(ab, dv, Ko[(2 * s + 1) * per + rem]);
  }
  const DevMod& m = R.m[l];
  out[(2 * o) * per + rem] = reduce128(am.hi, am.lo, m);
  out[(2 * o + 1) * per + rem] = reduce128(ab.hi, ab.lo, m);
}

// NS consecutive doubles or words of a thread: one 8- or 16-byte access.
template <int NS, class V, class T>
__device__ __forceinline__ void ld_slots(const T* p, T (&x)[NS]) {
  if constexpr (NS == 2) {
    const V v = __ldg(reinterpret_cast<const V*>(p));
    x[0] = v.x;
    x[1] = v.y;
  } else {
    x[0] = __ldg(p);
  }
}
template <int NS>
__device__ __forceinline__ void st_slots(u64* p, const u64 (&x)[NS]) {
  if constexpr (NS == 2)
    *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(x[0], x[1]);
  else
    *p = x[0];
}

// k_mac_ntt in double precision, for primes below 2^44 (ntt_fp.cuh): digits below 2 q, key
// residues below q, every product within 0.5625 q. NS slots a thread: two (16-byte accesses)
// once that leaves two blocks a SM. Bound by the digit and key bytes where each output has
// its own key, as external products in place: 4099 of them at q1 490 us in 128-bit integers, 303 us
// here (6.2 TB/s).
template <int NS>
__global__ void __launch_bounds__(256, NS == 1 ? 2 : 4) k_mac_fp(const u64* __restrict__ D, KeySel ks, u64* __restrict__ out, int T,
                                                int n, int nl, long nout, const __grid_constant__ DevRing R) {
  const long gid = ((long)blockIdx.x * blockDim.x + threadIdx.x) * NS;
  const long per = (long)nl * n;
  if (gid >= nout * per) return;
  const long o = gid / per;
  const int rem = (int)(gid % per);
  const int l = rem / n;
  const double q = R.t[l].qd, qinv = R.t[l].qinv;
  const u64* Ko = ks.base + ((o / ks.div) % ks.mod) * (ks.stride ? ks.stride : (long)T * 2 * per) + rem;
  const u64* Do = D + o * (long)T * per + rem;
  double m[NS], b[NS];
#pragma unroll
  for (int i = 0; i < NS; ++i) m[i] = b[i] = 0.0;
#pragma unroll(NS == 1 ? 9 : 3)
  for (int s = 0; s < T; ++s) {
    u64 d[NS], km[NS], kb[NS];
    ld_slots<NS, ulonglong2>(Do + s * per, d);
    ld_slots<NS, ulonglong2>(Ko + (2 * s) * per, km);
    ld_slots<NS, ulonglong2>(Ko + (2 * s + 1) * per, kb);
#pragma unroll
    for (int i = 0; i < NS; ++i) {
      const double x = fp_from_u64(d[i]);
      m[i] = __dadd_rn(m[i], fp_mulmod(x, fp_from_u64(km[i]), q, qinv));
      b[i] = __dadd_rn(b[i], fp_mulmod(x, fp_from_u64(kb[i]), q, qinv));
    }
  }
  u64 om[NS], ob[NS];
#pragma unroll
  for (int i = 0; i < NS; ++i) {
    om[i] = fp_to_u64(fp_canonical(m[i], q, qinv));
    ob[i] = fp_to_u64(fp_canonical(b[i], q, qinv));
  }
  st_slots(out + (2 * o) * per + rem, om);
  st_slots(out + (2 * o + 1) * per + rem, ob);
}

// Schoolbook (non-NTT ring) variant: negacyclic products, exact.
__global__ void k_mac_schoolbook(const u64* __restrict__ D, KeySel ks, u64* __restrict__ out, int T, int n, int nl,
                                 long nout, DevRing R) {
  long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  long per = (long)nl * n;
  if (gid >= nout * per) return;
  long o = gid / per;
  int rem = (int)(gid % per);
  int l = rem / n, t = rem % n;
  const u64* Ko = ks.base + ((o / ks.div) % ks.mod) * (ks.stride ? ks.stride : (long)T * 2 * per);
  const u64* Do = D + o * (long)T * per;
  const DevMod& m = R.m[l];
  const bool pow2 = m.log2q >= 0;
  u64 wm = 0, wb = 0;
  Acc128 pm{0, 0}, nm{0, 0}, pb{0, 0}, nb{0, 0};
  for (int s = 0; s < T; ++s) {
    const u64* dp = Do + s * per + (long)l * n;
    const u64* km = Ko + (2 * s) * per + (long)l * n;
    const u64* kb = Ko + (2 * s + 1) * per + (long)l * n;
    for (int j = 0; j < n; ++j) {
      u64 dv = dp[j];
      if (dv == 0) continue;
      int k = t - j;
      bool ng = k < 0;
      if (ng) k += n;
      if (pow2) {
        u64 a = dv * km[k], b = dv * kb[k];
        wm += ng ? (u64)0 - a : a;
        wb += ng ? (u64)0 - b : b;
      } else if (ng) {
        mac128(nm, dv, km[k]);
        mac128(nb, dv, kb[k]);
      } else {
        mac128(pm, dv, km[k]);
        mac128(pb, dv, kb[k]);
      }
    }
  }
  u64 rm, rb;
  if (pow2) {
    rm = wm & (m.q - 1);
    rb = wb & (m.q - 1);
  } else {
    rm = submod(reduce128(pm.hi, pm.lo, m), reduce128(nm.hi, nm.lo, m), m.q);
    rb = submod(reduce128(pb.hi, pb.lo, m), reduce128(nb.hi, nb.lo, m), m.q);
  }
  out[(2 * o) * per + rem] = rm;
  out[(2 * o + 1) * per + rem] = rb;
}

// ---------------------------------------------------------------------------
// Elementwise kernels. All buffers are [poly][limb][n].
// ---------------------------------------------------------------------------
// out[j] = a[j*sa] + sign * b[j*sb] for RLWEs (2 polys each); sign in {+1,-1}.
__global__ void k_rlwe_addsub(u64* out, const u64* a, long sa, const u64* b, long sb, int sign, long count, int n,
                              int nl, DevRing R) {
  long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  long per = 2L * nl * n;
  if (gid >= count * per) return;
  long j = gid / per;
  int rem = (int)(gid % per);
  int l = (rem / n) % nl;
  u64 q = R.m[l].q;
  u64 x = a[j * sa * per + rem], y = b[j * sb * per + rem];
  out[j * per + rem] = sign > 0 ? addmod(x, y, q) : submod(x, y, q);
}

// The trivial RLWE (0, delta) at q1 (answer.rs:181-191): zero mask, body = delta * X^0.
// `count` trivial RLWEs (0, d) with d the constant (d0, d1) in RNS form.
__global__ void k_set_trivial(u64* ct, long count, int n, int nl, u64 d0, u64 d1) {
  const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= count * 2 * nl * n) return;
  const long r = gid % (2L * nl * n);
  const int poly = (int)(r / (nl * n)), rem = (int)(r % (nl * n));
  const int l = rem / n, i = rem % n;
  ct[gid] = (poly == 1 && i == 0) ? (l == 0 ? d0 : d1) : 0;
}

// DMux combine (mux.rs:129-137, 222-251): out[2j] = in[j] - ext[j], out[2j+1] = ext[j].
__global__ void k_dmux_combine(u64* out, const u64* in, const u64* ext, long count, int n, int nl, DevRing R) {
  long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  long per = 2L * nl * n;
  if (gid >= count * per) return;
  long j = gid / per;
  int rem = (int)(gid % per);
  int l = (rem / n) % nl;
  u64 q = R.m[l].q;
  u64 e = ext[j * per + rem];
  out[(2 * j) * per + rem] = submod(in[j * per + rem], e, q);
  out[(2 * j + 1) * per + rem] = e;
}

// One DMux tree level in a single kernel (mux.rs:129-137, 222-251; the external
// product rgsw.rs:108-121 with the coefficient-form gadget product,
// rlev.rs:193-222), in double precision (ntt_fp.cuh). CTA (o, l) computes limb l
// of ext[o] = bit (x) in[o] and writes out[2o] = in[o] - ext, out[2o+1] = ext:
// the gadget digits (L = 2) of the mask and body coefficients (both limbs read,
// one CRT scaling per coefficient), forward transforms of the four digit
// polynomials at prime l, products with the RGSW samples (each within 0.5625 q;
// digit k of input half h with sample h L + L - 1 - k), and inverse transforms of
// the two sums. Buffers: [ct][2][nl][n], RGSW [2L][2][nl][n] eval at q1; nl = 2
// primes below 2^44. FP64-issue and latency bound: the levels of 256 to 1024 products
// of 64 queries took 728 us together with eight barriers a transform and 64-bit
// integer digit splits, 362 us with one barrier and splits on doubles, 295 us with all of a
// half's loads before its splits (each waited behind the previous split's rare branch; a level
// of 8192 products 1621 and 1217 us).
template <int LOGN>
__global__ void __launch_bounds__((1 << LOGN) / 8, LOGN >= 12 ? 1 : 2) k_dmux_fp(u64* __restrict__ out, const u64* __restrict__ in,
                                                                  KeySel ks, const __grid_constant__ DevRing R,
                                                                  const __grid_constant__ Gadget g) {
  constexpr int n = 1 << LOGN;
  constexpr int L = 2;
  constexpr int nl = 2;
  using L0 = NttPhase<LOGN, false, 0>;
  extern __shared__ __align__(16) double pair_sm[];  // the exchange areas of two transforms
  const int tid = threadIdx.x;
  const long o = blockIdx.x;
  const int l = blockIdx.y;
  const NttTable& T = R.t[l];
  const double q = T.qd, qinv = T.qinv;
  const u64* ct = in + o * 2 * nl * n;
  const u64* K = ks.base + ((o / ks.div) % ks.mod) * ks.stride;
  double a[2][8];  // mask and body sums
#pragma unroll
  for (int v = 0; v < 8; ++v) a[0][v] = a[1][v] = 0.0;
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {  // 0: mask digits (neg_s_m rows), 1: body digits (m rows)
    double e[2][8];
    u64 x0[8], x1[8];  // all loads before the splits, whose rare branch they would wait behind
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      const u64* c = ct + (long)h * nl * n + L0::index(v, tid);
      x0[v] = c[0];
      x1[v] = c[n];
    }
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      double val = fp_scaled2(fp_from_u64(x0[v]), fp_from_u64(x1[v]), g, R);
      e[0][v] = fp_next_digit(val, g);
      e[1][v] = fp_next_digit(val, g);
    }
    __syncthreads();  // the previous transforms' reads
    fp_forward2<LOGN>(e, tid, T, pair_sm);
#pragma unroll
    for (int k = 0; k < L; ++k)
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        u64 key[8];
        ld8_nc(K + ((long)(2 * (h * L + L - 1 - k) + part) * nl + l) * n + 8 * tid, key);
#pragma unroll
        for (int v = 0; v < 8; ++v)
          a[part][v] = __dadd_rn(a[part][v], fp_mulmod(e[k][v], fp_from_u64(key[v]), q, qinv));
      }
  }
  const u64 qi = R.m[l].q;
  u64* o0 = out + (2 * o) * 2 * nl * n;
  u64* o1 = o0 + 2 * nl * n;
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    a[0][v] = fp_reduce(a[0][v], q, qinv);
    a[1][v] = fp_reduce(a[1][v], q, qinv);
  }
  __syncthreads();
  fp_inverse2<LOGN>(a, tid, T, pair_sm);
#pragma unroll
  for (int part = 0; part < 2; ++part)
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      const long at = (long)(part * nl + l) * n + L0::index(v, tid);
      const u64 ext = fp_to_u64(fp_wrap(fp_mulmod(a[part][v], T.ninv_d[LOGN], q, qinv), q));
      o0[at] = submod(ct[at], ext, qi);
      o1[at] = ext;
    }
}

// Inverse transforms of RLWEs ext ([count][2][nl][n], eval form, canonical) in
// double precision (ntt_fp.cuh), one CTA per polynomial, with the consumer's
// elementwise step folded into the stores (coefficient form, canonical):
//   INTT_STORE: out[j] = ext[j]
//   INTT_DMUX:  out[2j] = base[j] - ext[j], out[2j+1] = ext[j]  (a DMux level)
//   INTT_ADD:   out[j] = base[j] + ext[j]                       (a CRot step)
enum { INTT_STORE = 0, INTT_DMUX = 1, INTT_ADD = 2 };
template <int LOGN, int MODE>
__global__ void __launch_bounds__((1 << LOGN) / 8) k_intt_fp_epi(const u64* __restrict__ ext, const u64* base,
                                                                 u64* out, const __grid_constant__ DevRing R) {
  constexpr int n = 1 << LOGN;
  using L0 = NttPhase<LOGN, false, 0>;
  __shared__ double ssm[n];
  const int tid = threadIdx.x;
  const int nl = R.nl;
  const long seg = blockIdx.x;  // ((j * 2) + part) * nl + limb
  const int l = (int)(seg % nl);
  const NttTable& T = R.t[l];
  const double q = T.qd, qinv = T.qinv;
  u64 x[8];
  ld8(ext + seg * n + 8 * tid, x);
  double e[8];
#pragma unroll
  for (int v = 0; v < 8; ++v) e[v] = fp_from_u64(x[v]);
  fp_inverse<LOGN>(e, tid, T, ssm);
  const u64 qi = R.m[l].q;
  const long per = 2L * nl * n, j = seg / (2 * nl), at0 = (seg % (2 * nl)) * n;
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    const int c = L0::index(v, tid);
    const u64 val = fp_to_u64(fp_wrap(fp_mulmod(e[v], T.ninv_d[LOGN], q, qinv), q));
    if constexpr (MODE == INTT_STORE) {
      out[seg * n + c] = val;
    } else if constexpr (MODE == INTT_DMUX) {
      out[(2 * j) * per + at0 + c] = submod(base[j * per + at0 + c], val, qi);
      out[(2 * j + 1) * per + at0 + c] = val;
    } else {
      out[seg * n + c] = addmod(base[seg * n + c], val, qi);
    }
  }
}

// Runs k_intt_fp_epi for `count` RLWEs; false (nothing launched) when the ring
// has no double-precision transform of this degree.
template <int MODE>
static bool intt_epi(const DevRing& R, const u64* ext, const u64* base, u64* out, long count, cudaStream_t st) {
  if (!R.ntt || !ntt_fp_ok(R.t[0], R.t[R.nl - 1])) return false;
  const unsigned grid = (unsigned)(count * 2 * R.nl);
  switch (R.n) {
    case 4096: k_intt_fp_epi<12, MODE><<<grid, 512, 0, st>>>(ext, base, out, R); break;
    case 2048: k_intt_fp_epi<11, MODE><<<grid, 256, 0, st>>>(ext, base, out, R); break;
    case 1024: k_intt_fp_epi<10, MODE><<<grid, 128, 0, st>>>(ext, base, out, R); break;
    case 512: k_intt_fp_epi<9, MODE><<<grid, 64, 0, st>>>(ext, base, out, R); break;
    default: return false;
  }
  VIA_LAUNCHED();
  return true;
}

// Rings whose inverse transforms k_intt_fp_epi serves.
static bool R_fp_small(const DevRing& R) {
  return R.ntt && ntt_fp_ok(R.t[0], R.t[R.nl - 1]) && (R.n == 512 || R.n == 1024 || R.n == 2048 || R.n == 4096);
}

static bool dmux_fp_ok(const DevRing& R, const Gadget& g) {
  return R.ntt && R.nl == 2 && g.L == 2 && g.fp && ntt_fp_ok(R.t[0], R.t[1]) && (R.n == 2048 || R.n == 4096);
}

// Modulus switch (prim/switching/kernels/mod_switch.rs:59-61):
// c' = floor((c * q_dst + floor(q_src/2)) / q_src) mod q_dst, c the canonical value.
__global__ void k_mod_switch(const u64* __restrict__ in, DevRing S, u64* __restrict__ out, DevMod dst, long ncoef,
                             int n, double dQs) {
  long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= ncoef) return;
  long p = gid / n;
  int i = (int)(gid % n);
  u128 v = S.nl == 2 ? crt2(in[(p * 2) * n + i], in[(p * 2 + 1) * n + i], S) : (u128)in[p * n + i];
  u128 Qs = S.Q();
  u128 num = v * dst.q + (Qs >> 1);
  u128 r;
  if (S.nl == 1 && S.m[0].log2q >= 0)
    r = num >> S.m[0].log2q;
  else
    r = div_exact(num, Qs, dQs);
  u64 rr = (u64)r;
  out[p * n + i] = rr >= dst.q ? rr - dst.q : rr;
}

// The same from a two-prime ring in double precision: round(c q_dst / Q) is fp_scaled2's value
// with q_dst for S, an integer within 1.2 q_dst of zero. Two coefficients a
// thread. Bound by its 24 bytes a coefficient: the 67 million coefficients of 64 queries'
// rows 830 us with 128-bit divisions, 251 here
__global__ void __launch_bounds__(256) k_mod_switch_fp(const u64* __restrict__ in, const __grid_constant__ DevRing S,
                                                       const __grid_constant__ Gadget g, u64* __restrict__ out,
                                                       double q, long ncoef, int n) {
  const long gid = ((long)blockIdx.x * blockDim.x + threadIdx.x) * 2;
  if (gid >= ncoef) return;
  const long p = gid / n;
  const int i = (int)(gid - p * n);
  const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(in + (p * 2) * n + i);
  const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(in + (p * 2 + 1) * n + i);
  double v[2] = {fp_scaled2(fp_from_u64(a.x), fp_from_u64(b.x), g, S),
                 fp_scaled2(fp_from_u64(a.y), fp_from_u64(b.y), g, S)};
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    if (v[k] < 0.0) v[k] = __dadd_rn(v[k], q);
    if (v[k] < 0.0) v[k] = __dadd_rn(v[k], q);
    if (v[k] >= q) v[k] = __dadd_rn(v[k], -q);
  }
  *reinterpret_cast<ulonglong2*>(out + gid) = make_ulonglong2(fp_to_u64(v[0]), fp_to_u64(v[1]));
}

// ---------------------------------------------------------------------------
// Cascade (prim/conversion/cascade.rs + conv.rs:122-148) helpers.
// ---------------------------------------------------------------------------
// LWE [lwe][nl*(n1+1)] -> rank-n1 MLWE of degree 1: masks [lwe][idx][nl], body [lwe][nl], residues of
// the query's words (any 64 bits).
__global__ void k_lwe_to_mlwe(const u64* __restrict__ q, int n1, int nl, long nlwe, DevRing R, u64* masks, u64* body) {
  long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  long per = (long)nl * (n1 + 1);
  if (gid >= nlwe * per) return;
  long w = gid / per;
  int r = (int)(gid % per);
  if (r < nl * n1) {
    int l = r / n1, idx = r % n1;
    masks[(w * n1 + idx) * nl + l] = reduce64(q[w * per + r], R.m[l]);
  } else {
    int l = r - nl * n1;
    body[w * nl + l] = reduce64(q[w * per + r], R.m[l]);
  }
}

// Regroups a batch's query LWEs: every query's first lwe_a LWEs (its DMux
// bits), query by query, then the rest of every query. Element-wise copy.
__global__ void k_permute_lwes(const u64* __restrict__ q, long nq, long n_lwe, long lwe_a, long lwe_len,
                               u64* __restrict__ out) {
  const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= nq * n_lwe * lwe_len) return;
  const long e = gid % lwe_len, lw = gid / lwe_len;
  const long qi = lw / n_lwe, j = lw % n_lwe;
  const long dst = j < lwe_a ? qi * lwe_a + j : nq * lwe_a + qi * (n_lwe - lwe_a) + (j - lwe_a);
  out[dst * lwe_len + e] = q[gid];
}

// After the step MAC: P [lwe][RANK_IN][2][nl][N] (eval). Produces
// masks_out[lwe][j] = -(P[j].mask + P[j+R].mask) for j < R and
// bsum[lwe] = sum_idx P[idx].body.
__global__ void k_cascade_reduce(const u64* __restrict__ P, int rank_in, int N, int nl, long nlwe, DevRing R,
                                 u64* __restrict__ masks_out, u64* __restrict__ bsum) {
  const int half = rank_in / 2;
  long per = (long)nl * N;
  long items = nlwe * (half + 1) * per;
  long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= items) return;
  long w = gid / ((half + 1) * per);
  long r = gid % ((half + 1) * per);
  int j = (int)(r / per);
  int rem = (int)(r % per);
  int l = rem / N;
  u64 q = R.m[l].q;
  const u64* Pw = P + w * rank_in * 2 * per;
  if (j < half) {
    u64 a = Pw[(2L * j) * per + rem], b = Pw[(2L * (j + half)) * per + rem];
    masks_out[(w * half + j) * per + rem] = negmod(addmod(a, b, q), q);
  } else {
    u64 acc = 0;
    for (int idx = 0; idx < rank_in; ++idx) acc = addmod(acc, Pw[(2L * idx + 1) * per + rem], q);
    bsum[w * per + rem] = acc;
  }
}

// One cascade step's key switches and rank reduction in a single pass
// (conv.rs:122-148): the digits D of the R input masks are transformed at the
// input degree n_in, where the eval form of embed_at(d, 0) (d(X^2) of degree
// 2 n_in) is d's own eval form with every slot repeated (slot t of the output
// degree reads slot t/2). For every output mask j < R/2 and slot t:
//   mask_out[j] = -(sum_s D[j][s] K_j[s].mask + D[j+R/2][s] K_{j+R/2}[s].mask)
//   bsum        =   sum_idx sum_s D[idx][s] K_idx[s].body
// D: [lwe][idx][L][nl][n_in]; keys: [idx][L][2][nl][n_out]; mask_out:
// [lwe][R/2][nl][n_out]. Block = TT slots x JJ output masks (TT * JJ = 256); the
// JJ lanes' body partials are summed in shared memory. Small batches give few
// blocks: the output masks j are then also split over JB blocks (blockIdx.x =
// slot block * JB + jb). Every block adds its body partial (canonical, so at
// most JB of them sum below 2^64) into this step's region of the zeroed
// accumulator bsk: bsk[(lwe nl + l) * bsk_stride + t]. The body itself is only
// needed after the last step (k_cascade_body_final).
__global__ void __launch_bounds__(256) k_cascade_mac(const u64* __restrict__ D, const u64* __restrict__ keys, int R,
                                                     int n_in, int L, int TT, int JB, DevRing Rg,
                                                     u64* __restrict__ mask_out, u64* __restrict__ bsk,
                                                     long bsk_stride) {
  __shared__ u64 part[256];
  const int nl = Rg.nl, n_out = 2 * n_in, half = R / 2;
  const int JJ = 256 / TT;
  const int jb = blockIdx.x % JB;
  const int tl = threadIdx.x % TT, jl = threadIdx.x / TT;
  const int t = (blockIdx.x / JB) * TT + tl;
  const int l = blockIdx.y;
  const long lwe = blockIdx.z;
  const DevMod& m = Rg.m[l];
  const long dper = (long)nl * n_in, kper = (long)nl * n_out;
  const u64* Dw = D + lwe * R * L * dper + (long)l * n_in + (t >> 1);
  const u64* Kl = keys + (long)l * n_out + t;
  Acc128 ab{0, 0};
  for (int j = jl + jb * JJ; j < half; j += JJ * JB) {
    Acc128 am{0, 0};
    const u64* d0 = Dw + (long)j * L * dper;
    const u64* d1 = Dw + (long)(j + half) * L * dper;
    const u64* k0 = Kl + (long)j * L * 2 * kper;
    const u64* k1 = Kl + (long)(j + half) * L * 2 * kper;
#pragma unroll 3
    for (int s = 0; s < L; ++s) {
      const u64 a = d0[s * dper], b = d1[s * dper];
      mac128(am, a, k0[(2 * s) * kper]);
      mac128(am, b, k1[(2 * s) * kper]);
      mac128(ab, a, k0[(2 * s + 1) * kper]);
      mac128(ab, b, k1[(2 * s + 1) * kper]);
    }
    mask_out[((lwe * half + j) * nl + l) * n_out + t] = negmod(reduce128(am.hi, am.lo, m), m.q);
  }
  part[threadIdx.x] = reduce128(ab.hi, ab.lo, m);
  __syncthreads();
  if (jl == 0) {
    u64 acc = part[tl];
    for (int x = 1; x < JJ; ++x) acc = addmod(acc, part[x * TT + tl], m.q);
    if (JB == 1)
      bsk[(lwe * nl + l) * bsk_stride + t] = acc;
    else
      atomicAdd(reinterpret_cast<unsigned long long*>(bsk + (lwe * nl + l) * bsk_stride + t),
                (unsigned long long)acc);
  }
}

// k_cascade_mac in double precision (ntt_fp.cuh): D holds the digits' signed
// double transforms (ntt_forward_i8_fp, below 2^48), keys the cascade
// key as exact doubles (below q). Every product is reduced to within 0.5625 q,
// so a mask's 2 L products stay below 1.125 L q; the body partial is brought
// back within q/2 after each output mask's 2 L products. Outputs as k_cascade_mac.
// I8 (the first step, n_in = 1): the digits are read as the signed bytes of
// k_decompose_i8, [lwe][idx][L], whose transform at degree 1 is the digit itself.
//
// A thread takes NS output slots (two: those of one input slot, which share its digits, with
// 16-byte key loads) for NL LWEs (which share the keys). TP threads along the slots x JJ
// output masks = 256. FP64-issue and load bound: with NS = NL = 2, 4 + 2 NL loads feed 8 NL
// products of 7 operations, where one slot and LWE a thread loaded 6 words for 4; a late
// step of 2688 LWEs 885 -> 644 us.
template <bool I8, int NL, int NS>
__global__ void __launch_bounds__(256, 2) k_cascade_mac_fp(const double* __restrict__ D, const int8_t* __restrict__ D8,
                                                        const double* __restrict__ keys, int R, int n_in, int L,
                                                        int TP, int JB, long nlwe, const __grid_constant__ DevRing Rg,
                                                        u64* __restrict__ mask_out, u64* __restrict__ bsk,
                                                        long bsk_stride) {
  __shared__ u64 part[NL][NS][256];
  const int nl = Rg.nl, n_out = 2 * n_in, half = R / 2;
  const int JJ = 256 / TP;
  const int jb = blockIdx.x % JB;
  const int tl = threadIdx.x % TP, jl = threadIdx.x / TP;
  const int t = ((blockIdx.x / JB) * TP + tl) * NS;  // first output slot
  const int u = t >> 1;                              // its input slot
  const int l = blockIdx.y;
  const DevMod& m = Rg.m[l];
  const double q = Rg.t[l].qd, qinv = Rg.t[l].qinv;
  const long dper = (long)nl * n_in, kper = (long)nl * n_out;
  long lwe[NL];  // past the end: the last LWE again, not stored
#pragma unroll
  for (int x = 0; x < NL; ++x) lwe[x] = min((long)blockIdx.z * NL + x, nlwe - 1);
  const double* Kl = keys + (long)l * n_out + t;
  double ab[NL][NS];
#pragma unroll
  for (int x = 0; x < NL; ++x)
#pragma unroll
    for (int h = 0; h < NS; ++h) ab[x][h] = 0.0;
  for (int j = jl + jb * JJ; j < half; j += JJ * JB) {
    double am[NL][NS];
#pragma unroll
    for (int x = 0; x < NL; ++x)
#pragma unroll
      for (int h = 0; h < NS; ++h) am[x][h] = 0.0;
#pragma unroll 1
    for (int i = 0; i < 2; ++i) {  // input masks j, j + half
      const int idx = j + i * half;
      const double* k = Kl + (long)idx * L * 2 * kper;
      const double* d[NL];
      const int8_t* e[NL];
#pragma unroll
      for (int x = 0; x < NL; ++x) {
        d[x] = D + ((lwe[x] * R + idx) * L) * dper + (long)l * n_in + u;
        e[x] = D8 + (lwe[x] * R + idx) * L;
      }
#pragma unroll(NS * NL == 1 ? 9 : 6)
      for (int s = 0; s < L; ++s) {
        double km[NS], kb[NS];
        ld_slots<NS, double2>(k + (2 * s) * kper, km);
        ld_slots<NS, double2>(k + (2 * s + 1) * kper, kb);
#pragma unroll
        for (int x = 0; x < NL; ++x) {
          const double a = I8 ? (double)e[x][s] : d[x][s * dper];
#pragma unroll
          for (int h = 0; h < NS; ++h) {
            am[x][h] = __dadd_rn(am[x][h], fp_mulmod(a, km[h], q, qinv));
            ab[x][h] = __dadd_rn(ab[x][h], fp_mulmod(a, kb[h], q, qinv));
          }
        }
      }
    }
#pragma unroll
    for (int x = 0; x < NL; ++x) {
      u64 out[NS];
#pragma unroll
      for (int h = 0; h < NS; ++h) {
        out[h] = negmod(fp_to_u64(fp_canonical(am[x][h], q, qinv)), m.q);
        ab[x][h] = fp_reduce(ab[x][h], q, qinv);
      }
      if ((long)blockIdx.z * NL + x < nlwe) st_slots(mask_out + ((lwe[x] * half + j) * nl + l) * n_out + t, out);
    }
  }
#pragma unroll
  for (int x = 0; x < NL; ++x)
#pragma unroll
    for (int h = 0; h < NS; ++h) part[x][h][threadIdx.x] = fp_to_u64(fp_canonical(ab[x][h], q, qinv));
  __syncthreads();
  if (jl == 0) {
#pragma unroll
    for (int x = 0; x < NL; ++x) {
      if ((long)blockIdx.z * NL + x >= nlwe) continue;
#pragma unroll
      for (int h = 0; h < NS; ++h) {
        u64 acc = part[x][h][tl];
        for (int y = 1; y < JJ; ++y) acc = addmod(acc, part[x][h][y * TP + tl], m.q);
        u64* o = bsk + (lwe[x] * nl + l) * bsk_stride + t + h;
        if (JB == 1)
          *o = acc;
        else
          atomicAdd(reinterpret_cast<unsigned long long*>(o), (unsigned long long)acc);
      }
    }
  }
}

// The cascade's final body in the eval domain, [lwe][nl][n1] (n1 = 2^K). Step k
// (output degree 2^(k+1)) maps body to embed_at(body, 0) - bsum_k, and the eval
// form of embed_at repeats every slot, so the steps from k0 on give
//   body[t] = b - sum_k bsum_k[t >> (K - 1 - k)]
// with b the LWE body (the degree-1 body, b0[lwe * b0_stride + l]) and bsum_k the step's
// accumulated sums, bsk[(lwe nl + l) * 2 n1 + 2^(k+1) - 2 + slot]. The steps before
// k0 (the GEMM steps) leave their sums in coefficient form (k_pack_rlwe).
__global__ void k_cascade_body_final(const u64* __restrict__ b0, long b0_stride, const u64* __restrict__ bsk, int k0,
                                     int K, int nl, long nlwe, DevRing Rg, u64* __restrict__ body) {
  const int n1 = 1 << K;
  const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= nlwe * nl * n1) return;
  const long ll = gid / n1;  // lwe * nl + l
  const int t = (int)(gid % n1), l = (int)(ll % nl);
  const DevMod& m = Rg.m[l];
  const u64* sk = bsk + ll * 2 * n1;
  u64 acc = 0;
  for (int k = k0; k < K; ++k) acc = addmod(acc, reduce64(sk[(2 << k) - 2 + (t >> (K - 1 - k))], m), m.q);
  body[gid] = submod(reduce64(b0[ll / nl * b0_stride + l], m), acc, m.q);  // the caller's word after GEMM steps
}

// body_out[lwe] = embed_at(body_in[lwe], N_out, 0) - bsum[lwe] (coefficient form).
__global__ void k_cascade_body(const u64* __restrict__ body_in, const u64* __restrict__ bsum, int n_in, int nl,
                               long nlwe, DevRing R, u64* __restrict__ body_out) {
  const int n_out = 2 * n_in;
  long per = (long)nl * n_out;
  long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= nlwe * per) return;
  long w = gid / per;
  int rem = (int)(gid % per);
  int l = rem / n_out, t = rem % n_out;
  u64 q = R.m[l].q;
  u64 e = (t & 1) ? 0 : body_in[(w * nl + l) * n_in + t / 2];
  body_out[w * per + rem] = submod(e, bsum[w * per + rem], q);
}

// Assemble cascade outputs into RLWEs [lwe][2][nl][n1]. The first k0 steps' body sums
// are in coefficient form (cascade_tc.cuh: gemm[((2^(k+1) - 2 + c) * 2 + l) * stride + lwe],
// pointing at the first of these LWEs): step k's coefficient c sits at coefficient
// c n1 / 2^(k+1).
__global__ void k_pack_rlwe(const u64* masks, const u64* body, const u64* __restrict__ gemm, long stride, int k0, int K,
                            long nlwe, int n1, int nl, DevRing Rg, u64* out) {
  long per = (long)nl * n1;
  long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= nlwe * per) return;
  long w = gid / per;
  int rem = (int)(gid % per);
  out[(2 * w) * per + rem] = masks[w * per + rem];
  u64 b = body[w * per + rem];
  const int l = rem / n1, i = rem % n1;
  for (int k = k0 - 1; k >= 0 && (i & ((1 << (K - 1 - k)) - 1)) == 0; --k) {
    const DevMod& m = Rg.m[l];
    b = submod(b, reduce64(gemm[(long)(((2 << k) - 2 + (i >> (K - 1 - k))) * 2 + l) * stride + w], m), m.q);
  }
  out[(2 * w + 1) * per + rem] = b;
}

// The cascade's RLWEs [lwe][2][nl][n1] in one kernel for double-precision rings (both primes
// below 2^40): per CTA (LWE, limb) the eval-form body of k_cascade_body_final, its inverse
// transform, the GEMM steps' sums of k_pack_rlwe, and the mask. Arguments as theirs; the GEMM
// steps' sums are loaded by one thread a coefficient that has any, all loads at once, while the
// transform has its own to wait for (one after the other in the epilogue 338 us of the 360 below
// stayed). 2688 LWEs of degree 2048 in 2 launches 360 us as three kernels (eval body, transform,
// assembly), 155 here: 64 KB in and 64 KB out an LWE at 2.3 TB/s, 35% of the copy bandwidth, as every
// CTA is a chain of loads, one transform and stores; 60 LWEs 27 us before, 16 here; 8 LWEs 15 and 9.5.
template <int LOGN>
__global__ void __launch_bounds__((1 << LOGN) / 8)
    k_cascade_rlwe_fp(const u64* __restrict__ masks, const u64* __restrict__ b0, long b0_stride,
                      const u64* __restrict__ bsk, const u64* __restrict__ gemm, long stride, int k0,
                      u64* __restrict__ out, const __grid_constant__ DevRing R) {
  constexpr int n = 1 << LOGN, K = LOGN;
  using L0 = NttPhase<LOGN, false, 0>;
  __shared__ double ssm[n];
  __shared__ u64 gsum[1 << 8];  // the GEMM steps' sums at the coefficients x << (K - k0)
  const int tid = threadIdx.x, nl = R.nl, l = blockIdx.y;
  const long w = blockIdx.x, per = (long)nl * n;
  const NttTable& T = R.t[l];
  const double q = T.qd, qinv = T.qinv;
  const DevMod& m = R.m[l];
  fp_prefetch_twiddles<LOGN>(tid, T);
  if (tid < (1 << k0)) {  // at most 8 sums below 2^49 each, all loads at once
    u64 s = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k < k0 && (tid & ((1 << (k0 - 1 - k)) - 1)) == 0)
        s += gemm[(long)(((2 << k) - 2 + (tid >> (k0 - 1 - k))) * 2 + l) * stride + w];
    gsum[tid] = reduce64(s, m);
  }
  const u64* sk = bsk + (w * nl + l) * 2 * n;
  const double b = fp_from_u64(reduce64(b0[w * b0_stride + l], m));  // the caller's word: any 64 bits
  double e[8];
#pragma unroll
  for (int v = 0; v < 8; ++v) e[v] = 0.0;
#pragma unroll 4
  for (int k = k0; k < K; ++k) {  // sums of at most 2^4 canonical terms each, below 2^44
    const u64* s = sk + (2 << k) - 2;
#pragma unroll
    for (int v = 0; v < 8; ++v) e[v] = __dadd_rn(e[v], fp_from_u64(s[(8 * tid + v) >> (K - 1 - k)]));
  }
#pragma unroll
  for (int v = 0; v < 8; ++v) e[v] = fp_reduce(__dadd_rn(b, -e[v]), q, qinv);
  fp_inverse<LOGN>(e, tid, T, ssm);  // its CTA barrier also publishes gsum
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    const int x = L0::index(v, tid);
    u64 c = fp_to_u64(fp_wrap(fp_mulmod(e[v], T.ninv_d[LOGN], q, qinv), q));
    if (k0 && (x & ((1 << (K - k0)) - 1)) == 0) c = submod(c, gsum[x >> (K - k0)], m.q);
    out[(2 * w + 1) * per + (long)l * n + x] = c;
    out[(2 * w) * per + (long)l * n + x] = masks[w * per + (long)l * n + x];
  }
}

// rlwe_to_rgsw assembly (prim/gates/convert.rs:162-178): for bit b, level i:
// neg_s_m[i] = (rlwe_i.body + gp_i.mask, gp_i.body), m[i] = rlwe_i.
// rlwe: [bits*L][2][nl][n]; gp: same shape; rgsw: [bits][2L][2][nl][n].
__global__ void k_assemble_rgsw(const u64* rlwe, const u64* gp, int L, long bits, int n, int nl, DevRing R, u64* rgsw) {
  long per = (long)nl * n;
  long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= bits * L * 2 * per) return;
  long w = gid / (2 * per);  // rlwe index = bit*L + i
  int rem = (int)(gid % (2 * per));
  int mb = rem / per;
  int r2 = rem % per;
  int l = r2 / n;
  long b = w / L;
  int i = (int)(w % L);
  u64 q = R.m[l].q;
  u64* dst_nsm = rgsw + ((b * 2 * L + i) * 2 + mb) * per + r2;
  u64* dst_m = rgsw + ((b * 2 * L + L + i) * 2 + mb) * per + r2;
  u64 g = gp[(2 * w + mb) * per + r2];
  if (mb == 0)
    *dst_nsm = addmod(rlwe[(2 * w + 1) * per + r2], g, q);
  else
    *dst_nsm = g;
  *dst_m = rlwe[(2 * w + mb) * per + r2];
}

// ---------------------------------------------------------------------------
// Host-side orchestration.
// ---------------------------------------------------------------------------
static inline unsigned blocks(long items, int threads = 256) { return (unsigned)((items + threads - 1) / threads); }

struct Workspace {
  long nlwe = 0, nbits = 0;  // per query
  int bmax = 1;              // queries the buffers are sized for
  // Cascade.
  DevBuf c_masks_a, c_masks_b, c_body_a, c_body_b, c_digits, c_P, c_bsum, c_rlwe;
  std::shared_ptr<const CtKeys> ct;  // the GEMM steps' keys (cascade_tc.cuh), null: none
  DevBuf c_gemm_body;                // their body sums
  DevBuf c_dig8;   // 8-bit cascade / conversion-key digits [lwe][n1 * L_CK] bytes (base <= 255)
  // RLWE -> RGSW.
  // RGSWs grouped by use: the DMux bits of every query ([q][nd]), then the
  // CMux and CRot bits ([q][nbits - nd]), each [2L][2][nl][n1] at q1.
  DevBuf g_digits, g_gp, rgsw_q1;
  DevBuf rgsw_q2;  // the same layout switched to q2: [2L][2][n1] per bit
  DevBuf q_perm;   // a batch's query LWEs in that grouped order (batches of two or more)
  // DMux.
  DevBuf dm_a, dm_b, dm_digits, dm_ext;
  // FirstDim / CMux.
  DevBuf sel, sel_bytes, fd_out, cm_diff, cm_digits, cm_ext, cm_b;
  // CRot / RespComp.
  DevBuf cr_ct, cr_diff, cr_digits, cr_ext, rs_ct3, rs_mproj, rs_bproj, rs_digits, rs_gp, rs_acc;
  Gadget g_ck, g_dmux, g_cmux, g_rsk;
  // Staging for the captured answer graphs: queries in, answers out.
  DevBuf q_in, a_mask, a_body;
  std::vector<std::pair<int, cudaGraphExec_t>> graphs;  // one per batch size
  std::vector<std::pair<int, unsigned long long>> graph_kernels;
  std::unique_ptr<struct RepackWs> repack;  // VIA-B buffers, made on the first batch answer
  cudaStream_t capture = nullptr;           // stream the answer graphs are captured on
  int graphs_gen = 0;                       // Server::plan_gen the graphs were captured under
  // A one-query answer expands its CMux / CRot bits on `side`, concurrently with
  // the DMux tree and the database scan on the answer's stream (fork / join).
  cudaStream_t side = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  ~Workspace() {
    for (auto& g : graphs) cudaGraphExecDestroy(g.second);
    if (capture) cudaStreamDestroy(capture);
    if (side) cudaStreamDestroy(side);
    if (ev_fork) cudaEventDestroy(ev_fork);
    if (ev_join) cudaEventDestroy(ev_join);
  }
};

void WorkspaceDeleter::operator()(Workspace* w) const { delete w; }
void workspace_destroy(Server& s) { s.ws.reset(); }
uint8_t* workspace_sel_bytes(Server& s) { return reinterpret_cast<uint8_t*>(s.ws->sel_bytes.p); }

void first_dim_queries(Server& s, const u64* sel_eval, u64* out_eval, int nq, uint8_t* scratch, cudaStream_t st,
                       bool tiled) {
  const via_params& p = s.prm;
  if (s.tensor_fd()) {
    fd_scan(s.fd, sel_eval, out_eval, nq, scratch, st, nullptr, tiled);
    return;
  }
  for (int q = 0; q < nq; ++q)
    first_dim_schoolbook(s.db->p, sel_eval + (size_t)q * p.num_rows * 2 * p.n1, out_eval + (size_t)q * p.num_cols * 2 * p.n1,
                         (int)p.num_rows, (int)p.num_cols, (int)p.n1, s.r2.m[0], st);
}

static bool cmux_fused_ok(const DevRing& R, const Gadget& g);

// Levels of at most this many CMuxes run on four-CTA clusters (cmux_fused).
constexpr long CMUX_CLUSTER_MAX = 64;
// DMux levels of at most this many coefficients (products x degree) run on a cluster per product
// and limb: 32 products of degree 2048 14.2 us against 15.8 us for one CTA each (k_dmux_fp); of
// degree 4096, whose CTAs fill an SM, 33.0 against 27.3.
constexpr long EXT_CLUSTER_MAX = 65536;

// Whether the scan of nq queries writes tiled columns, which the CMux tree's first level
// gathers: answers with the fused CMux and a first level of single-CTA CMuxes.
bool cmux_takes_tiles(Server& s, long nq) {
  const via_params& p = s.prm;
  return s.tensor_fd() && p.num_cols >= 2 && nq * (long)p.num_cols / 2 > CMUX_CLUSTER_MAX &&
         cmux_fused_ok(s.r2, make_gadget(p.b_cmux, (int)p.l_query, s.r2));
}

// Times every candidate scan tile for nq queries on the handle's workspace
// buffers (the workspace must hold batches of nq).
std::vector<FdTuneResult> workspace_measure_tiles(Server& s, Workspace& w, int nq, int reps) {
  if (w.bmax < nq) throw CudaError(100, "workspace smaller than the batch to tune");
  return fd_measure_tiles(s.fd, nq, w.sel.p, w.fd_out.p, reinterpret_cast<uint8_t*>(w.sel_bytes.p), s.stream, reps,
                          cmux_takes_tiles(s, nq));
}

// Allocates a workspace for batches of up to bmax queries, or (count_only)
// returns the bytes it would take.
static size_t workspace_build(Server& s, int bmax, Workspace* w, bool count_only) {
  const via_params& p = s.prm;
  size_t bytes = 0;
  auto A = [&](DevBuf& b, long count) {
    bytes += (size_t)std::max(0L, count) * 8;
    if (!count_only) b.alloc((size_t)std::max(0L, count));
  };
  const long n1 = p.n1, n2 = p.n2, nl = s.r1.nl, L = p.l_query, Lck = p.l_ck, I = p.num_rows, J = p.num_cols;
  const long B = std::max(1, bmax);
  w->bmax = (int)B;
  w->nlwe = (long)query_lwes(p);
  w->nbits = w->nlwe / L;
  const long nlwe = w->nlwe * B;  // LWEs of a full batch
  A(w->c_masks_a, nlwe * n1 * nl);
  A(w->c_masks_b, nlwe * n1 * nl);
  A(w->c_body_a, nlwe * n1 * nl);
  A(w->c_body_b, nlwe * n1 * nl);
  // NTT rings transform the cascade digits at the input degree (half of the
  // embedded degree); the other rings use the embedded digits and the P buffer.
  // The GEMM steps' two digit buffers lie in the same memory.
  w->ct = std::atomic_load(&s.ct);
  const long tc_words = w->ct ? 2 * (long)(ct_digit_bytes((int)n1) / 8) * ((nlwe + 7) / 8 * 8) : 0;
  A(w->c_digits, std::max(nlwe * (s.r1.ntt ? 1 : 2) * n1 * Lck * nl, tc_words));
  A(w->c_P, s.r1.ntt ? 0 : nlwe * 2 * n1 * 2 * nl);
  A(w->c_bsum, 2 * nlwe * n1 * nl);
  A(w->c_gemm_body, w->ct ? (long)ct_body_words(w->ct->steps) * nlwe : 0);
  A(w->c_dig8, p.ck_base <= 255 && s.r1.ntt ? (nlwe * n1 * Lck + 7) / 8 : 0);
  A(w->c_rlwe, nlwe * 2 * n1 * nl);
  A(w->g_digits, nlwe * Lck * nl * n1);
  A(w->g_gp, nlwe * 2 * nl * n1);
  A(w->rgsw_q1, B * w->nbits * 2 * L * 2 * nl * n1);
  A(w->rgsw_q2, B * w->nbits * 2 * L * 2 * n1);
  A(w->dm_a, B * I * 2 * nl * n1);
  A(w->dm_b, B * I * 2 * nl * n1);
  A(w->dm_digits, B * std::max(1L, I / 2) * 2 * L * nl * n1);
  A(w->dm_ext, B * std::max(1L, I / 2) * 2 * nl * n1);
  A(w->sel, B * I * 2 * n1);
  if (s.tensor_fd()) {
    size_t bytes = 0;  // the split selection grows with the batch; size it for every batch up to B
    for (int nq = 1; nq <= B; ++nq) bytes = std::max(bytes, fd_sel_bytes(s.fd, nq));
    A(w->sel_bytes, (bytes + 7) / 8);
  }
  A(w->fd_out, B * (s.tensor_fd() ? (long)s.fd.J_pad : J) * 2 * n1);  // tiled columns come in whole tiles
  const bool fused = cmux_fused_ok(s.r2, make_gadget(p.b_cmux, (int)p.l_query, s.r2));
  A(w->cm_diff, fused ? 0 : B * std::max(1L, J / 2) * 2 * n1);
  A(w->cm_digits, fused ? 0 : B * std::max(1L, J / 2) * 2 * L * n1);
  A(w->cm_ext, fused ? 0 : B * std::max(1L, J / 2) * 2 * n1);
  A(w->cm_b, B * std::max(1L, J / 2) * 2 * n1);
  A(w->cr_ct, B * 2 * n1);
  A(w->cr_diff, B * 2 * n1);
  A(w->cr_digits, B * 2 * L * n1);
  A(w->cr_ext, B * 2 * n1);
  A(w->rs_ct3, B * 2 * n1);
  long d = n1 / n2;
  A(w->rs_mproj, B * d * n2);
  A(w->rs_bproj, B * n2);
  A(w->rs_digits, B * d * p.l_rsk * n2);
  A(w->rs_gp, B * d * 2 * n2);
  A(w->rs_acc, B * 2 * n2);
  A(w->q_in, nlwe * lwe_len(p));
  A(w->q_perm, B > 1 ? nlwe * (long)lwe_len(p) : 0);
  A(w->a_mask, B * n2);
  A(w->a_body, B * n2);
  if (count_only) return bytes;
  w->g_ck = make_gadget(p.ck_base, (int)p.l_ck, s.r1);
  w->g_dmux = make_gadget(p.b_dmux, (int)p.l_query, s.r1);
  w->g_cmux = make_gadget(p.b_cmux, (int)p.l_query, s.r2);
  w->g_rsk = make_gadget(p.b_rsk, (int)p.l_rsk, s.r3);
  return bytes;
}

std::unique_ptr<Workspace, WorkspaceDeleter> workspace_make(Server& s, int bmax) {
  std::unique_ptr<Workspace, WorkspaceDeleter> w(new Workspace());
  bool built = true;
  try {
    workspace_build(s, bmax, w.get(), false);
  } catch (const CudaError& e) {
    if (e.status != 101) throw;
    w.reset(new Workspace());
    const size_t need = workspace_bytes(s, bmax) + ((size_t)96 << 20);  // about 48 allocations in pieces of 2 MiB
    size_t avail = 0, total = 0;
    VIA_CUDA(cudaMemGetInfo(&avail, &total));
    const std::shared_ptr<const CtKeys> ct = std::atomic_load(&s.ct);
    if (!ct || ct.use_count() > 2 || avail + ct->planes.n * 8 < need) throw;  // 2: the handle's and this one
    std::atomic_store(&s.ct, std::shared_ptr<const CtKeys>());
    built = false;
  }
  if (!built) workspace_build(s, bmax, w.get(), false);
  // The answer's own kernels go before the side stream's, which have until the CMux tree: five
  // queries at 64 x 1024 reached the scan after 950 us when both groups' cascades shared the
  // SMs evenly, and after 787 us this way (1390 -> 1340 us an answer). A graph's kernels keep the
  // priority of the stream they were captured on, whatever stream it is launched on.
  const StreamPriorities prio = stream_priorities();
  VIA_CUDA(cudaStreamCreateWithPriority(&w->capture, cudaStreamNonBlocking, prio.answer));
  VIA_CUDA(cudaStreamCreateWithPriority(&w->side, cudaStreamNonBlocking, prio.side));
  VIA_CUDA(cudaEventCreateWithFlags(&w->ev_fork, cudaEventDisableTiming));
  VIA_CUDA(cudaEventCreateWithFlags(&w->ev_join, cudaEventDisableTiming));
  return w;
}

size_t workspace_bytes(Server& s, int bmax) {
  Workspace scratch;
  return workspace_build(s, bmax, &scratch, true);
}

void workspace_create(Server& s, int bmax) { s.ws = workspace_make(s, bmax); }


int workspace_batch(Server& s) { return s.ws ? s.ws->bmax : 0; }

static void to_eval(const DevRing& R, u64* data, int n, long segments, cudaStream_t st) {
  if (R.ntt) ntt_forward(data, n, R.nl, segments, R.t[0], R.t[1], st);
}
// Eval form of gadget digits: the lazy forward transform, whose outputs are below 2 q on doubles
// (primes below 2^44, what k_mac_fp wants) and below (1 + 2 log2 n) q in integers; k_mac_ntt adds at
// most a few dozen products with key residues below q into 128-bit sums.
static void digits_to_eval(const DevRing& R, u64* data, int n, long segments, cudaStream_t st) {
  if (R.ntt) ntt_forward_lazy(data, n, R.nl, segments, R.t[0], R.t[1], st);
}
static void from_eval(const DevRing& R, u64* data, int n, long segments, cudaStream_t st) {
  if (R.ntt) ntt_inverse(data, n, R.nl, segments, R.t[0], R.t[1], st);
}

// Gadget products of `nout` outputs with T digit polys each (already in the eval
// domain) against keys: out eval [nout][2][nl][n].
static void mac(const DevRing& R, const u64* D, KeySel ks, u64* out, int T, int n, long nout, cudaStream_t st) {
  long items = nout * R.nl * n;
  // Two slots a thread where the buffers allow it (a primitive's caller may pass any 8-byte
  // address) and the grid stays wide: the 16 LWEs of one query's DMux bits took 8.2 us with one
  // slot a thread, 9.6 us with two.
  const bool wide = items / 512 >= 2 * 148 && (((uintptr_t)out | (uintptr_t)D | (uintptr_t)ks.base) & 15) == 0;
  const bool fp = R.ntt && ntt_fp_ok(R.t[0], R.t[R.nl - 1]) && T <= 128;
  if (fp && wide)
    k_mac_fp<2><<<blocks(items / 2), 256, 0, st>>>(D, ks, out, T, n, R.nl, nout, R);
  else if (fp)
    k_mac_fp<1><<<blocks(items), 256, 0, st>>>(D, ks, out, T, n, R.nl, nout, R);
  else if (R.ntt)
    k_mac_ntt<<<blocks(items), 256, 0, st>>>(D, ks, out, T, n, R.nl, nout, R);
  else
    k_mac_schoolbook<<<blocks(items), 256, 0, st>>>(D, ks, out, T, n, R.nl, nout, R);
  VIA_LAUNCHED();
}

static void decompose(const DevRing& R, const Gadget& g, const u64* in, int n_in, int stride, long npolys, u64* out,
                      cudaStream_t st) {
  k_decompose<<<blocks(npolys * n_in, 128), 128, 0, st>>>(in, n_in, stride, npolys, R, g, out);
  VIA_LAUNCHED();
}

static bool shared_key_fp(const DevRing& R, const int8_t* dig8, const u64* key, const u64* bodies, int L, long count,
                          u64* out, cudaStream_t st);

// Signed byte digits (bases up to 255); `in` is a 16-byte aligned buffer of canonical residues.
static void decompose_i8(const DevRing& R, const Gadget& g, const u64* in, int n_in, long npolys, int8_t* out,
                         cudaStream_t st) {
  if (n_in >= 4 && ct_digits_ok(g.base, (u32)g.L, R))
    k_ct_decompose<<<blocks(npolys * n_in / 4, 128), 128, 0, st>>>(in, n_in, npolys, ct_digits(g.base, R), out);
  else
    k_decompose_i8<<<blocks(npolys * n_in, 128), 128, 0, st>>>(in, n_in, npolys, R, g, out);
  VIA_LAUNCHED();
}

// Gadget products of `nout` outputs, each summing G decomposed input polys
// against its eval-form key samples: decompose -> transform -> multiply-accumulate
// through the `digits` scratch ([nout][G][L][nl][n]).
static void gadget_product(const DevRing& R, const Gadget& g, const u64* in, int n, int stride, int G, long nout,
                           KeySel ks, u64* out, u64* digits, cudaStream_t st) {
  decompose(R, g, in, n / stride, stride, (long)G * nout, digits, st);
  digits_to_eval(R, digits, n, (long)G * nout * g.L * R.nl, st);
  mac(R, digits, ks, out, G * g.L, n, nout, st);
}

static double to_double(u128 x) { return (double)(u64)(x >> 64) * 18446744073709551616.0 + (double)(u64)x; }

static void mod_switch(const DevRing& S, const u64* in, const DevRing& D, u64* out, long npolys, int n, cudaStream_t st) {
  long nco = npolys * n;
  // Odd primes below 2^44, a target below 2^40 and rounding ties that cannot happen.
  if (S.ntt && S.nl == 2 && ntt_fp_ok(S.t[0], S.t[1]) && D.m[0].q < (1ull << 40) && n % 2 == 0) {
    Gadget g{};
    g.dS = (double)D.m[0].q;
    g.ys[0] = (double)h_inv(S.m[1].q % S.m[0].q, S.m[0].q);
    g.ys[1] = (double)h_inv(S.m[0].q % S.m[1].q, S.m[1].q);
    k_mod_switch_fp<<<blocks(nco / 2), 256, 0, st>>>(in, S, g, out, (double)D.m[0].q, nco, n);
    VIA_LAUNCHED();
    return;
  }
  k_mod_switch<<<blocks(nco), 256, 0, st>>>(in, S, out, D.m[0], nco, n, to_double(S.Q()));
  VIA_LAUNCHED();
}

// Step 1: QueryDecomp (query_decomp.rs:39-95) of `nlwe` consecutive LWEs, the
// first being LWE lwe0 of the nlwe_all in the workspace (LWE-indexed buffers are used from that
// LWE's region on), forming the RGSWs of `nbits` query bits starting at bit
// bit0 -> rgsw_q1 [bit][2L][2][nl][n1] (coefficient form). Disjoint (lwe0,
// nlwe) ranges may run concurrently on different streams. Servers with GEMM
// steps (cascade_tc.cuh) have run those for every LWE (cascade_gemm): the
// cascade continues from their digits and body sums.
static void cascade_gemm(Server& s, Workspace& w, const u64* d_query, long nlwe, cudaStream_t st) {
  const long n1 = s.prm.n1;
  u64* body = w.c_gemm_body.p;
  uint8_t* da = reinterpret_cast<uint8_t*>(w.c_digits.p);
  uint8_t* db = da + ct_digit_bytes((int)n1) * ((nlwe + 7) / 8 * 8);
  VIA_CUDA(cudaMemsetAsync(body, 0, ct_body_words(ct_steps_for(w.ct->steps, nlwe)) * nlwe * 8, st));
  ct_run(s, *w.ct, d_query, nlwe, da, db, reinterpret_cast<int8_t*>(w.c_dig8.p), body, st);
}

static void query_decomp_range(Server& s, Workspace& w, const u64* d_query, long nlwe_all, long lwe0, long nlwe,
                               long bit0, long nbits, cudaStream_t st) {
  const via_params& p = s.prm;
  const DevRing& R = s.r1;
  const int n1 = p.n1, nl = R.nl, L = p.l_ck;
  const long lwe_n = (long)n1 * nl;  // per-LWE region of the mask / body / bsum buffers
  const long rgsw1 = 2L * p.l_query * 2 * nl * n1;
  u64 *mi = w.c_masks_a.p + lwe0 * lwe_n, *mo = w.c_masks_b.p + lwe0 * lwe_n;
  u64 *bi = w.c_body_a.p + lwe0 * lwe_n, *bo = w.c_body_b.p + lwe0 * lwe_n;
  u64* digits = w.c_digits.p + lwe0 * (R.ntt ? 1 : 2) * n1 * L * nl;
  u64* cP = R.ntt ? nullptr : w.c_P.p + lwe0 * 2 * n1 * 2 * nl;
  u64* bsum = w.c_bsum.p + lwe0 * lwe_n;
  // Eval rings: every step's body sums, [lwe][nl][2 n1] (step regions of 2, 4, .. n1).
  u64* bsk = w.c_bsum.p + lwe0 * 2 * lwe_n;
  u64* rlwe = w.c_rlwe.p + lwe0 * 2 * lwe_n;
  // Bases up to 255: digits as bytes, lifted and transformed by the 8-bit NTT.
  int8_t* dig8 = w.c_dig8.p ? reinterpret_cast<int8_t*>(w.c_dig8.p) + lwe0 * (long)n1 * L : nullptr;
  const int k0 = w.ct ? ct_steps_for(w.ct->steps, nlwe_all) : 0;  // steps already run as GEMMs
  const u64* query = d_query + lwe0 * (long)lwe_len(p);
  if (!k0) {
    k_lwe_to_mlwe<<<blocks(nlwe * nl * (n1 + 1)), 256, 0, st>>>(query, n1, nl, nlwe, R, mi, bi);
    VIA_LAUNCHED();
  }
  // Eval rings: how a step of input degree n_in spreads over the grid.
  const bool fp_mac = dig8 && s.cascade_eval_d.p;
  struct Split {
    int NS, NL, tt, JB;
    long slots, lwes;
  };
  const auto split = [&](int n_in) {
    const int n_out = 2 * n_in, rank_in = n1 / n_in;
    // fp: two output slots a thread from three blocks a SM on (with one: 60 LWEs 26 us a
    // step against 21, 18 LWEs 8.3 against 10.2), two LWEs as well from sixteen on.
    const long full = (long)n1 * nl * nlwe / 256;  // blocks with one slot and LWE a thread
    Split d;
    d.NS = fp_mac && n_in > 1 && full >= 3 * 148 ? 2 : 1;
    d.NL = d.NS == 2 && full >= 16 * 148 ? 2 : 1;
    const int jj = std::min(rank_in / 2, 8);
    d.tt = std::min(n_out / d.NS, 256 / jj);
    d.slots = n_out / d.NS / d.tt;
    // Split the output masks over JB blocks while the grid is below ~4 blocks
    // per SM and every block keeps at least one mask per thread row.
    d.lwes = (nlwe + d.NL - 1) / d.NL;
    const long base = d.slots * nl * d.lwes;
    const int rows = 256 / d.tt, iters = (rank_in / 2 + rows - 1) / rows;
    d.JB = 1;
    while (d.JB * 2 <= iters && base * d.JB * 2 <= CASCADE_SPLIT_BLOCKS) d.JB *= 2;
    return d;
  };
  // Blocks that share a step's body sums add to them; a step of one block a sum stores it (the
  // 134 MB of 2048 LWEs 315 us to clear).
  bool shared_sums = false;
  for (int n_in = 1 << k0; R.ntt && n_in < n1; n_in <<= 1) shared_sums |= split(n_in).JB > 1;
  if (shared_sums) VIA_CUDA(cudaMemsetAsync(bsk, 0, (size_t)nlwe * 2 * lwe_n * 8, st));
  const u64 step_len = (u64)2 * n1 * L * 2 * nl;
  int k = k0;
  for (int n_in = 1 << k0; n_in < n1; n_in <<= 1, ++k) {
    const int n_out = 2 * n_in, rank_in = n1 / n_in;
    const long polys = nlwe * rank_in;
    if (R.ntt) {
      // Digits at the input degree; see k_cascade_mac for the repeated slots.
      if (dig8 && (n_in > 1 || fp_mac)) {
        if (k != k0 || k0 == 0) {  // the last GEMM step left its successor's digits in dig8
          decompose_i8(R, w.g_ck, mi, n_in, polys, dig8, st);
        }
        if (n_in == 1)
          ;  // degree 1: the MAC reads the digits themselves
        else if (fp_mac)
          ntt_forward_i8_fp(dig8, reinterpret_cast<double*>(digits), n_in, nl, polys * L * nl, R.t[0], R.t[1], st);
        else
          ntt_forward_i8_lazy(dig8, digits, n_in, nl, polys * L * nl, R.t[0], R.t[1], st);
      } else {
        decompose(R, w.g_ck, mi, n_in, 1, polys, digits, st);
        if (n_in > 1) digits_to_eval(R, digits, n_in, polys * L * nl, st);
      }
      const Split d = split(n_in);
      const int tt = d.tt, JB = d.JB;
      dim3 grid((unsigned)(d.slots * JB), (unsigned)nl, (unsigned)d.lwes);
      u64* bsk_k = bsk + (n_out - 2);  // this step's region
      const double* kd = reinterpret_cast<const double*>(s.cascade_eval_d.p) + k * step_len;
      const double* dd = reinterpret_cast<const double*>(digits);
      if (fp_mac && n_in == 1)
        k_cascade_mac_fp<true, 1, 1><<<grid, 256, 0, st>>>(nullptr, dig8, kd, rank_in, n_in, L, tt, JB, nlwe, R, mo, bsk_k,
                                                        2L * n1);
      else if (d.NL == 2)
        k_cascade_mac_fp<false, 2, 2><<<grid, 256, 0, st>>>(dd, dig8, kd, rank_in, n_in, L, tt, JB, nlwe, R, mo, bsk_k,
                                                         2L * n1);
      else if (d.NS == 2)
        k_cascade_mac_fp<false, 1, 2><<<grid, 256, 0, st>>>(dd, dig8, kd, rank_in, n_in, L, tt, JB, nlwe, R, mo, bsk_k,
                                                            2L * n1);
      else if (fp_mac)
        k_cascade_mac_fp<false, 1, 1><<<grid, 256, 0, st>>>(dd, dig8, kd, rank_in, n_in, L, tt, JB, nlwe, R, mo, bsk_k,
                                                         2L * n1);
      else
        k_cascade_mac<<<grid, 256, 0, st>>>(digits, s.cascade_eval.p + k * step_len, rank_in, n_in, L, tt, JB, R, mo,
                                            bsk_k, 2L * n1);
      VIA_LAUNCHED();
      // The masks return to coefficient form for the next step's digits.
      from_eval(R, mo, n_out, nlwe * (rank_in / 2) * nl, st);
      std::swap(mi, mo);
      continue;
    } else {
      gadget_product(R, w.g_ck, mi, n_out, 2, 1, polys, keys_cyclic(s.cascade_eval.p + k * step_len, rank_in), cP,
                     digits, st);
      const long items = nlwe * (rank_in / 2 + 1) * nl * n_out;
      k_cascade_reduce<<<blocks(items), 256, 0, st>>>(cP, rank_in, n_out, nl, nlwe, R, mo, bsum);
      VIA_LAUNCHED();
      k_cascade_body<<<blocks(nlwe * nl * n_out), 256, 0, st>>>(bi, bsum, n_in, nl, nlwe, R, bo);
      VIA_LAUNCHED();
    }
    std::swap(mi, mo);
    std::swap(bi, bo);
  }
  // The cascade's body, from the LWE bodies and every step's sums.
  const u64* lwe_body = k0 ? query + (long)nl * n1 : bi;
  const long body_stride = k0 ? (long)lwe_len(p) : nl;
  const bool small_primes = R.ntt && R.m[0].q < (1ull << 40) && R.m[1].q < (1ull << 40) && k0 <= 8;
  if (small_primes && (n1 == 2048 || n1 == 4096)) {
    const dim3 grid((unsigned)nlwe, (unsigned)nl);
    const u64* gemm = w.c_gemm_body.p + lwe0;
    if (n1 == 2048)
      k_cascade_rlwe_fp<11><<<grid, 256, 0, st>>>(mi, lwe_body, body_stride, bsk, gemm, nlwe_all, k0, rlwe, R);
    else
      k_cascade_rlwe_fp<12><<<grid, 512, 0, st>>>(mi, lwe_body, body_stride, bsk, gemm, nlwe_all, k0, rlwe, R);
    VIA_LAUNCHED();
  } else {
    if (R.ntt) {
      k_cascade_body_final<<<blocks(nlwe * nl * n1), 256, 0, st>>>(lwe_body, body_stride, bsk, k0, k, nl, nlwe, R, bo);
      VIA_LAUNCHED();
      from_eval(R, bo, n1, nlwe * nl, st);
      std::swap(bi, bo);
    }
    k_pack_rlwe<<<blocks(nlwe * nl * n1), 256, 0, st>>>(mi, bi, w.c_gemm_body.p + lwe0, nlwe_all, k0, k, nlwe, n1, nl, R,
                                                        rlwe);
    VIA_LAUNCHED();
  }
  // RLWE -> RGSW with the conversion key (prim/gates/convert.rs:162-178); the
  // final rank-1 masks are already contiguous [lwe][nl][n1] in `mi`.
  u64* gp = w.g_gp.p + lwe0 * 2 * lwe_n;
  u64* gdig = w.g_digits.p + lwe0 * L * lwe_n;
  if (dig8) {
    decompose_i8(R, w.g_ck, mi, n1, nlwe, dig8, st);
    if (!shared_key_fp(R, dig8, s.conv_eval.p, nullptr, L, nlwe, gp, st)) {
      ntt_forward_i8_lazy(dig8, gdig, n1, nl, nlwe * L * nl, R.t[0], R.t[1], st);
      mac(R, gdig, keys_shared(s.conv_eval.p), gp, L, n1, nlwe, st);
      from_eval(R, gp, n1, nlwe * 2 * nl, st);
    }
  } else {
    gadget_product(R, w.g_ck, mi, n1, 1, 1, nlwe, keys_shared(s.conv_eval.p), gp, gdig, st);
    from_eval(R, gp, n1, nlwe * 2 * nl, st);
  }
  k_assemble_rgsw<<<blocks(nlwe * 2 * nl * n1), 256, 0, st>>>(rlwe, gp, (int)p.l_query, nbits, n1, nl, R,
                                                               w.rgsw_q1.p + bit0 * rgsw1);
  VIA_LAUNCHED();
}


// ext[o] = bit_o (x) cts[o] for `count` RLWEs (coefficient form); result in the
// eval domain unless `to_coeff`. The RGSW of output o is selected by `rgsw`.
static void external_products(const DevRing& R, const Gadget& g, KeySel rgsw, const u64* cts, long count, u64* digits,
                              u64* ext, bool to_coeff, cudaStream_t st) {
  const int n = R.n;
  // Mask and body of every RLWE are the G = 2 decomposed inputs; their digits
  // pair with the neg_s_m and m samples of the RGSW respectively.
  gadget_product(R, g, cts, n, 1, 2, count, rgsw, ext, digits, st);
  if (to_coeff) from_eval(R, ext, n, 2 * count * R.nl, st);
}

// One CMux of a tree level per CTA (mux.rs:75-84, 167-198; rgsw.rs:108-121),
// single-limb ring of degree 2^LOGN with a small gadget (gadget_scaled_small),
// 2^LOGN / 8 threads holding 8 residues each:
//   diff = in[2o+1] - in[2o] (eval) -> inverse NTT -> balanced digits of the
//   mask and body -> forward NTT of each digit polynomial -> products with the
//   RGSW samples (mask digits with neg_s_m, body digits with m, digit k with
//   sample L-1-k) -> out[o] = in[2o] + ext, eval form throughout.
// cur: [count*2][2][n]; nxt: [count][2][n]; the RGSW of CMux o ([2L][2][n],
// eval) is picked by `ks`. The digits never leave registers. Every transform,
// digit split and RGSW product is exact integer arithmetic on doubles (ntt_fp.cuh:
// FMA two-products and a floating-point quotient estimate; gadget_fp.cuh). For
// single primes q < 2^35 and small gadgets: differences of canonical residues are
// below q; the n^-1 product leaves coefficients within 0.5625 q, which the split
// takes as they are; each product with an RGSW sample (below q) is reduced to
// within 0.5625 q, so the 2L products and the input residue sum to less than
// (1 + 1.125 L) q before the final reduction.
//
// FP64-issue bound (about 2800 operations a thread, 2 CTAs of 8 warps an SM; 63% of the pipe).
// At n = 2048 the first exchange of a forward transform and the last of an inverse cross
// warps, the other two stay within one, and the inverse ends in the layout the forward
// starts in; transforms run two at a time (mask and body, then a half's two digits). 65536
// CMuxes 6.58 ms with single transforms, two barriers on every exchange and integer digit
// splits, 4.31 ms with one transform at a time, 4.08 ms with keys and inputs competing for L1,
// 3.89 ms with the inputs (read once) kept out of it, the keys (128 KB a selector, shared by
// neighbouring CTAs) held there and fetched into it while the digits are transformed; the
// tiled level of 131072 9.05 and 8.28 ms; 128 CMuxes (one a SM) 25, 20, 16.4 and 14.0 us.
//
// TILED (the first level): cur holds fd_scan's tiled columns of nq queries, where a pair's
// four residues of a slot are 32 consecutive bytes; in[2o] waits in shared memory.
template <int LOGN, bool TILED>
__global__ void __launch_bounds__((1 << LOGN) / 8, LOGN >= 12 ? 1 : 2) k_cmux_fp(const u64* __restrict__ cur,
                                                                                u64* __restrict__ nxt, KeySel ks,
                                                                                long nq, const __grid_constant__ DevRing R,
                                                                                const __grid_constant__ Gadget g) {
  constexpr int n = 1 << LOGN;
  extern __shared__ __align__(16) double pair_sm[];  // two transforms' exchange areas, then (TILED) in[2o]
  double* keep = pair_sm + 2 * n;
  const int tid = threadIdx.x;
  const long o = blockIdx.x;
  const NttTable& T = R.t[0];
  const double q = T.qd, qinv = T.qinv;
  const u64* in = cur + (2 * o) * 2 * n;
  const long tstep = 2 * FD_MT * nq;  // tiled: residues from a slot to the next
  if (TILED) {
    const long j = 2 * (o % ks.div), query = o / ks.div;  // ks.div CMuxes a query
    in = cur + (((j / FD_MT) * n + 8 * tid) * nq + query) * 2 * FD_MT + 2 * (j % FD_MT);
  }
  const u64* K = ks.base + ((o / ks.div) % ks.mod) * ks.stride;
  const int L = g.L;
  const bool dense = 4.0 * g.dB * q < 281474976710656.0;  // |digit| <= B / 2: fp_digit_phase's sums below 2^48
  double val[2][8];  // mask and body: difference, then scaled coefficients
  if (TILED) {
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      u64 x[4];  // in[2o] mask, body, in[2o+1] mask, body of slot 8 tid + v
      asm volatile("ld.global.L1::no_allocate.v4.u64 {%0, %1, %2, %3}, [%4];"
                   : "=l"(x[0]), "=l"(x[1]), "=l"(x[2]), "=l"(x[3])
                   : "l"(in + v * tstep));
      const double m = fp_from_u64(x[0]), b = fp_from_u64(x[1]);
      val[0][v] = __dadd_rn(fp_from_u64(x[2]), -m);
      val[1][v] = __dadd_rn(fp_from_u64(x[3]), -b);
      keep[v * (n / 8) + tid] = m;
      keep[n + v * (n / 8) + tid] = b;
    }
  } else {
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      u64 x[8], y[8];
      ld8_stream(in + 2 * n + p * n + 8 * tid, x);
      ld8_stream(in + p * n + 8 * tid, y);
#pragma unroll
      for (int v = 0; v < 8; ++v) val[p][v] = __dadd_rn(fp_from_u64(x[v]), -fp_from_u64(y[v]));
    }
  }
  fp_inverse2<LOGN>(val, tid, T, pair_sm);
#pragma unroll
  for (int p = 0; p < 2; ++p)
#pragma unroll
    for (int v = 0; v < 8; ++v)
      val[p][v] = fp_scaled(fp_mulmod(val[p][v], T.ninv_d[LOGN], q, qinv), g.dS, qinv);
  double a[2][8];  // mask and body sums
#pragma unroll
  for (int v = 0; v < 8; ++v) a[0][v] = a[1][v] = 0.0;
#pragma unroll 1
  for (int p = 0; p < 2; ++p) {  // 0: mask digits (neg_s_m rows), 1: body digits (m rows)
#pragma unroll 1
    for (int k = 0; k < L; k += 2) {
      double e[2][8];
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        e[0][v] = fp_next_digit(val[0][v], g);
        e[1][v] = fp_next_digit(val[0][v], g);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)  // the products' keys
#pragma unroll
        for (int part = 0; part < 2; ++part)
          if (k + i < L)
            fp_prefetch(K + (long)(2 * (p * L + L - 1 - k - i) + part) * n + 8 * tid);
      __syncthreads();  // the previous transforms' reads
      fp_forward_digits2<LOGN>(e, tid, T, pair_sm, dense);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if (k + i >= L) break;  // an odd depth's last digit comes alone
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          u64 key[8];
          ld8_nc(K + (long)(2 * (p * L + L - 1 - k - i) + part) * n + 8 * tid, key);
#pragma unroll
          for (int v = 0; v < 8; ++v)
            a[part][v] = __dadd_rn(a[part][v], fp_mulmod(e[i][v], fp_from_u64(key[v]), q, qinv));
        }
      }
    }
#pragma unroll
    for (int v = 0; v < 8; ++v) val[0][v] = val[1][v];
  }
#pragma unroll
  for (int part = 0; part < 2; ++part) {
    u64 x[8];
    if (!TILED) ld8_stream(in + part * n + 8 * tid, x);
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      const double y = TILED ? keep[part * n + v * (n / 8) + tid] : fp_from_u64(x[v]);
      x[v] = fp_to_u64(fp_canonical(__dadd_rn(y, a[part][v]), q, qinv));
    }
    st8_stream(nxt + o * 2 * n + part * n + 8 * tid, x);
  }
}

// The dynamic shared memory (`doubles` of it) of a kernel above, its limit raised where needed.
template <class K>
static size_t pair_smem(K kernel, size_t doubles) {
  const size_t bytes = doubles * 8;
  if (bytes > 48 * 1024)
    VIA_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  return bytes;
}

// The CMux of k_cmux_fp split over a cluster of four CTAs, for tree levels
// with too few CMuxes to fill the GPU, where one CMux's latency sets the level's
// time. CTA r of the cluster takes input half p = r & 1 (mask or body),
// inverse-transforms its difference, and forward-transforms its digit k = r >> 1;
// its products with the sample's mask and body (sample p L + L - 1 - k) are
// reduced mod q into its shared memory. After a cluster barrier, each rank
// adds in[2o] and the four partials of its half of the mask or body, read over
// distributed shared memory; a second barrier keeps every CTA's shared memory
// alive until those reads are done. Two transforms per CTA instead of six for
// one CTA. L = 2.
// In double precision with the bounds of k_cmux_fp: each CTA's products are
// signed residues within 0.5625 q, kept as doubles in shared memory.
// Latency-bound: an L2 wait for keys and twiddles in every phase until they are fetched into
// L1 with the inputs, and the final sums from conflict-free partials by all four ranks (two
// ranks, eight dependent rounds each, before): a CMux of degree 2048 8.5 us, 7.0 here, 64 of
// them 13.6 and 10.7; of degree 4096 23.4 us as one CTA, 11.5 here, 64 22.9 both ways.
template <int LOGN>
__global__ void __cluster_dims__(4, 1, 1) __launch_bounds__((1 << LOGN) / 8, LOGN >= 12 ? 1 : 2)
    k_cmux_cluster_fp(const u64* __restrict__ cur, u64* __restrict__ nxt, KeySel ks, const __grid_constant__ DevRing R,
                      const __grid_constant__ Gadget g) {
  namespace cg = cooperative_groups;
  constexpr int n = 1 << LOGN;
  extern __shared__ __align__(16) double cmux_sm[];
  double* ssm = cmux_sm;        // the inverse's exchanges, then the mask partial
  double* pbody = cmux_sm + n;  // the forward's exchanges, then the body partial
  cg::cluster_group cluster = cg::this_cluster();
  const int r = (int)cluster.block_rank();
  const int p = r & 1, k = r >> 1;
  const int tid = threadIdx.x;
  const long o = blockIdx.x / 4;
  const NttTable& T = R.t[0];
  const double q = T.qd, qinv = T.qinv;
  const u64* a = cur + (2 * o) * 2 * n;
  const int smp = p * 2 + 1 - k;  // sample L - 1 - k of half p (L = 2)
  const u64* K = ks.base + ((o / ks.div) % ks.mod) * ks.stride + (long)(2 * smp) * n + 8 * tid;
  const bool dense = 4.0 * g.dB * q < 281474976710656.0;
  double e[8];
  {
    u64 x[8], y[8];
    ld8(a + 2 * n + p * n + 8 * tid, x);
    ld8(a + p * n + 8 * tid, y);
    fp_prefetch_twiddles<LOGN>(tid, T);
    fp_prefetch(K);
    fp_prefetch(K + n);
#pragma unroll
    for (int v = 0; v < 8; ++v) e[v] = __dadd_rn(fp_from_u64(x[v]), -fp_from_u64(y[v]));
  }
  fp_inverse<LOGN>(e, tid, T, ssm);
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    double val = fp_scaled(fp_mulmod(e[v], T.ninv_d[LOGN], q, qinv), g.dS, qinv);
    e[v] = fp_next_digit(val, g);
    if (k) e[v] = fp_next_digit(val, g);
  }
  fp_forward_digits<LOGN>(e, tid, T, pbody, 0, dense);
  u64 km[8], kb[8];
  ld8_nc(K, km);
  ld8_nc(K + n, kb);
  __syncthreads();  // the exchanges; the partials' layout (slot 8 tid + v at v n / 8 + tid) crosses warps
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    ssm[v * (n / 8) + tid] = fp_mulmod(e[v], fp_from_u64(km[v]), q, qinv);
    pbody[v * (n / 8) + tid] = fp_mulmod(e[v], fp_from_u64(kb[v]), q, qinv);
  }
  cluster.sync();
  // Ranks 0 and 2 the output mask, 1 and 3 the body; four of a thread's eight slots each.
  const long at = p * n + 8 * tid + 4 * k;
  u64 x[4];
  asm volatile("ld.global.v4.u64 {%0, %1, %2, %3}, [%4];" : "=l"(x[0]), "=l"(x[1]), "=l"(x[2]), "=l"(x[3]) : "l"(a + at));
#pragma unroll
  for (int v = 0; v < 4; ++v) e[v] = fp_from_u64(x[v]);
#pragma unroll
  for (int y = 0; y < 4; ++y) {
    const double* part = cluster.map_shared_rank(p ? pbody : ssm, (r + y) & 3) + 4 * k * (n / 8) + tid;
#pragma unroll
    for (int v = 0; v < 4; ++v) e[v] = __dadd_rn(e[v], part[v * (n / 8)]);
  }
#pragma unroll
  for (int v = 0; v < 4; ++v) x[v] = fp_to_u64(fp_canonical(e[v], q, qinv));
  asm volatile("st.global.v4.u64 [%0], {%1, %2, %3, %4};" ::"l"(nxt + o * 2 * n + at), "l"(x[0]), "l"(x[1]), "l"(x[2]),
               "l"(x[3])
               : "memory");
  cluster.sync();
}

// One external product per four-CTA cluster and limb (rgsw.rs:108-121), coefficient form in
// and out, in double precision: levels and steps with too few products to fill the GPU,
// where one product's latency sets the time. CTA r takes input half p = r & 1 and digit
// k = r >> 1: one digit split, one forward transform, and its products with the sample's
// mask and body (sample p L + L - 1 - k, L = 2) in shared memory. After a cluster barrier
// ranks 0 and 1 sum the four partial masks / bodies over distributed shared memory and
// transform them back.
//   EXT_DMUX: out[2o] = in[o] - ext, out[2o+1] = ext            (a DMux level; mux.rs:129-137)
//   EXT_CROT: d = rot - in, rot = -X^shift in; out = in + bit (x) d, in place (a CRot step;
//             rotate.rs:128-150)
// in [ct][2][nl][n], RGSWs [2L][2][nl][n] eval. Latency-bound: a digit split, two transforms and
// two cluster barriers, where decompose, transform, multiply-accumulate and inverse kernels
// took about 24 us a DMux level and 32 us a CRot step (live, ring of 2048), 16 and 12 us in
// this kernel while keys and twiddles came from L2 and the partials' layout had bank
// conflicts, 12.5 and 9 us without, 10.5 us a DMux level with its loads before the splits
// (degree 4096: 26, 18 and 16.4 us).
enum { EXT_DMUX = 0, EXT_CROT = 1 };
template <int LOGN, int MODE>
__global__ void __cluster_dims__(4, 1, 1) __launch_bounds__((1 << LOGN) / 8)
    k_ext_cluster_fp(const u64* in, u64* out, KeySel ks, int shift, const __grid_constant__ DevRing R,
                     const __grid_constant__ Gadget g) {
  namespace cg = cooperative_groups;
  constexpr int n = 1 << LOGN;
  using L0 = NttPhase<LOGN, false, 0>;
  extern __shared__ __align__(16) double ext_sm[];
  double* pmask = ext_sm;      // the forward's exchanges, then the mask partial
  double* pbody = ext_sm + n;  // the body partial
  cg::cluster_group cluster = cg::this_cluster();
  const int r = (int)cluster.block_rank();
  const int p = r & 1, k = r >> 1;
  const int tid = threadIdx.x, nl = R.nl, l = blockIdx.y;
  const long o = blockIdx.x / 4;
  const NttTable& T = R.t[l];
  const double q = T.qd, qinv = T.qinv;
  const u64* ct = in + o * 2 * nl * n;
  const int smp = p * 2 + 1 - k;
  const u64* K = ks.base + ((o / ks.div) % ks.mod) * ks.stride + ((long)(2 * smp) * nl + l) * n + 8 * tid;
  fp_prefetch_twiddles<LOGN>(tid, T);
  fp_prefetch(K);
  fp_prefetch(K + (long)nl * n);
  // All loads before the splits, whose rare branch they would wait behind: x0, x1 the limbs of a
  // coefficient (DMUX), or it and the one `shift` places before (CROT).
  u64 x0[8], x1[8];
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    const int x = L0::index(v, tid);
    const u64* c = ct + (long)p * nl * n + x;
    x0[v] = c[0];
    if (MODE == EXT_DMUX)
      x1[v] = nl == 2 ? c[n] : 0;
    else
      x1[v] = c[x < shift ? n - shift : -shift];
  }
  double e[8];
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    double val;
    if (MODE == EXT_DMUX) {
      val = nl == 2 ? fp_scaled2(fp_from_u64(x0[v]), fp_from_u64(x1[v]), g, R)
                    : fp_scaled(fp_reduce(fp_from_u64(x0[v]), q, qinv), g.dS, qinv);
    } else {
      // rot[x] = -in[x - shift], or in[x - shift + n] where the index wraps.
      const double s = fp_from_u64(x1[v]);
      val = fp_scaled(fp_reduce(__dadd_rn(L0::index(v, tid) < shift ? s : -s, -fp_from_u64(x0[v])), q, qinv), g.dS, qinv);
    }
    e[v] = fp_next_digit(val, g);
    if (k) e[v] = fp_next_digit(val, g);
  }
  fp_forward<LOGN>(e, tid, T, pmask);
  u64 km[8], kb[8];
  ld8_nc(K, km);
  ld8_nc(K + (long)nl * n, kb);
  __syncthreads();  // the exchanges; the partials' layout (slot 8 tid + v at v n / 8 + tid) crosses warps
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    pmask[v * (n / 8) + tid] = fp_mulmod(e[v], fp_from_u64(km[v]), q, qinv);
    pbody[v * (n / 8) + tid] = fp_mulmod(e[v], fp_from_u64(kb[v]), q, qinv);
  }
  cluster.sync();
  if (r < 2) {
    double* mine = r ? pbody : pmask;
#pragma unroll
    for (int v = 0; v < 8; ++v) e[v] = mine[v * (n / 8) + tid];
#pragma unroll
    for (int y = 1; y < 4; ++y) {
      const double* peer = cluster.map_shared_rank(mine, (r + y) & 3);
#pragma unroll
      for (int v = 0; v < 8; ++v) e[v] = __dadd_rn(e[v], peer[v * (n / 8) + tid]);
    }
#pragma unroll
    for (int v = 0; v < 8; ++v) e[v] = fp_reduce(e[v], q, qinv);
  }
  cluster.sync();  // every CTA's partials have been read
  if (r >= 2) return;
  fp_inverse<LOGN>(e, tid, T, pmask);
  const u64 qi = R.m[l].q;
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    const long at = (long)(r * nl + l) * n + L0::index(v, tid);
    const u64 ext = fp_to_u64(fp_wrap(fp_mulmod(e[v], T.ninv_d[LOGN], q, qinv), q));
    if (MODE == EXT_DMUX) {
      out[(2 * o) * 2 * nl * n + at] = submod(ct[at], ext, qi);
      out[(2 * o + 1) * 2 * nl * n + at] = ext;
    } else {
      out[o * 2 * nl * n + at] = addmod(ct[at], ext, qi);
    }
  }
}

// ---------------------------------------------------------------------------
// Fused gadget products on the transform's registers, double precision (ntt_fp.cuh).
// ---------------------------------------------------------------------------
constexpr long SHARED_KEY_MIN = 512;  // CTAs from which k_shared_key_fp runs

// key (x) digits of one polynomial per CTA and limb, the key shared by all: signed digit
// bytes dig8 [c][L][n] -> forward transforms -> products with the eval-form samples
// [L][2][nl][n] -> inverse transforms of the two sums -> out [c][2][nl][n], coefficient
// form. Digits and products never reach memory; the key streams from L2.
//
// ROTATED (a key switch of rotated ciphertexts, keyswitch.rs:99-102): out =
// (-prod.mask, body - prod.body) with `bodies` [c][nl][n].
//
// FP64-issue bound: L + 2 transforms, two at a time, a CTA. 2048 key switches at q1 (L = 18)
// 1049 us in separate kernels (digit transforms, multiply-accumulate, inverse, sum), 781 us, and
// 760 with the keys fetched into L1 while the digits are transformed.
template <int LOGN, bool ROTATED>
__global__ void __launch_bounds__((1 << LOGN) / 8, LOGN >= 12 ? 1 : LOGN == 11 ? 2 : 1)
    k_shared_key_fp(const int8_t* __restrict__ dig8, const u64* __restrict__ key, const u64* __restrict__ bodies, int L,
                    u64* __restrict__ out, const __grid_constant__ DevRing R) {
  constexpr int n = 1 << LOGN;
  using L0 = NttPhase<LOGN, false, 0>;
  extern __shared__ __align__(16) double pair_sm[];
  const int tid = threadIdx.x, nl = R.nl, l = blockIdx.y;
  const long c = blockIdx.x;
  const NttTable& T = R.t[l];
  const double q = T.qd, qinv = T.qinv;
  const int8_t* d = dig8 + c * (long)L * n;
  const long per = (long)nl * n;
  const u64* K = key + (long)l * n + 8 * tid;
  const bool dense = q <= FP_DIGIT_Q;
  double a[2][8];  // mask and body sums
#pragma unroll
  for (int v = 0; v < 8; ++v) a[0][v] = a[1][v] = 0.0;
#pragma unroll 1
  for (int s = 0; s < L; s += 2) {
    const bool two = s + 1 < L;
    double e[2][8];
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      e[0][v] = (double)d[(long)s * n + L0::index(v, tid)];
      e[1][v] = two ? (double)d[(long)(s + 1) * n + L0::index(v, tid)] : 0.0;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)  // the products' keys
      if (r < 2 || two) fp_prefetch(K + (2 * s + r) * per);
    __syncthreads();  // the previous transforms' reads
    fp_forward_digits2<LOGN>(e, tid, T, pair_sm, dense);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      if (i && !two) break;
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        u64 k[8];
        ld8_nc(K + (2 * (s + i) + part) * per, k);
#pragma unroll
        for (int v = 0; v < 8; ++v)
          a[part][v] = __dadd_rn(a[part][v], fp_mulmod(e[i][v], fp_from_u64(k[v]), q, qinv));
      }
    }
  }
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    a[0][v] = fp_reduce(a[0][v], q, qinv);
    a[1][v] = fp_reduce(a[1][v], q, qinv);
  }
  __syncthreads();
  fp_inverse2<LOGN>(a, tid, T, pair_sm);
  const u64 qi = R.m[l].q;
#pragma unroll
  for (int part = 0; part < 2; ++part)
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      const int x = L0::index(v, tid);
      u64 w = fp_to_u64(fp_wrap(fp_mulmod(a[part][v], T.ninv_d[LOGN], q, qinv), q));
      if (ROTATED) w = part ? submod(bodies[c * per + (long)l * n + x], w, qi) : negmod(w, qi);
      out[(2 * c + part) * per + (long)l * n + x] = w;
    }
}

// External products with RGSWs of their own (rgsw.rs:108-121): per CTA (pair, limb) the gadget
// digits, the samples' forward transforms, products and inverse transforms. rgsw
// [c][2L][2][nl][n] and cts, out [c][2][nl][n], all in coefficient form at any 8-byte
// address. Each RGSW polynomial is read once and nothing else of its size is written.
// FP64-issue bound (6 L + 2 transforms, two at a time): 4099 pairs at q1, L = 2: 1.93 ms in
// separate kernels after a copy of the RGSWs, 1.80 ms with each sample word loaded, then
// checked, 1.21 ms with a polynomial's loads all in flight and the next one's lines fetched,
// 1.09 ms with the ciphertext's loads before its splits as well.
template <int LOGN>
__global__ void __launch_bounds__((1 << LOGN) / 8, LOGN >= 12 ? 1 : LOGN == 11 ? 2 : 1)
    k_external_fp(const u64* __restrict__ rgsw, const u64* __restrict__ cts, u64* __restrict__ out,
                  const __grid_constant__ DevRing R, const __grid_constant__ Gadget g) {
  constexpr int n = 1 << LOGN;
  using L0 = NttPhase<LOGN, false, 0>;
  extern __shared__ __align__(16) double pair_sm[];  // two exchange areas, then the scaled coefficients
  double* keep = pair_sm + 2 * n;
  const int tid = threadIdx.x, nl = R.nl, l = blockIdx.y, L = g.L;
  const long c = blockIdx.x, per = (long)nl * n;
  const NttTable& T = R.t[l];
  const double q = T.qd, qinv = T.qinv;
  const u64* ct = cts + c * 2 * per;
  const u64* K = rgsw + c * 2 * L * 2 * per + (long)l * n;
  // A sample's mask and body (2 n / 16 lines, one a thread) on their way while other polynomials
  // are transformed.
  const auto fetch = [&](int h, int k) {
    const long smp = h * L + L - 1 - k;
    fp_prefetch(K + (2 * smp + (tid >= n / 16)) * per + 16 * (tid % (n / 16)));
  };
  fetch(0, 0);
  const auto split = [&](u64 c0, u64 c1) {
    return nl == 2 ? fp_scaled2(fp_from_u64(c0), fp_from_u64(c1), g, R)
                   : fp_scaled(fp_reduce(fp_from_u64(c0), q, qinv), g.dS, qinv);
  };
  u64 any = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    u64 x0[8], x1[8];  // all loads before the splits, whose rare branch they would wait behind
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      const u64* x = ct + h * per + L0::index(v, tid);
      any |= x0[v] = x[0];
      any |= x1[v] = nl == 2 ? x[n] : 0;
    }
#pragma unroll
    for (int v = 0; v < 8; ++v) keep[h * n + v * (n / 8) + tid] = split(x0[v], x1[v]);
  }
  // Any 64-bit word, as of the samples below: split again from reduced words. (A check before the
  // splits made them wait for every load: 1024 products of degree 4096, L = 2, 666 -> 692 us.)
  if (any >= (1ull << 47)) {
#pragma unroll 1
    for (int i = 0; i < 16; ++i) {
      const u64* x = ct + (i >> 3) * per + L0::index(i & 7, tid);
      keep[(i >> 3) * n + (i & 7) * (n / 8) + tid] = split(x[0] % R.m[0].q, nl == 2 ? x[n] % R.m[1].q : 0);
    }
  }
  double a[2][8];  // mask and body sums
#pragma unroll
  for (int v = 0; v < 8; ++v) a[0][v] = a[1][v] = 0.0;
#pragma unroll 1
  for (int k = 0; k < L; ++k) {
    double e[2][8];  // digit k of the mask and of the body
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        double val = keep[h * n + v * (n / 8) + tid];
        e[h][v] = fp_next_digit(val, g);
        keep[h * n + v * (n / 8) + tid] = val;
      }
    __syncthreads();  // the previous transforms' reads
    fp_forward2<LOGN>(e, tid, T, pair_sm);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const long smp = h * L + L - 1 - k;
      u64 x[2][8], any = 0;  // the sample's mask and body
#pragma unroll
      for (int part = 0; part < 2; ++part)
#pragma unroll
        for (int v = 0; v < 8; ++v) any |= x[part][v] = K[(2 * smp + part) * per + L0::index(v, tid)];
      if (any >= (1ull << 47)) {  // as the transforms take any word
#pragma unroll
        for (int part = 0; part < 2; ++part)
#pragma unroll
          for (int v = 0; v < 8; ++v) x[part][v] %= T.q;
      }
      double f[2][8];
#pragma unroll
      for (int part = 0; part < 2; ++part)
#pragma unroll
        for (int v = 0; v < 8; ++v) f[part][v] = fp_from_u64(x[part][v]);
      if (h == 0)
        fetch(1, k);
      else if (k + 1 < L)
        fetch(0, k + 1);
      __syncthreads();
      fp_forward2<LOGN>(f, tid, T, pair_sm);
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        const double x = fp_reduce(e[h][v], q, qinv);  // the product's factor below q
        a[0][v] = __dadd_rn(a[0][v], fp_mulmod(f[0][v], x, q, qinv));
        a[1][v] = __dadd_rn(a[1][v], fp_mulmod(f[1][v], x, q, qinv));
      }
    }
  }
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    a[0][v] = fp_reduce(a[0][v], q, qinv);
    a[1][v] = fp_reduce(a[1][v], q, qinv);
  }
  __syncthreads();
  fp_inverse2<LOGN>(a, tid, T, pair_sm);
#pragma unroll
  for (int part = 0; part < 2; ++part)
#pragma unroll
    for (int v = 0; v < 8; ++v)
      out[(2 * c + part) * per + (long)l * n + L0::index(v, tid)] =
          fp_to_u64(fp_wrap(fp_mulmod(a[part][v], T.ninv_d[LOGN], q, qinv), q));
}

// Runs k_shared_key_fp (a key switch of rotated ciphertexts where `bodies` is given); false
// (nothing launched) for other rings, a key at an odd address, and products too few to fill
// the GPU, whose transforms in a row take longer than separate kernels side by side
// (240 CTAs 95 us, against 73 us).
static bool shared_key_fp(const DevRing& R, const int8_t* dig8, const u64* key, const u64* bodies, int L, long count,
                          u64* out, cudaStream_t st) {
  if (!R.ntt || !ntt_fp_ok(R.t[0], R.t[R.nl - 1]) || ((uintptr_t)key & 31) || count * R.nl < SHARED_KEY_MIN) return false;
  const dim3 grid((unsigned)count, (unsigned)R.nl);
#define VIA_SK_CASE(LG)                                                                                          \
  case 1 << LG:                                                                                                  \
    if (bodies)                                                                                                  \
      k_shared_key_fp<LG, true><<<grid, (1 << LG) / 8, pair_smem(k_shared_key_fp<LG, true>, 2 << LG), st>>>(     \
          dig8, key, bodies, L, out, R);                                                                         \
    else                                                                                                         \
      k_shared_key_fp<LG, false><<<grid, (1 << LG) / 8, pair_smem(k_shared_key_fp<LG, false>, 2 << LG), st>>>(   \
          dig8, key, bodies, L, out, R);                                                                         \
    break;
  switch (R.n) {
    VIA_SK_CASE(8)
    VIA_SK_CASE(9)
    VIA_SK_CASE(10)
    VIA_SK_CASE(11)
    VIA_SK_CASE(12)
    default: return false;
  }
#undef VIA_SK_CASE
  VIA_LAUNCHED();
  return true;
}

// CTAs from which k_external_fp runs whatever its gadget's depth. With fewer, a CTA's 3 L + 2 pairs of
// transforms in a row take longer than separate kernels side by side, except for shallow gadgets of
// small rings (us a call, fused and separate kernels; q1, two CTAs a product):
//   degree 2048: L = 2, 1 product 53, 55; L = 4, 1 64, 51, 16 65, 60, 32 66, 74; L = 11, 1 123, 54,
//     16 125, 77, 32 126, 116, 48 130, 151
//   degree 4096: L = 2, 1 73, 60, 16 73, 68, 24 73, 74, 32 74, 80; L = 8, 16 167, 100, 48 171, 217
//   degree 1024: L = 4, 1 46, 49; L = 8, 1 62, 51, 32 70, 68;  degree 256: L = 4, 1 42, 50; L = 8, 1 54, 48
// The many: 1024 products of degree 2048, L = 11, 1211 fused and about 3500 before there was this kernel.
constexpr long EXTERNAL_MIN = 64;

// Runs k_external_fp; false (nothing launched) for rings and gadgets it does not serve, for few products
// of a deep gadget (EXTERNAL_MIN), and for outputs that overlap an input: its CTAs write one limb
// while others may still read.
bool external_fp(const DevRing& R, const Gadget& g, const u64* rgsw, const u64* cts, long count, u64* out,
                 cudaStream_t st) {
  if (!R.ntt || !g.fp || !ntt_fp_ok(R.t[0], R.t[R.nl - 1])) return false;
  if ((g.L > 4 || g.L * R.n > 4096) && count * R.nl < EXTERNAL_MIN) return false;
  const size_t per = (size_t)R.nl * R.n, len = (size_t)count * 2 * per;
  const auto apart = [&](const u64* p, size_t words) { return out + len <= p || p + words <= out; };
  if (!apart(cts, len) || !apart(rgsw, len * 2 * g.L)) return false;
  const dim3 grid((unsigned)count, (unsigned)R.nl);
  switch (R.n) {
    case 4096: k_external_fp<12><<<grid, 512, pair_smem(k_external_fp<12>, 4 << 12), st>>>(rgsw, cts, out, R, g); break;
    case 2048: k_external_fp<11><<<grid, 256, pair_smem(k_external_fp<11>, 4 << 11), st>>>(rgsw, cts, out, R, g); break;
    case 1024: k_external_fp<10><<<grid, 128, pair_smem(k_external_fp<10>, 4 << 10), st>>>(rgsw, cts, out, R, g); break;
    case 512: k_external_fp<9><<<grid, 64, pair_smem(k_external_fp<9>, 4 << 9), st>>>(rgsw, cts, out, R, g); break;
    case 256: k_external_fp<8><<<grid, 32, pair_smem(k_external_fp<8>, 4 << 8), st>>>(rgsw, cts, out, R, g); break;
    default: return false;
  }
  VIA_LAUNCHED();
  return true;
}

// Rings and gadgets k_ext_cluster_fp serves. Raises its shared-memory limit (n = 4096: 64 KB) on the
// current device.
static bool ext_cluster_ok(const DevRing& R, const Gadget& g) {
  return R.ntt && g.L == 2 && g.fp && ntt_fp_ok(R.t[0], R.t[R.nl - 1]) && (R.n == 2048 || R.n == 4096);
}

template <int MODE>
static void ext_cluster(const DevRing& R, const Gadget& g, const u64* in, u64* out, KeySel ks, int shift, long count,
                        cudaStream_t st) {
  const dim3 grid((unsigned)(4 * count), (unsigned)R.nl);
  const int smem = 2 * R.n * 8;
  if (R.n == 4096) {
    VIA_CUDA(cudaFuncSetAttribute(k_ext_cluster_fp<12, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    k_ext_cluster_fp<12, MODE><<<grid, 512, smem, st>>>(in, out, ks, shift, R, g);
  } else {
    k_ext_cluster_fp<11, MODE><<<grid, 256, smem, st>>>(in, out, ks, shift, R, g);
  }
  VIA_LAUNCHED();
}

// CMux level o < count: fused kernel when the ring has one NTT limb of a
// supported degree and a small gadget, else diff -> external product -> add.
static bool cmux_fused_ok(const DevRing& R, const Gadget& g) {
  return R.ntt && R.nl == 1 && g.small && g.S < ((u128)1 << 32) && R.m[0].q < (1ull << 35) &&
         (R.n == 4096 || R.n == 2048 || R.n == 1024 || R.n == 512);
}

// tiled_nq > 0: cur holds the tiled columns of that many queries (cmux_takes_tiles).
static void cmux_fused(const DevRing& R, const Gadget& g, const u64* cur, u64* nxt, KeySel ks, long count,
                       long tiled_nq, cudaStream_t st) {
  // Levels of at most 64 CMuxes leave most SMs idle: split each CMux over a
  // four-CTA cluster to cut its latency (both sides measured at k_cmux_cluster_fp).
  if (count <= CMUX_CLUSTER_MAX && g.L == 2 && !tiled_nq) {
#define VIA_CMUX_CASE(LG)                                                                                       \
  k_cmux_cluster_fp<LG><<<(unsigned)(4 * count), (1 << LG) / 8, pair_smem(k_cmux_cluster_fp<LG>, 2 << LG), st>>>( \
      cur, nxt, ks, R, g);                                                                                      \
  break;
    switch (R.n) {
      case 4096: VIA_CMUX_CASE(12)
      case 2048: VIA_CMUX_CASE(11)
      case 1024: VIA_CMUX_CASE(10)
      default: VIA_CMUX_CASE(9)
    }
#undef VIA_CMUX_CASE
    VIA_LAUNCHED();
    return;
  }
#define VIA_CMUX_CASE(LG)                                                                                        \
  if (tiled_nq)                                                                                                 \
    k_cmux_fp<LG, true><<<(unsigned)count, (1 << LG) / 8, pair_smem(k_cmux_fp<LG, true>, 4 << LG), st>>>(       \
        cur, nxt, ks, tiled_nq, R, g);                                                                          \
  else                                                                                                          \
    k_cmux_fp<LG, false><<<(unsigned)count, (1 << LG) / 8, pair_smem(k_cmux_fp<LG, false>, 2 << LG), st>>>(     \
        cur, nxt, ks, 0, R, g);                                                                                 \
  break;
  switch (R.n) {
    case 4096: VIA_CMUX_CASE(12)
    case 2048: VIA_CMUX_CASE(11)
    case 1024: VIA_CMUX_CASE(10)
    default: VIA_CMUX_CASE(9)
  }
#undef VIA_CMUX_CASE
  VIA_LAUNCHED();
}

// CRot diff for nq RLWEs (rotate.rs:128-150): rot = -(X^k * ct), diff = rot - ct, with
// (X^k * a)[i] = a[i-k], negated on wrap.
__global__ void k_crot_diff_batch(const u64* ct, int n, int k, long nq, DevMod m, u64* diff) {
  long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= nq * 2 * n) return;
  long p = gid / n;
  int i = (int)(gid % n);
  int src = i - k;
  bool wrap = src < 0;
  if (wrap) src += n;
  u64 v = ct[p * n + src];
  u64 xk = wrap ? negmod(v, m.q) : v;
  diff[p * n + i] = submod(negmod(xk, m.q), ct[p * n + i], m.q);
}

// Ring switch inputs (prim/switching/ring_switch.rs:358-385): for j < d,
// mask_proj_j[t] = (X^j * mask)[d t]; body_proj_0[t] = body[d t].
__global__ void k_ring_switch_proj_batch(const u64* ct, int n1, int n2, long nq, DevMod m, u64* mask_proj,
                                         u64* body_proj) {
  const int d = n1 / n2;
  long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= nq * (d + 1) * n2) return;
  long q = gid / ((d + 1) * n2);
  int r = (int)(gid % ((d + 1) * n2));
  int j = r / n2, t = r % n2;
  const u64* c = ct + q * 2 * n1;
  if (j == d) {
    body_proj[q * n2 + t] = c[n1 + d * t];
    return;
  }
  int src = d * t - j;
  bool wrap = src < 0;
  if (wrap) src += n1;
  u64 v = c[src];
  mask_proj[(q * d + j) * n2 + t] = wrap ? negmod(v, m.q) : v;
}

// The sums over j of gp_j (eval or coefficient form).
__global__ void k_ring_switch_sum_batch(const u64* gp, int d, int n2, long nq, DevMod m, u64* acc) {
  long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= nq * 2 * n2) return;
  long q = gid / (2 * n2);
  int r = (int)(gid % (2 * n2));
  int mb = r / n2, t = r % n2;
  u64 sacc = 0;
  for (int j = 0; j < d; ++j) sacc = addmod(sacc, gp[((q * d + j) * 2 + mb) * n2 + t], m.q);
  acc[q * 2 * n2 + mb * n2 + t] = sacc;
}

__global__ void k_ring_switch_finish_batch(const u64* acc, const u64* body_proj, int n2, long nq, DevMod m3, DevMod m4,
                                           double dq3, u64* out_mask, u64* out_body) {
  long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= nq * n2) return;
  long q = gid / n2;
  int t = (int)(gid % n2);
  const u64 q3 = m3.q;
  const u64* a = acc + q * 2 * n2;
  out_mask[q * n2 + t] = negmod(a[t], q3);  // mask: q3 -> q3 is the identity rescale
  u64 body = submod(body_proj[q * n2 + t], a[n2 + t], q3);
  // body: q3 -> q4 (mod_switch_asym, prim/switching/mod_switch.rs:124-154).
  u128 num = (u128)body * m4.q + q3 / 2;
  u64 r = (u64)div_exact(num, (u128)q3, dq3);
  out_body[q * n2 + t] = r >= m4.q ? r - m4.q : r;
}

// Step 7, RespComp (resp_comp.rs:46-76), of B RLWEs at (q2, n1) in coefficient
// form: q2 -> q3, ring switch n1 -> n2 with the RSK, body q3 -> q4.
static void resp_comp(Server& s, Workspace& w, const u64* ct_q2, long B, u64* d_mask, u64* d_body,
                      cudaStream_t st) {
  const via_params& p = s.prm;
  const int n1 = p.n1, n2 = p.n2;
  mod_switch(s.r2, ct_q2, s.r3n1, w.rs_ct3.p, B * 2, n1, st);
  const int d = n1 / n2;
  k_ring_switch_proj_batch<<<blocks(B * (d + 1) * n2), 256, 0, st>>>(w.rs_ct3.p, n1, n2, B, s.r3.m[0], w.rs_mproj.p,
                                                                      w.rs_bproj.p);
  VIA_LAUNCHED();
  gadget_product(s.r3, w.g_rsk, w.rs_mproj.p, n2, 1, 1, B * d, keys_cyclic(s.rsk_eval.p, d), w.rs_gp.p,
                 w.rs_digits.p, st);
  k_ring_switch_sum_batch<<<blocks(B * 2 * n2), 256, 0, st>>>(w.rs_gp.p, d, n2, B, s.r3.m[0], w.rs_acc.p);
  VIA_LAUNCHED();
  from_eval(s.r3, w.rs_acc.p, n2, B * 2, st);
  k_ring_switch_finish_batch<<<blocks(B * n2), 256, 0, st>>>(w.rs_acc.p, w.rs_bproj.p, n2, B, s.r3.m[0], s.r4.m[0],
                                                             (double)p.q3, d_mask, d_body);
  VIA_LAUNCHED();
}

// Runs the pipeline for nq queries (d_query: nq queries back to back; d_mask,
// d_body: [nq][n2]). When stop_stage > 0 (nq == 1 only), copies that stage's
// output in coefficient form to `dump` and returns early. Stages: 1 cascade
// RLWEs, 2 query RGSWs at q1, 3 DMux outputs, 4 mod-switched rows at q2,
// 5 FirstDim columns, 6 CMux output, 7 CRot output.
void answer_device_stages(Server& s, Workspace& w, const u64* d_query, int nq, u64* d_mask, u64* d_body,
                          cudaStream_t st, int stop_stage, u64* dump) {
  const via_params& p = s.prm;
  const int n1 = p.n1, L = p.l_query, nl = s.r1.nl;
  const long I = p.num_rows, J = p.num_cols, B = nq;
  const int nd = ilog2(I), nc = ilog2(J);
  const int nr = (int)(w.nbits - nd - nc);
  const long rgsw1 = 2L * L * 2 * nl * n1, rgsw2 = 2L * L * 2 * n1;
  if (nq < 1 || nq > w.bmax) throw CudaError(100, "batch larger than the workspace");
  auto copy_out = [&](const u64* src, size_t count) {
    VIA_CUDA(cudaMemcpyAsync(dump, src, count * 8, cudaMemcpyDeviceToDevice, st));
  };
  // ---- Step 1: QueryDecomp. The LWEs are taken grouped by use (every query's
  // DMux bits, then every query's CMux and CRot bits), so the RGSWs come out in
  // the grouped layout of rgsw_q1 and each group is one contiguous range.
  const long nb = w.nbits - nd;                 // CMux + CRot bits per query
  const long lwe_a = (long)nd * L, nlwe_all = w.nlwe * B;
  const u64* qsrc = d_query;
  if (B > 1) {
    const long ll = (long)lwe_len(p);
    k_permute_lwes<<<blocks(nlwe_all * ll), 256, 0, st>>>(d_query, B, w.nlwe, lwe_a, ll, w.q_perm.p);
    VIA_LAUNCHED();
    qsrc = w.q_perm.p;
  }
  u64* const rgsw_b1 = w.rgsw_q1.p + B * nd * rgsw1;  // the CMux / CRot bits' group
  u64* const rgsw_b2 = w.rgsw_q2.p + B * nd * rgsw2;
  if (w.ct) cascade_gemm(s, w, qsrc, nlwe_all, st);
  // Answers that run to the end expand the CMux / CRot bits (the rest of their cascades,
  // RGSWs and q1 -> q2 switch) on the side stream while the DMux tree and the
  // database scan run on `st`; `st` waits for them before the CMux tree. The
  // two groups' LWEs, buffer regions and scratch are disjoint.
  const bool split = (stop_stage == 0 || stop_stage == STOP_AFTER_CROT) && nd > 0 && nb > 0 && s.r1.ntt;
  if (split) {
    VIA_CUDA(cudaEventRecord(w.ev_fork, st));
    VIA_CUDA(cudaStreamWaitEvent(w.side, w.ev_fork, 0));
    query_decomp_range(s, w, qsrc, nlwe_all, B * lwe_a, nlwe_all - B * lwe_a, B * nd, B * nb, w.side);
    mod_switch(s.r1, rgsw_b1, s.r2, rgsw_b2, B * nb * 2 * L * 2, n1, w.side);
    to_eval(s.r2, rgsw_b2, n1, B * nb * 2 * L * 2, w.side);
    VIA_CUDA(cudaEventRecord(w.ev_join, w.side));
    query_decomp_range(s, w, qsrc, nlwe_all, 0, B * lwe_a, 0, B * nd, st);
    to_eval(s.r1, w.rgsw_q1.p, n1, B * nd * 2 * L * 2 * nl, st);
  } else {
    query_decomp_range(s, w, qsrc, nlwe_all, 0, nlwe_all, 0, B * w.nbits, st);
    if (stop_stage == 1) return copy_out(w.c_rlwe.p, (size_t)w.nlwe * 2 * nl * n1);
    if (stop_stage == 2) return copy_out(w.rgsw_q1.p, (size_t)w.nbits * rgsw1);  // one query: bit order

    // ---- mod_switch_rgsw q1 -> q2 of every bit (convert.rs:223-240; only the
    // CMux / CRot bits are used at q2), then eval form for both moduli.
    mod_switch(s.r1, w.rgsw_q1.p, s.r2, w.rgsw_q2.p, B * w.nbits * 2 * L * 2, n1, st);
    to_eval(s.r2, w.rgsw_q2.p, n1, B * w.nbits * 2 * L * 2, st);
    to_eval(s.r1, w.rgsw_q1.p, n1, B * w.nbits * 2 * L * 2 * nl, st);
  }

  // ---- Step 2: DMux tree at q1 from the trivial RLWE(0, delta) (answer.rs:181-191).
  {
    u128 Q1 = s.r1.Q();
    u128 delta = (Q1 + p.p - 1) / p.p;
    k_set_trivial<<<blocks(B * 2 * nl * n1), 256, 0, st>>>(w.dm_a.p, B, n1, nl, (u64)(delta % s.r1.m[0].q),
                                                           (u64)(delta % s.r1.m[1].q));
    VIA_LAUNCHED();
    u64 *in = w.dm_a.p, *out = w.dm_b.p;
    for (int i = 0; i < nd; ++i) {
      const long active = 1L << i;  // per query
      KeySel bit{w.rgsw_q1.p + i * rgsw1, active, B, nd * rgsw1};
      // One cluster per product and limb for few products (EXT_CLUSTER_MAX), one CTA above.
      if (B * active * n1 <= EXT_CLUSTER_MAX && ext_cluster_ok(s.r1, w.g_dmux)) {
        ext_cluster<EXT_DMUX>(s.r1, w.g_dmux, in, out, bit, 0, B * active, st);
        std::swap(in, out);
        continue;
      }
      if (dmux_fp_ok(s.r1, w.g_dmux)) {
        const dim3 grid((unsigned)(B * active), 2);
        if (n1 == 4096)
          k_dmux_fp<12><<<grid, 512, pair_smem(k_dmux_fp<12>, 2 * n1), st>>>(out, in, bit, s.r1, w.g_dmux);
        else
          k_dmux_fp<11><<<grid, 256, pair_smem(k_dmux_fp<11>, 2 * n1), st>>>(out, in, bit, s.r1, w.g_dmux);
        VIA_LAUNCHED();
        std::swap(in, out);
        continue;
      }
      if (R_fp_small(s.r1)) {
        external_products(s.r1, w.g_dmux, bit, in, B * active, w.dm_digits.p, w.dm_ext.p, false, st);
        intt_epi<INTT_DMUX>(s.r1, w.dm_ext.p, in, out, B * active, st);
        std::swap(in, out);
        continue;
      }
      external_products(s.r1, w.g_dmux, bit, in, B * active, w.dm_digits.p, w.dm_ext.p, true, st);
      k_dmux_combine<<<blocks(B * active * 2 * nl * n1), 256, 0, st>>>(out, in, w.dm_ext.p, B * active, n1, nl, s.r1);
      VIA_LAUNCHED();
      std::swap(in, out);
    }
    if (stop_stage == 3) return copy_out(in, (size_t)I * 2 * nl * n1);
    // ---- Step 3: ModSwitch q1 -> q2 (answer.rs:194-199) into the selection rows.
    mod_switch(s.r1, in, s.r2, w.sel.p, B * 2 * I, n1, st);
  }
  if (stop_stage == 4) return copy_out(w.sel.p, (size_t)I * 2 * n1);

  // ---- Step 4: FirstDim (answer.rs:204-205), one pass over the database for
  // the whole batch; the columns stay in the eval domain.
  to_eval(s.r2, w.sel.p, n1, B * 2 * I, st);
  const bool tiled = stop_stage != 5 && cmux_takes_tiles(s, B);
  first_dim_queries(s, w.sel.p, w.fd_out.p, nq, reinterpret_cast<uint8_t*>(w.sel_bytes.p), st, tiled);
  if (stop_stage == 5) {
    copy_out(w.fd_out.p, (size_t)J * 2 * n1);
    from_eval(s.r2, dump, n1, 2 * J, st);
    return;
  }

  if (split) VIA_CUDA(cudaStreamWaitEvent(st, w.ev_join, 0));  // the CMux / CRot RGSWs are ready

  // ---- Step 5: CMux tree (mux.rs:167-198), level by level in the eval domain:
  // diff = in[2j+1] - in[2j] (eval) -> coeff -> gadget product -> out[j] = in[2j] + ext.
  u64* cur = w.fd_out.p;
  for (int i = 0; i < nc; ++i) {
    const long half = (J >> i) / 2;  // CMuxes per query at this level
    KeySel bit{rgsw_b2 + i * rgsw2, half, B, nb * rgsw2};
    u64* nxt = cur == w.fd_out.p ? w.cm_b.p : w.fd_out.p;  // ping-pong between fd_out and cm_b
    if (cmux_fused_ok(s.r2, w.g_cmux)) {
      cmux_fused(s.r2, w.g_cmux, cur, nxt, bit, B * half, tiled && i == 0 ? B : 0, st);
      cur = nxt;
      continue;
    }
    k_rlwe_addsub<<<blocks(B * half * 2 * n1), 256, 0, st>>>(w.cm_diff.p, cur + 2 * n1, 2, cur, 2, -1, B * half, n1, 1,
                                                             s.r2);
    VIA_LAUNCHED();
    from_eval(s.r2, w.cm_diff.p, n1, B * 2 * half, st);
    external_products(s.r2, w.g_cmux, bit, w.cm_diff.p, B * half, w.cm_digits.p, w.cm_ext.p, false, st);
    k_rlwe_addsub<<<blocks(B * half * 2 * n1), 256, 0, st>>>(nxt, cur, 2, w.cm_ext.p, 1, +1, B * half, n1, 1, s.r2);
    VIA_LAUNCHED();
    cur = nxt;
  }
  // Selected columns back to coefficient form.
  if (!intt_epi<INTT_STORE>(s.r2, cur, nullptr, w.cr_ct.p, B, st)) {
    VIA_CUDA(cudaMemcpyAsync(w.cr_ct.p, cur, (size_t)B * 2 * n1 * 8, cudaMemcpyDeviceToDevice, st));
    from_eval(s.r2, w.cr_ct.p, n1, B * 2, st);
  }
  if (stop_stage == 6) return copy_out(w.cr_ct.p, 2 * (size_t)n1);

  // ---- Step 6: CRot, SlotExtract (rotate.rs:128-150).
  for (int i = 0; i < nr; ++i) {
    KeySel bit{rgsw_b2 + (nc + i) * rgsw2, 1, B, nb * rgsw2};
    if (ext_cluster_ok(s.r2, w.g_cmux) && w.g_cmux.small) {
      ext_cluster<EXT_CROT>(s.r2, w.g_cmux, w.cr_ct.p, w.cr_ct.p, bit, n1 - (1 << i), B, st);
      continue;
    }
    k_crot_diff_batch<<<blocks(B * 2 * n1), 256, 0, st>>>(w.cr_ct.p, n1, n1 - (1 << i), B, s.r2.m[0], w.cr_diff.p);
    VIA_LAUNCHED();
    if (R_fp_small(s.r2)) {
      external_products(s.r2, w.g_cmux, bit, w.cr_diff.p, B, w.cr_digits.p, w.cr_ext.p, false, st);
      intt_epi<INTT_ADD>(s.r2, w.cr_ext.p, w.cr_ct.p, w.cr_ct.p, B, st);
      continue;
    }
    external_products(s.r2, w.g_cmux, bit, w.cr_diff.p, B, w.cr_digits.p, w.cr_ext.p, true, st);
    k_rlwe_addsub<<<blocks(B * 2 * n1), 256, 0, st>>>(w.cr_ct.p, w.cr_ct.p, 1, w.cr_ext.p, 1, +1, B, n1, 1, s.r2);
    VIA_LAUNCHED();
  }
  if (stop_stage == 7) return copy_out(w.cr_ct.p, 2 * (size_t)n1);
  if (stop_stage == STOP_AFTER_CROT) return;
  resp_comp(s, w, w.cr_ct.p, B, d_mask, d_body, st);
}

void answer_device_stages(Server& s, const u64* d_query, int nq, u64* d_mask, u64* d_body, cudaStream_t st,
                          int stop_stage, u64* dump) {
  answer_device_stages(s, *s.ws, d_query, nq, d_mask, d_body, st, stop_stage, dump);
}

void answer_device(Server& s, const u64* d_query, u64* d_mask, u64* d_body, cudaStream_t st) {
  answer_device_stages(s, d_query, 1, d_mask, d_body, st, 0, nullptr);
}

u64* ws_query(Workspace& w) { return w.q_in.p; }
u64* ws_answer_mask(Workspace& w) { return w.a_mask.p; }
u64* ws_answer_body(Workspace& w) { return w.a_body.p; }
u64* workspace_query(Server& s) { return s.ws->q_in.p; }
u64* workspace_answer_mask(Server& s) { return s.ws->a_mask.p; }
u64* workspace_answer_body(Server& s) { return s.ws->a_body.p; }

// The whole answer for nq queries (~220 kernels) on the workspace buffers,
// captured once per batch size into a CUDA graph and replayed.
// st == nullptr captures (if needed) without launching.
void answer_graph(Server& s, Workspace& w, int nq, cudaStream_t st) {
  cudaGraphExec_t exec = nullptr;
  unsigned long long kernels = 0;
  if (w.graphs_gen != s.plan_gen) {  // the scan tiles changed since these were captured
    for (auto& g : w.graphs) cudaGraphExecDestroy(g.second);
    w.graphs.clear();
    w.graph_kernels.clear();
    w.graphs_gen = s.plan_gen;
  }
  for (size_t i = 0; i < w.graphs.size(); ++i)
    if (w.graphs[i].first == nq) {
      exec = w.graphs[i].second;
      kernels = w.graph_kernels[i].second;
    }
  if (!exec) {
    cudaGraph_t g;
    unsigned long long before = __atomic_load_n(&g_kernel_launches, __ATOMIC_RELAXED);
    VIA_CUDA(cudaStreamBeginCapture(w.capture, cudaStreamCaptureModeThreadLocal));
    try {
      answer_device_stages(s, w, w.q_in.p, nq, w.a_mask.p, w.a_body.p, w.capture, 0, nullptr);
    } catch (...) {
      cudaStreamEndCapture(w.capture, &g);
      throw;
    }
    VIA_CUDA(cudaStreamEndCapture(w.capture, &g));
    kernels = __atomic_load_n(&g_kernel_launches, __ATOMIC_RELAXED) - before;
    __atomic_sub_fetch(&g_kernel_launches, kernels, __ATOMIC_RELAXED);  // captured, not run
    cudaError_t e = cudaGraphInstantiate(&exec, g, cudaGraphInstantiateFlagUseNodePriority);
    cudaGraphDestroy(g);
    VIA_CUDA(e);
    w.graphs.push_back({nq, exec});
    w.graph_kernels.push_back({nq, kernels});
  }
  if (!st) return;
  VIA_CUDA(cudaGraphLaunch(exec, st));
  __atomic_add_fetch(&g_kernel_launches, kernels, __ATOMIC_RELAXED);
}

void answer_graph(Server& s, int nq, cudaStream_t st) { answer_graph(s, *s.ws, nq, st ? st : s.stream); }


// ===========================================================================
// VIA-B: repack of T CRot outputs into one RLWE (crates/via-primitives/src/
// conversion/repack.rs, crates/via-server/src/batch.rs:72-163).
//
// A level's list of MLWEs is stored as masks [count][rank][deg] and bodies
// [count][deg] at q2, coefficient form. Extr_{n_rec} turns each CRot output into
// an (n1/n_rec, n_rec)-MLWE; input t goes to position bitrev(t) (the reference
// swaps the T inputs into bit-reversed order) and positions >= T are zero
// MLWEs. Each level pairs entries (2p, 2p+1): embed_d interleaves the pair
// (slots 0 and 1), every embedded mask is key-switched with the level's
// q2-switched cascade keys, and conv_step's slot reduction gives
// masks_out[j] = -(P[j].mask + P[j+R/2].mask), body = embed_d(bodies) - sum P.body.
// Pairs of two zero MLWEs give zero MLWEs (zero digits), so only the leading
// nonzero entries are processed.
// ===========================================================================

// masks/bodies of the level-0 list from the CRot outputs ct [T][2][n1].
__global__ void k_repack_extr(const u64* __restrict__ ct, int T, int lt, int n1, int g, DevMod m, u64* __restrict__ masks,
                              u64* __restrict__ bodies) {
  const int D = n1 / g;
  const long total = (long)T * (D + 1) * g;
  const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= total) return;
  const int i = (int)(gid % g);
  const int k = (int)((gid / g) % (D + 1));
  const int t = (int)(gid / ((long)g * (D + 1)));
  int pos = 0;
  for (int b = 0; b < lt; ++b) pos |= ((t >> b) & 1) << (lt - 1 - b);
  const u64* mask = ct + (long)t * 2 * n1;
  const u64* body = mask + n1;
  if (k == D) {
    bodies[(long)pos * g + i] = body[(long)D * i];
    return;
  }
  u64 v;
  if (k == 0) {
    v = mask[(long)D * i];
  } else {
    // (X * pi_{D-k}(A))[i]: pi[i-1], and -pi[g-1] at i = 0.
    const int slot = D - k;
    v = i == 0 ? negmod(mask[(long)D * (g - 1) + slot], m.q) : mask[(long)D * (i - 1) + slot];
  }
  masks[((long)pos * D + k) * g + i] = v;
}

// embed_d (d = 2) of `pairs` pairs: emb_masks [pair][rank][2 n_in], emb_body [pair][2 n_in].
__global__ void k_repack_embed(const u64* __restrict__ masks, const u64* __restrict__ bodies, long pairs, int rank,
                               int n_in, u64* __restrict__ emb_masks, u64* __restrict__ emb_body) {
  const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= pairs * (rank + 1) * n_in) return;
  const int i = (int)(gid % n_in);
  const int k = (int)((gid / n_in) % (rank + 1));
  const long pr = gid / ((long)n_in * (rank + 1));
  const int n_out = 2 * n_in;
  if (k == rank) {
    emb_body[pr * n_out + 2 * i] = bodies[(2 * pr) * n_in + i];
    emb_body[pr * n_out + 2 * i + 1] = bodies[(2 * pr + 1) * n_in + i];
    return;
  }
  u64* o = emb_masks + (pr * rank + k) * n_out;
  o[2 * i] = masks[((2 * pr) * rank + k) * n_in + i];
  o[2 * i + 1] = masks[((2 * pr + 1) * rank + k) * n_in + i];
}

__global__ void k_sub_polys(const u64* __restrict__ a, const u64* __restrict__ b, long count, DevMod m,
                            u64* __restrict__ out) {
  const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= count) return;
  out[gid] = submod(a[gid], b[gid], m.q);
}

// The repack keys: for every output degree nout = 2 n_rec .. n1 the cascade step
// of that degree (rank_in = 2 n1 / nout RLevs of L_CK samples), switched from q1
// to q2 sample by sample (mod_switch_rlev, repack.rs:684-739) and transformed at
// q2. Must run before the cascade key itself is transformed.
void derive_repack_keys(Server& s) {
  const via_params& p = s.prm;
  if (via_b_batch(p) < 2 || !s.cascade_eval.p) return;
  const int n1 = p.n1, L = p.l_ck, nl = s.r1.nl;
  const u64 step_len = (u64)2 * n1 * L * 2 * nl;
  size_t total = 0;
  s.repack_off.clear();
  for (int nout = 2 * (int)p.n_rec; nout <= n1; nout <<= 1) {
    s.repack_off.push_back(total);
    total += (size_t)(2 * n1 / nout) * L * 2 * nout;
  }
  s.repack_eval.alloc(total);
  int level = 0;
  for (int nout = 2 * (int)p.n_rec; nout <= n1; nout <<= 1, ++level) {
    const int k = ilog2(nout);  // cascade step k has output degree 2^k
    const long polys = (long)(2 * n1 / nout) * L * 2;
    u64* dst = s.repack_eval.p + s.repack_off[level];
    mod_switch(s.r1, s.cascade_eval.p + (k - 1) * step_len, s.r2, dst, polys, nout, s.stream);
    to_eval(s.r2, dst, nout, polys, s.stream);
  }
}

struct RepackWs {
  int T = 0;
  DevBuf la_m, la_b, lb_m, lb_b, emb_m, emb_b, digits, P, bsum, packed;
  DevBuf crot_all;  // CRot outputs of a batch run in chunks [T * groups][2][n1]
  Gadget g;
};

// Called with the workspace owned by the caller.
static RepackWs& repack_ws(Server& s, Workspace& w) {
  if (!w.repack) {
    const via_params& p = s.prm;
    auto r = std::make_unique<RepackWs>();
    const long T = via_b_batch(p), n1 = p.n1, L = p.l_ck;
    const long pairs = std::max(1L, T / 2);
    r->T = (int)T;
    // Level lists hold at most T (+1 zero partner) entries of n1 + deg residues.
    r->la_m.alloc((T + 2) * n1);
    r->la_b.alloc((T + 2) * n1);
    r->lb_m.alloc((T + 2) * n1);
    r->lb_b.alloc((T + 2) * n1);
    r->emb_m.alloc(pairs * 2 * n1);
    r->emb_b.alloc(pairs * n1);
    r->digits.alloc(pairs * 2 * n1 * L);
    r->P.alloc(pairs * 4 * n1);
    r->bsum.alloc(pairs * n1);
    r->g = make_gadget(p.ck_base, (int)p.l_ck, s.r2);
    if (T > w.bmax) r->crot_all.alloc(T * 2 * n1);  // one batch runs in chunks of bmax queries
    w.repack = std::move(r);
  }
  return *w.repack;
}

static void repack(Server& s, Workspace& w, const u64* crot, u64* out_rlwe, cudaStream_t st) {
  const via_params& p = s.prm;
  RepackWs& r = repack_ws(s, w);
  const int n1 = p.n1, g = (int)p.n_rec, T = r.T, D = n1 / g;
  int lt = 0;
  while ((1 << lt) < T) ++lt;
  u64 *cm = r.la_m.p, *cb = r.la_b.p, *nm = r.lb_m.p, *nb = r.lb_b.p;
  {
    const long total = (long)T * (D + 1) * g;
    k_repack_extr<<<blocks(total), 256, 0, st>>>(crot, T, lt, n1, g, s.r2.m[0], cm, cb);
    VIA_LAUNCHED();
  }
  long active = T;  // leading nonzero entries of the current list
  int rank = D, level = 0;
  for (int n_in = g; n_in < n1; n_in <<= 1, rank >>= 1, ++level) {
    const int n_out = 2 * n_in;
    if (active & 1) {  // the last pair's partner is a zero MLWE
      VIA_CUDA(cudaMemsetAsync(cm + active * rank * n_in, 0, (size_t)rank * n_in * 8, st));
      VIA_CUDA(cudaMemsetAsync(cb + active * n_in, 0, (size_t)n_in * 8, st));
    }
    const long pairs = (active + 1) / 2;
    k_repack_embed<<<blocks(pairs * (rank + 1) * n_in), 256, 0, st>>>(cm, cb, pairs, rank, n_in, r.emb_m.p, r.emb_b.p);
    VIA_LAUNCHED();
    gadget_product(s.r2, r.g, r.emb_m.p, n_out, 1, 1, pairs * rank,
                   keys_cyclic(s.repack_eval.p + s.repack_off[level], rank), r.P.p, r.digits.p, st);
    const long items = pairs * (rank / 2 + 1) * n_out;
    k_cascade_reduce<<<blocks(items), 256, 0, st>>>(r.P.p, rank, n_out, 1, pairs, s.r2, nm, r.bsum.p);
    VIA_LAUNCHED();
    from_eval(s.r2, nm, n_out, pairs * (rank / 2), st);
    from_eval(s.r2, r.bsum.p, n_out, pairs, st);
    k_sub_polys<<<blocks(pairs * n_out), 256, 0, st>>>(r.emb_b.p, r.bsum.p, pairs * n_out, s.r2.m[0], nb);
    VIA_LAUNCHED();
    std::swap(cm, nm);
    std::swap(cb, nb);
    active = pairs;
  }
  // The rank-1 MLWE of degree n1 is the RLWE (mask, body).
  VIA_CUDA(cudaMemcpyAsync(out_rlwe, cm, (size_t)n1 * 8, cudaMemcpyDeviceToDevice, st));
  VIA_CUDA(cudaMemcpyAsync(out_rlwe + n1, cb, (size_t)n1 * 8, cudaMemcpyDeviceToDevice, st));
}

// answer_batch (srv/batch.rs:72-163): the prefix through CRot for the T queries
// (sharing one database scan), the repack, and RespComp once.
// `groups` VIA-B batches of T queries each (d_queries back to back); answer g
// goes to d_mask/d_body + g * n2.
void answer_batch_device(Server& s, Workspace& w, const u64* d_queries, int groups, u64* d_mask, u64* d_body,
                         cudaStream_t st) {
  const int T = via_b_batch(s.prm);
  const int n1 = s.prm.n1;
  if (T < 2) throw CudaError(100, "answer_batch: the server was set up for VIA-C (n_rec = n2)");
  if (!s.repack_eval.p) throw CudaError(100, "answer_batch: no repack keys");
  RepackWs& r = repack_ws(s, w);
  const int total = T * groups;
  const u64* crot = w.cr_ct.p;
  if (total <= w.bmax) {
    answer_device_stages(s, w, d_queries, total, nullptr, nullptr, st, STOP_AFTER_CROT, nullptr);
  } else {
    // More queries than the workspace holds: the prefix runs in chunks of bmax
    // queries (each chunk shares one database scan) and the CRot outputs are
    // gathered for the repack. Memory stays that of a bmax-query workspace.
    if (r.crot_all.n < (size_t)total * 2 * n1) {
      VIA_CUDA(cudaStreamSynchronize(st));
      r.crot_all.alloc((size_t)total * 2 * n1);
    }
    const size_t qlen = (size_t)query_lwes(s.prm) * lwe_len(s.prm);
    for (int q0 = 0; q0 < total; q0 += w.bmax) {
      const int nc = std::min(w.bmax, total - q0);
      answer_device_stages(s, w, d_queries + (size_t)q0 * qlen, nc, nullptr, nullptr, st, STOP_AFTER_CROT, nullptr);
      VIA_CUDA(cudaMemcpyAsync(r.crot_all.p + (size_t)q0 * 2 * n1, w.cr_ct.p, (size_t)nc * 2 * n1 * 8,
                               cudaMemcpyDeviceToDevice, st));
    }
    crot = r.crot_all.p;
  }
  if (!r.packed.p || r.packed.n < (size_t)groups * 2 * n1) r.packed.alloc((size_t)groups * 2 * n1);
  for (int g = 0; g < groups; ++g)
    repack(s, w, crot + (size_t)g * T * 2 * n1, r.packed.p + (size_t)g * 2 * n1, st);
  resp_comp(s, w, r.packed.p, groups, d_mask, d_body, st);
}

void answer_batch_device(Server& s, const u64* d_queries, u64* d_mask, u64* d_body, cudaStream_t st) {
  answer_batch_device(s, *s.ws, d_queries, 1, d_mask, d_body, st);
}


// ===========================================================================
// Standalone primitives (the reference's own kernel-level operations, on
// caller buffers; coefficient form in and out).
// ===========================================================================

// External products ext[c] = rgsw[c] (x) ct[c] (crates/via-primitives/src/
// encryption/rgsw.rs:108-121): every RGSW is transformed once per call (the
// reference re-transforms its samples per call too, rlev.rs:211-219), then the
// mask and body digits meet the neg_s_m and m samples.
//   rgsw [count][2L][2][nl][n], cts/out [count][2][nl][n].
// For what external_fp declines. Scratch: rgsw_eval (count * 2L * 2 * nl * n), digits (count * 2L * nl * n).
void prim_external_products(const DevRing& R, const Gadget& g, const u64* rgsw, const u64* cts, long count, u64* out,
                            u64* rgsw_eval, u64* digits, cudaStream_t st) {
  const long per = (long)R.nl * R.n;
  VIA_CUDA(cudaMemcpyAsync(rgsw_eval, rgsw, (size_t)count * 2 * g.L * 2 * per * 8, cudaMemcpyDeviceToDevice, st));
  to_eval(R, rgsw_eval, R.n, count * 2 * g.L * 2 * R.nl, st);
  external_products(R, g, KeySel{rgsw_eval, 1, count, 0}, cts, count, digits, out, true, st);
}

// X^k a (negacyclic) of mask and body, split into masks [count][nl][n] and
// bodies [count][nl][n] (element.rs:328, ops.rs:147-180).
__global__ void k_rotate_split(const u64* __restrict__ cts, const u64* __restrict__ shifts, long count, int n, int nl,
                               DevRing R, u64* __restrict__ masks, u64* __restrict__ bodies) {
  const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long per = (long)nl * n;
  if (gid >= count * 2 * per) return;
  const long c = gid / (2 * per);
  const int part = (int)((gid / per) % 2);
  const int l = (int)((gid % per) / n), i = (int)(gid % n);
  const u64 k = shifts[c] % (u64)(2 * n);
  u64 v = cts[gid];
  // A mask is split into digits, by steps on doubles among others: any 64-bit word mod q here.
  if (part == 0 && v >= R.m[l].q) v = reduce64(v, R.m[l]);
  const u64 pos = (u64)i + k;  // < 3n
  const int dst = (int)(pos % (u64)n);
  const bool neg = ((pos / (u64)n) & 1) != 0;
  const u64 q = R.m[l].q;
  u64* o = (part == 0 ? masks : bodies) + c * per + (long)l * n;
  o[dst] = neg && v ? q - v : v;
}

// out = (-prod.mask, body - prod.body) (keyswitch.rs:99-102).
__global__ void k_key_switch_finish(const u64* __restrict__ prod, const u64* __restrict__ bodies, long count, int n,
                                    int nl, DevRing R, u64* __restrict__ out) {
  const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long per = (long)nl * n;
  if (gid >= count * per) return;
  const long c = gid / per;
  const long r = gid % per;
  const int l = (int)(r / n);
  const u64 q = R.m[l].q;
  const u64 pm = prod[(2 * c) * per + r], pb = prod[(2 * c + 1) * per + r];
  out[(2 * c) * per + r] = pm ? q - pm : 0;
  out[(2 * c + 1) * per + r] = submod(bodies[c * per + r], pb, q);
}

// Key switches of rotated ciphertexts: out[c] = key_switch(K, X^{shift[c]} ct[c]).
//   key: RLev of L samples [L][2][nl][n] (coefficient form), shared by all.
// Scratch: key_eval (L * 2 * nl * n), masks/bodies (count * nl * n each),
// digits (count * L * nl * n), prod (count * 2 * nl * n).
void prim_key_switches(const DevRing& R, const Gadget& g, const u64* key, const u64* cts, const u64* shifts, long count,
                       u64* out, u64* key_eval, u64* masks, u64* bodies, u64* digits, u64* prod, cudaStream_t st) {
  const int n = R.n;
  const long per = (long)R.nl * n;
  VIA_CUDA(cudaMemcpyAsync(key_eval, key, (size_t)g.L * 2 * per * 8, cudaMemcpyDeviceToDevice, st));
  to_eval(R, key_eval, n, (long)g.L * 2 * R.nl, st);
  k_rotate_split<<<blocks(count * 2 * per), 256, 0, st>>>(cts, shifts, count, n, R.nl, R, masks, bodies);
  VIA_LAUNCHED();
  if (n >= 4 && ct_digits_ok(g.base, (u32)g.L, R)) {
    // Digits as bytes (in the product's memory, which the products then overwrite).
    int8_t* dig8 = reinterpret_cast<int8_t*>(prod);
    static_assert(CT_L <= 2 * 2 * 8, "18 bytes of digits fit the product's 32 bytes a coefficient");
    decompose_i8(R, g, masks, n, count, dig8, st);
    if (shared_key_fp(R, dig8, key_eval, bodies, g.L, count, out, st)) return;
    ntt_forward_i8_lazy(dig8, digits, n, R.nl, count * g.L * R.nl, R.t[0], R.t[1], st);
    mac(R, digits, keys_shared(key_eval), prod, g.L, n, count, st);
  } else {
    gadget_product(R, g, masks, n, 1, 1, count, keys_shared(key_eval), prod, digits, st);
  }
  from_eval(R, prod, n, count * 2 * R.nl, st);
  k_key_switch_finish<<<blocks(count * per), 256, 0, st>>>(prod, bodies, count, n, R.nl, R, out);
  VIA_LAUNCHED();
}

}  // namespace via
