// The first steps of the LWE -> RLWE cascade (crates/via-primitives/src/conversion/
// cascade.rs:388-404, conv.rs:122-148) as exact integer GEMMs on the tensor cores.
//
// A step of input degree n key-switches R = n1 / n masks. Output mask j < R / 2 is
//   -sum over i in {j, j + R/2}, s < L, c < n of d_i,s[c] K_i,s.mask X^2c  (degree 2 n)
// with small digits d and the key K the same for every LWE, so for all LWEs together it
// is one matrix product per j: rows the LWEs, K dimension the (i, s, c) digits, columns the
// 2 n output coefficients with the entries +-K_i,s[y - 2c]. Residues are split into five
// unsigned bytes; digits are stored unsigned (w = d + o in [0, B)), and the constant part
// o * (column sum) is subtracted in the epilogue. Every byte product sum is exact in 32
// bits. Nothing is transformed: the epilogue folds the five sums into a residue per prime,
// splits it into the next step's digits and writes those, so a step is one kernel.
//
// The epilogue never forms the 75-bit coefficient c in [0, Q). With y_l = c_l (Q / q_l)^-1
// mod q_l, c / Q = y_0 / q_0 + y_1 / q_1 (mod 1); the inverses (and the minus sign of the
// masks) are folded into the key bytes. round(c S / Q) mod S, S = B^18 = T^3, then follows
// by three exact steps T y_l = p q_l + y_l' per prime, and the balanced digits are the
// plain base-B digits of that value plus o (1 + B + ... ), less o each.
#pragma once
#include <vector>

#include "gadget_fp.cuh"
#include "server.cuh"

namespace via {

constexpr int CT_L = 18;              // gadget depth (every NTT preset's)
constexpr int CT_LP = CT_L / 3;       // digits per piece
constexpr int CT_ROWS = 16;           // output coefficients per work unit
constexpr int CT_N = 2 * 5 * CT_ROWS; // MMA columns of a unit: [limb][byte][coefficient]
constexpr int CT_KC = 96;             // K bytes per pipeline stage
constexpr int CT_M = 128;             // LWEs per tile

// Geometry of the step of input degree n.
struct CtStep {
  int n, half;    // half = output masks
  int kp;         // K bytes of one output mask's digits (2 * L * n, padded to 16)
  int G;          // output masks per unit (units of n < 8 hold several)
  int chunks;     // pipeline stages per unit
  int units;      // mask units; as many body units follow
  int chain;      // body units summed in one accumulator: body items are units / chain
  __host__ __device__ int items() const { return units + units / chain; }
};

constexpr int CT_MANY = 3;  // LWE tiles from which body chains are long

inline CtStep ct_step(int n1, int n, int mtiles = 1) {
  CtStep s{};
  s.n = n;
  s.half = n1 / n / 2;
  s.kp = (2 * CT_L * n + 15) / 16 * 16;
  s.G = n < 8 ? 8 / n : 1;
  s.chunks = (s.G * s.kp + CT_KC - 1) / CT_KC;
  s.units = n1 / CT_ROWS;
  // Body sums run over every output mask, so units of the same coefficients chain in one
  // accumulator: fewer epilogues and atomics (seven steps of 2688 LWEs 1700 us without
  // chains, 1300 us with). With one or two tiles of LWEs, 128 mask units fill the GPU once
  // and a chain must not outlast a mask unit, which shorter chains of larger steps
  // keep to (18 LWEs, input degrees 16, 32, 64: 18.8, 23.5 and 28.3 us with the long
  // chains, 16.3, 18 and 25.6 with these).
  const int most = (mtiles >= CT_MANY ? 128 : n < 32 ? 64 : 32) / n;
  s.chain = most < 1 ? 1 : (most < 8 ? most : 8);
  return s;
}

// Digit split constants (see the head of this file).
struct CtDigits {
  double q[2], qinv[2], c24[2], yscale[2];
  u64 qi[2];
  double T;
  u32 Ti, base, o, M;  // M = ceil(2^(32 + sh) / T), 2^31 <= M < 2^32
  int sh;
  u32 off;             // o (T - 1) / (B - 1) + 2 T
};

// The fixed-point fractions f[piece] (32 bits, rounded up by less than 3 ulp) of
// the three base-T pieces of round(c S / Q) + o (S - 1) / (B - 1) mod S, most
// significant piece first, for c / Q = y0 / q0 + y1 / q1 mod 1, |y_l| <= 0.5625 q_l.
__device__ __forceinline__ void ct_pieces(double y0, double y1, const CtDigits& D, u32 (&f)[3]) {
  int p[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    // T y = qt q + r exactly, |r| <= 0.5625 q (fp_mulmod with its quotient kept);
    // the quotient's low word is read off the rounding sum.
    const double h0 = __dmul_rn(D.T, y0), h1 = __dmul_rn(D.T, y1);
    const double l0 = __fma_rn(D.T, y0, -h0), l1 = __fma_rn(D.T, y1, -h1);
    const double u0 = __fma_rn(h0, D.qinv[0], FP_ROUND), u1 = __fma_rn(h1, D.qinv[1], FP_ROUND);
    p[i] = __double2loint(u0) + __double2loint(u1);
    y0 = __dadd_rn(__fma_rn(-__dadd_rn(u0, -FP_ROUND), D.q[0], h0), l0);
    y1 = __dadd_rn(__fma_rn(-__dadd_rn(u1, -FP_ROUND), D.q[1], h1), l1);
  }
  // Rounding: the remainder y0 / q0 + y1 / q1 to the nearest integer (no ties: Q is odd).
  const double s = __fma_rn(y0, D.qinv[0], __dmul_rn(y1, D.qinv[1]));
  const double us = __dadd_rn(s, FP_ROUND);
  int rnd = __double2loint(us);
  if (fabs(__dadd_rn(s, -__dadd_rn(us, -FP_ROUND))) > 0.5 - 1e-12) {  // too near to tell in doubles (2^-38)
    const i128 num = (i128)(i64)y0 * (i128)D.qi[1] + (i128)(i64)y1 * (i128)D.qi[0];
    const i128 Q = (i128)D.qi[0] * D.qi[1];
    rnd = 2 * num > Q ? 1 : (2 * num < -Q ? -1 : 0);
  }
  // Pieces lie in (-1.2 T, 1.2 T); with off (below 3 T, at least 2 T) they are
  // nonnegative and below 4.3 T < 2^29, where umulhi(x, M) >> sh = floor(x / T).
  u32 carry = 2;
#pragma unroll
  for (int i = 2; i >= 0; --i) {
    const u32 x = (u32)p[i] + (i == 2 ? (u32)rnd : 0u) + D.off + carry - 2;
    carry = __umulhi(x, D.M) >> D.sh;
    const u32 u = x - carry * D.Ti;
    const u64 m = (u64)u * D.M;
    f[i] = (u32)(m >> D.sh) + 1;
  }
}

// The next base-B digit of a fraction, most significant first.
__device__ __forceinline__ u32 ct_digit(u32& f, u32 base) {
  const u64 m = (u64)f * base;
  f = (u32)m;
  return (u32)(m >> 32);
}

// Signed bytes of four unsigned digits w below 256: w - o.
__device__ __forceinline__ u32 ct_signed(u32 w, u32 o) { return (w + (128 - o) * 0x01010101u) ^ 0x80808080u; }

// Bytes per LWE of the digit buffers: the largest step's K bytes, and the slack a
// stage of the last unit may read past it.
inline size_t ct_digit_bytes(int n1) {
  size_t b = 0;
  for (int n = 1; n < n1; n <<= 1) {
    const CtStep s = ct_step(n1, n);
    const size_t k = (size_t)s.half * s.kp;
    b = k > b ? k : b;
  }
  return b + CT_KC;
}

// Whether the digit split above serves this gadget, and its constants.
bool ct_digits_ok(u64 base, u32 L, const DevRing& R);
CtDigits ct_digits(u64 base, const DevRing& R);
// Whether the GEMM steps serve this server's cascade.
bool ct_supported(const via_params& p, const DevRing& R);
// Leading steps prepared as GEMMs: input degrees 1 .. 128 (the last cascade step stays on
// transforms). Their key planes take 409 MB at n1 = 2048, 818 MB at 4096.
inline int ct_steps(const via_params& p) { return ilog2(p.n1) - 1 < 8 ? ilog2(p.n1) - 1 : 8; }
// Steps run as GEMMs for nlwe LWEs, of `prepared`: input degree 128 from two tiles on, where
// its 189 MB of planes serve enough of them (2688 LWEs: 513 us against 1370 us in the four
// transform kernels, 180 LWEs 59 against 95; one query's 42 against 26).
inline int ct_steps_for(int prepared, long nlwe) { return prepared > 7 && nlwe <= CT_M ? 7 : prepared; }
// Builds s.ct from the coefficient-form cascade key; leaves it null where the steps do not serve
// the server or its memory does not hold them. `base` (a view's) lends its own where they are equal.
void ct_prepare(Server& s, const Server* base);
// Raises the kernel's shared-memory limit on the current device.
void ct_prepare_device();
// Runs the leading steps for nlwe LWEs of d_query ([lwe][nl (n1 + 1)]): leaves the
// next step's signed digits in dig8 ([lwe][rank][L][degree]) and adds every step's body
// sums (coefficient form) to body[((2 n - 2 + y) * 2 + limb) * nlwe + lwe] (n the step's
// input degree, y < 2 n; ct_body_words(steps) words per LWE, zeroed by the caller), so that
// the lanes of a warp, which are LWEs, add to consecutive words. da and db are
// digit buffers of ct_digit_bytes(n1) bytes per LWE, LWEs rounded up to 8.
void ct_run(Server& s, const CtKeys& keys, const u64* d_query, long nlwe, uint8_t* da, uint8_t* db, int8_t* dig8, u64* body,
            cudaStream_t st);
inline size_t ct_body_words(int steps) { return (((size_t)2 << steps) - 2) * 2; }

}  // namespace via
