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

#include "gadget.cuh"
#include "ntt_fp.cuh"
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
  size_t b_off;   // byte offset of its units in the key planes
  size_t c_off;   // its column constants: [item][2][16] doubles
  __host__ __device__ int items() const { return units + units / chain; }
};

inline CtStep ct_step(int n1, int n) {
  CtStep s{};
  s.n = n;
  s.half = n1 / n / 2;
  s.kp = (2 * CT_L * n + 15) / 16 * 16;
  s.G = n < 8 ? 8 / n : 1;
  s.chunks = (s.G * s.kp + CT_KC - 1) / CT_KC;
  s.units = n1 / CT_ROWS;
  // Body sums run over every output mask, so units of the same coefficients chain in
  // one accumulator: fewer epilogues and atomics, and with 128 mask units one item per SM
  // for a single tile. Longer chains of the larger steps would outlast a mask item.
  s.chain = n >= 128 ? 1 : (128 / n < 8 ? 128 / n : 8);
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

bool ct_supported(const via_params& p, const DevRing& R);
// Number of leading steps run as GEMMs.
int ct_steps(const via_params& p);
// Builds the key planes and column constants from the coefficient-form cascade key.
void ct_prepare(Server& s);
// Raises the kernel's shared-memory limit on the current device.
void ct_prepare_device();
// Runs the leading ct.steps steps for nlwe LWEs of d_query ([lwe][nl (n1 + 1)]): leaves the
// next step's signed digits in dig8 ([lwe][rank][L][degree]) and adds every step's body
// sums (coefficient form) to body[((2 n - 2 + y) * 2 + limb) * nlwe + lwe] (n the step's
// input degree, y < 2 n; ct_body_words(steps) words per LWE, zeroed by the caller), so that
// the lanes of a warp, which are LWEs, add to consecutive words. da and db are
// digit buffers of ct_digit_bytes(n1) bytes per LWE, LWEs rounded up to 8.
void ct_run(Server& s, const u64* d_query, long nlwe, uint8_t* da, uint8_t* db, int8_t* dig8, u64* body,
            cudaStream_t st);
inline size_t ct_body_words(int steps) { return (((size_t)2 << steps) - 2) * 2; }

}  // namespace via
