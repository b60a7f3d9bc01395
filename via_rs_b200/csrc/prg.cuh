// The reference's PRG (crates/via-primitives/src/sampling/prg.rs:57-205, SHAKE-256
// from the sha3 0.10.9 / keccak 0.1.6 crates): counter mode,
// block b = SHAKE256(seed || le64(b))[0..136), bytes served in order. Keccak-f[1600]
// is written from FIPS 202. Shared by the wire decoder and the device client.
#pragma once
#include <stdint.h>

#include <cmath>

#include "common.cuh"

namespace via {

constexpr int SHAKE_RATE = 136;  // bytes per block (SHAKE256)
constexpr int RATE_LANES = SHAKE_RATE / 8;

// Keccak-f[1600] (FIPS 202 section 3): round constants from the rc(t) LFSR
// (Algorithm 5) and rotation offsets from the (x, y) -> (y, 2x + 3y) walk
// (Algorithm 2), both evaluated at compile time.
struct KeccakConsts {
  u64 rc[24];
  int rot[25];
};

constexpr bool rc_bit(int t) {
  if (t % 255 == 0) return true;
  unsigned r = 1;  // R = 10000000 as bits r0..r7 with r0 the low bit
  for (int i = 1; i <= t % 255; ++i) {
    // R = 0 || R, then r0 ^= r8, r4 ^= r8, r5 ^= r8, r6 ^= r8, R = Trunc8(R).
    r <<= 1;
    const unsigned r8 = (r >> 8) & 1;
    r ^= r8;
    r ^= r8 << 4;
    r ^= r8 << 5;
    r ^= r8 << 6;
    r &= 0xFF;
  }
  return r & 1;
}

constexpr KeccakConsts make_keccak_consts() {
  KeccakConsts k{};
  for (int i = 0; i < 24; ++i) {
    u64 c = 0;
    for (int j = 0; j <= 6; ++j)
      if (rc_bit(j + 7 * i)) c |= (u64)1 << ((1 << j) - 1);
    k.rc[i] = c;
  }
  for (int i = 0; i < 25; ++i) k.rot[i] = 0;
  int x = 1, y = 0;
  for (int t = 0; t < 24; ++t) {
    k.rot[x + 5 * y] = ((t + 1) * (t + 2) / 2) % 64;
    const int nx = y, ny = (2 * x + 3 * y) % 5;
    x = nx;
    y = ny;
  }
  return k;
}

static __constant__ KeccakConsts c_keccak = make_keccak_consts();

__host__ __device__ inline const KeccakConsts& keccak_consts() {
#ifdef __CUDA_ARCH__
  return c_keccak;
#else
  static constexpr KeccakConsts k = make_keccak_consts();
  return k;
#endif
}

__host__ __device__ __forceinline__ u64 rotl64(u64 v, int s) { return s == 0 ? v : (v << s) | (v >> (64 - s)); }

__host__ __device__ inline void keccak_f1600(u64 (&A)[25]) {
  constexpr KeccakConsts R = make_keccak_consts();  // rotation amounts fold into the instructions
  const KeccakConsts& K = keccak_consts();
#pragma unroll 1
  for (int r = 0; r < 24; ++r) {
    u64 C[5], D[5], B[25];
#pragma unroll
    for (int x = 0; x < 5; ++x) C[x] = A[x] ^ A[x + 5] ^ A[x + 10] ^ A[x + 15] ^ A[x + 20];
#pragma unroll
    for (int x = 0; x < 5; ++x) D[x] = C[(x + 4) % 5] ^ rotl64(C[(x + 1) % 5], 1);
#pragma unroll
    for (int i = 0; i < 25; ++i) A[i] ^= D[i % 5];
#pragma unroll
    for (int x = 0; x < 5; ++x)
#pragma unroll
      for (int y = 0; y < 5; ++y) B[y + 5 * ((2 * x + 3 * y) % 5)] = rotl64(A[x + 5 * y], R.rot[x + 5 * y]);
#pragma unroll
    for (int x = 0; x < 5; ++x)
#pragma unroll
      for (int y = 0; y < 5; ++y) A[x + 5 * y] = B[x + 5 * y] ^ (~B[(x + 1) % 5 + 5 * y] & B[(x + 2) % 5 + 5 * y]);
    A[0] ^= K.rc[r];
  }
}

// One PRG block: SHAKE256(seed || le64(counter)) truncated to 136 bytes, as 17
// little-endian lanes. seed || counter (at most 72 bytes) fits one absorbed block.
__host__ __device__ inline void prg_block(const uint8_t* seed, int seed_len, u64 counter, u64 (&out)[RATE_LANES]) {
  u64 A[25];
#pragma unroll
  for (int i = 0; i < 25; ++i) A[i] = 0;
  // seed || counter || 0x1F as little-endian words (at most 73 bytes), then the last pad bit.
#pragma unroll
  for (int l = 0; l < 10; ++l) {
    u64 v = 0;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const int i = 8 * l + b, c = i - seed_len;
      const u64 byte = i < seed_len ? seed[i] : c < 8 ? (counter >> (8 * c)) & 0xFF : c == 8 ? 0x1F : 0;
      v |= byte << (8 * b);
    }
    A[l] = v;
  }
  A[RATE_LANES - 1] ^= (u64)0x80 << 56;
  keccak_f1600(A);
#pragma unroll
  for (int l = 0; l < RATE_LANES; ++l) out[l] = A[l];
}

// ---------------------------------------------------------------------------
// Rejection sampling of a whole mask by one CTA (uniform_below, prg.rs:160-206).
//
// Every limb's draw takes the same nb bytes, so candidate c sits at byte
// pos + c nb of the stream whatever was rejected before it; only the limb it is
// tried against (draw index mod nl) depends on the earlier candidates. That
// dependence is a function of the parity alone, (start parity) -> (accepted
// candidates), and these functions compose associatively, so a prefix scan over
// the threads finds every candidate's draw index. Thread i of a chunk takes
// WALK_V consecutive candidates (WALK_V nb bytes: whole words).
//
// A draw rejected 64 times in a row must end the stream with an error. Such a
// run covers at least seven whole threads, so any seven neighbours of a warp
// without an accepted candidate, or four at a warp's edge, return
// WALK_UNDECIDED (2^-46 a warp at an acceptance of 0.63, the secure preset's
// primes; 2^-31 at 1/2, the least a prime can have), as does a stream longer
// than `avail` bytes: the caller then takes the sequential path, which decides
// it exactly.
// ---------------------------------------------------------------------------
// 4608 candidates a chunk: a mask of 4096 draws and its few rejections in one (512 threads need
// a second chunk for nearly every mask: 24 queries of 40 masks 261 us, 195 with 576).
constexpr int WALK_THREADS = 576;
constexpr int WALK_V = 8;
constexpr long WALK_UNDECIDED = -1;

struct WalkLimbs {
  u64 q[2], mask[2];
  int nb, nl;
};

// Bytes to generate ahead for `draws` accepted draws of `nbytes` bytes below q:
// the mean (draws / acceptance) and eight standard deviations.
inline double walk_bytes(double draws, u64 q, int nbytes) {
  const int bits = 64 - __builtin_clzll(q);
  const double a = (double)q / (bits == 64 ? 18446744073709551616.0 : (double)((u64)1 << bits));
  return nbytes * (draws / a + 8.0 * std::sqrt(draws * (1.0 - a)) / a);
}

struct WalkShared {
  u32 warp_cnt[WALK_THREADS / 32];  // accepted from parity 0 | from parity 1 << 16
  long end;                         // candidates consumed once the last draw is accepted
  int undecided, total;
  u64 draw[WALK_THREADS * WALK_V];  // a chunk's draws, on their way to coalesced stores
};

// Accepted candidates of `acc` (bit i: limb 0; bit 8 + i: limb 1) from parity s.
__device__ __forceinline__ int walk_count(u32 acc, int nl, int s) {
  int cnt = 0;
#pragma unroll
  for (int i = 0; i < WALK_V; ++i) cnt += (acc >> (i + 8 * (nl == 2 ? ((s + cnt) & 1) : 0))) & 1;
  return cnt;
}

// a then b, both packed as in WalkShared::warp_cnt.
__device__ __forceinline__ u32 walk_compose(u32 a, u32 b) {
  const u32 a0 = a & 0xFFFF, a1 = a >> 16;
  const u32 r0 = a0 + ((a0 & 1) ? b >> 16 : b & 0xFFFF);
  const u32 r1 = a1 + ((a1 & 1) ? b & 0xFFFF : b >> 16);
  return r0 | (r1 << 16);
}

// Draws the n1 * nl mask coefficients (row-major, limb 0 first) from the stream
// `words` (little-endian, `avail` bytes, a multiple of 8) at byte `pos` into out
// [nl][n1]. Returns the candidates consumed. Called by all WALK_THREADS threads.
__device__ inline long walk_mask(const u64* __restrict__ words, u64 avail, u64 pos, const WalkLimbs& W, int n1,
                                 u64* __restrict__ out, WalkShared& sh) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int total = n1 * W.nl;
  if (tid == 0) {
    sh.end = WALK_UNDECIDED;
    sh.undecided = 0;
  }
  int base = 0;  // draws accepted so far
  for (long c0 = 0; base < total; c0 += (long)WALK_THREADS * WALK_V) {
    const u64 at = pos + (u64)(c0 + (long)tid * WALK_V) * W.nb;
    const bool have = at + (u64)WALK_V * W.nb <= avail;
    // The next chunk or, after the last, what the caller draws next.
    if (lane % 2 == 0 && at + (u64)WALK_THREADS * WALK_V * W.nb < avail)
      asm volatile("prefetch.global.L1 [%0];" ::"l"(words + ((at + (u64)WALK_THREADS * WALK_V * W.nb) >> 3)));
    u64 w[9];
    const int sh8 = 8 * (int)(at & 7);
#pragma unroll
    for (int i = 0; i < 9; ++i) {
      const u64 k = (at >> 3) + i;
      w[i] = (have && i <= W.nb && k < avail / 8) ? words[k] : 0;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (sh8) w[i] = (w[i] >> sh8) | (w[i + 1] << (64 - sh8));
    u64 v[WALK_V];
    u32 acc = 0;
    switch (W.nb) {  // candidate i starts at byte i nb of w
#define VIA_WALK_CASE(NB)                                                                    \
  case NB: {                                                                                 \
    _Pragma("unroll") for (int i = 0; i < WALK_V; ++i) {                                     \
      constexpr int B = 8 * NB;                                                              \
      const int bit = i * B, lo = bit >> 6, off = bit & 63;                                  \
      u64 x = w[lo] >> off;                                                                  \
      if (off + B > 64) x |= w[lo + 1] << ((64 - off) & 63);                                 \
      v[i] = x;                                                                              \
    }                                                                                        \
  } break;
      VIA_WALK_CASE(1)
      VIA_WALK_CASE(2)
      VIA_WALK_CASE(3)
      VIA_WALK_CASE(4)
      VIA_WALK_CASE(5)
      VIA_WALK_CASE(6)
      VIA_WALK_CASE(7)
      default:
        VIA_WALK_CASE(8)
#undef VIA_WALK_CASE
    }
    if (have) {
#pragma unroll
      for (int i = 0; i < WALK_V; ++i) {
        acc |= (u32)((v[i] & W.mask[0]) < W.q[0]) << i;
        acc |= (u32)((v[i] & W.mask[1]) < W.q[1]) << (8 + i);
      }
    }
    // No rejected draw in the chunk (six masks of ten with the paper preset's primes, 2^-20 and
    // 2^-12 short of a power of two): candidate and draw index coincide.
    const int s0 = W.nl == 2 ? base & 1 : 0;
    u32 need = 0;  // the thread's candidates that are draws then
#pragma unroll
    for (int i = 0; i < WALK_V; ++i)
      if (base + tid * WALK_V + i < total) need |= 1u << (i + (W.nl == 2 ? 8 * ((s0 + i) & 1) : 0));
    if (__syncthreads_and((acc & need) == need)) {
      // Through shared memory, so that a warp's stores are consecutive (a thread's own eight
      // draws would be 32 bytes apart from its neighbour's).
      const auto slot = [](int x) { return x ^ ((x >> 4) & 15); };
#pragma unroll
      for (int i = 0; i < WALK_V; ++i) sh.draw[slot(tid * WALK_V + i)] = v[i] & W.mask[W.nl == 2 ? (s0 + i) & 1 : 0];
      __syncthreads();
#pragma unroll
      for (int i = 0; i < WALK_V; ++i) {
        const int x = i * WALK_THREADS + tid, d = base + x, l = W.nl == 2 ? d & 1 : 0;
        if (d < total) out[(size_t)l * n1 + (W.nl == 2 ? d >> 1 : d)] = sh.draw[slot(x)];
      }
      if (base + WALK_THREADS * WALK_V >= total) return c0 + (total - base);
      base += WALK_THREADS * WALK_V;
      continue;
    }
    const u32 own = (u32)walk_count(acc, W.nl, 0) | ((u32)walk_count(acc, W.nl, 1) << 16);
    u32 incl = own;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const u32 o = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl = walk_compose(o, incl);
    }
    u32 excl = __shfl_up_sync(0xffffffffu, incl, 1);
    if (lane == 0) excl = 0;
    __syncthreads();  // the previous chunk's readers are done with sh
    if (lane == 31) sh.warp_cnt[warp] = incl;
    __syncthreads();
    // Every warp scans the warps' counts itself.
    u32 wi = lane < WALK_THREADS / 32 ? sh.warp_cnt[lane] : 0;
#pragma unroll
    for (int d = 1; d < WALK_THREADS / 32; d <<= 1) {
      const u32 o = __shfl_up_sync(0xffffffffu, wi, d);
      if (lane >= d) wi = walk_compose(o, wi);
    }
    const u32 all = __shfl_sync(0xffffffffu, wi, WALK_THREADS / 32 - 1);
    const u32 before = warp ? __shfl_sync(0xffffffffu, wi, warp - 1) : 0;
    const auto from = [](u32 f, int s) { return (int)(s ? f >> 16 : f & 0xFFFF); };
    int d = base + from(walk_compose(before, excl), s0);
    const int d0 = d;
#pragma unroll
    for (int i = 0; i < WALK_V; ++i) {
      const int l = W.nl == 2 ? d & 1 : 0;
      if ((acc >> (i + 8 * l)) & 1) {
        if (d < total) {
          out[(size_t)l * n1 + (W.nl == 2 ? d >> 1 : d)] = v[i] & W.mask[l];
          if (d == total - 1) sh.end = c0 + (long)tid * WALK_V + i + 1;
        }
        ++d;
      }
    }
    // Threads before the end of the mask that accepted nothing.
    const u32 none = __ballot_sync(0xffffffffu, d == d0 && d0 < total);
    const u32 r2 = none & (none >> 1), r4 = r2 & (r2 >> 2), r7 = r4 & (r4 >> 3);
    if (lane == 0 && (r7 || (none & 0xF) == 0xF || (none >> 28) == 0xF)) sh.undecided = 1;
    base += from(all, s0);
    __syncthreads();
    if (sh.undecided) {
      __syncthreads();
      return WALK_UNDECIDED;
    }
  }
  const long end = sh.end;
  __syncthreads();  // the next mask resets sh
  return end;
}

}  // namespace via
