// Exact integer GEMMs of the cascade's first steps (cascade_tc.cuh).
#include "cascade_tc.cuh"

#include <algorithm>

#include "tc.cuh"

namespace via {
namespace {

constexpr int CT_EPI = 16;  // epilogue warps: four per TMEM lane quadrant, four coefficients each
constexpr int CT_THREADS = 64 + 32 * CT_EPI;
constexpr int CT_ACC = 3;   // accumulator sets of CT_N TMEM columns
constexpr int CT_STAGE_A = CT_M * CT_KC, CT_STAGE_B = CT_N * CT_KC, CT_STAGE = CT_STAGE_A + CT_STAGE_B;
constexpr int CT_STAGES = 7;
constexpr int CT_SMEM = CT_STAGES * CT_STAGE + 256;
static_assert(CT_SMEM <= 227 * 1024, "shared memory per block");

struct CtParams {
  CtStep st;
  CtDigits D;
  const uint8_t* a;   // digits of this step
  const uint8_t* b;   // key planes of this step
  const double* c;    // column constants of this step
  uint8_t* out;       // next GEMM step's digits, or null
  int8_t* dig8;       // signed digits [lwe][half][L][2 n] when this is the last GEMM step
  u64* body;          // this step's body accumulators [2 n][2][nlwe]
  int* err;
  long nlwe;
  size_t a_tile, out_tile;  // bytes per 128-LWE tile
  int mtiles, out_kp, out_half;
  unsigned fault_ns;  // test hook: > 0 makes the epilogue's first wait run out after this long
};

// Item -> its first unit, and its units. Units 0 .. units - 1 are mask units.
__host__ __device__ __forceinline__ int ct_item(const CtStep& S, int item, int& len) {
  len = item < S.units ? 1 : S.chain;
  return item < S.units ? item : S.units + (item - S.units) * S.chain;
}

// First output mask of a unit. Mask units of n >= 8 run over the coefficient blocks of
// one output mask, body units over the output masks of one coefficient block.
__host__ __device__ __forceinline__ int ct_first_mask(const CtStep& S, int unit) {
  const int mu = unit < S.units ? unit : unit - S.units;
  if (S.n < 8) return mu * S.G;
  return unit < S.units ? mu / (2 * S.n / CT_ROWS) : mu % S.half;
}

// First step's digits from the query: K position j kp + which L + s of LWE w holds
// digit s of mask which * half + j. Thread = (8-LWE group, j, LWE of the group).
__global__ void __launch_bounds__(256) k_ct_digits(const u64* __restrict__ q, long nlwe, long lwe_len, int n1,
                                                   CtStep st, CtDigits D, size_t tile, uint8_t* __restrict__ out) {
  const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const int l8 = (int)(gid & 7);
  const int j = (int)((gid >> 3) % st.half);
  const long grp = (gid >> 3) / st.half;
  const long w = grp * 8 + l8;
  if (w >= nlwe) return;
  constexpr int KP = (2 * CT_L + 15) / 16 * 16;
  u32 word[KP / 4];
#pragma unroll
  for (int i = 0; i < KP / 4; ++i) word[i] = 0;
#pragma unroll
  for (int which = 0; which < 2; ++which) {
    const u64* src = q + w * lwe_len + j + which * st.half;
    u64 a0 = src[0], a1 = src[n1];
    if (a0 >= (1ull << 47)) a0 %= D.qi[0];  // as the integer path: any 64-bit input word
    if (a1 >= (1ull << 47)) a1 %= D.qi[1];
    u32 f[3];
    ct_pieces(fp_mulmod(fp_from_u64(a0), D.yscale[0], D.q[0], D.qinv[0]),
              fp_mulmod(fp_from_u64(a1), D.yscale[1], D.q[1], D.qinv[1]), D, f);
#pragma unroll
    for (int s = 0; s < CT_L; ++s) {
      const int at = which * CT_L + s;
      word[at / 4] |= ct_digit(f[s / CT_LP], D.base) << (8 * (at % 4));
    }
  }
  const long mt = w / CT_M;
  const long left = nlwe - mt * CT_M;
  const int ng = (int)(((left < CT_M ? left : CT_M) + 7) / 8);
  uint8_t* o = out + mt * tile + ((size_t)j * (KP / 16) * ng + (w % CT_M) / 8) * 128 + (w & 7) * 16;
#pragma unroll
  for (int b = 0; b < KP / 16; ++b)
    *reinterpret_cast<uint4*>(o + (size_t)b * ng * 128) =
        make_uint4(word[4 * b], word[4 * b + 1], word[4 * b + 2], word[4 * b + 3]);
}

// One step. Persistent CTAs walk the (unit, LWE tile) items, tiles fastest, so the CTAs
// that run together share a unit's key planes in L2. Warp 0 copies the (digit, key) chunks
// into a ring of shared-memory stages, warp 1 issues the MMAs into one of three TMEM
// accumulator sets, sixteen epilogue warps fold the previous one.
//
// Bounds: up to n = 32 the epilogue (128 x 16 coefficients, 64 FP64 and about 200 integer
// instructions each, 10000 cycles a mask unit) is longer than the MMAs (36 n K bytes, 166
// cycles for 32 of them: kind::i8 runs at 4000 multiply-adds a cycle and SM here); from
// n = 64 on the MMAs are. One query (18 LWEs): 11 to 15 us a step up to n = 16, of which
// 5 us are launch and first loads and 5 us one epilogue. 2688 LWEs: 116 us (n = 8) to 360 us
// (n = 64) a step, against 2400 us in four kernels on transforms.
__global__ void __launch_bounds__(CT_THREADS, 1) k_ct_step(const __grid_constant__ CtParams P) {
  extern __shared__ __align__(1024) uint8_t smem[];
  u64* full = reinterpret_cast<u64*>(smem + CT_STAGES * CT_STAGE);
  u64* empty = full + CT_STAGES;
  u64* acc_full = empty + CT_STAGES;
  u64* acc_empty = acc_full + CT_ACC;
  u64* drain = acc_empty + CT_ACC;
  u64* never = drain + 1;  // the test hook's barrier: initialised, never arrived on
  u32* tmem_slot = reinterpret_cast<u32*>(never + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < CT_STAGES; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, 1);
    }
    for (int a = 0; a < CT_ACC; ++a) {
      mbar_init(acc_full + a, 1);
      mbar_init(acc_empty + a, CT_EPI * 32);
    }
    mbar_init(drain, 1);
    mbar_init(never, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const u32 tmem = *tmem_slot;
  const CtStep& S = P.st;
  const int items = S.items() * P.mtiles;
  const int upj = S.n >= 8 ? 2 * S.n / CT_ROWS : 1;  // units per output mask (n >= 8)

  if (warp == 0) {
    if (lane == 0) {
      int s = 0;
      u32 ph = 0, armed = 0, armed_par = 0;
      bool ok = true;
      for (int it = blockIdx.x; ok && it < items; it += gridDim.x) {
        const int mt = it % P.mtiles;
        int len;
        const int unit0 = ct_item(S, it / P.mtiles, len);
        const long left = P.nlwe - (long)mt * CT_M;
        const u32 ng = (u32)((min(left, (long)CT_M) + 7) / 8);
        const u32 abytes = CT_KC / 16 * ng * 128;
        const uint8_t* asrc = nullptr;
        const uint8_t* bsrc = P.b + (size_t)unit0 * S.chunks * CT_STAGE_B;
        for (int i = 0, kc = 0; i < len * S.chunks; ++i) {
          if (kc == 0) asrc = P.a + mt * P.a_tile + (size_t)ct_first_mask(S, unit0 + i / S.chunks) * S.kp / 16 * ng * 128;
          if (!mbar_wait(empty + s, ph ^ 1, abort_flag)) {
            ok = false;
            break;
          }
          uint8_t* dst = smem + s * CT_STAGE;
          mbar_expect_tx(full + s, abytes + CT_STAGE_B);
          bulk_g2s(dst, asrc + (size_t)kc * abytes, abytes, full + s);
          bulk_g2s(dst + CT_STAGE_A, bsrc + (size_t)i * CT_STAGE_B, CT_STAGE_B, full + s);
          if (++kc == S.chunks) kc = 0;
          armed |= 1u << s;
          armed_par = (armed_par & ~(1u << s)) | (ph << s);
          if (++s == CT_STAGES) {
            s = 0;
            ph ^= 1;
          }
        }
      }
      if (!ok) {
        atomicOr(P.err, 16);
        *abort_flag = 1;
      }
      // Every copy started here lands before the CTA can exit.
      for (int k = 0; k < CT_STAGES; ++k)
        if ((armed >> k) & 1)
          if (!mbar_wait(full + k, (armed_par >> k) & 1, abort_flag, false)) atomicOr(P.err, 16);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int s = 0, a = 0;
      u32 ph = 0, aph = 0;
      bool ok = true;
      const u32 idesc = idesc_u8(CT_N);
      constexpr u32 lbo_b = CT_N / 8 * 128;
      for (int it = blockIdx.x; ok && it < items; it += gridDim.x) {
        const long left = P.nlwe - (long)(it % P.mtiles) * CT_M;
        // Tiles of fewer than 128 LWEs: rows past the last 8-LWE group read what
        // follows in the stage; their accumulator lanes are never used.
        const u32 lbo_a = (u32)((min(left, (long)CT_M) + 7) / 8) * 128;
        if (!mbar_wait(acc_empty + a, aph ^ 1, abort_flag)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const u32 dacc = tmem + (u32)(a * CT_N);
        int nk;
        ct_item(S, it / P.mtiles, nk);
        nk *= S.chunks;
        for (int kc = 0; kc < nk; ++kc) {
          if (!mbar_wait(full + s, ph, abort_flag)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const u32 sa = smem_addr(smem + s * CT_STAGE), sb = sa + CT_STAGE_A;
#pragma unroll
          for (int ks = 0; ks < CT_KC / 32; ++ks)
            mma_i8(dacc, smem_desc(sa + ks * 2 * lbo_a, lbo_a, 128), smem_desc(sb + ks * 2 * lbo_b, lbo_b, 128), idesc,
                   kc == 0 && ks == 0 ? 0u : 1u);
          mma_commit(empty + s);
          if (++s == CT_STAGES) {
            s = 0;
            ph ^= 1;
          }
        }
        if (!ok) break;
        mma_commit(acc_full + a);
        if (++a == CT_ACC) {
          a = 0;
          aph ^= 1;
        }
      }
      if (!ok) {
        atomicOr(P.err, 32);
        *abort_flag = 1;
      }
      mma_commit(drain);
      if (!mbar_wait(drain, 0, abort_flag, false)) atomicOr(P.err, 32);
    }
  } else {
    const int quad = warp & 3, part = (warp - 2) >> 2;
    const int m = quad * 32 + lane;  // LWE of the tile
    const int n_out = 2 * S.n;
    int a = 0;
    u32 aph = 0;
    bool ok = P.fault_ns == 0 || mbar_wait_never(never, P.fault_ns);
    for (int it = blockIdx.x; ok && it < items; it += gridDim.x) {
      const int mt = it % P.mtiles;
      int len;
      const int unit = ct_item(S, it / P.mtiles, len);
      const long w = (long)mt * CT_M + m;
      double cr[2][4];  // the column constants, on their way while the accumulator fills
      {
        const double* cc = P.c + (size_t)(it / P.mtiles) * 2 * CT_ROWS + part * 4;
#pragma unroll
        for (int l = 0; l < 2; ++l)
#pragma unroll
          for (int r = 0; r < 4; r += 2) {
            const double2 x = __ldg(reinterpret_cast<const double2*>(cc + l * CT_ROWS + r));
            cr[l][r] = x.x;
            cr[l][r + 1] = x.y;
          }
      }
      if (!__all_sync(0xffffffffu, mbar_wait(acc_full + a, aph, abort_flag))) {
        ok = false;
        break;
      }
      tc_fence_after();
      const bool quad_live = (long)mt * CT_M + quad * 32 < P.nlwe;  // warp-uniform
      u32 v[2][5][4];
      if (quad_live) {
        const u32 tb = tmem + (u32)(a * CT_N) + ((u32)(quad * 32) << 16) + part * 4;
#pragma unroll
        for (int l = 0; l < 2; ++l)
#pragma unroll
          for (int k = 0; k < 5; ++k) tmem_ld4(tb + (u32)((l * 5 + k) * CT_ROWS), v[l][k]);
        tmem_wait_ld();
#pragma unroll
        for (int l = 0; l < 2; ++l)
#pragma unroll
          for (int k = 0; k < 5; ++k) pin(v[l][k]);
      }
      tc_fence_before();
      mbar_arrive(acc_empty + a);
      if (++a == CT_ACC) {
        a = 0;
        aph ^= 1;
      }
      if (!quad_live || w >= P.nlwe) continue;
      // Fold: five byte sums (below 2^31) less the digit offset's constant, mod q_l,
      // |y| <= q / 2 + 1.
      double y[2][4];
#pragma unroll
      for (int l = 0; l < 2; ++l) {
        const double q = P.D.q[l], qinv = P.D.qinv[l];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const u64 lo = (u64)v[l][0][r] + ((u64)v[l][1][r] << 8) + ((u64)v[l][2][r] << 16);
          const u64 hi = (u64)v[l][3][r] + ((u64)v[l][4][r] << 8);
          const double x = __dadd_rn(__dadd_rn(fp_from_u64(lo), fp_mulmod(fp_from_u64(hi), P.D.c24[l], q, qinv)), -cr[l][r]);
          y[l][r] = __fma_rn(-__dadd_rn(__fma_rn(x, qinv, FP_ROUND), -FP_ROUND), q, x);
        }
      }
      const int r0 = part * 4;
      if (unit >= S.units) {  // body sums, canonical, added over the items of the same coefficients
        const int yy = S.n >= 8 ? (unit - S.units) / S.half * CT_ROWS + r0 : r0 % n_out;
        unsigned long long* o = reinterpret_cast<unsigned long long*>(P.body) + (size_t)yy * 2 * P.nlwe + w;
#pragma unroll
        for (int l = 0; l < 2; ++l) {
          u64 b[4];
#pragma unroll
          for (int r = 0; r < 4; ++r) b[r] = __double2ull_rn(fp_canonical(y[l][r], P.D.q[l], P.D.qinv[l]));
          if (S.n == 1) {
            b[0] += b[2];
            b[1] += b[3];
          }
#pragma unroll
          for (int r = 0; r < 4; ++r)
            if (S.n > 1 || r < 2) atomicAdd(o + (size_t)(2 * r + l) * P.nlwe, b[r]);
        }
        continue;
      }
      // Rows part * 4 .. + 3 of the unit: output mask jj, coefficients yy .. (n >= 2),
      // or masks jj, jj + 1 of two coefficients each (n = 1).
      const int jj = S.n >= 8 ? unit / upj : unit * S.G + r0 / n_out;
      const int yy = S.n >= 8 ? (unit % upj) * CT_ROWS + r0 : r0 % n_out;
      u32 f[4][3];
#pragma unroll
      for (int r = 0; r < 4; ++r) ct_pieces(y[0][r], y[1][r], P.D, f[r]);
      if (P.out) {
        const int which = jj / P.out_half, j2 = jj % P.out_half;
        const long left = P.nlwe - (long)mt * CT_M;
        const u32 ngb = (u32)((min(left, (long)CT_M) + 7) / 8) * 128;
        uint8_t* base = P.out + mt * P.out_tile + (m / 8) * 128 + (m & 7) * 16;
        u32 pos = (u32)(j2 * P.out_kp + which * CT_L * n_out + yy);
        uint8_t* o = base + (size_t)(pos >> 4) * ngb + (pos & 15);  // n >= 8: s steps by whole 16-byte rows
        const u32 step = (u32)(n_out >> 4) * ngb;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int k = 0; k < CT_LP; ++k) {
            const u32 d = ct_digit(f[0][i], P.D.base) | ct_digit(f[1][i], P.D.base) << 8 |
                          ct_digit(f[2][i], P.D.base) << 16 | ct_digit(f[3][i], P.D.base) << 24;
            if (S.n >= 8) {
              *reinterpret_cast<u32*>(o) = d;
              o += step;
            } else if (S.n > 1) {
              *reinterpret_cast<u32*>(base + ((pos >> 4) * ngb + (pos & 15))) = d;
              pos += n_out;
            } else {
              *reinterpret_cast<uint16_t*>(base + ((pos >> 4) * ngb + (pos & 15))) = (uint16_t)d;
              const u32 p2 = pos + P.out_kp;
              *reinterpret_cast<uint16_t*>(base + ((p2 >> 4) * ngb + (p2 & 15))) = (uint16_t)(d >> 16);
              pos += n_out;
            }
          }
      } else {
        int8_t* o = P.dig8 + ((w * S.half + jj) * CT_L) * (long)n_out + yy;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int k = 0; k < CT_LP; ++k, o += n_out) {
            u32 d = 0;
#pragma unroll
            for (int r = 0; r < 4; ++r) d |= ct_digit(f[r][i], P.D.base) << (8 * r);
            d = ct_signed(d, P.D.o);
            if (S.n == 1) {
              *reinterpret_cast<uint16_t*>(o) = (uint16_t)d;
              *reinterpret_cast<uint16_t*>(o + CT_L * n_out) = (uint16_t)(d >> 16);
            } else {
              *reinterpret_cast<u32*>(o) = d;
            }
          }
      }
    }
    if (!ok) {
      atomicOr(P.err, 64);
      *abort_flag = 1;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// Key planes of one step: thread = (unit, 16 K bytes, limb, row), five 16-byte core-matrix
// rows each. key: the step's coefficient-form samples [R][L][2][2][n_out]. Mask entries
// are -K (Q / q_l)^-1 mod q_l, body entries K. CHECK: sets *differs where `planes` holds others.
template <bool CHECK>
__global__ void k_ct_planes(const u64* __restrict__ key, CtStep st, DevRing R, u64 inv0, u64 inv1,
                            uint8_t* __restrict__ planes, int* differs) {
  const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const int k16s = st.chunks * (CT_KC / 16);
  if (gid >= (long)2 * st.units * k16s * 32) return;
  const int r = (int)(gid & 15), l = (int)((gid >> 4) & 1);
  const int k16 = (int)((gid >> 5) % k16s), unit = (int)((gid >> 5) / k16s);
  const int mb = unit >= st.units, mu = unit - mb * st.units;
  const int n_out = 2 * st.n, L = CT_L;
  const int g_row = st.n >= 8 ? 0 : r / n_out;
  const int j = ct_first_mask(st, unit) + g_row;
  const int y = st.n >= 8 ? (mb ? mu / st.half : mu % (n_out / CT_ROWS)) * CT_ROWS + r : r % n_out;
  const DevMod& m = R.m[l];
  const u64 inv = l ? inv1 : inv0;
  u32 word[5][4];
#pragma unroll
  for (int k = 0; k < 5; ++k) word[k][0] = word[k][1] = word[k][2] = word[k][3] = 0;
#pragma unroll
  for (int x = 0; x < 16; ++x) {
    const int kk = k16 * 16 + x;
    const int g = kk / st.kp, e = kk % st.kp;
    if (g != g_row || e >= 2 * L * st.n) continue;
    const int which = e / (L * st.n), s = (e / st.n) % L, c = e % st.n;
    int at = y - 2 * c;
    const bool wrap = at < 0;
    if (wrap) at += n_out;
    u64 v = key[((((long)(j + which * st.half) * L + s) * 2 + mb) * 2 + l) * n_out + at];
    v = reduce64(v, m);
    if (mb == 0) v = mulmod(v, inv, m);
    if (wrap != (mb == 0)) v = negmod(v, m.q);
#pragma unroll
    for (int k = 0; k < 5; ++k) word[k][x >> 2] |= (u32)((v >> (8 * k)) & 0xFF) << (8 * (x & 3));
  }
  const int kc = k16 / (CT_KC / 16), kb = k16 % (CT_KC / 16);
  uint8_t* base = planes + ((size_t)unit * st.chunks + kc) * CT_STAGE_B + (size_t)kb * (CT_N / 8) * 128;
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const int row = (l * 5 + k) * CT_ROWS + r;
    uint4* at = reinterpret_cast<uint4*>(base + (row / 8) * 128 + (row % 8) * 16);
    if (CHECK) {
      const uint4 v = *at;
      if (v.x != word[k][0] || v.y != word[k][1] || v.z != word[k][2] || v.w != word[k][3]) *differs = 1;
    } else {
      *at = make_uint4(word[k][0], word[k][1], word[k][2], word[k][3]);
    }
  }
}

// Column constants o * (sum of the item's key entries of the column) mod q_l, one warp per
// (item, limb, row): read back from the planes.
__global__ void k_ct_consts(const uint8_t* __restrict__ planes, CtStep st, DevRing R, u32 o, double* __restrict__ out) {
  const long gid = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (gid >= (long)st.items() * 32) return;
  const int r = (int)(gid & 15), l = (int)((gid >> 4) & 1), item = (int)(gid >> 5);
  int len;
  const int unit0 = ct_item(st, item, len);
  u64 sum[5] = {0, 0, 0, 0, 0};
  for (int k16 = lane; k16 < len * st.chunks * (CT_KC / 16); k16 += 32) {
    const uint8_t* base = planes + ((size_t)unit0 * st.chunks + k16 / (CT_KC / 16)) * CT_STAGE_B +
                          (size_t)(k16 % (CT_KC / 16)) * (CT_N / 8) * 128;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const int row = (l * 5 + k) * CT_ROWS + r;
      const uint4 v = *reinterpret_cast<const uint4*>(base + (row / 8) * 128 + (row % 8) * 16);
      const u32 w[4] = {v.x, v.y, v.z, v.w};
      for (int i = 0; i < 4; ++i)
        for (int b = 0; b < 4; ++b) sum[k] += (w[i] >> (8 * b)) & 0xFF;
    }
  }
#pragma unroll
  for (int k = 0; k < 5; ++k)
    for (int d = 16; d; d >>= 1) sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], d);
  if (lane == 0) {
    const DevMod& m = R.m[l];
    u64 acc = 0;
    for (int k = 4; k >= 0; --k) acc = reduce64((acc << 8) + reduce64(sum[k], m), m);
    out[((size_t)item * 2 + l) * CT_ROWS + r] = (double)mulmod(acc, o, m);
  }
}

}  // namespace

CtDigits ct_digits(u64 base, const DevRing& R) {
  CtDigits D{};
  for (int l = 0; l < 2; ++l) {
    const u64 q = R.m[l].q;
    D.qi[l] = q;
    D.q[l] = (double)q;
    D.qinv[l] = 1.0 / (double)q;
    D.c24[l] = (double)(((u64)1 << 24) % q);
    D.yscale[l] = (double)h_inv(R.m[1 - l].q % q, q);
  }
  u64 T = 1;
  for (int i = 0; i < CT_LP; ++i) T *= base;
  D.T = (double)T;
  D.Ti = (u32)T;
  D.base = (u32)base;
  D.o = (u32)(base - 1 - base / 2);
  int sh = 0;
  while (((u64)1 << (sh + 1)) < T) ++sh;  // 2^sh < T <= 2^(sh + 1)
  D.sh = sh;
  D.M = (u32)((((u128)1 << (32 + sh)) + T - 1) / T);
  D.off = (u32)(D.o * ((T - 1) / (base - 1)) + 2 * T);
  return D;
}

// Two-prime NTT rings, primes of 26 to 40 bits (five bytes; a quotient of T y / q fits the low
// word), gadgets of 18 digits with B^6 < 2^26 (a piece's arithmetic fits 32 bits; B up to 20, and
// the test on B alone keeps B^6 within 64 bits).
bool ct_digits_ok(u64 base, u32 L, const DevRing& R) {
  if (!R.ntt || R.nl != 2 || L != CT_L || base < 3 || base > 255) return false;
  u64 T = 1;
  for (int i = 0; i < CT_LP; ++i) T *= base;
  if (T >= (1ull << 26)) return false;
  for (int l = 0; l < 2; ++l)
    if (R.m[l].q >= (1ull << 40) || R.m[l].q < (1ull << 26)) return false;
  return true;
}

bool ct_supported(const via_params& p, const DevRing& R) {
  return p.n1 >= 256 && ct_digits_ok(p.ck_base, p.l_ck, R);
}

void ct_prepare_device() {
  VIA_CUDA(cudaFuncSetAttribute(k_ct_step, cudaFuncAttributeMaxDynamicSharedMemorySize, CT_SMEM));
}

void ct_prepare(Server& s, const Server* base) {
  const via_params& p = s.prm;
  if (!ct_supported(p, s.r1) || !s.cascade_eval.p || !s.fd_err.p) return;
  const int K = ct_steps(p), n1 = (int)p.n1;
  ct_prepare_device();
  const CtDigits D = ct_digits(p.ck_base, s.r1);
  const u64 step_len = (u64)2 * n1 * CT_L * 2 * 2;
  const u64 inv0 = (u64)D.yscale[0], inv1 = (u64)D.yscale[1];
  const auto plane_bytes = [](const CtStep& st) { return (size_t)2 * st.units * st.chunks * CT_STAGE_B; };
  const auto plane_blocks = [](const CtStep& st) {
    return (unsigned)(((long)2 * st.units * st.chunks * (CT_KC / 16) * 32 + 255) / 256);
  };
  const std::shared_ptr<const CtKeys> lent = base ? std::atomic_load(&base->ct) : nullptr;
  if (lent) {
    DevBuf differs(1);
    VIA_CUDA(cudaMemsetAsync(differs.p, 0, 8, s.stream));
    uint8_t* planes = reinterpret_cast<uint8_t*>(lent->planes.p);
    for (int k = 0; k < K; ++k) {
      const CtStep st = ct_step(n1, 1 << k);
      k_ct_planes<true><<<plane_blocks(st), 256, 0, s.stream>>>(s.cascade_eval.p + k * step_len, st, s.r1, inv0, inv1,
                                                                planes, reinterpret_cast<int*>(differs.p));
      VIA_LAUNCHED();
      planes += plane_bytes(st);
    }
    int other = 0;
    VIA_CUDA(cudaMemcpyAsync(&other, differs.p, sizeof(int), cudaMemcpyDeviceToHost, s.stream));
    VIA_CUDA(cudaStreamSynchronize(s.stream));
    if (!other) {
      std::atomic_store(&s.ct, lent);
      return;
    }
  }
  size_t bytes = 0, consts = 0;
  for (int k = 0; k < K; ++k) {
    const CtStep st = ct_step(n1, 1 << k);
    bytes += plane_bytes(st);
    consts += (size_t)2 * st.units * 2 * CT_ROWS;  // room for items of one unit
  }
  auto keys = std::make_shared<CtKeys>();
  try {
    keys->planes.alloc(bytes / 8);
    keys->consts.alloc(2 * consts);  // for few and for many tiles
  } catch (const CudaError& e) {
    if (e.status != 101) throw;
    return;  // no room: the transforms need no planes
  }
  uint8_t* planes = reinterpret_cast<uint8_t*>(keys->planes.p);
  double* cc = reinterpret_cast<double*>(keys->consts.p);
  for (int k = 0; k < K; ++k) {
    const CtStep st = ct_step(n1, 1 << k);
    k_ct_planes<false><<<plane_blocks(st), 256, 0, s.stream>>>(s.cascade_eval.p + k * step_len, st, s.r1, inv0, inv1,
                                                               planes, nullptr);
    VIA_LAUNCHED();
    for (int many = 0; many < 2; ++many) {
      const CtStep c = ct_step(n1, 1 << k, many ? CT_MANY : 1);
      const long warps = (long)c.items() * 32;
      k_ct_consts<<<(unsigned)((warps * 32 + 255) / 256), 256, 0, s.stream>>>(planes, c, s.r1, D.o,
                                                                             cc + many * consts);
      VIA_LAUNCHED();
    }
    planes += plane_bytes(st);
    cc += (size_t)2 * st.units * 2 * CT_ROWS;
  }
  keys->steps = K;
  std::atomic_store(&s.ct, std::shared_ptr<const CtKeys>(std::move(keys)));
}

void ct_run(Server& s, const CtKeys& keys, const u64* d_query, long nlwe, uint8_t* da, uint8_t* db, int8_t* dig8, u64* body,
            cudaStream_t st) {
  const via_params& p = s.prm;
  const int n1 = (int)p.n1;
  const CtDigits D = ct_digits(p.ck_base, s.r1);
  const int mtiles = (int)((nlwe + CT_M - 1) / CT_M);
  CtStep cur = ct_step(n1, 1, mtiles);
  const long threads = (nlwe + 7) / 8 * 8 * cur.half;
  k_ct_digits<<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(d_query, nlwe, (long)lwe_len(p), n1, cur, D,
                                                                (size_t)CT_M * cur.half * cur.kp, da);
  VIA_LAUNCHED();
  size_t b_off = 0, c_off = mtiles >= CT_MANY ? keys.consts.n / 2 : 0;
  const int steps = ct_steps_for(keys.steps, nlwe);
  for (int k = 0; k < steps; ++k) {
    const CtStep nxt = ct_step(n1, 2 << k, mtiles);
    const bool last = k + 1 == steps;
    CtParams P{};
    P.st = cur;
    P.D = D;
    P.a = da;
    P.b = reinterpret_cast<const uint8_t*>(keys.planes.p) + b_off;
    P.c = reinterpret_cast<const double*>(keys.consts.p) + c_off;
    P.out = last ? nullptr : db;
    P.dig8 = dig8;
    P.body = body + ((2L << k) - 2) * 2 * nlwe;
    P.err = reinterpret_cast<int*>(s.fd_err.p);
    P.nlwe = nlwe;
    P.a_tile = (size_t)CT_M * cur.half * cur.kp;
    P.out_tile = (size_t)CT_M * nxt.half * nxt.kp;
    P.mtiles = mtiles;
    P.fault_ns = s.fd.fault_wait_ns;
    P.out_kp = nxt.kp;
    P.out_half = nxt.half;
    const int items = cur.items() * mtiles;
    k_ct_step<<<std::min(items, s.fd.grid), CT_THREADS, CT_SMEM, st>>>(P);
    VIA_LAUNCHED();
    b_off += (size_t)2 * cur.units * cur.chunks * CT_STAGE_B;
    c_off += (size_t)2 * cur.units * 2 * CT_ROWS;
    std::swap(da, db);
    cur = nxt;
  }
}

}  // namespace via
