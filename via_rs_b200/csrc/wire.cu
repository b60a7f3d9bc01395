// Query wire formats (crates/via-protocol/src/wire/format.rs:93-190) and the
// device-side mask regeneration of the PRG-compressed format.
//
// A query on the wire is n_lwe packets, one per LWE ciphertext, each starting
// with the format tag of format.rs:
//   0x00 Uncompressed : [0x00][count: u64 LE][count u64 LE]   count = nl * (n1 + 1)
//                       (the LWE verbatim: mask polynomial limb-major, then body)
//   0x01 PrgCompressed: [0x01][seed: 32 bytes][count: u64 LE][count u64 LE]   count = nl
//                       (the body verbatim; the mask is regenerated)
// Mask regeneration (format.rs:20-27,146-160): Shake256Prg(seed), then
// uniform_below(q_l) for every mask coefficient in row-major order, one draw
// per limb, limb 0 first (prim/sampling/prg.rs:108-206). The PRG's byte stream
// is counter-mode, block b = SHAKE256(seed || le64(b))[0..136), so every block
// is one Keccak-f[1600] permutation and the device computes all blocks of all
// packets in parallel; one CTA per packet then takes its mask from the stream
// (walk_mask; an accepted draw consumes ceil(bitlen(q) / 8) bytes).
#include <cstring>
#include <string>
#include <vector>

#include "prg.cuh"
#include "server.cuh"

namespace via {
namespace {

constexpr int SEED_LEN = 32;

// All PRG blocks of all compressed packets: blocks [pkt][nblk][17].
__global__ void k_prg_blocks(const uint8_t* __restrict__ seeds, int npkt, int nblk, u64* __restrict__ blocks) {
  const long gid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= (long)npkt * nblk) return;
  const int pkt = (int)(gid / nblk), b = (int)(gid % nblk);
  u64 out[RATE_LANES];
  prg_block(seeds + (size_t)pkt * SEED_LEN, SEED_LEN, (u64)b, out);
  u64* dst = blocks + gid * RATE_LANES;
#pragma unroll
  for (int l = 0; l < RATE_LANES; ++l) dst[l] = out[l];
}

struct Sampler {
  u64 q[2];
  u64 mask[2];
  int nbytes[2];
};

// The mask and the body of one compressed packet per CTA: LWE lwe[pkt] of `query`
// ([nl][n1] limb-major, then nl body residues). err: 2 where walk_mask could not
// decide. Latency-bound: a chunk of 4608 candidates is one pass of the paper
// preset's mask, several of the secure preset's. Against one thread walking each
// stream (k_prg_masks): 40 packets of the paper preset 3412 us there, 6.5 here.
__global__ void __launch_bounds__(WALK_THREADS) k_prg_masks_scan(const u64* __restrict__ blocks,
                                                                 const u64* __restrict__ bodies,
                                                                 const int* __restrict__ lwe, int nblk, int n1,
                                                                 u64 lwe_len, WalkLimbs W, u64* __restrict__ query,
                                                                 int* __restrict__ err) {
  __shared__ WalkShared sh;
  const int pkt = blockIdx.x;
  u64* out = query + (size_t)lwe[pkt] * lwe_len;
  if (threadIdx.x < W.nl) out[(size_t)W.nl * n1 + threadIdx.x] = bodies[(size_t)pkt * W.nl + threadIdx.x];
  const u64 avail = (u64)nblk * SHAKE_RATE;
  const long used = walk_mask(blocks + (size_t)pkt * nblk * RATE_LANES, avail, 0, W, n1, out, sh);
  if (used == WALK_UNDECIDED && threadIdx.x == 0) atomicMax(err, 2);
}

// The general walk, for limbs whose draws take different numbers of bytes and
// for streams walk_mask leaves undecided. One thread per compressed packet:
// uniform_below over the packet's stream, writing the mask polynomial of LWE
// lwe[pkt] ([nl][n1] limb-major) and its body. Blocks beyond the precomputed
// nblk (a run of rejections) are computed here.
__global__ void k_prg_masks(const u64* __restrict__ blocks, const uint8_t* __restrict__ seeds,
                            const u64* __restrict__ bodies, const int* __restrict__ lwe, int npkt, int nblk, int n1, int nl, u64 lwe_len, Sampler S,
                            u64* __restrict__ query, int* __restrict__ err) {
  const int pkt = blockIdx.x * blockDim.x + threadIdx.x;
  if (pkt >= npkt) return;
  const u64* blk = blocks + (size_t)pkt * nblk * RATE_LANES;
  u64 extra[RATE_LANES];
  long extra_idx = -1;
  u64 pos = 0;  // byte position in the stream
  auto byte_at = [&](u64 p) -> unsigned {
    const long b = (long)(p / SHAKE_RATE);
    const int o = (int)(p % SHAKE_RATE);
    u64 lane;
    if (b < nblk) {
      lane = blk[(size_t)b * RATE_LANES + o / 8];
    } else {
      if (b != extra_idx) {
        prg_block(seeds + (size_t)pkt * SEED_LEN, SEED_LEN, (u64)b, extra);
        extra_idx = b;
      }
      lane = extra[o / 8];
    }
    return (unsigned)((lane >> (8 * (o % 8))) & 0xFF);
  };
  u64* out = query + (size_t)lwe[pkt] * lwe_len;
  for (int l = 0; l < nl; ++l) out[(size_t)nl * n1 + l] = bodies[(size_t)pkt * nl + l];
  for (int k = 0; k < n1; ++k)
    for (int l = 0; l < nl; ++l) {
      // q >= 2^(bits-1) accepts at least half of the draws, so 64 rejections in
      // a row (probability below 2^-64) end the packet with an error instead.
      u64 v = 0;
      bool ok = false;
      for (int attempt = 0; attempt < 64 && !ok; ++attempt) {
        v = 0;
        for (int b = 0; b < S.nbytes[l]; ++b) v |= (u64)byte_at(pos + b) << (8 * b);
        pos += S.nbytes[l];
        v &= S.mask[l];
        ok = v < S.q[l];
      }
      if (!ok) {
        atomicExch(err, 1);
        return;
      }
      out[(size_t)l * n1 + k] = v;
    }
}

struct ApiErr : std::runtime_error {
  via_status code;
  ApiErr(via_status c, const std::string& m) : std::runtime_error(m), code(c) {}
};

u64 rd64(const uint8_t* p) {
  u64 v = 0;
  for (int i = 0; i < 8; ++i) v |= (u64)p[i] << (8 * i);
  return v;
}

// A parsed wire query. Compressed packets leave their LWE to the device and are
// listed in seeds / bodies / lwes; `flat` (the flat layout) is made when an
// uncompressed packet comes.
struct WireQuery {
  std::vector<u64> flat, bodies;
  std::vector<uint8_t> seeds;
  std::vector<int> lwes;
};

void parse_wire(const via_params& p, const uint8_t* wire, u64 len, WireQuery& Q) {
  const u64 n_lwe = query_lwes(p), ll = lwe_len(p), nl = p.q1_1 ? 2 : 1;
  u64 off = 0;
  for (u64 w = 0; w < n_lwe; ++w) {
    if (off >= len) throw ApiErr(VIA_ERR_BUFFER_TOO_SHORT, "wire query: " + std::to_string(w) + " of " +
                                                               std::to_string(n_lwe) + " LWE packets present");
    const uint8_t tag = wire[off];
    if (tag == 0x00) {
      if (len - off < 9) throw ApiErr(VIA_ERR_BUFFER_TOO_SHORT, "wire query: truncated packet header");
      const u64 count = rd64(wire + off + 1);
      if (count != ll) throw ApiErr(VIA_ERR_DIM_MISMATCH, "wire query: uncompressed LWE length mismatch");
      if ((len - off - 9) / 8 < count) throw ApiErr(VIA_ERR_BUFFER_TOO_SHORT, "wire query: truncated LWE");
      Q.flat.resize(n_lwe * ll);
      std::memcpy(Q.flat.data() + w * ll, wire + off + 9, count * 8);  // little-endian words
      off += 9 + 8 * count;
    } else if (tag == 0x01) {
      if (len - off < 1 + SEED_LEN + 8) throw ApiErr(VIA_ERR_BUFFER_TOO_SHORT, "wire query: truncated packet header");
      const u64 count = rd64(wire + off + 1 + SEED_LEN);
      if (count != nl) throw ApiErr(VIA_ERR_DIM_MISMATCH, "wire query: compressed body length mismatch");
      if ((len - off - 1 - SEED_LEN - 8) / 8 < count) throw ApiErr(VIA_ERR_BUFFER_TOO_SHORT, "wire query: truncated body");
      Q.seeds.insert(Q.seeds.end(), wire + off + 1, wire + off + 1 + SEED_LEN);
      Q.lwes.push_back((int)w);
      for (u64 i = 0; i < count; ++i) Q.bodies.push_back(rd64(wire + off + 1 + SEED_LEN + 8 + 8 * i));
      off += 1 + SEED_LEN + 8 + 8 * count;
    } else {
      throw ApiErr(VIA_ERR_UNKNOWN_FORMAT_TAG, "wire query: unknown format tag " + std::to_string(tag));
    }
  }
  if (off != len) throw ApiErr(VIA_ERR_QUERY_LENGTH_MISMATCH, "wire query: bytes after the last of " +
                                                                  std::to_string(n_lwe) + " LWE packets");
}

Sampler make_sampler(const via_params& p) {
  Sampler S{};
  const u64 qs[2] = {p.q1_0, p.q1_1 ? p.q1_1 : p.q1_0};
  for (int l = 0; l < 2; ++l) {
    const int bits = 64 - __builtin_clzll(qs[l]);
    S.q[l] = qs[l];
    S.nbytes[l] = (bits + 7) / 8;
    S.mask[l] = bits == 64 ? ~(u64)0 : (((u64)1 << bits) - 1);
  }
  return S;
}

// Decodes a wire query into the device buffer d_query (flat layout).
void decode_to_device(Server& s, const uint8_t* wire, u64 len, u64* d_query, cudaStream_t st) {
  const via_params& p = s.prm;
  const u64 ll = lwe_len(p);
  const int nl = p.q1_1 ? 2 : 1;
  WireQuery Q;
  parse_wire(p, wire, len, Q);
  if (!Q.flat.empty())
    VIA_CUDA(cudaMemcpyAsync(d_query, Q.flat.data(), Q.flat.size() * 8, cudaMemcpyHostToDevice, st));
  const int npkt = (int)Q.lwes.size();
  if (npkt == 0) {
    VIA_CUDA(cudaStreamSynchronize(st));  // Q is freed on return
    return;
  }
  const Sampler S = make_sampler(p);
  WalkLimbs W{{S.q[0], S.q[1]}, {S.mask[0], S.mask[1]}, S.nbytes[0], nl};
  const bool scan = nl == 1 || S.nbytes[0] == S.nbytes[1];
  double need = 0;
  for (int l = 0; l < nl; ++l) need += walk_bytes((double)p.n1, S.q[l], S.nbytes[l]);
  // A whole number of the scan's thread loads past the last draw, as well.
  const int nblk = (int)((need + WALK_V * 8) / SHAKE_RATE + 2);
  // One upload and one scratch: bodies, seeds, LWE numbers, error word, then the blocks.
  const size_t w_seeds = Q.bodies.size(), w_lwes = w_seeds + Q.seeds.size() / 8, w_err = w_lwes + (npkt + 1) / 2;
  std::vector<u64> head(w_err + 1, 0);
  std::memcpy(head.data(), Q.bodies.data(), Q.bodies.size() * 8);
  std::memcpy(head.data() + w_seeds, Q.seeds.data(), Q.seeds.size());
  std::memcpy(head.data() + w_lwes, Q.lwes.data(), Q.lwes.size() * sizeof(int));
  ScratchLease d(s.wire_scratch, head.size() + (size_t)npkt * nblk * RATE_LANES);
  VIA_CUDA(cudaMemcpyAsync(d.p, head.data(), head.size() * 8, cudaMemcpyHostToDevice, st));
  const uint8_t* seeds = reinterpret_cast<const uint8_t*>(d.p + w_seeds);
  const int* lwes = reinterpret_cast<const int*>(d.p + w_lwes);
  int* d_err = reinterpret_cast<int*>(d.p + w_err);
  u64* blocks = d.p + head.size();
  const long nb = (long)npkt * nblk;
  k_prg_blocks<<<(unsigned)((nb + 127) / 128), 128, 0, st>>>(seeds, npkt, nblk, blocks);
  VIA_LAUNCHED();
  int err = 2;
  if (scan) {
    k_prg_masks_scan<<<npkt, WALK_THREADS, 0, st>>>(blocks, d.p, lwes, nblk, p.n1, ll, W, d_query, d_err);
    VIA_LAUNCHED();
    VIA_CUDA(cudaMemcpyAsync(&err, d_err, sizeof(int), cudaMemcpyDeviceToHost, st));
    VIA_CUDA(cudaStreamSynchronize(st));  // the temporaries are freed on return
  }
  if (err == 2) {
    VIA_CUDA(cudaMemsetAsync(d_err, 0, 8, st));
    k_prg_masks<<<(unsigned)((npkt + 63) / 64), 64, 0, st>>>(blocks, seeds, d.p, lwes, npkt, nblk, p.n1, nl, ll, S,
                                                            d_query, d_err);
    VIA_LAUNCHED();
    VIA_CUDA(cudaMemcpyAsync(&err, d_err, sizeof(int), cudaMemcpyDeviceToHost, st));
    VIA_CUDA(cudaStreamSynchronize(st));
  }
  if (err) throw ApiErr(VIA_ERR_INVALID_PRG_SEED, "wire query: a PRG seed's stream rejected 64 draws in a row");
}

template <class F>
via_status wire_guarded(F&& f) {
  try {
    f();
    return VIA_OK;
  } catch (const ApiErr& e) {
    set_last_error(e.what());
    return e.code;
  } catch (const CudaError& e) {
    set_last_error(e.what());
    return e.status == 101 ? VIA_ERR_OUT_OF_MEMORY : VIA_ERR_CUDA;
  } catch (const std::exception& e) {
    set_last_error(e.what());
    return VIA_ERR_INVALID_ARGUMENT;
  }
}

}  // namespace

}  // namespace via

using namespace via;

extern "C" {

via_status via_query_from_wire(via_server* s, const uint8_t* wire, uint64_t len, uint64_t* out_query,
                               uint64_t out_len) {
  return wire_guarded([&] {
    if (!s || !wire || !out_query) throw ApiErr(VIA_ERR_INVALID_ARGUMENT, "null argument");
    const via_params& p = s->prm;
    const u64 total = query_lwes(p) * lwe_len(p);
    if (out_len < total) throw ApiErr(VIA_ERR_BUFFER_TOO_SHORT, "output shorter than one query");
    DevBuf d(total);
    decode_to_device(*s, wire, len, d.p, s->stream);
    VIA_CUDA(cudaMemcpyAsync(out_query, d.p, total * 8, cudaMemcpyDeviceToHost, s->stream));
    VIA_CUDA(cudaStreamSynchronize(s->stream));
  });
}

via_status via_server_answer_wire(via_server* s, const uint8_t* wire, uint64_t len, uint64_t* out_mask,
                                  uint64_t* out_body) {
  return wire_guarded([&] {
    if (!s || !wire || !out_mask || !out_body) throw ApiErr(VIA_ERR_INVALID_ARGUMENT, "null argument");
    if (!s->cascade_eval.p) throw ApiErr(VIA_ERR_SETUP_NOT_COMPLETE, "server has no public keys");
    const via_params& p = s->prm;
    std::lock_guard<std::mutex> g(s->mu);
    decode_to_device(*s, wire, len, workspace_query(*s), s->stream);
    answer_graph(*s, 1, s->stream);
    VIA_CUDA(cudaMemcpyAsync(out_mask, workspace_answer_mask(*s), p.n2 * 8, cudaMemcpyDeviceToHost, s->stream));
    VIA_CUDA(cudaMemcpyAsync(out_body, workspace_answer_body(*s), p.n2 * 8, cudaMemcpyDeviceToHost, s->stream));
    const std::string e = device_flags(*s, s->stream);
    if (!e.empty()) throw ApiErr(VIA_ERR_TIMEOUT, e);
  });
}

}  // extern "C"
