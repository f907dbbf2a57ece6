// ans_codec.cu -- byte rANS over 4 KiB blocks for sm_100a: histogram,
// encode (with single-pass output compaction) and decode.
//
// Stream layout and arithmetic are those of include/ans (GpuANSCodec.h,
// GpuANSEncode.h, GpuANSDecode.h); the kernels are organised differently:
//  * encode writes the final coalesced stream directly: each warp collects its
//    block's words in shared memory and a slot in L2, learns its word offset
//    through a decoupled look-back over per-block flags, and stores 16-byte
//    vectors. The reference instead writes an uncoalesced scratch (5,248-byte
//    stride), scans with up to three kernels and copies with a fourth.
//  * the table is normalised by the last CTA of the histogram kernel, not by
//    a separate launch;
//  * decode validates the header on the device and reports a status instead
//    of device asserts, and checks that every block consumes exactly its
//    words and returns to the start state.
#include "ans_dev.cuh"
#include <cstdlib>
#include "mans_internal.h"

namespace mans {

// ------------------------------------------------------------------------
// Histogram of a raw byte buffer (GpuANSStatistics.h:24-151), with per-warp
// shared-memory bins merged into the global histogram once per CTA.
// ------------------------------------------------------------------------
constexpr int kHistThreads = 256;

__device__ __forceinline__ void hist_word(uint32_t* h, uint32_t w) {
  atomicAdd(&h[w & 0xff], 1u);
  atomicAdd(&h[(w >> 8) & 0xff], 1u);
  atomicAdd(&h[(w >> 16) & 0xff], 1u);
  atomicAdd(&h[w >> 24], 1u);
}

__global__ __launch_bounds__(kHistThreads) void hist_bytes_kernel(const uint8_t* __restrict__ in,
                                                                  uint64_t n, Ctrl* ctrl,
                                                                  int prob_bits) {
  kernel_begin();
  __shared__ uint32_t s_h[kHistThreads / 32][kAnsSyms];
  const int t = threadIdx.x, warp = t >> 5;
  for (int i = t; i < (kHistThreads / 32) * kAnsSyms; i += kHistThreads) (&s_h[0][0])[i] = 0;
  __syncthreads();
  uint32_t* h = s_h[warp];
  const uint64_t n16 = n >> 4;
  const uint4* in4 = reinterpret_cast<const uint4*>(in);
  for (uint64_t i = (uint64_t)blockIdx.x * kHistThreads + t; i < n16;
       i += (uint64_t)gridDim.x * kHistThreads) {
    uint4 v = __ldcs(in4 + i);
    hist_word(h, v.x);
    hist_word(h, v.y);
    hist_word(h, v.z);
    hist_word(h, v.w);
  }
  if (blockIdx.x == 0) {
    uint64_t i = (n16 << 4) + t;
    if (i < n) atomicAdd(&h[in[i]], 1u);
  }
  hist_merge_and_normalize(s_h, kHistThreads / 32, ctrl, n, 0, prob_bits);
}

// ------------------------------------------------------------------------
// Encode: one warp per 4 KiB block. The block arrives in the warp's shared
// stage with one bulk (TMA) copy from L2, where it was prefetched one grid of
// warps earlier; symbols are read eight steps ahead of use. Blocks are
// claimed one at a time (a claim held while another block is encoded would
// stall every later block's look-back).
// ------------------------------------------------------------------------
// One CTA of up to 32 warps per SM shares the 32 KiB table; small inputs take
// smaller CTAs, so that their blocks spread over the SMs.
constexpr int kEncMinWarps = 4, kEncMaxWarps = 32, kEncMaxThreads = kEncMaxWarps * 32;

// Empty input: header and a zero pdf only (GpuANSEncode.h:201-237).
__device__ __forceinline__ void encode_empty(uint8_t* __restrict__ out, uint64_t out_cap, int p,
                                             const uint32_t* __restrict__ pdf,
                                             unsigned long long* out_size64, uint32_t* out_size32,
                                             const Sink& sink, int lane) {
  const uint64_t over = ans_overhead(0);
  if (over > out_cap) {
    if (lane == 0) report(sink, MANS_ERR_OUTPUT_OVERFLOW, over);
    return;
  }
  if (lane < 8) {
    const uint32_t hv = lane == 0 ? kAnsMagicVersion : (lane == 4 ? (uint32_t)p : 0u);
    reinterpret_cast<uint32_t*>(out)[lane] = hv;
  }
  for (int i = lane; i < kAnsSyms; i += 32)
    reinterpret_cast<uint16_t*>(out + kAnsHeaderBytes)[i] = (uint16_t)pdf[i];
  if (lane == 0) {
    if (out_size64) *out_size64 = over;
    if (out_size32) *out_size32 = (uint32_t)over;
  }
}

// The last CTA resets the work counters and advances the epoch: the call's
// flags are then stale.
__device__ __forceinline__ void encode_done(Ctrl* ctrl, uint32_t epoch) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&ctrl->done_counter[1], 1u) == gridDim.x - 1) {
      ctrl->tile_counter[1] = 0;
      ctrl->done_counter[1] = 0;
      ctrl->epoch = (epoch + 1) & 0x3fffffffu;
    }
  }
}

// kGather: the input's records lie in slots (enc_gather).
template <int kP, bool kGather>
__global__ __launch_bounds__(kEncMaxThreads, 1) void ans_encode_slots_kernel(
    const uint8_t* __restrict__ in, uint8_t* __restrict__ out, uint64_t out_cap,
    unsigned long long* out_size64, uint32_t* out_size32, Ctrl* ctrl, unsigned long long* flags,
    uint8_t* __restrict__ slots, const AnsGather gather) {
  kernel_begin();
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  EncWarp& sw = reinterpret_cast<EncWarp*>(smem_raw + kEncTableBytes)[warp];
  if (lane == 0) mbar_init(&sw.bar);
  uint32_t parity = 0;
  const Sink sink = sink_of(ctrl);
  const bool failed = sink_failed(sink);
  const uint32_t epoch = *((volatile uint32_t*)&ctrl->epoch);
  const uint64_t n = __ldcg(&ctrl->merged_size);
  const uint64_t nb = div_up_u64(n, kAnsBlock);
  enc_fill_table(smem_raw, ctrl->enc_table, kP);
  // Fewer blocks than warps were launched for: as many warps of every CTA as
  // spread them evenly take part (claimed by all, the blocks crowd on the SMs
  // that come first; 6 M small uint32 values 51.0 us a call, so 43.6).
  const bool idle = failed || (warp >= kEncMinWarps && (uint32_t)warp * gridDim.x >= (uint32_t)nb);
  __syncthreads();
  if (!failed && nb == 0 && blockIdx.x == 0 && warp == 0)
    encode_empty(out, out_cap, kP, ctrl->pdf, out_size64, out_size32, sink, lane);

  const uint32_t warps = blockDim.x >> 5, ahead = gridDim.x * warps;
  // Two word slots per warp. A block's words wait in one slot for its
  // stream offset while the warp encodes its next block into the other;
  // the look-back of the waiting block then runs after that next block's
  // aggregate is published, when its predecessors have usually finished,
  // instead of stalling the warp. Every claimed block publishes its
  // aggregate as soon as it is encoded, before any wait, so the deferred
  // look-backs always complete.
  uint16_t* const slot0 = reinterpret_cast<uint16_t*>(
      slots + ((uint64_t)blockIdx.x * warps + warp) * 2 * kEncSlotBytes);
  EncPending pend{0xffffffffu, 0, 0, nullptr};
  uint32_t cur = 0;
  while (!idle) {
    const uint32_t b = warp_claim(&ctrl->tile_counter[1], lane);
    if (b >= nb) break;
    if (!kGather && lane == 0 && (uint64_t)b + ahead < nb) {
      const uint64_t s1 = ((uint64_t)b + ahead) * kAnsBlock;
      prefetch_l2(in + s1, (uint32_t)min_u64(kAnsBlock, n - s1));
    }
    uint16_t* const sout = slot0 + cur * (kEncSlotBytes / 2);
    uint32_t x;
    const uint32_t nw = encode_words_rep<kP, kGather>(in, n, b, smem_raw, sw, parity, sout, sink,
                                                      lane, x, gather, (uint64_t)b + ahead);
    if (lane == 0)
      st_flag(&flags[b], make_flag(b == 0 ? kFlagIncl : kFlagAgg, epoch, (nw + 7) & ~7u));
    if (pend.b != 0xffffffffu)
      encode_finish<true>(out, out_cap, n, out_size64, out_size32, ctrl->pdf, flags, epoch, kP,
                          sink, pend, lane);
    pend = EncPending{b, nw, x, sout};
    cur ^= 1u;
  }
  if (pend.b != 0xffffffffu)
    encode_finish<true>(out, out_cap, n, out_size64, out_size32, ctrl->pdf, flags, epoch, kP, sink,
                        pend, lane);
  encode_done(ctrl, epoch);
}

// The same with each block's words compacted in shared memory (no scratch in
// global memory, no deferral), for the allocation-free call. With a concentrated
// symbol distribution most lanes of a step look up the same few entries, and the
// expanded 16-byte entries save integer work; with a flat one the lanes spread
// over many entries, and the packed 8-byte entries cost fewer shared-memory
// wavefronts. The effective number of symbols 2^(2p) / sum(pdf^2) decides (<= 16:
// expanded; 60 MB of two symbols at p = 10: packed 144.1 us, this 137.8).
__global__ __launch_bounds__(kEncThreads, 2) void ans_encode_shared_kernel(
    const uint8_t* __restrict__ in, uint8_t* __restrict__ out, uint64_t out_cap,
    unsigned long long* out_size64, uint32_t* out_size32, Ctrl* ctrl,
    unsigned long long* flags, int p) {
  kernel_begin();
  extern __shared__ __align__(16) uint8_t smem_raw[];
  EncSmem& ss = *reinterpret_cast<EncSmem*>(smem_raw);
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  uint64_t* bar = &ss.bar[warp];
  if (lane == 0) mbar_init(bar);
  uint32_t parity = 0;
  const Sink sink = sink_of(ctrl);
  const bool failed = sink_failed(sink);
  const uint32_t epoch = *((volatile uint32_t*)&ctrl->epoch);
  const uint64_t n = __ldcg(&ctrl->merged_size);
  const uint64_t nb = div_up_u64(n, kAnsBlock);
  __shared__ uint32_t s_sq[kEncWarps];
  const uint32_t q = ctrl->pdf[t], sq = __reduce_add_sync(0xffffffffu, q * q);
  const uint2 packed = ctrl->enc_table[t];
  if (lane == 0) s_sq[warp] = sq;
  __syncthreads();
  uint32_t total = 0;  // 2^22 at most
  for (int w = 0; w < kEncWarps; ++w) total += s_sq[w];
  const bool expanded = total * 16ull >= 1ull << (2 * p);
  if (expanded) ss.expanded[t] = expand_enc_entry(packed, p);
  else ss.packed[t] = packed;
  __syncthreads();
  if (!failed && nb == 0 && blockIdx.x == 0 && warp == 0)
    encode_empty(out, out_cap, p, ctrl->pdf, out_size64, out_size32, sink, lane);
  const uint32_t ahead = gridDim.x * kEncWarps;
  while (!failed) {
    const uint32_t b = warp_claim(&ctrl->tile_counter[1], lane);
    if (b >= nb) break;
    if (lane == 0 && (uint64_t)b + ahead < nb) {
      const uint64_t s1 = ((uint64_t)b + ahead) * kAnsBlock;
      prefetch_l2(in + s1, (uint32_t)min_u64(kAnsBlock, n - s1));
    }
    if (expanded)
      encode_block(in, n, out, out_cap, out_size64, out_size32, ctrl->pdf, flags, epoch, p, sink,
                   ss.expanded, ss.in[warp], bar, parity, ss.out[warp], b, lane);
    else
      encode_block(in, n, out, out_cap, out_size64, out_size32, ctrl->pdf, flags, epoch, p, sink,
                   ss.packed, ss.in[warp], bar, parity, ss.out[warp], b, lane);
  }
  encode_done(ctrl, epoch);
}

// ------------------------------------------------------------------------
// Decode: a warp decodes a block, or two together, from the last step to the
// first. What bounds it: per step 21 to 22 instructions (24 at p = 11; block
// overhead included) of which 7 go to the half-rate integer ALU, two population
// counts, the lookup's shared-memory wavefronts, and a chain of two shared-memory
// loads, a vote and a population count (about 130 cycles) that only other chains
// can hide. Two kernels:
//  * full: one CTA of 32 warps per SM around a replicated table of 128 KiB,
//    pairs of blocks (CTAs of eight warps around one copy of a 4-byte table, words
//    staged whole, took 0.575 ms on 1 GiB of detector frames, here 0.517; 1.092 on a
//    2 GiB uint16 volume, 1.028; 131 us on 100 MB of bytes at p = 11, 95);
//  * light: CTAs of eight warps, three to an SM, one copy of the 4-byte table,
//    each block's words staged whole, a block per warp. Its table is built sooner,
//    and kernels of several streams share an SM, for which the full one leaves
//    no room.
// ------------------------------------------------------------------------
constexpr int kDecFullWarps = 32, kDecLightWarps = 8, kDecLightCtas = 3;
constexpr size_t kDecFullStage = (size_t)kDecFullWarps * 2 * sizeof(DecWarp);
constexpr size_t kDecLightStage = (size_t)kDecLightWarps * sizeof(DecWhole);
constexpr size_t kDecFullSmem = kDecLutBytes + kDecFullStage;
constexpr size_t kDecLightSmem = kDecLutOneBytes + kDecLightStage;

// Each warp's first blocks are fixed and the rest is claimed: a small input then
// takes no claim at all (4,736 warps on one counter cost 5 us). They are spread
// over the CTAs, or (`spread` false) fill CTA by CTA, so that a small input builds
// few tables (four streams of 8 MiB uint16 calls: 11.4 us a call, spread 16.8).
// Full: two blocks are taken at a time and decoded together,
// one at a time once less than a block per warp of the grid is left, so that the
// last wave is short. The next claim and its prefetches come in the middle of
// the current blocks, where other warps hide their latency.
template <int kP, bool kLight>
__device__ __forceinline__ void decode_blocks(const uint8_t* __restrict__ in, uint32_t nb, uint32_t n,
                                              uint32_t cw, uint8_t* __restrict__ out,
                                              const uint8_t* lut, uint8_t* stage, bool spread,
                                              Ctrl* ctrl, const Sink& sink, int lane) {
  constexpr int kBlocks = kLight ? 1 : 2;
  constexpr DecTab kTab = kLight ? kTabOne : dec_many(kP);
  constexpr uint32_t kWhole = (kLight ? kDecLightStage : kDecFullStage) / sizeof(DecWhole);
  auto bad = [&](uint32_t k) { report(sink, MANS_ERR_CORRUPT, k); };
  const uint32_t warp = threadIdx.x >> 5;
  const uint32_t order = spread ? warp * gridDim.x + blockIdx.x : blockIdx.x * kDecLightWarps + warp;
  if ((uint64_t)kWhole * gridDim.x >= nb) {
    // a block per warp at most, and room to stage its words whole
    if (order < nb)
      decode_block<kP, kTab, 1>(in, nb, n, cw, out, lut, reinterpret_cast<DecWhole*>(stage) + warp,
                                order, lane, [](int) {}, bad);
    return;
  }
  DecWarp* const ws = reinterpret_cast<DecWarp*>(stage) + kBlocks * warp;
  const uint8_t* states = in + kAnsHeaderBytes + 2 * kAnsSyms;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  const uint32_t first = kBlocks == 2 && nb > warps ? 2u : 1u;  // blocks per warp at the start
  auto claim = [&](uint32_t seen, uint32_t& take) {
    take = kBlocks == 2 && seen < nb && nb - seen > warps ? 2u : 1u;
    if (first * warps >= nb) return nb;
    uint32_t v = 0;
    if (lane == 0) v = first * warps + atomicAdd(&ctrl->tile_counter[2], take);
    return __shfl_sync(0xffffffffu, v, 0);
  };
  uint32_t take = first;
  uint32_t b = first * order;
  while (b < nb) {
    uint32_t nxt = 0, nxt_take = 0;  // nxt_take 0: not claimed yet
    auto hook = [&](int c) {
      if (c != 3) return;
      nxt = claim(b, nxt_take);
      if (lane < kBlocks && lane < nxt_take && nxt + lane < nb) {
        const uint2 bn = __ldg(reinterpret_cast<const uint2*>(states + 128ull * nb) + nxt + lane);
        prefetch_l2(states + 128ull * (nxt + lane), 128);
        const uint32_t wn = ((bn.x & 0xffffu) + 7) & ~7u;
        if ((uint64_t)bn.y + wn <= cw) prefetch_l2(in + ans_overhead(nb) + 2ull * bn.y, 2 * wn);
      }
    };
    if constexpr (kLight) {
      decode_block<kP, kTab, 1>(in, nb, n, cw, out, lut, ws, b, lane, hook, bad);
    } else {
      bool pair = take == 2 && b + 2 < nb;
      if (pair) pair = decode_block<kP, kTab, 2>(in, nb, n, cw, out, lut, ws, b, lane, hook, bad);
      if (!pair)  // one by one (the last block may be short, and has no fixed chunks)
        for (uint32_t k = b; k < nb && k < b + take; ++k)
          decode_block<kP, kTab, 1>(in, nb, n, cw, out, lut, ws, k, lane, [](int) {}, bad);
    }
    if (!nxt_take) nxt = claim(b, nxt_take);  // the hook has not run
    b = nxt;
    take = nxt_take;
  }
}

template <bool kLight>
__global__ __launch_bounds__((kLight ? kDecLightWarps : kDecFullWarps) * 32,
                             kLight ? kDecLightCtas : 1) void ans_decode_kernel(
    const uint8_t* __restrict__ in, uint64_t in_size, uint8_t* __restrict__ out, uint64_t out_cap,
    Ctrl* ctrl, int expect_p, int record) {
  kernel_begin();
  extern __shared__ __align__(16) uint8_t smem_raw[];
  __shared__ uint32_t s_incl[kAnsSyms];
  __shared__ int s_ok;
  const int t = threadIdx.x, lane = t & 31;
  uint8_t* const lut = smem_raw;  // below every warp's words (see decode_block)
  uint8_t* const stage = smem_raw + (kLight ? kDecLutOneBytes : kDecLutBytes);
  const Sink sink = sink_of(ctrl);

  // ---- header validation (GpuANSCodec.h:106-113 asserts, GpuANSDecode.h:220-227)
  uint32_t h[5] = {0, 0, 0, 0, 0};
  uint32_t pdf = 0;
  bool ok = in_size >= kAnsHeaderBytes + 2 * kAnsSyms;
  if (ok) {
#pragma unroll
    for (int i = 0; i < 5; ++i) h[i] = __ldg(reinterpret_cast<const uint32_t*>(in) + i);
    pdf = dec_pdf(in);
  }
  const uint32_t nb = h[1], n = h[2], cw = h[3];
  const int p = (int)(h[4] & 0xfu);
  ok = ok && h[0] == kAnsMagicVersion && p >= 9 && p <= kMaxProbBits &&
       (expect_p < 0 || p == expect_p) && (uint64_t)nb == div_up_u64(n, kAnsBlock) &&
       ans_overhead(nb) + 2ull * cw <= in_size && (uint64_t)n <= out_cap;
  const bool failed_before = sink_failed(sink);
  if (t == 0) s_ok = ok && !failed_before;
  if (!ok && blockIdx.x == 0 && t == 0 && !failed_before) report(sink, MANS_ERR_BAD_STREAM, 0);
  if (record && ok && blockIdx.x == 0 && t == 0) ctrl->merged_size = n;
  __syncthreads();

  // A CTA without a block builds no table. The light kernel fills CTA by CTA up to
  // two thirds of the grid's warps (two CTAs per SM) and spreads the blocks from
  // there on, so that the SMs have the same number (10 MB of bytes: 17.0 us a call,
  // filled 17.5).
  const bool spread = !kLight || 3ull * nb > 2ull * kDecLightWarps * gridDim.x;
  if (s_ok && (spread ? blockIdx.x : blockIdx.x * kDecLightWarps) < nb) {
    const bool tables_ok = dec_build_lut(pdf, p, kLight ? kTabOne : dec_many(p), lut, s_incl);
    if (!tables_ok && blockIdx.x == 0 && t == 0) report(sink, MANS_ERR_BAD_STREAM, 1);
    __syncthreads();
    if (tables_ok) {
      switch (p) {
        case 9: decode_blocks<9, kLight>(in, nb, n, cw, out, lut, stage, spread, ctrl, sink, lane); break;
        case 10: decode_blocks<10, kLight>(in, nb, n, cw, out, lut, stage, spread, ctrl, sink, lane); break;
        default: decode_blocks<11, kLight>(in, nb, n, cw, out, lut, stage, spread, ctrl, sink, lane); break;
      }
    }
  }

  // Where every block is some warp's first, nothing has been claimed, and there is
  // no counter to reset (ok and nb are the same in every CTA): 0.8 us of a small call.
  if (!ok || nb <= gridDim.x * (blockDim.x >> 5)) return;
  __syncthreads();
  if (t == 0) {
    __threadfence();
    if (atomicAdd(&ctrl->done_counter[2], 1u) == gridDim.x - 1) {
      ctrl->tile_counter[2] = 0;
      ctrl->done_counter[2] = 0;
    }
  }
}

// ------------------------------------------------------------------------
// Host launchers
// ------------------------------------------------------------------------
static int occupancy(const void* fn, int threads, size_t smem) {
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, threads, smem) != cudaSuccess) n = 1;
  return n > 0 ? n : 1;
}

void init_ans_launch_cfg(LaunchCfg& cfg) {
  for (auto* k : {ans_encode_slots_kernel<9, false>, ans_encode_slots_kernel<10, false>,
                  ans_encode_slots_kernel<11, false>, ans_encode_slots_kernel<9, true>,
                  ans_encode_slots_kernel<10, true>, ans_encode_slots_kernel<11, true>})
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)enc_smem_bytes(kEncMaxWarps));
  cudaFuncSetAttribute(ans_encode_shared_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)sizeof(EncSmem));
  cfg.enc_ctas = occupancy((const void*)ans_encode_shared_kernel, kEncThreads, sizeof(EncSmem));
  cudaFuncSetAttribute(ans_decode_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)kDecLightSmem);
  cudaFuncSetAttribute(ans_decode_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)kDecFullSmem);
  cfg.hist_ctas = occupancy((const void*)hist_bytes_kernel, kHistThreads, 0);
}

cudaError_t launch_hist_bytes(const uint8_t* in, uint64_t n, Ctrl* ctrl, int prob_bits,
                              const LaunchCfg& cfg, cudaStream_t s) {
  uint64_t want = div_up_u64(n >> 4, kHistThreads);
  uint64_t cap = (uint64_t)cfg.sms * cfg.hist_ctas;
  unsigned grid = (unsigned)(want < 1 ? 1 : (want < cap ? want : cap));
  return launch(hist_bytes_kernel, grid, kHistThreads, 0, s, in, n, ctrl, prob_bits);
}

uint64_t ans_encode_slot_bytes(const LaunchCfg& cfg) {
  return (uint64_t)cfg.sms * kEncMaxWarps * 2 * kEncSlotBytes;  // two per warp
}

cudaError_t launch_ans_encode(const uint8_t* in, uint8_t* out, uint64_t out_cap,
                              unsigned long long* out_size64, uint32_t* out_size32, Ctrl* ctrl,
                              unsigned long long* flags, int prob_bits, uint64_t likely_blocks,
                              uint64_t max_blocks, const LaunchCfg& cfg, cudaStream_t s,
                              uint8_t* slots, const AnsGather* gather) {
  if (slots) {
    // one CTA per SM with as many warps as spread the blocks evenly
    uint64_t warps = div_up_u64(likely_blocks, (uint64_t)cfg.sms);
    warps = warps < kEncMinWarps ? kEncMinWarps : warps < kEncMaxWarps ? warps : kEncMaxWarps;
    const uint64_t want = div_up_u64(max_blocks, warps);
    const unsigned grid =
        (unsigned)(want < 1 ? 1 : (want < (uint64_t)cfg.sms ? want : (uint64_t)cfg.sms));
    auto* k = prob_bits == 9    ? ans_encode_slots_kernel<9, false>
              : prob_bits == 10 ? ans_encode_slots_kernel<10, false>
                                : ans_encode_slots_kernel<11, false>;
    if (gather)
      k = prob_bits == 9    ? ans_encode_slots_kernel<9, true>
          : prob_bits == 10 ? ans_encode_slots_kernel<10, true>
                            : ans_encode_slots_kernel<11, true>;
    return launch(k, grid, (unsigned)warps * 32, enc_smem_bytes((int)warps), s, in, out, out_cap,
                  out_size64, out_size32, ctrl, flags, slots, gather ? *gather : AnsGather{});
  } else {
    const uint64_t want = div_up_u64(max_blocks, kEncWarps);
    const uint64_t cap = (uint64_t)cfg.sms * cfg.enc_ctas;
    const unsigned grid = (unsigned)(want < 1 ? 1 : (want < cap ? want : cap));
    return launch(ans_encode_shared_kernel, grid, kEncThreads, sizeof(EncSmem), s, in, out, out_cap,
                  out_size64, out_size32, ctrl, flags, prob_bits);
  }
}

// Up to this many likely blocks per SM (its resident warps) the light kernel
// decodes them. Per call, light / full: 4 MiB of bytes 14.6 / 15.5 us, 8 MB 15.4 /
// 15.6, 12 MB 17.9 / 18.1; four streams of 16 MiB uint32 calls 24.4 / 28.5, of 12 MB
// of bytes 15.4 / 17.0. With more blocks its warps take several (32 MiB of uint32
// frames, 37 per SM: 47.7 / 43.3).
constexpr uint64_t kDecLightBlocks = (uint64_t)kDecLightWarps * kDecLightCtas;

cudaError_t launch_ans_decode(const uint8_t* in, uint64_t in_size, uint8_t* out, uint64_t out_cap,
                              Ctrl* ctrl, int expect_p, int record, uint64_t likely_blocks,
                              uint64_t max_blocks, const LaunchCfg& cfg, cudaStream_t s) {
  const uint64_t sms = (uint64_t)cfg.sms;
  const bool light = likely_blocks <= sms * kDecLightBlocks;
  // more than two CTAs per SM: as many as fit, so that every SM has the same number
  const bool even = light && likely_blocks > sms * kDecLightWarps * (kDecLightCtas - 1);
  const uint64_t want = light && !even ? div_up_u64(max_blocks, kDecLightWarps) : max_blocks;
  const uint64_t cap = light ? sms * kDecLightCtas : sms;
  const unsigned grid = (unsigned)(want < 1 ? 1 : (want < cap ? want : cap));
  if (light)
    return launch(ans_decode_kernel<true>, grid, kDecLightWarps * 32, kDecLightSmem, s, in, in_size,
                  out, out_cap, ctrl, expect_p, record);
  return launch(ans_decode_kernel<false>, grid, kDecFullWarps * 32, kDecFullSmem, s, in, in_size, out,
                out_cap, ctrl, expect_p, record);
}

}  // namespace mans
