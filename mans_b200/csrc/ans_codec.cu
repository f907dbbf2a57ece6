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
constexpr int kEncMaxWarps = 32, kEncMaxThreads = kEncMaxWarps * 32;

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
  while (!failed) {
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
// global memory, no deferral), for the allocation-free call.
__global__ __launch_bounds__(kEncThreads) void ans_encode_shared_kernel(
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
  if (!failed) ss.table[t] = ctrl->enc_table[t];
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
    encode_block<false>(in, n, out, out_cap, out_size64, out_size32, ctrl->pdf, flags, epoch, p,
                        sink, ss.table, ss.in[warp], bar, parity, ss.out[warp], b, lane);
  }
  encode_done(ctrl, epoch);
}

// ------------------------------------------------------------------------
// Decode: a warp decodes a block, or two together, from the last step to the
// first. One CTA of up to 32 warps per SM shares the replicated slot table
// (128 KiB). What bounds it: per step 22 instructions (block overhead included)
// of which 7 go to the half-rate integer ALU, two population counts, and a chain of two
// shared-memory loads, a vote and a population count (about 130 cycles) that
// only other chains can hide. The former kernel (22 instructions, 12 of them
// ALU, table conflicts on 40% of its shared wavefronts, 32 chains per SM
// instead of 64) took 0.575 ms on 1 GiB of detector frames (here 0.525), 1.092
// on a 2 GiB uint16 volume (1.042), 27.7 us on 8 MiB of uint16 (21.0) and 131 us
// on 100 MB of skewed bytes at p = 11 (105; its drop-in call also launched half
// a resident wave). A single block takes 14.4 us instead of 13.4.
// ------------------------------------------------------------------------
constexpr int kDecMaxWarps = 32, kDecMinWarps = 8;
constexpr size_t kDecStageMax = (size_t)kDecMaxWarps * 2 * sizeof(DecWarp);
constexpr size_t dec_stage_bytes(size_t warps, int blocks) {
  return warps * sizeof(DecWhole) <= kDecStageMax ? warps * sizeof(DecWhole)
                                                  : warps * blocks * sizeof(DecWarp);
}

// kBlocks: blocks that a warp takes at a time and decodes together (one at a
// time once less than a block per warp of the grid is left, so that the last
// wave is short). Each warp's first blocks are fixed, spread over the CTAs, and
// the rest is claimed: a small input then takes no claim at all (4,736 warps on
// one counter cost 5 us). The next claim and its prefetches come in the middle
// of the current blocks, where other warps hide their latency.
template <int kP, int kBlocks>
__device__ __forceinline__ void decode_blocks(const uint8_t* __restrict__ in, uint32_t nb, uint32_t n,
                                              uint32_t cw, uint8_t* __restrict__ out,
                                              const uint8_t* lut, uint8_t* stage, uint32_t stage_bytes,
                                              Ctrl* ctrl, const Sink& sink, int lane) {
  auto bad = [&](uint32_t k) { report(sink, MANS_ERR_CORRUPT, k); };
  const uint32_t warp = threadIdx.x >> 5;
  if ((uint64_t)stage_bytes / sizeof(DecWhole) * gridDim.x >= nb) {
    // a block per warp at most, and room to stage its words whole
    const uint32_t k = warp * gridDim.x + blockIdx.x;
    if (k < nb)
      decode_block<kP, 1>(in, nb, n, cw, out, lut, reinterpret_cast<DecWhole*>(stage) + warp, k, lane,
                          [](int) {}, bad);
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
  uint32_t b = first * (warp * gridDim.x + blockIdx.x);
  while (b < nb) {
    uint32_t nxt = 0, nxt_take = 0;
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
    bool pair = kBlocks == 2 && take == 2 && b + 2 < nb;
    if (pair) pair = decode_block<kP, kBlocks>(in, nb, n, cw, out, lut, ws, b, lane, hook, bad);
    if (!pair) {
      // one by one (the last block may be short, and has no fixed chunks); the
      // hook has not run, so the next claim is made here
      for (uint32_t k = b; k < nb && k < b + take; ++k)
        decode_block<kP, 1>(in, nb, n, cw, out, lut, ws, k, lane, [](int) {}, bad);
      nxt = claim(b, nxt_take);
    }
    b = nxt;
    take = nxt_take;
  }
}

template <int kBlocks>
__global__ __launch_bounds__(kDecMaxWarps * 32, 1) void ans_decode_kernel(
    const uint8_t* __restrict__ in, uint64_t in_size, uint8_t* __restrict__ out, uint64_t out_cap,
    Ctrl* ctrl, int expect_p, int record, uint32_t stage_bytes) {
  kernel_begin();
  extern __shared__ __align__(16) uint8_t smem_raw[];
  __shared__ uint32_t s_incl[kAnsSyms];
  __shared__ int s_ok;
  const int t = threadIdx.x, lane = t & 31;
  uint8_t* const lut = smem_raw;  // below every warp's words (see decode_block)
  uint8_t* const stage = smem_raw + kDecLutBytes;
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

  if (s_ok && blockIdx.x < nb) {  // CTA k holds block k at least
    const bool tables_ok = dec_build_lut(pdf, p, lut, s_incl);
    if (!tables_ok && blockIdx.x == 0 && t == 0) report(sink, MANS_ERR_BAD_STREAM, 1);
    __syncthreads();
    if (tables_ok) {
      switch (p) {
        case 9: decode_blocks<9, kBlocks>(in, nb, n, cw, out, lut, stage, stage_bytes, ctrl, sink, lane); break;
        case 10: decode_blocks<10, kBlocks>(in, nb, n, cw, out, lut, stage, stage_bytes, ctrl, sink, lane); break;
        default: decode_blocks<11, kBlocks>(in, nb, n, cw, out, lut, stage, stage_bytes, ctrl, sink, lane); break;
      }
    }
  }

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
  cudaFuncSetAttribute(ans_decode_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)(kDecLutBytes + kDecStageMax));
  cudaFuncSetAttribute(ans_decode_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)(kDecLutBytes + kDecStageMax));
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
    warps = warps < 4 ? 4 : warps < kEncMaxWarps ? warps : kEncMaxWarps;
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

cudaError_t launch_ans_decode(const uint8_t* in, uint64_t in_size, uint8_t* out, uint64_t out_cap,
                              Ctrl* ctrl, int expect_p, int record, uint64_t likely_blocks,
                              uint64_t max_blocks, const LaunchCfg& cfg, cudaStream_t s) {
  // One CTA per SM with as many warps as spread the blocks evenly; a warp takes
  // two blocks together once a block per warp does not hold them all (16 M
  // uint16 values, 30 blocks per SM: decode 31 us one by one, 36 in pairs; 24 M,
  // 45 per SM: 50 and 40; 1 GiB of detector frames: 0.591 and 0.525 ms).
  const int blocks = likely_blocks > (uint64_t)cfg.sms * kDecMaxWarps ? 2 : 1;
  uint64_t warps = div_up_u64(likely_blocks, (uint64_t)cfg.sms * blocks);
  warps = warps < kDecMinWarps ? kDecMinWarps : warps < kDecMaxWarps ? warps : kDecMaxWarps;
  const uint64_t want = div_up_u64(max_blocks, warps * blocks);
  const unsigned grid =
      (unsigned)(want < 1 ? 1 : (want < (uint64_t)cfg.sms ? want : (uint64_t)cfg.sms));
  auto* k = blocks == 2 ? ans_decode_kernel<2> : ans_decode_kernel<1>;
  const size_t stage = dec_stage_bytes(warps, blocks);
  return launch(k, grid, (unsigned)warps * 32, kDecLutBytes + stage, s, in, in_size, out, out_cap,
                ctrl, expect_p, record, (uint32_t)stage);
}

}  // namespace mans
