// ans_dev.cuh -- per-block work of the byte rANS codec for sm_100a (encode
// with in-place output compaction, decode), shared by the single-buffer and
// batched kernels.
//
// Arithmetic and layout: include/ans/GpuANSEncode.h:25-164 and :181-284,
// include/ans/GpuANSDecode.h:27-302 (see ans_codec.cu for the organisation).
#pragma once

#include "ans_table.cuh"
#include "mans_internal.h"
#include "smem_io.cuh"

namespace mans {

constexpr int kEncWarps = 8;
constexpr int kEncThreads = kEncWarps * 32;
constexpr uint32_t kEncOutWords = kAnsMaxBlockWords + 8;
// A block's words compacted in global memory: slots of whole 128-byte lines.
constexpr uint32_t kEncSlotBytes = (kEncOutWords * 2 + 127) / 128 * 128;

constexpr uint32_t kEncStageBytes = kAnsBlock + 16;  // a block plus its 16-byte phase

// The encoder's per-symbol entry in shared memory, expanded from the packed
// table (make_enc_entry) so that a step needs almost no field extraction:
// {reciprocal, renormalisation threshold pdf << (31 - p), bias,
//  shift | cmpl << 5}. The quotient's shift is taken from the low five bits
// of the last word by a wrapping funnel shift.
struct alignas(16) EncEntry4 {
  uint32_t rcp, thr, bias, cs;
};
__device__ __forceinline__ EncEntry4 expand_enc_entry(uint2 e, int p) {
  const uint32_t cmpl = e.y >> 20;
  return EncEntry4{e.x, ((1u << p) - cmpl) << (kAnsStateBits - p), (e.y >> 5) & 0x1fffu,
                   (e.y & 31u) | (cmpl << 5)};
}

struct EncSmem {  // words compacted in shared memory
  union {
    uint2 packed[kAnsSyms];
    EncEntry4 expanded[kAnsSyms];
  };
  alignas(16) uint8_t in[kEncWarps][kEncStageBytes];
  uint64_t bar[kEncWarps];
  alignas(16) uint16_t out[kEncWarps][kEncOutWords];
};

// The coding step's symbol arithmetic for precision kP:
// x' = (xr / pdf << p) + xr % pdf + cdf = xr + bias + q * cmpl, q = xr / pdf.
template <int kP>
__device__ __forceinline__ uint32_t enc_code(uint32_t xr, const uint2& e) {
  const uint32_t q = __funnelshift_r(__umulhi(xr, e.x), 0u, e.y);  // shift = y & 31
  return xr + ((e.y >> 5) & 0x1fffu) + q * (e.y >> 20);
}
template <int kP>
__device__ __forceinline__ uint32_t enc_code(uint32_t xr, const EncEntry4& e) {
  const uint32_t q = __funnelshift_r(__umulhi(xr, e.rcp), 0u, e.cs);  // shift = cs & 31
  return xr + e.bias + q * (e.cs >> 5);
}
template <int kP>
__device__ __forceinline__ uint32_t enc_threshold(const uint2& e) {
  return ((1u << kP) - (e.y >> 20)) << (kAnsStateBits - kP);
}
template <int kP>
__device__ __forceinline__ uint32_t enc_threshold(const EncEntry4& e) {
  return e.thr;
}
// One interleaved step: renormalise (emit 16 bits, lanes in ascending order
// into the compacted word buffer), then code the symbol.
// kGuard: drop words past the buffer (see encode_words).
template <int kP, bool kGuard, bool kShared, typename Entry>
__device__ __forceinline__ void enc_step(bool valid, uint32_t& x, uint32_t sym,
                                         const Entry* __restrict__ tab, uint16_t* __restrict__ out,
                                         uint32_t& nw, uint32_t ltmask) {
  const Entry e = tab[sym];
  const bool wr = valid && x >= enc_threshold<kP>(e);
  const uint32_t vote = __ballot_sync(0xffffffffu, wr);
  const uint32_t idx = nw + __popc(vote & ltmask);
  const bool st = wr && (!kGuard || idx < kEncOutWords);
  if constexpr (kShared) {
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n @q st.shared.u16 [%0], %1;\n}\n"
                 ::"r"((uint32_t)__cvta_generic_to_shared(out + idx)), "h"((uint16_t)x),
                 "r"((uint32_t)st)
                 : "memory");
  } else {
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n @q st.global.u16 [%0], %1;\n}\n"
                 ::"l"(out + idx), "h"((uint16_t)x), "r"((uint32_t)st)
                 : "memory");
  }
  nw += __popc(vote);
  const uint32_t xr = wr ? (x >> 16) : x;
  x = valid ? enc_code<kP>(xr, e) : xr;
}

__device__ __forceinline__ void discard_l2_line(const void* p) {
  asm volatile("discard.global.L2 [%0], 128;" ::"l"(p) : "memory");
}

// The coding of one staged block (syms: the lane's first symbol in the stage,
// bs bytes) at precision kP. kShared: sout is in shared memory (else a
// global slot). Returns the word count; x receives the lane's final state.
template <int kP, bool kShared, typename Entry>
__device__ __forceinline__ uint32_t encode_staged(const uint8_t* syms, uint32_t bs,
                                                  const Entry* table, uint16_t* sout, int lane,
                                                  uint32_t& x) {
  const uint32_t ltmask = lanemask_lt();
  x = kAnsStartState;
  uint32_t nw = 0;
  const uint32_t full = bs >> 5;
  uint32_t j = 0;
  // Each step adds at most 32 words, and nw is the same in every lane: while
  // nw <= kRoom the next eight steps fit in the buffer without a check. The
  // eight symbol loads of a round do not depend on the state, so they issue
  // ahead of the round's coding chain.
  constexpr uint32_t kRoom = kEncOutWords - 8 * 32;
  for (; j + 8 <= full && nw <= kRoom; j += 8) {
#pragma unroll
    for (int u = 0; u < 8; ++u)
      enc_step<kP, false, kShared>(true, x, syms[(j + u) * 32], table, sout, nw, ltmask);
  }
  const bool tail_valid = (uint32_t)lane < (bs & 31);
  if (nw <= kRoom) {  // at most seven more steps and the partial one
    for (; j < full; ++j)
      enc_step<kP, false, kShared>(true, x, syms[j * 32], table, sout, nw, ltmask);
    if (bs & 31)
      enc_step<kP, false, kShared>(tail_valid, x, tail_valid ? syms[j * 32] : 0u, table, sout, nw,
                                   ltmask);
  } else {
    for (; j < full; ++j)
      enc_step<kP, true, kShared>(true, x, syms[j * 32], table, sout, nw, ltmask);
    if (bs & 31)
      enc_step<kP, true, kShared>(tail_valid, x, tail_valid ? syms[j * 32] : 0u, table, sout, nw,
                                  ltmask);
  }
  return nw;
}

// Encode block b of one buffer (one warp) into the warp's word buffer sout
// (kSharedOut: in shared memory, else a per-warp slot in global memory,
// which stays in L2): one bulk copy of the block into the warp's stage, then the
// interleaved coding; the word count is padded to a 16-byte multiple with
// zeros (GpuANSEncode.h:275). Returns the number of words; x receives the
// lane's final state.
template <bool kSharedOut, typename Entry>
__device__ __forceinline__ uint32_t encode_words(const uint8_t* __restrict__ in, uint64_t n,
                                                 uint32_t b, const Entry* table, uint8_t* stage,
                                                 uint64_t* bar, uint32_t& parity, uint16_t* sout,
                                                 int p, const Sink& sink, int lane, uint32_t& x) {
  const uint64_t start = (uint64_t)b * kAnsBlock;
  const uint32_t bs = (uint32_t)min_u64(kAnsBlock, n - start);
  // one bulk copy of the block (rounded out to 16-byte boundaries) into this
  // warp's stage; the previous block's reads of the stage are complete
  __syncwarp();
  if (lane == 0) {
    const uintptr_t a0 = reinterpret_cast<uintptr_t>(in + start) & ~uintptr_t(15);
    const uintptr_t a1 = (reinterpret_cast<uintptr_t>(in + start) + bs + 15) & ~uintptr_t(15);
    bulk_load(stage, reinterpret_cast<const void*>(a0), (uint32_t)(a1 - a0), bar);
  }
  if (!mbar_wait(bar, parity) && lane == 0) report(sink, MANS_ERR_TIMEOUT, b);
  parity ^= 1u;
  const uint8_t* syms = stage + phase16(in + start) + lane;
  uint32_t nw;
  switch (p) {
    case 9: nw = encode_staged<9, kSharedOut>(syms, bs, table, sout, lane, x); break;
    case 10: nw = encode_staged<10, kSharedOut>(syms, bs, table, sout, lane, x); break;
    default: nw = encode_staged<11, kSharedOut>(syms, bs, table, sout, lane, x); break;
  }
  // A table that fits the block's bytes keeps each lane within its bound of
  // words (kAnsMaxBlockWords / 32); only a table built from other bytes (two
  // calls racing on one scratch area) can exceed it. Word writes past the
  // buffer are dropped above, and the block is reported.
  if (nw > kAnsMaxBlockWords) {
    if (lane == 0) report(sink, MANS_ERR_CORRUPT, b);
    nw = kAnsMaxBlockWords;
  }
  const uint32_t padded = (nw + 7) & ~7u;
  if ((uint32_t)lane < padded - nw) sout[nw + lane] = 0;
  return nw;
}

// ---- asynchronous copies global -> shared ----
__device__ __forceinline__ void cp_async16(uint32_t smem, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t smem, const void* g) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// ---- encode with replicated tables (word slots in global memory) ----
// The step's integer instructions bound the coder (the ALU pipe issues at half
// rate), and shared-memory wavefronts come next. 16-byte entries need the
// fewest instructions (24 per step, block overhead included; 29 with the
// packed 8-byte entry) and the copies below keep a lookup at four wavefronts
// for any distribution (unreplicated: 5 to 10 on a flat one). On 1 GiB of
// detector frames 0.695 -> 0.641 ms, a 2 GiB uint16 volume 1.622 -> 1.321 ms,
// 100 MB of skewed bytes 151 -> 113 us, 8 MiB of uint16 37.5 -> 21 us against
// a table per CTA of eight warps in one of two layouts, with each step's words
// stored to the slot in global memory.
// Expanded entries (EncEntry4) in 8 copies: entry s of copy c at 128 s + 16 c.
// A lane reads copy lane % 8, so the four quarter-warps of a 16-byte load
// never conflict, whatever symbols they look up.
constexpr uint32_t kEncTableBytes = kAnsSyms * 128;
// A block's words collect in shared memory and leave for the slot in pieces
// of 256 words (one 16-byte store per lane), checked every eight steps: at
// most 255 words are left over, and eight steps add at most 256.
constexpr uint32_t kEncPieceWords = 256;
// Steps whose table entries are loaded ahead of the coding chain (eight spill
// at 64 registers, and 24 warps per SM with 80 registers are slower: 0.696 ms
// on the detector frames).
constexpr int kEncAhead = 4;
struct EncWarp {
  alignas(16) uint8_t in[kEncStageBytes];
  alignas(16) uint16_t words[2 * kEncPieceWords];
  alignas(16) uint64_t bar;
};
inline size_t enc_smem_bytes(int warps) { return kEncTableBytes + (size_t)warps * sizeof(EncWarp); }

// Fill the table from 256 packed entries (all threads of the CTA; the caller
// synchronises). Rotated, so that the lanes of a store spread over the banks.
__device__ __forceinline__ void enc_fill_table(uint8_t* tab, const uint2* __restrict__ enc, int p) {
  // each entry is loaded once (a load per copy cost a small input 16 round trips
  // to L2, one after the other)
#pragma unroll 2
  for (uint32_t sym = threadIdx.x; sym < kAnsSyms; sym += blockDim.x) {
    const EncEntry4 e = expand_enc_entry(enc[sym], p);
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c)
      *reinterpret_cast<EncEntry4*>(tab + 128 * sym + 16 * ((c + sym) & 7)) = e;
  }
}

// One interleaved step: renormalise (16 bits of each lane whose state is at
// its threshold, in lane order, to shared address wa on), then code. In PTX,
// so that one predicate serves the vote, the store and the shift: the integer
// ALU, which issues at half rate, bounds the coder.
template <int kP>
__device__ __forceinline__ void enc_step_rep(uint32_t& x, const EncEntry4& e, uint32_t& wa,
                                             uint32_t ltmask) {
  asm volatile(
      "{\n .reg .pred p;\n .reg .b32 v, r;\n"
      " setp.ge.u32 p, %0, %2;\n"
      " vote.sync.ballot.b32 v, p, 0xffffffff;\n"
      " and.b32 r, v, %3;\n popc.b32 r, r;\n mad.lo.u32 r, r, 2, %1;\n"
      " @p st.shared.u16 [r], %0;\n"
      " popc.b32 v, v;\n mad.lo.u32 %1, v, 2, %1;\n"
      " @p shr.u32 %0, %0, 16;\n}\n"
      : "+r"(x), "+r"(wa) : "r"(e.thr), "r"(ltmask) : "memory");
  x = enc_code<kP>(x, e);
}
// The same for a partial step: only lanes with `valid` hold a symbol.
template <int kP>
__device__ __forceinline__ void enc_step_part(bool valid, uint32_t& x, const EncEntry4& e,
                                              uint32_t& wa,
                                              uint32_t ltmask) {
  const bool wr = valid && x >= e.thr;
  const uint32_t vote = __ballot_sync(0xffffffffu, wr);
  if (wr) {
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(wa + 2u * __popc(vote & ltmask)), "r"(x) : "memory");
    x >>= 16;
  }
  wa += 2u * __popc(vote);
  if (valid) x = enc_code<kP>(x, e);
}

// Encode a staged block (syms: the lane's first symbol in the stage, bs bytes)
// into its word slot, padded to a multiple of eight words with zeros. Returns
// the word count; x receives the lane's final state.
template <int kP>
__device__ __forceinline__ uint32_t encode_staged_rep(const uint8_t* syms, uint32_t bs,
                                                      const uint8_t* tab, uint16_t* words,
                                                      uint8_t* slot, int lane, uint32_t& x) {
  const uint32_t ltmask = lanemask_lt();
  const uint32_t wb = smem_addr(words);
  const uint8_t* const tl = tab + 16 * (lane & 7);
  auto entry = [&](uint32_t sym) { return *reinterpret_cast<const EncEntry4*>(tl + 128 * sym); };
  x = kAnsStartState;
  uint32_t wa = wb, done = 0;  // shared address of the next word; bytes in the slot
  const uint32_t full = bs >> 5;
  uint32_t j = 0;
#pragma unroll 1
  for (; j + 8 <= full; j += 8) {
#pragma unroll
    for (int h = 0; h < 8; h += kEncAhead) {
      EncEntry4 e[kEncAhead];
#pragma unroll
      for (int u = 0; u < kEncAhead; ++u) e[u] = entry(syms[(j + h + u) * 32]);
#pragma unroll
      for (int u = 0; u < kEncAhead; ++u) enc_step_rep<kP>(x, e[u], wa, ltmask);
    }
    if (wa - wb >= 2 * kEncPieceWords) {
      __syncwarp();
      const uint4* src = reinterpret_cast<const uint4*>(words) + lane;
      const uint4 v = src[0], r = src[32];
      // a slot holds any block whose words fit the bound; more only come from
      // a table that does not belong to the bytes, and are dropped
      if (done + 2 * kEncPieceWords <= kEncSlotBytes)
        *reinterpret_cast<uint4*>(slot + done + 16 * lane) = v;
      __syncwarp();
      reinterpret_cast<uint4*>(words)[lane] = r;
      __syncwarp();
      wa -= 2 * kEncPieceWords;
      done += 2 * kEncPieceWords;
    }
  }
  for (; j < full; ++j) enc_step_rep<kP>(x, entry(syms[j * 32]), wa, ltmask);
  if (bs & 31) {
    const bool valid = (uint32_t)lane < (bs & 31);
    enc_step_part<kP>(valid, x, entry(valid ? syms[j * 32] : 0u), wa, ltmask);
  }
  const uint32_t rem = (wa - wb) >> 1;  // < 512
  const uint32_t padded = (rem + 7) & ~7u;
  __syncwarp();
  if ((uint32_t)lane < padded - rem) words[rem + lane] = 0;
  __syncwarp();
  for (uint32_t i = lane; i < padded / 8; i += 32)
    if (done + 16 * i + 16 <= kEncSlotBytes)
      *reinterpret_cast<uint4*>(slot + done + 16 * i) = reinterpret_cast<const uint4*>(words)[i];
  return done / 2 + rem;
}

// Stage block [b0, b1) of a mapped uint32 buffer whose records lie in slots
// (AnsGather): all parts begin and end on 8-byte boundaries. A full group has
// 512 record bytes at least, so a block holds parts of ten groups at most (and
// of one short last group). Also prefetches the records of block `later` into
// L2 (past the last block: nothing).
__device__ __forceinline__ void enc_gather(const uint8_t* __restrict__ in, uint64_t n, uint32_t b,
                                           uint64_t later, const AnsGather& src, uint8_t* stage,
                                           int lane) {
  const uint64_t b0 = (uint64_t)b * kAnsBlock, b1 = min_u64(b0 + kAnsBlock, n);
  const uint64_t rb = 40 * src.groups;
  const uint32_t* off = reinterpret_cast<const uint32_t*>(in);
  const uint32_t total = (uint32_t)(n - rb);
  const uint64_t l0 = later * kAnsBlock, l1 = min_u64(l0 + kAnsBlock, n);
  const bool ahead = l0 < n && l1 > rb;
  const uint32_t f = b1 > rb ? src.first_group[b] : 0u;
  const uint32_t lf = ahead ? src.first_group[later] : 0u;
  auto offset = [&](uint64_t k) { return k < src.groups ? off[k] : total; };
  const uint32_t o = offset((uint64_t)f + lane);
  const uint32_t lo = offset((uint64_t)lf + lane), lo1 = __shfl_down_sync(0xffffffffu, lo, 1);
  if (ahead && lane < 12 && lo < lo1 && rb + lo < l1)
    prefetch_l2(src.slots + ((uint64_t)lf + lane) * 4096, lo1 - lo);
  const uint32_t dst = smem_addr(stage);
  if (b0 < rb) {
    const uint32_t h = (uint32_t)(min_u64(b1, rb) - b0);
    for (uint32_t i = 8 * lane; i < h; i += 256) cp_async8(dst + i, in + b0 + i);
  }
  if (b1 > rb) {
    // lane k: its group's part of record bytes [r0, r1), in the slots and in
    // the stage
    const uint32_t r0 = (uint32_t)(b0 > rb ? b0 - rb : 0), r1 = (uint32_t)(b1 - rb);
    const uint32_t o1 = __shfl_down_sync(0xffffffffu, o, 1);
    const uint32_t p0 = max(o, r0), len = min(o1, r1) - p0;
    const uint32_t from = 4096u * lane + p0 - o;
    const uint32_t to = dst + (uint32_t)(b0 > rb ? 0 : rb - b0) + p0 - r0;
    const uint32_t parts = __popc(__ballot_sync(0xffffffffu, lane < 31 && o < r1));
    const uint8_t* const g = src.slots + (uint64_t)f * 4096 + 8 * lane;
    for (uint32_t k = 0; k < parts; ++k) {
      const uint32_t n8 = __shfl_sync(0xffffffffu, len, k);
      const uint8_t* p = g + __shfl_sync(0xffffffffu, from, k);
      uint32_t q = __shfl_sync(0xffffffffu, to, k) + 8 * lane;
      for (uint32_t i = 8 * lane; i < n8; i += 1024, p += 1024, q += 1024) {
        cp_async8(q, p);
#pragma unroll
        for (uint32_t u = 256; u < 1024; u += 256)
          if (i + u < n8) cp_async8(q + u, p + u);
      }
    }
  }
  cp_async_wait_all();
}

// encode_words for the replicated table: block b of one buffer (one warp).
// kGather: the block's bytes come from slots (src), and block `later` is
// prefetched.
template <int kP, bool kGather>
__device__ __forceinline__ uint32_t encode_words_rep(const uint8_t* __restrict__ in, uint64_t n,
                                                     uint32_t b, const uint8_t* tab, EncWarp& sw,
                                                     uint32_t& parity, uint16_t* slot,
                                                     const Sink& sink, int lane, uint32_t& x,
                                                     const AnsGather& src, uint64_t later) {
  const uint64_t start = (uint64_t)b * kAnsBlock;
  const uint32_t bs = (uint32_t)min_u64(kAnsBlock, n - start);
  __syncwarp();  // the previous block's reads of the stage are complete
  if (kGather) {
    enc_gather(in, n, b, later, src, sw.in, lane);
    __syncwarp();
  } else if (lane == 0) {
    const uintptr_t a0 = reinterpret_cast<uintptr_t>(in + start) & ~uintptr_t(15);
    const uintptr_t a1 = (reinterpret_cast<uintptr_t>(in + start) + bs + 15) & ~uintptr_t(15);
    bulk_load(sw.in, reinterpret_cast<const void*>(a0), (uint32_t)(a1 - a0), &sw.bar);
  }
  if (!kGather) {
    if (!mbar_wait(&sw.bar, parity) && lane == 0) report(sink, MANS_ERR_TIMEOUT, b);
    parity ^= 1u;
  }
  uint32_t nw = encode_staged_rep<kP>(sw.in + phase16(in + start) + lane, bs, tab, sw.words,
                                      reinterpret_cast<uint8_t*>(slot), lane, x);
  if (nw > kAnsMaxBlockWords) {  // see encode_words
    if (lane == 0) report(sink, MANS_ERR_CORRUPT, b);
    nw = kAnsMaxBlockWords;
  }
  return nw;
}

// Store block b, whose nw words (padded to padded) start at word `prefix` of
// the stream's data section: lane states, block word entry, the words, and
// for the buffer's last block the header, pdf and size. Then the slot's
// lines are dropped from L2 without write-back.
template <bool kSlots>
__device__ __forceinline__ void encode_store(uint8_t* __restrict__ out, uint64_t out_cap,
                                             uint64_t n, int p, const uint32_t* __restrict__ pdf,
                                             unsigned long long* out_size64, uint32_t* out_size32,
                                             const Sink& sink, uint32_t b, uint32_t nw,
                                             uint32_t prefix, uint32_t x, const uint16_t* sout,
                                             int lane) {
  const uint64_t nb = div_up_u64(n, kAnsBlock);
  const uint64_t over = ans_overhead(nb);
  const uint32_t bs = (uint32_t)min_u64(kAnsBlock, n - (uint64_t)b * kAnsBlock);
  const uint32_t padded = (nw + 7) & ~7u;
  const uint64_t end = over + 2ull * ((uint64_t)prefix + padded);
  const bool last = (uint64_t)b + 1 == nb;
  if (last && end > out_cap && lane == 0) report(sink, MANS_ERR_OUTPUT_OVERFLOW, end);
  if (end <= out_cap) {
    uint32_t* states = reinterpret_cast<uint32_t*>(out + kAnsHeaderBytes + 2 * kAnsSyms);
    states[(uint64_t)b * 32 + lane] = x;
    uint2* bw = reinterpret_cast<uint2*>(out + kAnsHeaderBytes + 2 * kAnsSyms + 128 * nb);
    if (lane == 0) bw[b] = make_uint2((bs << 16) | nw, prefix);
    uint4* dst = reinterpret_cast<uint4*>(out + over + 2ull * prefix);
    const uint4* src = reinterpret_cast<const uint4*>(sout);
    const uint32_t cnt = padded / 8;
    if (kSlots) {  // four loads in flight per lane
      for (uint32_t i = lane; i < cnt; i += 128) {
        uint4 v[4];
#pragma unroll
        for (uint32_t h = 0; h < 4; ++h)
          if (i + 32 * h < cnt) v[h] = __ldcg(src + i + 32 * h);
#pragma unroll
        for (uint32_t h = 0; h < 4; ++h)
          if (i + 32 * h < cnt) dst[i + 32 * h] = v[h];
      }
    } else {
      for (uint32_t i = lane; i < cnt; i += 32) dst[i] = src[i];
    }
    if (last) {
      if (lane < 8) {
        const uint32_t hv = lane == 0 ? kAnsMagicVersion
                          : lane == 1 ? (uint32_t)nb
                          : lane == 2 ? (uint32_t)n
                          : lane == 3 ? prefix + padded
                          : lane == 4 ? (uint32_t)p : 0u;
        reinterpret_cast<uint32_t*>(out)[lane] = hv;
      }
      for (int i = lane; i < kAnsSyms; i += 32)
        reinterpret_cast<uint16_t*>(out + kAnsHeaderBytes)[i] = (uint16_t)pdf[i];
      if (lane == 0 && (nb & 1)) bw[nb] = make_uint2(0, 0);
      if (lane == 0) {
        if (out_size64) *out_size64 = end;
        if (out_size32) *out_size32 = (uint32_t)end;
      }
    }
  }
  __syncwarp();
  if (kSlots) {
    // the slot's lines are consumed: drop them from L2 without write-back
    const uint32_t lines = (2 * padded + 127) / 128;
    if ((uint32_t)lane < lines) discard_l2_line(reinterpret_cast<const uint8_t*>(sout) + 128 * lane);
    if ((uint32_t)lane + 32 < lines)
      discard_l2_line(reinterpret_cast<const uint8_t*>(sout) + 128 * (lane + 32));
    __syncwarp();
  }
}

// A block whose words wait in their slot for the block's stream offset.
struct EncPending {
  uint32_t b;      // block index (0xffffffff: none)
  uint32_t nw;     // its words
  uint32_t x;      // the lane's final state
  uint16_t* sout;  // its word slot
};

// The second half of a block: the exclusive word prefix from the decoupled
// look-back, the block's inclusive prefix, and the store.
template <bool kSlots>
__device__ __forceinline__ void encode_finish(
    uint8_t* __restrict__ out, uint64_t out_cap, uint64_t n, unsigned long long* out_size64,
    uint32_t* out_size32, const uint32_t* __restrict__ pdf, unsigned long long* flags,
    uint32_t epoch, int p, const Sink& sink, const EncPending& pb, int lane) {
  const uint32_t padded = (pb.nw + 7) & ~7u;
  uint32_t prefix = 0;
  if (pb.b > 0) {
    prefix = lookback_exclusive(flags, pb.b, epoch, sink);
    if (lane == 0) st_flag(&flags[pb.b], make_flag(kFlagIncl, epoch, prefix + padded));
  }
  __syncwarp();
  encode_store<kSlots>(out, out_cap, n, p, pdf, out_size64, out_size32, sink, pb.b, pb.nw, prefix,
                       pb.x, pb.sout, lane);
}

// One block, its words in shared memory: encode, publish the aggregate, look
// back, store (flags per block).
template <typename Entry>
__device__ __forceinline__ void encode_block(
    const uint8_t* __restrict__ in, uint64_t n, uint8_t* __restrict__ out, uint64_t out_cap,
    unsigned long long* out_size64, uint32_t* out_size32, const uint32_t* __restrict__ pdf,
    unsigned long long* flags, uint32_t epoch, int p, const Sink& sink, const Entry* table,
    uint8_t* stage, uint64_t* bar, uint32_t& parity, uint16_t* sout, uint32_t b, int lane) {
  uint32_t x;
  const uint32_t nw =
      encode_words<true>(in, n, b, table, stage, bar, parity, sout, p, sink, lane, x);
  const uint32_t padded = (nw + 7) & ~7u;
  if (lane == 0) st_flag(&flags[b], make_flag(b == 0 ? kFlagIncl : kFlagAgg, epoch, padded));
  encode_finish<false>(out, out_cap, n, out_size64, out_size32, pdf, flags, epoch, p, sink,
                       EncPending{b, nw, x, sout}, lane);
}

// ---- decode ----
constexpr int kMaxProbBits = 11;

// The slot table of a stream's pdf: for slot s = x mod 2^p of symbol y, what
// turns the state x into pdf * (x >> p) + (s - cdf) (GpuANSDecode.h:307-377).
// Slots are uniformly distributed whatever the data, so with one copy the 32
// lookups of a step conflict; a lane that reads its own copy (lane modulo the
// copies) takes fewer shared-memory wavefronts. Three forms:
//  kTabWide: {P = pdf << (32 - p), D << 8 | y}, D = (s - cdf) - (s * pdf >> p)
//    (signed): the new state is umulhi(x, P) + D, since umulhi(x, P) = x * pdf
//    >> p = pdf * (x >> p) + (s * pdf >> p), exactly, and the second term depends
//    on s alone. (pdf = 2^p, a single symbol: P = 2^32 - 1 and D = 1, since the
//    state x >= 1 stays as it is.) 8 bytes, 16 copies, 2 wavefronts: the fewest
//    instructions, for p <= 10.
//  kTabMany: {s - cdf:12, y:8, pdf:12} (one instruction per field, and one between
//    the load and the multiplication), 4 bytes, 16 copies, 2 wavefronts: for p =
//    11, where the wide form has room for 8 copies only (4 wavefronts; 100 MB of
//    bytes 103.0 us, here 94.8).
//  kTabOne: the same entries, one copy (about 3.5 wavefronts): at most 8 KiB, quick
//    to build and small beside other kernels on the SM.
enum DecTab { kTabWide, kTabMany, kTabOne };
constexpr int kDecCopyBits = 4;
constexpr uint32_t kDecLutBytes = 128u << 10;                // kTabWide, kTabMany
constexpr uint32_t kDecLutOneBytes = 4u << kMaxProbBits;     // kTabOne
__host__ __device__ constexpr DecTab dec_many(int p) { return p <= 10 ? kTabWide : kTabMany; }
__device__ __forceinline__ uint2 make_dec_entry(uint32_t pdf, uint32_t s, uint32_t cdf, uint32_t sym,
                                                int p) {
  if (pdf >> p) return make_uint2(0xffffffffu, (1u << 8) | sym);
  return make_uint2(pdf << (32 - p), ((s - cdf - ((s * pdf) >> p)) << 8) | sym);
}

// Build the table (all threads of a CTA of at least 256; pdf: symbol
// threadIdx.x's, dec_pdf; s_incl: 256 words of shared scratch). Each slot finds its symbol by bisection of the inclusive
// prefix sums, so a concentrated pdf costs no more than a flat one. Returns
// false, in every thread, when the pdf does not sum to 2^p. The caller
// synchronises before the table is read.
__device__ __forceinline__ uint32_t dec_pdf(const uint8_t* __restrict__ in) {
  return threadIdx.x < kAnsSyms
             ? __ldg(reinterpret_cast<const uint16_t*>(in + kAnsHeaderBytes) + threadIdx.x)
             : 0u;
}
__device__ __forceinline__ bool dec_build_lut(uint32_t pdf, int p, DecTab tab, uint8_t* lut,
                                              uint32_t* s_incl) {
  __shared__ uint32_t s_sum[8];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  uint32_t incl = pdf;
  __syncthreads();  // earlier readers of the table and the scratch are done
  if (t < kAnsSyms) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) s_sum[warp] = incl;
  }
  __syncthreads();
  uint32_t base = 0, total = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    if (w < warp) base += s_sum[w];
    total += s_sum[w];
  }
  if (t < kAnsSyms) s_incl[t] = base + incl;
  __syncthreads();
  if (total != (1u << p)) return false;
#pragma unroll 4
  for (uint32_t s = t; s < (1u << p); s += blockDim.x) {
    uint32_t sym = 0;  // the first symbol whose inclusive sum exceeds s
#pragma unroll
    for (uint32_t h = 128; h > 0; h >>= 1)
      if (s_incl[sym + h - 1] <= s) sym += h;
    const uint32_t hi = s_incl[sym], lo = sym ? s_incl[sym - 1] : 0u;
    const uint32_t e = (s - lo) << 20 | sym << 12 | (hi - lo);
    if (tab == kTabOne) {
      reinterpret_cast<uint32_t*>(lut)[s] = e;
    } else {
      // a row of copies, rotated so that the lanes of a store spread over the banks
      const uint2 w = tab == kTabWide ? make_dec_entry(hi - lo, s, lo, sym, p) : make_uint2(e, e);
      const uint32_t n16 = tab == kTabWide ? 8u : 4u;
      uint4* row = reinterpret_cast<uint4*>(lut) + s * n16;
      for (uint32_t c = 0; c < n16; ++c) row[(c + lane) & (n16 - 1)] = make_uint4(w.x, w.y, w.x, w.y);
    }
  }
  return true;
}

// A block's words are read backwards through a window of two pieces of 256
// words: eight steps read at most one piece, so it is checked every eight
// steps whether the lower piece has been entered, which then moves up, while
// the piece below it, loaded a move ahead, takes its place.
constexpr uint32_t kDecPieceWords = 256;
// Decoded bytes leave through a per-warp 512-byte stage, 16 steps at a time,
// as one 16-byte store per lane.
constexpr int kDecChunkSteps = 16;
constexpr uint32_t kDecChunkBytes = kDecChunkSteps * 32;

struct DecWarp {
  static constexpr bool kWhole = false;
  alignas(16) uint16_t words[2 * kDecPieceWords];
  alignas(16) uint8_t out[kDecChunkBytes + 16];  // a chunk at its destination's phase
};
// Where few warps share the shared memory, a block's words are staged whole,
// without the window's moves and checks.
struct DecWhole {
  static constexpr bool kWhole = true;
  alignas(16) uint16_t words[kEncOutWords];
  alignas(16) uint8_t out[kDecChunkBytes + 16];
};

// Store one decoded 512-byte chunk from the warp's stage, where it sits at
// offset ph = g & 15 (the destination's phase), to g: 16-byte stores for the
// whole 16-byte units and byte stores for a partial first and last unit (the
// mapped buffer that a MANS decode writes starts at any phase).
__device__ __forceinline__ void dec_flush_chunk(uint8_t* __restrict__ g, const uint8_t* ostage,
                                                uint32_t ph, int lane) {
  if (ph == 0) {
    reinterpret_cast<uint4*>(g)[lane] = reinterpret_cast<const uint4*>(ostage)[lane];
    return;
  }
  uint8_t* g0 = g - ph;  // 16-byte aligned; stage unit u <-> g0 + 16 u
  if (lane >= 1) reinterpret_cast<uint4*>(g0)[lane] = reinterpret_cast<const uint4*>(ostage)[lane];
  if (lane < 16) {
    if ((uint32_t)lane >= ph) g0[lane] = ostage[lane];                  // unit 0
    else g0[kDecChunkBytes + lane] = ostage[kDecChunkBytes + lane];      // unit 32
  }
}

__device__ __forceinline__ uint4 ld_shared_v4(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void st_shared_v4(uint32_t a, const uint4& v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z),
               "r"(v.w) : "memory");
}

// The window over a block's words.
struct DecWindow {
  const uint4* below;  // this lane's unit (16 bytes) of the piece below the window
  uint4 next;          // ... loaded
  uint32_t base;       // pieces below the window
  uint32_t wb, wa;     // shared addresses: the window, one past the next word to read

  // Load `next` where want holds. A predicated load in straight-line code: on a
  // branch of its own, the merge with the old value would wait for the load.
  __device__ __forceinline__ void fetch(bool want) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.u32 p, %5, 0;\n"
        " @p ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];\n}\n"
        : "+r"(next.x), "+r"(next.y), "+r"(next.z), "+r"(next.w)
        : "l"(below), "r"((uint32_t)want));
  }
  // The caller synchronises the warp before (the memory's previous readers)
  // and after.
  __device__ __forceinline__ void open(const uint16_t* data, uint32_t nw, uint16_t* w, int lane) {
    const uint4* g = reinterpret_cast<const uint4*>(data);
    const uint32_t total = (nw + 7) / 8;  // units of the block
    base = nw > 2 * kDecPieceWords ? (nw - 1) / kDecPieceWords - 1 : 0u;
    wb = smem_addr(w);
    wa = wb + 2 * (nw - base * kDecPieceWords);
    next = make_uint4(0, 0, 0, 0);
    const uint32_t lo = base * (kDecPieceWords / 8) + lane;
    below = g + lo - (kDecPieceWords / 8);
    fetch(base != 0);
    // past L1, of which the table and the windows leave little
    if (lo < total) cp_async16(wb + 16 * lane, g + lo);
    if (lo + kDecPieceWords / 8 < total)
      cp_async16(wb + 2 * kDecPieceWords + 16 * lane, g + lo + kDecPieceWords / 8);
    cp_async_wait_all();
  }
  __device__ __forceinline__ void open_whole(const uint16_t* data, uint32_t nw, uint16_t* w,
                                             int lane) {
    base = 0;
    wb = smem_addr(w);
    wa = wb + 2 * nw;
    for (uint32_t i = lane; i < (nw + 7) / 8; i += 32)
      cp_async16(wb + 16 * i, reinterpret_cast<const uint4*>(data) + i);
    cp_async_wait_all();
  }
  // Before at most eight steps.
  __device__ __forceinline__ void advance(int lane) {
    const bool move = base != 0 && wa - wb < 2 * kDecPieceWords;
    if (move) {
      __syncwarp();
      // each unit is read and written by one lane
      st_shared_v4(wb + 2 * kDecPieceWords + 16 * lane, ld_shared_v4(wb + 16 * lane));
      st_shared_v4(wb + 16 * lane, next);
      __syncwarp();
      wa += 2 * kDecPieceWords;
      --base;
      below -= kDecPieceWords / 8;
    }
    fetch(move && base != 0);
  }
};

// Renormalise: lanes whose state fell below 2^15 read one word each, the
// highest reading lane first (GpuANSDecode.h:78-92). Every lane loads (a lane
// that reads nothing, its next word): a predicated load takes more
// instructions. A lane's load may lie one word past the words, which is the
// warp's own memory still.
__device__ __forceinline__ void dec_read(uint32_t& x, uint32_t& wa, uint32_t gemask) {
  asm volatile(
      "{\n .reg .pred p;\n .reg .b32 v, r, w;\n"
      " setp.lt.u32 p, %0, 32768;\n"
      " vote.sync.ballot.b32 v, p, 0xffffffff;\n"
      " and.b32 r, v, %2;\n popc.b32 r, r;\n mad.lo.u32 r, r, -2, %1;\n"
      " ld.shared.u16 w, [r];\n"
      " popc.b32 v, v;\n mad.lo.u32 %1, v, -2, %1;\n"
      " @p prmt.b32 %0, w, %0, 0x5410;\n}\n"
      : "+r"(x), "+r"(wa) : "r"(gemask) : "memory");
}

// A block's entry and start state, checked against the stream's header.
struct DecBlock {
  const uint16_t* words;
  uint32_t nw, bs, x;
  __device__ __forceinline__ bool load(const uint8_t* __restrict__ in, uint32_t nb, uint32_t n,
                                       uint32_t cw, uint32_t b, int lane) {
    const uint32_t* states = reinterpret_cast<const uint32_t*>(in + kAnsHeaderBytes + 2 * kAnsSyms);
    x = __ldg(states + (uint64_t)b * 32 + lane);
    const uint2 bw = __ldg(reinterpret_cast<const uint2*>(states + 32ull * nb) + b);
    const uint32_t pre = bw.y;
    nw = bw.x & 0xffffu;
    bs = bw.x >> 16;
    words = reinterpret_cast<const uint16_t*>(in + ans_overhead(nb)) + pre;
    const uint32_t expect = (b + 1 == nb) ? n - b * kAnsBlock : kAnsBlock;
    const uint32_t padded = (nw + 7) & ~7u;
    return bs == expect && (uint64_t)pre + padded <= cw && padded <= kEncOutWords && !(pre & 7);
  }
};

// One step's lookup: slot of the state, table entry, new state. Returns the
// symbol in the low byte.
template <int kP, DecTab kTab>
__device__ __forceinline__ uint32_t dec_lookup(uint32_t& x, const uint8_t* lut_lane) {
  constexpr uint32_t kShift = (kTab == kTabWide ? 3 : 2) + (kTab == kTabOne ? 0 : kDecCopyBits);
  constexpr uint32_t kMask = ((1u << kP) - 1u) << kShift;
  const uint8_t* const at = lut_lane + ((x << kShift) & kMask);
  if constexpr (kTab == kTabWide) {
    const uint2 e = *reinterpret_cast<const uint2*>(at);
    asm("mad.hi.u32 %0, %0, %1, %2;" : "+r"(x) : "r"(e.x), "r"((uint32_t)((int)e.y >> 8)));
    return e.y;
  } else {
    const uint32_t e = *reinterpret_cast<const uint32_t*>(at);
    x = (e & 0xfffu) * (x >> kP) + (e >> 20);
    return e >> 12;
  }
}

// Decode kBlocks (1 or 2) consecutive blocks, b on, of one stream (one warp)
// into out + 4096 b. in: the stream (header validated by the caller: nb
// blocks, n bytes, cw words); lut: its slot table for precision kP. A step is a chain of two shared-memory loads, a vote and
// a population count; two blocks at a time give the warp two chains. With
// kBlocks = 2 both blocks are full, and where an entry of the two does not fit
// the stream nothing is decoded or reported and the result is false: the
// caller then takes the blocks one by one, so that a damaged block costs no
// other. (kBlocks = 1: an entry that does not fit is reported.)
// A corrupt stream can move the window's wa below the warp's words, by at most
// 128 steps x 32 words = 8 KiB; the slot table's memory (8 KiB at least) lies
// below every warp's words in the CTA's shared memory, so such reads stay
// inside it, and the final position check reports the block.
// Stage: DecWarp (kBlocks of them) or DecWhole, the warp's shared memory.
// hook(c) runs before chunk c (the block's chunks count down to 0); bad(b) in
// lane 0 reports block b as corrupt.
template <int kP, DecTab kTab, int kBlocks, typename Stage, typename Hook, typename Bad>
__device__ __forceinline__ bool decode_block(const uint8_t* __restrict__ in, uint32_t nb, uint32_t n,
                                             uint32_t cw, uint8_t* __restrict__ out,
                                             const uint8_t* lut, Stage* ws, uint32_t b, int lane,
                                             Hook hook, Bad bad) {
  DecBlock k[kBlocks];
  bool fits = true;
#pragma unroll
  for (int u = 0; u < kBlocks; ++u) {
    const bool f = k[u].load(in, nb, n, cw, b + u, lane);
    if (kBlocks == 1 && !f && lane == 0) bad(b);
    fits = fits && f;
  }
  if (!fits) return false;
  uint8_t* dst = out + (uint64_t)b * kAnsBlock;
  const uint32_t gemask = lanemask_ge();
  const uint8_t* const ll = lut + (kTab == kTabWide ? 8u : 4u) *
                                      (kTab == kTabOne ? 0u : lane & ((1u << kDecCopyBits) - 1));
  DecWindow w[kBlocks];
  __syncwarp();
#pragma unroll
  for (int u = 0; u < kBlocks; ++u) {
    if (Stage::kWhole) w[u].open_whole(k[u].words, k[u].nw, ws[u].words, lane);
    else w[u].open(k[u].words, k[u].nw, ws[u].words, lane);
  }
  __syncwarp();
  int chunks = kAnsStepsPerBlock / kDecChunkSteps;
  if (kBlocks == 1) {
    const uint32_t bs = k[0].bs;
    chunks = (int)(bs / kDecChunkBytes);
    // a last block's other steps, one by one
    for (int j = (int)((bs + 31) >> 5) - 1; j >= chunks * kDecChunkSteps; --j) {
      if (!Stage::kWhole) w[0].advance(lane);
      uint32_t xs = kAnsStartState;  // a lane without a symbol reads nothing
      const bool valid = 32u * j + lane < bs;
      if (valid) {
        xs = k[0].x;
        dst[j * 32 + lane] = (uint8_t)dec_lookup<kP, kTab>(xs, ll);
      }
      dec_read(xs, w[0].wa, gemask);
      if (valid) k[0].x = xs;
    }
  }
  const uint32_t ph = phase16(dst);  // the phase of every chunk
#pragma unroll 1
  for (int c = chunks - 1; c >= 0; --c) {
    hook(c);
#pragma unroll
    for (int i = kDecChunkSteps - 1; i >= 0; --i) {
      if (!Stage::kWhole && (i & 7) == 7) {
#pragma unroll
        for (int u = 0; u < kBlocks; ++u) w[u].advance(lane);
      }
#pragma unroll
      for (int u = 0; u < kBlocks; ++u)
        ws[u].out[ph + lane + i * 32] = (uint8_t)dec_lookup<kP, kTab>(k[u].x, ll);
#pragma unroll
      for (int u = 0; u < kBlocks; ++u) dec_read(k[u].x, w[u].wa, gemask);
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < kBlocks; ++u)
      dec_flush_chunk(dst + u * kAnsBlock + kDecChunkBytes * c, ws[u].out, ph, lane);
    __syncwarp();
  }
#pragma unroll
  for (int u = 0; u < kBlocks; ++u) {
    const bool ok = w[u].base == 0 && w[u].wa == w[u].wb && k[u].x == kAnsStartState;
    if (__any_sync(0xffffffffu, !ok) && lane == 0) bad(b + u);
  }
  return true;
}

}  // namespace mans
