// adm_u32.cu -- single-buffer kernels of the uint32 ADM mapping (per-group
// work in adm_u32.cuh).
#include "adm_u32.cuh"
#include "mans_internal.h"

namespace mans {

// One warp maps one group at a time. Groups are claimed in order, one at a
// time (a claim held while another group is mapped would stall every later
// group's look-back), and the group one grid of warps ahead is prefetched
// into L2 for whichever warp claims it. The warp publishes its group's record
// bytes as soon as they are counted, builds the records in shared memory
// while its predecessors finish, and only then reads its offset from the
// decoupled look-back and stores the records (8-byte aligned) to M.
__global__ __launch_bounds__(kMap32Threads) void adm_u32_map_kernel(
    const uint32_t* __restrict__ in, uint64_t n, uint8_t* __restrict__ M, uint64_t m_cap,
    Ctrl* ctrl, unsigned long long* flags, int prob_bits) {
  kernel_begin();
  extern __shared__ __align__(16) uint8_t smem_raw[];
  Map32Smem& sm = *reinterpret_cast<Map32Smem*>(smem_raw);
  __shared__ uint32_t s_h[kMap32Warps][kAnsSyms];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  for (int i = t; i < kMap32Warps * kAnsSyms; i += kMap32Threads) (&s_h[0][0])[i] = 0;
  __syncthreads();
  const uint64_t g = div_up_u64(n, kAdmGroup);
  const Sink sink = sink_of(ctrl);
  const bool failed = sink_failed(sink);
  const uint32_t epoch = *((volatile uint32_t*)&ctrl->epoch);
  const uint32_t ahead = gridDim.x * kMap32Warps;
  while (!failed) {
    const uint32_t grp = warp_claim(&ctrl->tile_counter[0], lane);
    if (grp >= g) break;
    if (lane == 0 && (uint64_t)grp + ahead < g) {
      const uint64_t ns = ((uint64_t)grp + ahead) * kAdmGroup;
      prefetch_l2(in + ns, (uint32_t)(4 * min_u64(kAdmGroup, n - ns)));
    }
    map32_group(in, n, M, m_cap, flags, &ctrl->merged_size, grp, epoch, sink, s_h[warp],
                sm.stage[warp], lane);
  }
  hist_merge_and_normalize(s_h, kMap32Warps, ctrl, g == 0 ? 0ull : ~0ull, 0, prob_bits);
}

__global__ __launch_bounds__(kUnmap32Threads) void adm_u32_unmap_kernel(
    const uint8_t* __restrict__ M, uint64_t n, uint32_t* __restrict__ out, Ctrl* ctrl) {
  kernel_begin();
  extern __shared__ __align__(16) uint8_t smem_raw[];
  Unmap32Smem& sm = *reinterpret_cast<Unmap32Smem*>(smem_raw);
  const Sink sink = sink_of(ctrl);
  if (sink_failed(sink)) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint64_t g = div_up_u64(n, kAdmGroup);
  const uint64_t msize = __ldcg(&ctrl->merged_size);
  const uint64_t rec_base = 40 * g;
  if (msize < rec_base) {
    if (blockIdx.x == 0 && threadIdx.x == 0) report(sink, MANS_ERR_CORRUPT, msize);
    return;
  }
  const uint64_t warps = (uint64_t)gridDim.x * kUnmap32Warps;
  for (uint64_t grp = (uint64_t)blockIdx.x * kUnmap32Warps + warp; grp < g; grp += warps)
    unmap32_group(M, n, msize - rec_base, out, grp, sink, sm.stage[warp], lane);
}

// ------------------------------------------------------------------------
// The map of large inputs for an encoder that gathers: groups are taken in a
// fixed order and their records left in slots (map32_slot), then one small scan
// turns record bytes into offsets and tells the encoder, for every 4 KiB block
// of the mapped buffer, the group whose records the block starts with. The
// single-pass map above spends its time waiting: a group's look-back needs
// every earlier group's length (23% of it by itself), and making the groups
// cheaper does not shorten that chain. 1 GiB of detector frames: map 0.945 ->
// 0.626 ms (scan included, about 15 us), encode 0.642 -> 0.708 for the gathering.
// Data without groups of one-byte codes lose what those gain elsewhere (1 GiB of
// Laplace codes: 1.102 + 0.740 -> 1.138 + 0.816 ms); the host cannot tell.
// ------------------------------------------------------------------------
__global__ __launch_bounds__(kMap32Threads) void adm_u32_split_kernel(
    const uint32_t* __restrict__ in, uint64_t n, uint8_t* __restrict__ M,
    uint8_t* __restrict__ slots, Ctrl* ctrl) {
  kernel_begin();
  extern __shared__ __align__(16) uint8_t smem_raw[];
  Map32Smem& sm = *reinterpret_cast<Map32Smem*>(smem_raw);
  __shared__ uint32_t s_h[kMap32Warps][kAnsSyms];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  for (int i = t; i < kMap32Warps * kAnsSyms; i += kMap32Threads) (&s_h[0][0])[i] = 0;
  __syncthreads();
  const uint64_t g = div_up_u64(n, kAdmGroup), warps = (uint64_t)gridDim.x * kMap32Warps;
  for (uint64_t grp = (uint64_t)blockIdx.x * kMap32Warps + warp; grp < g; grp += warps) {
    if (lane == 0 && grp + warps < g) {
      const uint64_t ns = (grp + warps) * kAdmGroup;
      prefetch_l2(in + ns, (uint32_t)(4 * min_u64(kAdmGroup, n - ns)));
    }
    map32_slot(in, n, M, slots + grp * kGroupRecMax, grp, s_h[warp], sm.stage[warp], lane);
  }
  __syncthreads();
  uint32_t v = 0;
  for (int w = 0; w < kMap32Warps; ++w) v += s_h[w][t];
  if (v) atomicAdd(&ctrl->hist[t], v);
}

// Offsets of the groups' records (single-pass look-back over tiles of 2,048
// groups claimed in order), their bytes' histogram, the group at the start of
// each block, the merged size; the last CTA normalises.
constexpr int kScan32Per = 8, kScan32Tile = kMap32Threads * kScan32Per;

__global__ __launch_bounds__(kMap32Threads) void adm_u32_scan_kernel(
    uint8_t* __restrict__ M, uint64_t n, uint32_t* __restrict__ first_group, Ctrl* ctrl,
    unsigned long long* flags, int prob_bits) {
  kernel_begin();
  __shared__ uint32_t s_h[kMap32Warps][kAnsSyms];
  __shared__ uint32_t s_tile, s_warp[kMap32Warps], s_prefix;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  for (int i = t; i < kMap32Warps * kAnsSyms; i += kMap32Threads) (&s_h[0][0])[i] = 0;
  const uint64_t g = div_up_u64(n, kAdmGroup), rec_base = 40 * g;
  uint32_t* const off = reinterpret_cast<uint32_t*>(M);
  const Sink sink = sink_of(ctrl);
  const uint32_t epoch = *((volatile uint32_t*)&ctrl->epoch);
  while (true) {
    __syncthreads();
    if (t == 0) s_tile = atomicAdd(&ctrl->tile_counter[6], 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    const uint64_t base = (uint64_t)tile * kScan32Tile + (uint64_t)warp * 32 * kScan32Per;
    if ((uint64_t)tile * kScan32Tile >= g) break;
    // the warp's 256 groups in eight rows of 32
    uint32_t v[kScan32Per], incl[kScan32Per], sum = 0;
#pragma unroll
    for (int i = 0; i < kScan32Per; ++i) {
      const uint64_t k = base + 32 * i + lane;
      v[i] = k < g ? off[k] : 0u;
    }
#pragma unroll
    for (int i = 0; i < kScan32Per; ++i) {
      incl[i] = v[i];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl[i], o);
        if (lane >= o) incl[i] += y;
      }
      incl[i] += sum;
      sum = __shfl_sync(0xffffffffu, incl[i], 31);
    }
    if (lane == 0) s_warp[warp] = sum;
    __syncthreads();
    uint32_t wbase = 0, total = 0;
    for (int w = 0; w < kMap32Warps; ++w) {
      if (w < warp) wbase += s_warp[w];
      total += s_warp[w];
    }
    if (warp == 0) {
      if (lane == 0) st_flag(&flags[tile], make_flag(tile == 0 ? kFlagIncl : kFlagAgg, epoch, total));
      uint32_t pre = 0;
      if (tile > 0) {
        pre = lookback_exclusive(flags, tile, epoch, sink);
        if (lane == 0) st_flag(&flags[tile], make_flag(kFlagIncl, epoch, pre + total));
      }
      if (lane == 0) {
        s_prefix = pre;
        if (((uint64_t)tile + 1) * kScan32Tile >= g) ctrl->merged_size = rec_base + pre + total;
      }
    }
    __syncthreads();
    const uint32_t pre = s_prefix + wbase;
#pragma unroll
    for (int i = 0; i < kScan32Per; ++i) {
      const uint64_t k = base + 32 * i + lane;
      const uint32_t o = pre + incl[i] - v[i];
      if (k < g) {
        off[k] = o;
        // the block that begins inside the group's records, if any (4,096 bytes at most)
        const uint64_t a0 = rec_base + o, a1 = a0 + v[i];
        for (uint64_t b = div_up_u64(a0, kAnsBlock); b * kAnsBlock < a1; ++b) first_group[b] = (uint32_t)k;
        if (k == 0) first_group[rec_base / kAnsBlock] = 0;
      }
#pragma unroll
      for (int y = 0; y < 4; ++y) {
        const uint32_t byte = (o >> (8 * y)) & 0xffu;
        if (y >= 2 && base + 32 * i + 32 <= g &&
            __all_sync(0xffffffffu, byte == __shfl_sync(0xffffffffu, byte, 0))) {
          if (lane == 0) atomicAdd(&s_h[warp][byte], 32u);  // high bytes mostly agree
        } else if (k < g) {
          atomicAdd(&s_h[warp][byte], 1u);
        }
      }
    }
  }
  hist_merge_and_normalize(s_h, kMap32Warps, ctrl, ~0ull, 6, prob_bits);
}

// ------------------------------------------------------------------------
static int occupancy32(const void* fn, int threads, size_t smem) {
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, threads, smem) != cudaSuccess) {
    cudaGetLastError();
    n = 1;
  }
  return n > 0 ? n : 1;
}

// Called once per device (with the device current) by init_launch_cfg; the
// results live in the caller's LaunchCfg, so launches on several devices or
// from several host threads read no shared mutable state.
void init_adm_u32_launch_cfg(LaunchCfg& cfg) {
  cudaFuncSetAttribute(adm_u32_map_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)sizeof(Map32Smem));
  cudaFuncSetAttribute(adm_u32_unmap_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)sizeof(Unmap32Smem));
  cudaFuncSetAttribute(adm_u32_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)sizeof(Map32Smem));
  cfg.split32_ctas =
      occupancy32((const void*)adm_u32_split_kernel, kMap32Threads, sizeof(Map32Smem));
  cfg.map32_ctas = occupancy32((const void*)adm_u32_map_kernel, kMap32Threads, sizeof(Map32Smem));
  cfg.unmap32_ctas =
      occupancy32((const void*)adm_u32_unmap_kernel, kUnmap32Threads, sizeof(Unmap32Smem));
}

static unsigned grid_for(uint64_t want, uint64_t cap) {
  return (unsigned)(want < 1 ? 1 : (want < cap ? want : cap));
}

cudaError_t launch_adm_u32_map(const uint32_t* in, uint64_t n, uint8_t* m, uint64_t m_cap,
                               Ctrl* ctrl, unsigned long long* flags, int prob_bits,
                               const LaunchCfg& cfg, cudaStream_t s) {
  const int occ = cfg.map32_ctas > 0 ? cfg.map32_ctas : 1;
  const uint64_t ctas = div_up_u64(div_up_u64(n, kAdmGroup), kMap32Warps);
  return launch(adm_u32_map_kernel, grid_for(ctas, (uint64_t)cfg.sms * occ), kMap32Threads,
                sizeof(Map32Smem), s, in, n, m, m_cap, ctrl, flags, prob_bits);
}

uint64_t adm_u32_split_bytes(uint64_t n) {
  const uint64_t g = div_up_u64(n, kAdmGroup);
  return div_up_u64(40 * g, 16) * 16 + (uint64_t)kGroupRecMax * g;
}

cudaError_t launch_adm_u32_split(const uint32_t* in, uint64_t n, uint8_t* m, uint32_t* first_group,
                                 Ctrl* ctrl, unsigned long long* flags, int prob_bits,
                                 const LaunchCfg& cfg, cudaStream_t s, AnsGather* gather) {
  const uint64_t g = div_up_u64(n, kAdmGroup);
  gather->slots = m + div_up_u64(40 * g, 16) * 16;
  gather->first_group = first_group;
  gather->groups = g;
  cudaError_t e = launch(adm_u32_split_kernel,
                         grid_for(div_up_u64(g, kMap32Warps), (uint64_t)cfg.sms * cfg.split32_ctas),
                         kMap32Threads, sizeof(Map32Smem), s, in, n, m,
                         const_cast<uint8_t*>(gather->slots), ctrl);
  if (e != cudaSuccess) return e;
  return launch(adm_u32_scan_kernel, grid_for(div_up_u64(g, kScan32Tile), (uint64_t)cfg.sms * 4),
                kMap32Threads, 0, s, m, n, first_group, ctrl, flags, prob_bits);
}

cudaError_t launch_adm_u32_unmap(const uint8_t* m, uint64_t n, uint32_t* out, Ctrl* ctrl,
                                 const LaunchCfg& cfg, cudaStream_t s) {
  const int occ = cfg.unmap32_ctas > 0 ? cfg.unmap32_ctas : 1;
  const uint64_t groups = div_up_u64(n, kAdmGroup);
  return launch(adm_u32_unmap_kernel,
                grid_for(div_up_u64(groups, kUnmap32Warps), (uint64_t)cfg.sms * occ),
                kUnmap32Threads, sizeof(Unmap32Smem), s, m, n, out, ctrl);
}

}  // namespace mans
