// bd_kernels.cu -- the per-timestep kernels of the Brownian-dynamics step.
//
// A step of a reacting system is a chain of kernels with no host
// synchronisation, all counts on the device; their phases are the functions of
// bd_step.cuh, which bd_resident.cu runs in one kernel for small systems.
//
// Binned sort (the default), 5 launches, 6 with surface panels:
//   k_bin          streaming  diffuse + reflect + first-order reactions + cell
//                             key, each record into the next place of its
//                             cell's bin; births last (diffuse, uniReact,
//                             adjustPositions, calcHashD: particles_kernel.cu:
//                             61-95, 127-207, reaction_kernel.cuh:263-342;
//                             zeroReact + poisrandF on the host in the
//                             reference, reaction_cpu.cpp:36-63, stats.cpp:
//                             234-275)
//   k_bin_surface  streaming  the records whose move meets a panel
//   k_scan         one wave   exclusive scan of the cell counts = cell starts
//                             (replaces RadixSort's 5 passes + CUDPP scans,
//                             radixsort.cu:1045-1143, and the cellStart memset)
//   k_pairs_cells  streaming  canonical order inside each cell + pair search
//                             over the neighbour cells within the binding
//                             radius (reorderDataAndFindCellStartD, collideD,
//                             collideCell: particles_kernel.cu:212-272,
//                             318-497)
//   k_pairs_big    one wave   the same for cells of more than kBigCell records
//   k_match        32 CTAs    one reaction per particle (greedy matching in
//                             pair order), product placement, counters, commit
//                             (bimReact, resetNonInteracting:
//                             reaction_kernel.cuh:202-258,
//                             particles_kernel.cu:499-508)
// More births than kFewBirths a step are counted by k_zeroth before it.
//
// Compact sort (when the bins would not fit), 6 launches: k_count and
// k_scatter in place of k_bin; k_scatter recomputes k_count's records
// (counter-based RNG makes them identical) and puts each into its cell's range
// (compactPosAndTypeD, particles_kernel.cu:98-123).
//
// HBM traffic per particle-step: k_bin R16 + W16, k_pairs R16 + W16 = 64 B,
// plus 12 B per cell for the counts and the starts; compact 16 B more.
//
// Diffusion alone (no first- or second-order reaction, one instance):
// k_diffuse_steps takes many steps of each record in one launch; with
// zeroth-order births k_diffuse updates the records in place and k_append
// adds the births.
#include "bd_step.cuh"

#include <algorithm>

namespace bd {
namespace {

// ---------------------------------------------------------------- kernels

__global__ void __launch_bounds__(1024) k_zeroth(KParams p, int check_append) {
  __shared__ uint32_t s_total;
  DevCtrl* c = p.ctrl;
  const uint32_t nz = p.n_inst * p.Z;
  if (p.n_inst == 1 && nz <= 4u) {
    // One instance, at most four reactions: the entries come from the
    // kernel parameters and the status, step and flags are loaded
    // together, so the counts wait on one round of global loads (the
    // CDFs) instead of a chain of four.  Counting as below.
    __shared__ uint32_t s_part[32], s_cnt[4];
    const uint32_t status = ld_u32(&c->status), step = p.inst_step[0];
    const bool adv = advancing(p.inst_flags[0]);
    const uint32_t G = nz > 2u ? 256u : (nz > 1u ? 512u : 1024u);  // threads per entry
    const uint32_t g = threadIdx.x / G, t = threadIdx.x % G;
    uint32_t off, len, rxn;
    int32_t kmin;
    uint32_t le = 0;
    if (g < nz && adv) {
      zero0_entry(p, g, off, len, kmin, rxn);
      const U4 r = philox(U4{g, step, kTagZeroCount, 0u}, p.inst0.key_lo, p.inst0.key_hi);
      const double u = u53_to_unit(r.x, r.y);
      const double* cdf = p.cdf + off;
      for (uint32_t k = t; k < len; k += G) le += cdf[k] <= u ? 1u : 0u;
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) le += __shfl_xor_sync(kFull, le, d);
    if ((threadIdx.x & 31u) == 0) s_part[threadIdx.x >> 5] = le;
    __syncthreads();
    if (threadIdx.x < nz) {
      uint32_t cnt = 0;
      if (adv) {
        zero0_entry(p, threadIdx.x, off, len, kmin, rxn);
        uint32_t below = 0;
        for (uint32_t w = 0; w < G / 32u; ++w) below += s_part[threadIdx.x * (G / 32u) + w];
        cnt = (uint32_t)kmin + min(below, len - 1u);
        if (cnt && !status) atomicAdd(&p.pending[rxn], (unsigned long long)cnt);
      }
      s_cnt[threadIdx.x] = cnt;
    }
    __syncthreads();
    if (threadIdx.x == 0 && !status) {
      uint32_t carry = 0;
      for (uint32_t e = 0; e < nz; ++e) {
        p.zero_off[e] = carry;
        carry += s_cnt[e];
      }
      p.zero_off[nz] = carry;
      c->n_virtual = carry;
      if (check_append && (uint64_t)c->n_slots + carry > p.capacity) atomicOr(&c->status, kStatCapacity);
    }
    return;
  }
  if (ld_u32(&c->status)) return;
  if (nz <= 32u) {
    // Few entries (one instance, a few reactions): a group of at least 32
    // threads per entry counts the CDF values at or below u.  The CDF does
    // not decrease, so that count is the smallest k with CDF(k) > u, the
    // index the binary search below finds, and its loads are all in flight
    // at once instead of one dependent load per halving.
    __shared__ uint32_t s_part[32], s_cnt[32];
    uint32_t groups = 1;
    while (groups < nz) groups <<= 1;
    const uint32_t G = 1024u / groups;  // threads per entry, a multiple of 32
    const uint32_t g = threadIdx.x / G, t = threadIdx.x % G;
    uint32_t le = 0;
    if (g < nz) {
      const uint32_t inst = g / p.Z, zr = g % p.Z;
      const DevInstance& I = p.inst[inst];
      if (advancing(p.inst_flags[inst])) {
        const DevZero& Zr = p.zero[I.block * p.Z + zr];
        const U4 r = philox(U4{zr, p.inst_step[inst], kTagZeroCount, 0u}, I.key_lo, I.key_hi);
        const double u = u53_to_unit(r.x, r.y);
        const double* cdf = p.cdf + Zr.cdf_off;
        for (uint32_t k = t; k < Zr.cdf_len; k += G) le += cdf[k] <= u ? 1u : 0u;
      }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) le += __shfl_xor_sync(kFull, le, d);
    if ((threadIdx.x & 31u) == 0) s_part[threadIdx.x >> 5] = le;
    __syncthreads();
    if (threadIdx.x < nz) {
      const uint32_t e = threadIdx.x, inst = e / p.Z, zr = e % p.Z;
      const DevInstance& I = p.inst[inst];
      uint32_t cnt = 0;
      if (advancing(p.inst_flags[inst])) {
        const DevZero& Zr = p.zero[I.block * p.Z + zr];
        uint32_t below = 0;
        for (uint32_t w = 0; w < G / 32u; ++w) below += s_part[e * (G / 32u) + w];
        cnt = (uint32_t)Zr.kmin + min(below, Zr.cdf_len - 1u);
        if (cnt) atomicAdd(&p.pending[(size_t)inst * p.R + Zr.rxn], (unsigned long long)cnt);
      }
      s_cnt[e] = cnt;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t carry = 0;
      for (uint32_t e = 0; e < nz; ++e) {
        p.zero_off[e] = carry;
        carry += s_cnt[e];
      }
      p.zero_off[nz] = carry;
      c->n_virtual = carry;
      if (check_append && (uint64_t)c->n_slots + carry > p.capacity) atomicOr(&c->status, kStatCapacity);
    }
    return;
  }
  uint32_t carry = 0;
  for (uint32_t base = 0; base < nz; base += 1024) {
    const uint32_t e = base + threadIdx.x;
    uint32_t cnt = 0;
    if (e < nz) {
      const uint32_t inst = e / p.Z, zr = e % p.Z;
      const DevInstance& I = p.inst[inst];
      if (advancing(p.inst_flags[inst])) {
        const DevZero& Zr = p.zero[I.block * p.Z + zr];
        const U4 r = philox(U4{zr, p.inst_step[inst], kTagZeroCount, 0u}, I.key_lo, I.key_hi);
        const double u = u53_to_unit(r.x, r.y);
        // inversion: smallest k with CDF(k) > u
        const double* cdf = p.cdf + Zr.cdf_off;
        uint32_t lo = 0, hi = Zr.cdf_len - 1;
        while (lo < hi) {
          const uint32_t mid = (lo + hi) >> 1;
          if (cdf[mid] > u) hi = mid;
          else lo = mid + 1;
        }
        cnt = (uint32_t)Zr.kmin + lo;
        if (cnt) atomicAdd(&p.pending[(size_t)inst * p.R + Zr.rxn], (unsigned long long)cnt);
      }
    }
    uint32_t tot;
    const uint32_t ex = block_exclusive_scan<1024>(cnt, &s_total);
    tot = s_total;
    if (e < nz) p.zero_off[e] = carry + ex;
    carry += tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    p.zero_off[nz] = carry;
    c->n_virtual = carry;
    if (check_append && (uint64_t)c->n_slots + carry > p.capacity) atomicOr(&c->status, kStatCapacity);
  }
}

// kMinBlocks 4 / 6 cap registers at 64 / 40 (50% / 75% occupancy, the
// latter with a few spills); the launch shape picks the variant.
template <bool kTable, int kMinBlocks, bool kSingle, int kSurf = 0>
__global__ void __launch_bounds__(256, kMinBlocks) k_count(KParams p) {
  __shared__ DevSpecies s_species[kSingle ? kCtxSpecies : 1];
  __shared__ DevUni s_uni[kSingle ? kCtxUni : 1];
  SingleCtx ctx{};
  if (kSingle) ctx = single_ctx(p, s_species, s_uni);
  DevCtrl* c = p.ctrl;
  if (ctrl_status_warp(c)) return;
  const uint32_t cur = ld_u32(&c->cur);
  const float4* __restrict__ st = cur_state(p, cur);
  const uint32_t n_real = ld_u32(&c->n_slots), n_total = n_real + ld_u32(&c->n_virtual);
  stream_records<false>(st, n_real, n_total, [&](uint32_t i, const float4& rec) {
    Out2 o;
    o.n = 0;
    if (i < n_real) advance_rec<kTable, true, kSingle, kSurf>(p, ctx, rec, i, o);
    else if (i < n_total) advance_virtual<kSingle>(p, ctx, i - n_real, o);
    warp_count(p.cell_count, o.n > 0 ? o.key[0] : kNoKey);
    if (__any_sync(kFull, o.n > 1)) warp_count(p.cell_count, o.n > 1 ? o.key[1] : kNoKey);
  });
}

template <bool kTable, int kMinBlocks, bool kSingle, int kSurf = 0>
__global__ void __launch_bounds__(256, kMinBlocks) k_scatter(KParams p) {
  __shared__ DevSpecies s_species[kSingle ? kCtxSpecies : 1];
  __shared__ DevUni s_uni[kSingle ? kCtxUni : 1];
  SingleCtx ctx{};
  if (kSingle) ctx = single_ctx(p, s_species, s_uni);
  DevCtrl* c = p.ctrl;
  if (ctrl_status_warp(c)) return;
  const uint32_t cur = ld_u32(&c->cur);
  const float4* __restrict__ st = cur_state(p, cur);
  const uint32_t n_real = ld_u32(&c->n_slots), n_total = n_real + ld_u32(&c->n_virtual);
  stream_records<false>(st, n_real, n_total, [&](uint32_t i, const float4& rec) {
    Out2 o;
    o.n = 0;
    if (i < n_real) advance_rec<kTable, false, kSingle, kSurf>(p, ctx, rec, i, o);
    else if (i < n_total) advance_virtual<kSingle>(p, ctx, i - n_real, o);
    const int kmax = __any_sync(kFull, o.n > 1) ? 2 : 1;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (k >= kmax) break;  // warp-uniform
      const uint32_t key = o.n > k ? o.key[k] : kNoKey;
      const uint32_t off = warp_claim(p.cell_count, key);
      if (key != kNoKey) {
        const uint32_t slot = p.cell_start[key] + off;
        if (slot < p.capacity) p.scatter[slot] = o.r[k];
        else atomicOr(&c->status, kStatBounds);
      }
    }
  });
}

template <bool kSingle>
__device__ __noinline__ void bin_births(const KParams& p, DevCtrl* c, const SingleCtx& ctx, uint32_t n) {
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t v0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); v0 < n; v0 += stride) {  // whole warps
    const uint32_t v = v0 + lane_id();
    Out2 o;
    o.n = 0;
    if (v < n) advance_virtual<kSingle>(p, ctx, v, o);
    claim_retire(p, c, claim_issue(p.cell_count, o.n > 0 ? o.key[0] : kNoKey, o.r[0]));
    if (__any_sync(kFull, o.n > 1)) claim_retire(p, c, claim_issue(p.cell_count, o.n > 1 ? o.key[1] : kNoKey, o.r[1]));
  }
}

// Bound by its stores, 16 bytes each into sectors that stay partly empty (a
// bare kernel with the same copy, atomics and stores takes 188 us at 16M, 106
// when it only copies and counts); the issue slots are half busy.  16M c3 step:
// 227 us -> 202 by taking out of the record's path what rarely applies (the
// first-order loop behind a bound on the coin's word, one in-box test for the
// three axes, no lower cell bound, births) and what can be laid out (Philox
// round keys).  Advancing the few records that react in a call instead, to
// free registers for a fifth CTA per SM, was slower (219 us at four CTAs, 269
// at five: the call's conventions spill the loop).
// Births: those k_zeroth counted, dealt out over the grid; with
// births_in_bin the last CTA counts and bins them itself, after its records
// (no k_zeroth: one launch of 4 us less).
template <bool kTable, int kMinBlocks, bool kSingle, int kSurf = 0>
__global__ void __launch_bounds__(256, kMinBlocks) k_bin(const __grid_constant__ KParams p) {
  __shared__ DevSpecies s_species[kSingle ? kCtxSpecies : 1];
  __shared__ DevUni s_uni[kSingle ? kCtxUni : 1];
  __shared__ DeferBuffer s_defer[kSurf == 2 ? 8 : 1];  // one per warp (blocks of at most 256 threads)
  DeferBuffer& defer_buf = s_defer[kSurf == 2 ? threadIdx.x >> 5 : 0];
  // One answer for the whole CTA: records binned by the other CTAs may raise
  // a status bit at any time, and zeroth_births has barriers and a scan that
  // every warp takes part in.
  __shared__ uint32_t s_stop;
  DevCtrl* c = p.ctrl;
  if (threadIdx.x == 0) s_stop = ld_u32(&c->status);
  SingleCtx ctx{};
  if (kSingle) ctx = single_ctx(p, s_species, s_uni);
  else __syncthreads();
  if (s_stop) return;
  const uint32_t cur = ld_u32(&c->cur);
  const float4* __restrict__ st = cur_state(p, cur);
  const uint32_t n_real = ld_u32(&c->n_slots);
  bin_records<kTable, kSingle, kSurf, false>(p, c, ctx, defer_buf, st, n_real, p.cell_count);
  if (p.births_in_bin) {
    if (blockIdx.x == gridDim.x - 1u) zeroth_births<kSingle>(p, c, ctx, p.cell_count);
  } else if (p.Z) {
    bin_births<kSingle>(p, c, ctx, ld_u32(&c->n_virtual));
  }
}

// Binned path with surfaces, pass 1b: the records k_bin queued because
// their move meets a panel box, advanced with the surface walk (the same
// Philox counters, so the same step) and put into their bins.  A walk's
// cost varies with the panels near the record (one sphere against a mesh
// of many triangles), and the queue holds neighbouring records together,
// so warps take 32 queue entries at a time from a counter until the queue
// is empty: a warp of slow walks does not hold the others' share.  Bound by
// the latency of its load chains.  c3 in a cell, 2M / 16M particles: 84 / 102
// us before the finer panel grid and the panel heads in one load; then 39 /
// 66 us at four CTAs per SM (64 registers, 92 to 144 bytes of spills), 36 / 60
// at three (80 registers, 16 to 72 bytes), 36 / 65 at two.
template <bool kTable, bool kSingle>
__global__ void __launch_bounds__(256, 3) k_bin_surface(KParams p) {
  __shared__ DevSpecies s_species[kSingle ? kCtxSpecies : 1];
  __shared__ DevUni s_uni[kSingle ? kCtxUni : 1];
  SingleCtx ctx{};
  if (kSingle) ctx = single_ctx(p, s_species, s_uni);
  DevCtrl* c = p.ctrl;
  if (ctrl_status_warp(c)) return;
  const float4* __restrict__ st = cur_state(p, ld_u32(&c->cur));
  const uint32_t n = min(ld_u32(&c->n_surf), p.capacity);
  const uint32_t lane = lane_id();
  // first products keep k_bin's deferred claim (consumed one record later)
  PendingClaim pending;
  pending.key = kNoKey;
  pending.old = 0;
  pending.leader = 0;
  pending.rank = 0;
  for (;;) {  // warp-uniform trip count
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(&c->surf_ticket, 32u);
    base = __shfl_sync(kFull, base, 0);
    if (base >= n) break;
    const uint32_t e = base + lane;
    Out2 o;
    o.n = 0;
    if (e < n) {
      const uint32_t i = p.surf_queue[e];
      advance_rec<kTable, true, kSingle, 1>(p, ctx, st[i], i, o);
    }
    const PendingClaim next = claim_issue(p.cell_count, o.n > 0 ? o.key[0] : kNoKey, o.r[0]);
    if (__any_sync(kFull, o.n > 1)) claim_retire(p, c, claim_issue(p.cell_count, o.n > 1 ? o.key[1] : kNoKey, o.r[1]));
    claim_retire(p, c, pending);
    pending = next;
  }
  claim_retire(p, c, pending);
}

// Bulk global -> shared copies completed on an mbarrier (the copy engine
// moves the bytes; no thread issues a load per word).
__device__ __forceinline__ uint32_t smem_u32(const void* ptr) {
  return (uint32_t)__cvta_generic_to_shared(ptr);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// One thread: announce `bytes` and start the copy that will deliver them.
// The fence orders this thread's earlier generic-proxy accesses of the
// buffer (the warp's reads of its previous contents) before the copy.
__device__ __forceinline__ void bulk_to_smem(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// Wait for the phase with parity `parity` of `bar` to complete; false after
// 2^20 polls (each poll suspends the thread for at most a short
// hardware-defined time).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  for (uint32_t it = 0; it < (1u << 20); ++it) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Exclusive scan of the cell counts into cell_start, by a cooperative grid
// of two CTAs per SM (every CTA resident).  CTA b owns a contiguous range of
// cells and moves it through shared memory in chunks of up to kScanChunk
// counts, each brought in by one bulk copy (the copy engine, not a load
// per word): pass 1 sums the range, a contiguous run of counts per thread,
// and publishes the sum (tile_sums[b]); after one grid barrier, pass 2 adds
// the sums of the CTAs before it, scans each chunk in shared memory and
// writes it out by one bulk copy.  On the 16M c3 step a range is one chunk,
// so pass 2 finds it still in shared memory and its threads know where their
// runs start.  The last 1..3 counts of the grid that do not fill 16 bytes go
// by plain loads and stores.  What bounds it: its launch (6 us when it does
// nothing) and the chain status, copy, barrier, sums, store.  c3 steps of 2M,
// 4M, 14.5M and 16M particles: 9.9, 12.0, 17.9 and 18.0 us.  Runs of any
// length, which meet in one bank when it is a multiple of 16, with a second
// pass over the counts took 15.4, 19.8, 41.2 and 20.7 us.  At that time chunks
// of 49,152 counts (one CTA per SM) took 22.4 us, of 12,288 (four) 26.3 us at
// 16M.  Earlier forms: a
// single-pass scan by decoupled look-back, 27 us (643 tiles, and the
// frontier of known prefixes moved by the 32 flags one poll reads per round
// trip); this grid scan reading tiles of 8,192 counts with vector loads
// instead of staging them, 24.6 us.
constexpr uint32_t kScanChunk = 24576;  // counts per chunk: 96 KiB of shared memory
constexpr uint32_t kScanSmem = kScanChunk * 4u;  // dynamic shared memory of k_scan

__device__ __forceinline__ void bulk_to_global(void* dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_u32(src)),
               "r"(bytes)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

// Chunk [c0, c0 + len) of the counts into s_cnt: the 16-byte-aligned part
// by one bulk copy on `bar` (scan_fetch, thread 0), the rest by plain loads.
__device__ __forceinline__ void scan_fetch(const KParams& p, uint32_t* s_cnt, uint64_t* bar, uint32_t c0, uint32_t len) {
  const uint32_t bulk = len & ~3u;
  if (bulk && threadIdx.x == 0) bulk_to_smem(s_cnt, p.cell_count + c0, bulk * 4u, bar);
}

// The fetched chunk is there.  False when the copy's wait runs out.
__device__ __forceinline__ bool scan_landed(const KParams& p, uint32_t* s_cnt, uint64_t* bar, uint32_t c0, uint32_t len,
                                            uint32_t& phase) {
  const uint32_t bulk = len & ~3u;
  if (threadIdx.x < len - bulk) s_cnt[bulk + threadIdx.x] = __ldcg(&p.cell_count[c0 + bulk + threadIdx.x]);
  bool ok = true;
  if (bulk) {
    ok = mbar_wait(bar, phase);
    if (!ok) mbar_wait(bar, phase);  // give the copy in flight more time to land before the CTA leaves
    phase ^= 1u;
  }
  // one answer for the whole CTA, so that its threads leave or go on together
  return __syncthreads_and(ok) != 0;
}

__global__ void __launch_bounds__(1024) k_scan(KParams p) {
  extern __shared__ __align__(128) uint32_t s_cnt[];
  __shared__ __align__(8) uint64_t s_bar;
  __shared__ uint32_t s_stop, s_total, s_warp[32];
  DevCtrl* c = p.ctrl;
  // ranges of a multiple of 4 counts (16-byte aligned bulk copies)
  const uint32_t per = ((p.n_cells + gridDim.x - 1u) / gridDim.x + 3u) & ~3u;
  const uint32_t lo = min(blockIdx.x * per, p.n_cells), hi = min(lo + per, p.n_cells);
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  uint32_t phase = 0;
  if (threadIdx.x == 0) {
    const uint32_t status = ld_u32(&c->status);
    mbar_init(&s_bar);
    mbar_init_fence();
    // the first chunk is on its way while the status is
    if (lo < hi) scan_fetch(p, s_cnt, &s_bar, lo, min(kScanChunk, hi - lo));
    s_stop = status != 0u;
  }
  __syncthreads();
  // The status is the previous kernels' and the same for every CTA: all
  // return here together or none does, once the copy has landed.
  if (s_stop) {
    if (lo < hi) scan_landed(p, s_cnt, &s_bar, lo, min(kScanChunk, hi - lo), phase);
    return;
  }
  if (p.scan_withhold && blockIdx.x == 0) {  // test switch: CTA 0 never arrives
    if (lo < hi) scan_landed(p, s_cnt, &s_bar, lo, min(kScanChunk, hi - lo), phase);
    if (gridDim.x == 1 && threadIdx.x == 0) atomicOr(&c->status, kStatTimeout);
    return;
  }
  bool ok = true;
  // A thread's run of a chunk is of odd length, so that a warp's runs start
  // in different banks.
  auto run_of = [](uint32_t len) { return ((len + 1023u) >> 10) | 1u; };
  // pass 1: the range's sum, each thread over its run
  uint32_t sum = 0;
  for (uint32_t c0 = lo; c0 < hi && ok; c0 += kScanChunk) {
    const uint32_t len = min(kScanChunk, hi - c0), q = run_of(len);
    if (c0 != lo) {
      __syncthreads();  // the previous chunk is summed
      scan_fetch(p, s_cnt, &s_bar, c0, len);
    }
    ok = scan_landed(p, s_cnt, &s_bar, c0, len, phase);
    const uint32_t b0 = min(threadIdx.x * q, len), b1 = min(b0 + q, len);
    for (uint32_t i = b0; i < b1; ++i) sum += s_cnt[i];
  }
  if (!ok) {
    if (threadIdx.x == 0) atomicOr(&c->status, kStatTimeout);
    return;
  }
  // counts of the range before the thread's runs: its start in the chunk,
  // when the range is one chunk
  const uint32_t before = block_exclusive_scan<1024>(sum, &s_total);
  if (threadIdx.x == 0) p.tile_sums[blockIdx.x] = s_total;
  if (!grid_barrier(c)) return;
  // the counts before the range: all sums asked for at once, and every warp
  // adds up the warps' sums for itself
  uint32_t v = 0;
  for (uint32_t b = threadIdx.x; b < blockIdx.x; b += 1024u) v += __ldcg(&p.tile_sums[b]);
  v = __reduce_add_sync(kFull, v);
  if (lane == 0) s_warp[warp] = v;
  __syncthreads();
  uint32_t carry = __reduce_add_sync(kFull, s_warp[lane]);
  // pass 2: each chunk's starts in shared memory, a run of q counts per thread
  const bool resident = hi - lo <= kScanChunk;  // the one chunk is still staged
  for (uint32_t c0 = lo; c0 < hi; c0 += kScanChunk) {
    const uint32_t len = min(kScanChunk, hi - c0);
    if (!resident) {
      __syncthreads();
      if (threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // last chunk's store has read its source
      __syncthreads();
      scan_fetch(p, s_cnt, &s_bar, c0, len);
      if (!scan_landed(p, s_cnt, &s_bar, c0, len, phase)) {
        if (threadIdx.x == 0) atomicOr(&c->status, kStatTimeout);
        break;
      }
    }
    const uint32_t q = run_of(len);
    const uint32_t b0 = min(threadIdx.x * q, len), b1 = min(b0 + q, len);
    uint32_t run = carry + before, total = s_total;
    if (!resident) {
      uint32_t s = 0;
      for (uint32_t i = b0; i < b1; ++i) s += s_cnt[i];
      run = carry + block_exclusive_scan<1024>(s, &s_total);
      total = s_total;
    }
    carry += total;
    for (uint32_t i = b0; i < b1; ++i) {
      const uint32_t x = s_cnt[i];
      s_cnt[i] = run;
      run += x;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the writes above, seen by the bulk copy
    __syncthreads();
    const uint32_t bulk = len & ~3u;
    if (threadIdx.x == 0 && bulk) bulk_to_global(p.cell_start + c0, s_cnt, bulk * 4u);
    if (threadIdx.x < len - bulk) p.cell_start[c0 + bulk + threadIdx.x] = s_cnt[bulk + threadIdx.x];
  }
  if (threadIdx.x == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  if (blockIdx.x == gridDim.x - 1u && threadIdx.x == 0) {  // every count lies at or before its range's end
    p.cell_start[p.n_cells] = carry;
    c->n_sorted = carry;
    if (carry > p.capacity) atomicOr(&c->status, kStatCapacity);
  }
}

template <bool kHasBim, bool kBinned, bool kSingle>
__global__ void __launch_bounds__(256, 4) k_pairs_cells(KParams p) {
  __shared__ PairShared<kHasBim, 8> s_pair;
  __shared__ PairSpecies<kSingle> s_species;
  pair_species<kSingle>(p, s_species);  // before any warp may leave
  const bool adv0 = kSingle ? advancing(ld_u32(&p.inst_flags[0])) : true;
  DevCtrl* c = p.ctrl;
  if (ctrl_status_warp(c)) return;
  pair_cells<kHasBim, kBinned, kSingle, false, 8>(p, c, next_state(p, ld_u32(&c->cur)), adv0, s_pair, s_species,
                                                  p.cell_start, p.cell_count);
}

// Large cells: part 1 (sort) by every CTA, a grid barrier, part 2 (pairs)
// by every CTA, in one launch, cooperative whether there are pairs to find
// or not (the merge passes of the sort have barriers too), so that a
// barrier waits only on resident CTAs.  Every CTA reads the
// same final count of queued cells, so when none is large they all leave
// at once: one empty launch per step instead of two (the two empty
// launches cost 3.3 us per 16M c3 step; the one measured within noise of
// them).  The first step that queues a cell without big_scratch in place
// raises kStatScratch; the host allocates it and replays the step.
// 64 registers: at the 114 the compiler asks for, the two CTAs per SM hold
// nearly every register, so that the launch, which needs all of them resident
// at once, waits for the other handles' kernels to drain (8 handles of 40,000
// particles, us a step of each: 70 with 114 registers, 50 with 64, 57 before
// the units; 16 handles 142 / 99 / 113).  Its own time rises by 1 to 5%.
template <bool kHasBim, bool kBinned>
__global__ void __launch_bounds__(256, 4) k_pairs_big(KParams p) {
  __shared__ unsigned long long s_key[kBigChunk];
  DevCtrl* c = p.ctrl;
  if (stop_block(c)) return;
  const unsigned long long queued = __ldcg(&c->big_queue);
  const uint32_t nbig = min((uint32_t)queued, p.big_cap), units = (uint32_t)(queued >> 32);
  if (nbig == 0) return;
  if (p.big_scratch_cap < 2ull * p.capacity) {
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&c->status, kStatScratch);
    return;
  }
  if (!big_sort<kBinned>(p, c, nbig, units, s_key)) return;
  if (!kHasBim) return;
  if (!grid_barrier(c)) return;
  big_pairs<kBinned, 256>(p, c, nbig, units);
}

template <bool kSurf>
__global__ void __launch_bounds__(1024) k_match(KParams p) {
  __shared__ MatchShared s_match;
  DevCtrl* c = p.ctrl;
  // loaded together (in a failed step the pairs mean nothing)
  const uint32_t status = ld_u32(&c->status), K = ld_u32(&c->n_pairs);
  const DevPair mine = match_pair(p);
  if (status) return;
  if (K > p.pair_cap) {
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&c->status, kStatPairs);
    return;
  }
  const bool grid = gridDim.x > 1 && K > kMatchOneCta;  // the same in every CTA
  if (!grid && blockIdx.x != 0) return;
  match_commit<kSurf>(p, c, K, mine, grid, s_match);
}

// Nothing in a diffusion-only step depends on another record, so a record
// takes all its steps in registers: one read and one write whatever their
// number, one launch, and no k_finalize_inplace (the last CTA to finish
// commits).  Bound by the issue of Philox and Box-Muller, 3.7 us a step of 1M
// records (4.3 before the rows of philox_row, two steps unrolled, one in-box
// test and the subnormal cases left out of the normals), beside a memory floor
// of 5 us in all: 16 steps took 224 us as 32 launches, 80 with those, 76 now.
// Same operations in the same order as advance_rec, so the same bits.
// Without zeroth-order reactions; with them the slot count changes every
// step.
constexpr uint32_t kDiffuseCtas = 8;  // per SM

template <bool kTable>
__global__ void __launch_bounds__(256, (int)kDiffuseCtas) k_diffuse_steps(const __grid_constant__ KParams p, uint32_t nsteps) {
  DevCtrl* c = p.ctrl;
  if (ctrl_status_warp(c)) return;
  const uint32_t n = ld_u32(&c->n_slots), cur = ld_u32(&c->cur);
  const uint32_t flags = ld_u32(&p.inst_flags[0]), step0 = ld_u32(&p.inst_step[0]), base = ld_u32(&p.inst_slot_base[0]);
  const uint32_t target = ld_u32(&p.inst_target[0]);
  // the instance freezes at its target, and takes a step if it has not yet
  const uint32_t take = advancing(flags) ? min(nsteps, max(target, step0 + 1u) - step0) : 0u;
  float4* st = cur ? p.state[1] : p.state[0];
  const DevInstance& I = p.inst0;
  // 32 records at a time, dealt to the CTAs in turn: what is left for a last
  // round is spread over the SMs
  const uint32_t first = ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32u + lane_id();
  for (uint64_t at = first; at < n; at += gridDim.x * blockDim.x) {
    const uint32_t i = (uint32_t)at;
    float4 r = st[i];
    const uint32_t w = rec_w(r);
    if (w == kDead || take == 0) continue;
    const float sigma = __ldg(&p.species[I.block * p.S + (w & kSpeciesMask)].sigma);
    const PhiloxRow row = philox_row(i - base, kTagDiffuse, p.keys0);
#pragma unroll 2
    for (uint32_t k = 0; k < take; ++k) {
      const U4 rn = philox_of_row(row, step0 + k, kTagDiffuse, p.keys0);
      float g0, g1, g2;
      normals3<kTable>(rn, p.gauss, g0, g1, g2);
      r.x = __fmaf_rn(sigma, g0, r.x);
      r.y = __fmaf_rn(sigma, g1, r.y);
      r.z = __fmaf_rn(sigma, g2, r.z);
      // one branch for the three axes
      if (!(r.x >= I.lo[0] && r.x <= I.hi[0] && r.y >= I.lo[1] && r.y <= I.hi[1] && r.z >= I.lo[2] &&
            r.z <= I.hi[2])) {
        r.x = reflect(r.x, I.lo[0], I.hi[0]);
        r.y = reflect(r.y, I.lo[1], I.hi[1]);
        r.z = reflect(r.z, I.lo[2], I.hi[2]);
      }
    }
    st[i] = r;
  }
  // every CTA has read the control words before the last one commits
  __syncthreads();
  if (threadIdx.x != 0) return;
  __threadfence();
  if (atomicAdd(&c->bar_count, 1u) != gridDim.x - 1u) return;
  c->bar_count = 0u;
  if (take) {
    p.inst_step[0] = step0 + take;
    if (step0 + take >= target) {
      p.inst_flags[0] = flags | kInstFrozen;
      p.inst_frozen[0] = (uint32_t)c->step + take - 1u;
    }
  }
  c->n_virtual = 0;
  c->n_pairs_last = 0;
  c->deaths_last = 0;
  c->step += nsteps;
  c->steps_done += nsteps;
}

template <bool kTable>
__global__ void __launch_bounds__(256) k_diffuse(KParams p) {
  const DevCtrl* c = p.ctrl;
  if (ctrl_status_warp(c)) return;
  const uint32_t cur = ld_u32(&c->cur);
  float4* st = cur ? p.state[1] : p.state[0];
  const uint32_t n = ld_u32(&c->n_slots);
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    Out2 o;
    advance_rec<kTable, false, false>(p, SingleCtx{}, st[i], i, o);
    if (o.n > 0) st[i] = o.r[0];
  }
}

__global__ void __launch_bounds__(256) k_append(KParams p) {
  const DevCtrl* c = p.ctrl;
  if (ctrl_status_warp(c)) return;
  const uint32_t cur = ld_u32(&c->cur);
  float4* st = cur ? p.state[1] : p.state[0];
  const uint32_t n = ld_u32(&c->n_slots), nv = ld_u32(&c->n_virtual);
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += stride) {
    Out2 o;
    advance_virtual<false>(p, SingleCtx{}, v, o);
    st[n + v] = make_float4(o.r[0].x, o.r[0].y, o.r[0].z, __uint_as_float(rec_w(o.r[0]) & ~kNewborn));
  }
}

__global__ void k_finalize_inplace(KParams p) {
  DevCtrl* c = p.ctrl;
  if (ld_u32(&c->status)) return;
  const uint32_t step_now = (uint32_t)*(volatile uint64_t*)&c->step;
  commit_events(p);
  for (uint32_t inst = threadIdx.x; inst < p.n_inst; inst += blockDim.x) advance_instance_step(p, inst, step_now);
  __syncthreads();  // every thread has read the step before thread 0 advances it
  if (threadIdx.x == 0) {
    c->n_slots += c->n_virtual;
    c->n_virtual = 0;
    c->n_pairs_last = 0;
    c->deaths_last = 0;
    c->step += 1;
    c->steps_done += 1;
  }
}

__global__ void __launch_bounds__(256) k_instance_counts(KParams p, unsigned long long* counts) {
  const DevCtrl* c = p.ctrl;
  const uint32_t cur = ld_u32(&c->cur);
  const float4* st = cur_state(p, cur);
  const uint32_t n = ld_u32(&c->n_slots);
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += stride) {
    const uint32_t i = base + threadIdx.x;
    uint32_t key = kNoKey;
    if (i < n) {
      const uint32_t w = rec_w(st[i]);
      if (w != kDead) key = w >> 16;
    }
    const uint32_t peers = __match_any_sync(kFull, key);
    if (key != kNoKey && lane_id() == (uint32_t)(__ffs(peers) - 1))
      atomicAdd(&counts[key], (unsigned long long)__popc(peers));
  }
}

__global__ void __launch_bounds__(256) k_species_counts(KParams p, unsigned long long* counts) {
  const DevCtrl* c = p.ctrl;
  const uint32_t cur = ld_u32(&c->cur);
  const float4* st = cur_state(p, cur);
  const uint32_t n = ld_u32(&c->n_slots);
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += stride) {
    const uint32_t i = base + threadIdx.x;
    uint32_t key = kNoKey;
    if (i < n) {
      const uint32_t w = rec_w(st[i]);
      if (w != kDead) key = (w >> 16) * p.S + (w & kSpeciesMask);
    }
    const uint32_t peers = __match_any_sync(kFull, key);
    if (key != kNoKey && lane_id() == (uint32_t)(__ffs(peers) - 1))
      atomicAdd(&counts[key], (unsigned long long)__popc(peers));
  }
}

// Squared diffusion moves of the coming step, summed per (instance,
// species): the step's own Philox counters, normals and wall reflections
// (advance_rec, before its reactions), read only.  An observable
// (bd_measure_msd), launched before a step, not part of it.  Sums go
// through shared memory when the (instance, species) table fits.
constexpr uint32_t kMsdShared = 512;

template <bool kTable>
__global__ void __launch_bounds__(256) k_msd(KParams p, double* sum, unsigned long long* cnt) {
  __shared__ double s_sum[kMsdShared];
  __shared__ unsigned long long s_cnt[kMsdShared];
  const DevCtrl* c = p.ctrl;
  if (ld_u32(&c->status)) return;  // the step will not run: nothing to measure
  const uint32_t keys = p.n_inst * p.S;
  const bool in_smem = keys <= kMsdShared;
  if (in_smem)
    for (uint32_t k = threadIdx.x; k < keys; k += blockDim.x) {
      s_sum[k] = 0.0;
      s_cnt[k] = 0ull;
    }
  __syncthreads();
  const uint32_t cur = ld_u32(&c->cur);
  const float4* st = cur_state(p, cur);
  const uint32_t n = ld_u32(&c->n_slots);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float4 rec = st[i];
    const uint32_t w = rec_w(rec);
    if (w == kDead) continue;
    const uint32_t inst = w >> 16, sp = w & kSpeciesMask;
    if (!advancing(p.inst_flags[inst])) continue;
    const DevInstance& I = p.inst[inst];
    const uint32_t local = i - p.inst_slot_base[inst];
    const float sigma = p.species[I.block * p.S + sp].sigma;
    const U4 rn = philox(U4{local, p.inst_step[inst], kTagDiffuse, 0u}, I.key_lo, I.key_hi);
    float g0, g1, g2;
    normals3<kTable>(rn, p.gauss, g0, g1, g2);
    const double dx = (double)reflect(__fmaf_rn(sigma, g0, rec.x), I.lo[0], I.hi[0]) - rec.x;
    const double dy = (double)reflect(__fmaf_rn(sigma, g1, rec.y), I.lo[1], I.hi[1]) - rec.y;
    const double dz = (double)reflect(__fmaf_rn(sigma, g2, rec.z), I.lo[2], I.hi[2]) - rec.z;
    const double d2 = dx * dx + dy * dy + dz * dz;
    const uint32_t key = inst * p.S + sp;
    if (in_smem) {
      atomicAdd(&s_sum[key], d2);
      atomicAdd(&s_cnt[key], 1ull);
    } else {
      atomicAdd(&sum[key], d2);
      atomicAdd(&cnt[key], 1ull);
    }
  }
  __syncthreads();
  if (in_smem)
    for (uint32_t k = threadIdx.x; k < keys; k += blockDim.x)
      if (s_cnt[k]) {
        atomicAdd(&sum[k], s_sum[k]);
        atomicAdd(&cnt[k], s_cnt[k]);
      }
}

}  // namespace

// The matcher, cooperatively over shape.grid_match CTAs (all resident, so
// its grid barriers cannot wait on a CTA that never runs).
void launch_match(const KParams& p, const LaunchShape& shape, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(shape.grid_match > 1 ? shape.grid_match : 1));
  cfg.blockDim = dim3(1024);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeCooperative;
  attr.val.cooperative = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = shape.grid_match > 1 ? 1 : 0;
  if (p.n_panels) cudaLaunchKernelEx(&cfg, k_match<true>, p);
  else cudaLaunchKernelEx(&cfg, k_match<false>, p);
}

// The large-cell kernel over shape.grid_big CTAs, cooperatively (its grid
// barriers wait only on resident CTAs).
void launch_big(const KParams& p, bool has_bim, bool binned, const LaunchShape& shape, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)std::max(shape.grid_big, 1));
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeCooperative;
  attr.val.cooperative = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = shape.grid_big > 1 ? 1 : 0;
  if (has_bim) {
    if (binned) cudaLaunchKernelEx(&cfg, k_pairs_big<true, true>, p);
    else cudaLaunchKernelEx(&cfg, k_pairs_big<true, false>, p);
  } else {
    if (binned) cudaLaunchKernelEx(&cfg, k_pairs_big<false, true>, p);
    else cudaLaunchKernelEx(&cfg, k_pairs_big<false, false>, p);
  }
}

// The cell scan, cooperatively over at most shape.grid_scan CTAs (all
// resident) and at most one per kScanTile cells.
void launch_scan(const KParams& p, const LaunchShape& shape, cudaStream_t s) {
  const uint32_t g = std::max(1u, std::min((uint32_t)std::max(shape.grid_scan, 1), p.n_tiles));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(g);
  cfg.blockDim = dim3(1024);
  cfg.dynamicSmemBytes = kScanSmem;
  cfg.stream = s;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeCooperative;
  attr.val.cooperative = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = g > 1 ? 1 : 0;
  cudaLaunchKernelEx(&cfg, k_scan, p);
}

void enqueue_diffuse(const KParams& p, bool table, uint32_t nsteps, uint64_t n_slots, cudaStream_t s) {
  // Few steps: one wave, since a CTA's reads of the control words, its fence
  // and its count take longer than a record's step.  Many: a CTA per 256
  // records, since the last round of a wave runs half empty.  One wave and a
  // CTA per 256 records, us: 1M records 1 step 17 / 51, 8 steps 43 / 59, 16
  // steps 75 / 77, 25 steps 111 / 107; 4M 34 / 182, 140 / 204, 262 / 271,
  // 406 / 384.  With little work in all the wave itself has fewer CTAs, since
  // they count themselves on one word: 300,000 records, 1 step, three / eight
  // per SM 10.4 / 16.7 (12.6 as k_diffuse and k_finalize_inplace), 1M 1 step
  // 14.9 / 17.6, 4 steps 27.6 / 28.2; 4M, 4 steps 83 / 78.
  const uint64_t ctas = std::max<uint64_t>((n_slots + 255u) / 256u, 1u);
  const unsigned wave = 152u * (n_slots * nsteps <= 4000000u ? 3u : kDiffuseCtas);
  const unsigned grid = (unsigned)std::min<uint64_t>(ctas, nsteps < 20u ? wave : 1u << 20);
  if (table) k_diffuse_steps<true><<<grid, 256, 0, s>>>(p, nsteps);
  else k_diffuse_steps<false><<<grid, 256, 0, s>>>(p, nsteps);
}

int enqueue_step(const KParams& p, Path path, bool table, bool has_zero, bool has_uni, bool has_bim,
                 const LaunchShape& shape, cudaStream_t s, StageHook hook, void* ctx) {
  (void)has_uni;
  const int gs = shape.grid_stream, bs = shape.block_stream;
  int n = 0;
  auto done = [&](const char* name) {
    ++n;
    if (hook) hook(ctx, name);
  };
  if (has_zero && !(path == Path::kBinned && p.births_in_bin)) {
    k_zeroth<<<1, 1024, 0, s>>>(p, path == Path::kDiffuseOnly ? 1 : 0);
    done("k_zeroth");
  }
  if (path == Path::kDiffuseOnly) {
    if (!has_zero) {
      enqueue_diffuse(p, table, 1, p.capacity, s);
      done("k_diffuse_steps");
      return n;
    }
    if (table) k_diffuse<true><<<gs, bs, 0, s>>>(p);
    else k_diffuse<false><<<gs, bs, 0, s>>>(p);
    done("k_diffuse");
    if (has_zero) {
      k_append<<<gs, bs, 0, s>>>(p);
      done("k_append");
    }
    k_finalize_inplace<<<1, 256, 0, s>>>(p);
    done("k_finalize_inplace");
    return n;
  }
  // Register-capped variants of the streaming kernels, picked by the launch
  // shape's resident CTAs per SM: 1 = no cap, 4 = 64 registers, 6 = 40.
#define BD_STREAM_LAUNCH3(KERNEL, MINB, SURF)                                              \
  do {                                                                                     \
    if (single) {                                                                          \
      if (table) KERNEL<true, MINB, true, SURF><<<gs, bs, 0, s>>>(p);                       \
      else KERNEL<false, MINB, true, SURF><<<gs, bs, 0, s>>>(p);                            \
    } else {                                                                               \
      if (table) KERNEL<true, MINB, false, SURF><<<gs, bs, 0, s>>>(p);                      \
      else KERNEL<false, MINB, false, SURF><<<gs, bs, 0, s>>>(p);                           \
    }                                                                                      \
  } while (0)
  // With surfaces: one variant per kernel, no register cap.
#define BD_STREAM_LAUNCH(KERNEL, SURF)                   \
  do {                                                   \
    switch (shape.min_blocks) {                          \
      case 6: BD_STREAM_LAUNCH3(KERNEL, 6, SURF); break; \
      case 4: BD_STREAM_LAUNCH3(KERNEL, 4, SURF); break; \
      default: BD_STREAM_LAUNCH3(KERNEL, 1, SURF);       \
    }                                                    \
  } while (0)
  // The compact path walks the surfaces inline: one variant per kernel, no
  // register cap.
#define BD_STREAM_LAUNCH_COMPACT(KERNEL)          \
  do {                                            \
    if (p.n_panels) BD_STREAM_LAUNCH3(KERNEL, 1, 1); \
    else BD_STREAM_LAUNCH(KERNEL, 0);             \
  } while (0)
#define BD_PAIRS_LAUNCH(BINNED)                                                                      \
  do {                                                                                               \
    if (single) {                                                                                    \
      if (has_bim) k_pairs_cells<true, BINNED, true><<<shape.grid_pairs, 256, 0, s>>>(p);  \
      else k_pairs_cells<false, BINNED, true><<<shape.grid_pairs, 256, 0, s>>>(p);         \
    } else {                                                                                         \
      if (has_bim) k_pairs_cells<true, BINNED, false><<<shape.grid_pairs, 256, 0, s>>>(p); \
      else k_pairs_cells<false, BINNED, false><<<shape.grid_pairs, 256, 0, s>>>(p);        \
    }                                                                                                \
  } while (0)
  const bool single = p.n_inst == 1 && p.S <= kCtxSpecies && p.U <= kCtxUni;
  if (path == Path::kBinned) {
    if (p.n_panels) {
      BD_STREAM_LAUNCH(k_bin, 2);
      done("k_bin");
      if (single) {
        if (table) k_bin_surface<true, true><<<gs, bs, 0, s>>>(p);
        else k_bin_surface<false, true><<<gs, bs, 0, s>>>(p);
      } else {
        if (table) k_bin_surface<true, false><<<gs, bs, 0, s>>>(p);
        else k_bin_surface<false, false><<<gs, bs, 0, s>>>(p);
      }
      done("k_bin_surface");
    } else {
      BD_STREAM_LAUNCH(k_bin, 0);
      done("k_bin");
    }
    launch_scan(p, shape, s);
    done("k_scan");
    BD_PAIRS_LAUNCH(true);
    done("k_pairs_cells");
    launch_big(p, has_bim, true, shape, s);
    done("k_pairs_big");
    launch_match(p, shape, s);
    done("k_match");
    return n;
  }
  BD_STREAM_LAUNCH_COMPACT(k_count);
  done("k_count");
  launch_scan(p, shape, s);
  done("k_scan");
  BD_STREAM_LAUNCH_COMPACT(k_scatter);
  done("k_scatter");
  BD_PAIRS_LAUNCH(false);
  done("k_pairs_cells");
#undef BD_STREAM_LAUNCH
#undef BD_STREAM_LAUNCH_COMPACT
#undef BD_STREAM_LAUNCH3
#undef BD_PAIRS_LAUNCH
  launch_big(p, has_bim, false, shape, s);
  done("k_pairs_big");
  launch_match(p, shape, s);
  done("k_match");
  return n;
}

void enqueue_instance_counts(const KParams& p, unsigned long long* counts, cudaStream_t s) {
  k_instance_counts<<<152 * 4, 256, 0, s>>>(p, counts);
}

// At most kMatchGrid CTAs: on the dense smoke step (24,509 candidates, 119
// rounds) 32 CTAs took 0.985 ms against 1.06 ms for 152 (one per SM) and
// 1.07 ms for 16, and a grid launch costs the small-K steps of c3 about
// 2 us over a single CTA (14.3 against 12.3 us) with 16 to 64 CTAs, 4 us
// with 152.
constexpr int kMatchGrid = 32;

int match_grid(int n_sm) {
  int a = 0, b = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_match<false>, 1024, 0) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_match<true>, 1024, 0) != cudaSuccess)
    return 1;
  const int per_sm = a < b ? a : b;
  const int resident = per_sm > 0 ? per_sm * n_sm : 1;
  return resident < kMatchGrid ? resident : kMatchGrid;
}

int big_grid(int n_sm) {
  int a[4] = {0, 0, 0, 0};
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a[0], k_pairs_big<true, true>, 256, 0) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a[1], k_pairs_big<true, false>, 256, 0) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a[2], k_pairs_big<false, true>, 256, 0) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a[3], k_pairs_big<false, false>, 256, 0) != cudaSuccess)
    return 1;
  const int resident = *std::min_element(a, a + 4) * n_sm;
  return resident < 1 ? 1 : (resident < kBigGrid ? resident : kBigGrid);
}

int scan_grid(int n_sm) {
  int a = 0;
  if (cudaFuncSetAttribute(k_scan, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kScanSmem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_scan, 1024, kScanSmem) != cudaSuccess || a < 1)
    return 0;
  return a * n_sm;
}

void enqueue_species_counts(const KParams& p, unsigned long long* counts, cudaStream_t s) {
  k_species_counts<<<152 * 4, 256, 0, s>>>(p, counts);
}

void enqueue_msd(const KParams& p, bool table, double* sum, unsigned long long* counts, cudaStream_t s) {
  if (table) k_msd<true><<<152 * 4, 256, 0, s>>>(p, sum, counts);
  else k_msd<false><<<152 * 4, 256, 0, s>>>(p, sum, counts);
}

}  // namespace bd
