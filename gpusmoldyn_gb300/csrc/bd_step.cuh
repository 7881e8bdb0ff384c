// bd_step.cuh -- the phases of one timestep as device functions: advance and
// bin, order and search pairs, large cells, match and commit.  bd_kernels.cu
// launches them as one kernel each; bd_resident.cu runs them in one
// persistent kernel for small systems.
#pragma once
#include "bd_device.cuh"
#include "bd_kernels.h"
#include "bd_surface.cuh"

namespace bd {
namespace {

constexpr uint32_t kNoKey = 0xFFFFFFFFu;
constexpr unsigned long long kFree64 = ~0ull;  // matcher word of a record not in a pending pair
constexpr unsigned kFull = 0xFFFFFFFFu;

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }

__device__ __forceinline__ uint32_t ld_u32(const uint32_t* p) { return __ldcg(p); }

// Data that a step kernel only reads and an earlier kernel wrote: through
// the read-only path, unless the including file runs several phases in one
// launch (BD_PHASES_IN_ONE_LAUNCH), where a phase reads what an earlier
// phase of the same launch wrote.
template <class T>
__device__ __forceinline__ T ld_step(const T* q) {
#ifdef BD_PHASES_IN_ONE_LAUNCH
  return *q;
#else
  return __ldg(q);
#endif
}

// What a CTA met in a phase, for the barrier that ends it (one launch for
// all phases); nothing when every phase is a kernel.
enum PhaseFlag : uint32_t { kFlagStop = 0, kFlagPairs = 1, kFlagBig = 2, kFlagGrid = 3, kPhaseFlags = 4 };
#ifdef BD_PHASES_IN_ONE_LAUNCH
__device__ __forceinline__ uint32_t* phase_flags() {
  __shared__ uint32_t s_flags[kPhaseFlags];
  return s_flags;
}
__device__ __forceinline__ void flag_phase(PhaseFlag f) { *(volatile uint32_t*)(phase_flags() + f) = 1u; }
#else
__device__ __forceinline__ void flag_phase(PhaseFlag) {}
#endif

// Set status bits: the step stops and does not commit.
__device__ __forceinline__ void raise(DevCtrl* c, uint32_t bits) {
  atomicOr(&c->status, bits);
  flag_phase(kFlagStop);
}

// ctrl words are written by earlier kernels and read here through L2.
__device__ __forceinline__ uint32_t ctrl_status_warp(const DevCtrl* c) {
  uint32_t s = 0;
  if (lane_id() == 0) s = ld_u32(&c->status);
  return __shfl_sync(kFull, s, 0);
}

// Grid-stride loop over the records [0, n_total) of the step: body(i, rec)
// with rec the current record for i < n_real (indices from n_real on are the
// step's zeroth-order births).  The next iteration's record is loaded before
// the body runs, so each thread keeps two 16-byte loads in flight.  Every
// thread of a warp makes the same number of calls (warp collectives allowed).
// kSpread deals the records to the CTAs 32 at a time, so that a system with
// fewer records than threads keeps every SM busy; else a CTA takes blockDim
// records in a row.
template <bool kSpread, class Body>
__device__ __forceinline__ void stream_records(const float4* __restrict__ st, uint32_t n_real, uint32_t n_total,
                                               Body&& body) {
  const uint32_t stride = gridDim.x * blockDim.x;
  uint32_t base = kSpread ? ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32u : blockIdx.x * blockDim.x;
  const uint32_t own = kSpread ? lane_id() : threadIdx.x;
  const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  float4 next = base + own < n_real ? __ldcs(&st[base + own]) : none;
  for (; base < n_total; base += stride) {
    const uint32_t i = base + own;
    const float4 rec = next;
    const uint32_t ahead = i + stride;
    next = ahead < n_real && ahead > i ? __ldcs(&st[ahead]) : none;
    // and the record after that towards L2
    const uint32_t far = ahead + stride;
    if (far < n_real && far > ahead) asm volatile("prefetch.global.L2 [%0];" ::"l"(st + far));
    body(i, rec);
  }
}

__device__ __forceinline__ const float4* cur_state(const KParams& p, uint32_t cur) {
  return cur ? p.state[1] : p.state[0];
}
__device__ __forceinline__ float4* next_state(const KParams& p, uint32_t cur) {
  return cur ? p.state[0] : p.state[1];
}

// An instance advances when it is active, not frozen and not removed.
__device__ __forceinline__ bool advancing(uint32_t flags) {
  return (flags & kInstActive) && !(flags & (kInstFrozen | kInstRemoved));
}

// Commit one step (global index `step`) of an instance; it freezes when it
// reaches its target, so a request never runs past the step count it asked
// for, and the step it froze at is kept (inst_frozen: the state is in
// canonical order again after one more step).
__device__ __forceinline__ void advance_instance_step(const KParams& p, uint32_t inst, uint32_t step) {
  // loaded together: the commit waits on one round trip
  const uint32_t f = p.inst_flags[inst], s = p.inst_step[inst] + 1, target = p.inst_target[inst];
  if (!advancing(f)) return;
  p.inst_step[inst] = s;
  if (s >= target) {
    p.inst_flags[inst] = f | kInstFrozen;
    p.inst_frozen[inst] = step;
  }
}

struct Out2 {
  float4 r[2];
  uint32_t key[2];
  int n;
};

__device__ __forceinline__ uint32_t word_of(const U4& c, uint32_t k) {
  switch (k & 3u) {
    case 0: return c.x;
    case 1: return c.y;
    case 2: return c.z;
    default: return c.w;
  }
}

// Instance parameters.  kSingle (a handle with one instance) reads the copy
// in the kernel parameters, which the compiler folds into constant-bank
// operands; ensembles read the instance table in global memory.
template <bool kSingle>
__device__ __forceinline__ const DevInstance& inst_of(const KParams& p, uint32_t inst) {
  if (kSingle) return p.inst0;
  // rows of 80 bytes: fields side by side come in one load (64 c4 instances:
  // k_pairs_cells 194.8 -> 190.2 us)
  static_assert(sizeof(DevInstance) % 16 == 0, "16-byte rows");
  return *static_cast<const DevInstance*>(__builtin_assume_aligned(&p.inst[inst], 16));
}

// What every record of a one-instance handle reads, loaded once per CTA:
// the instance's flags, step and first slot in registers, its species and
// first-order tables in shared memory (at most kCtxSpecies / kCtxUni
// entries; larger networks run the generic kernels).
constexpr uint32_t kCtxSpecies = 64, kCtxUni = 64;
struct SingleCtx {
  uint32_t flags, step, slot_base;
  const DevSpecies* species;
  const DevUni* uni;
};

// A word above it cannot be accepted as the coin of the species' only
// first-order reaction (u32_to_unit rounds by at most 128); 0 without one,
// all ones with several, whose other coins have to be drawn.
__device__ __forceinline__ uint32_t first_coin_bound(const DevSpecies& s, const DevUni* uni) {
  if (s.uni_count != 1u) return s.uni_count ? 0xFFFFFFFFu : 0u;
  const double bound = (double)uni[s.uni_begin].prob * 4294967296.0 + 256.0;
  return bound < 4294967295.0 ? (uint32_t)bound : 0xFFFFFFFFu;
}

// Fills the shared tables (all threads of the CTA call it; one barrier).  The
// species' max_r, which the advance does not need, holds the bits of
// first_coin_bound.
__device__ __forceinline__ SingleCtx single_ctx(const KParams& p, DevSpecies* s_species, DevUni* s_uni) {
  for (uint32_t t = threadIdx.x; t < p.S; t += blockDim.x) {
    DevSpecies s = p.species[t];
    s.max_r = __uint_as_float(first_coin_bound(s, p.uni));
    s_species[t] = s;
  }
  for (uint32_t t = threadIdx.x; t < p.U; t += blockDim.x) s_uni[t] = p.uni[t];
  __syncthreads();
  return SingleCtx{ld_u32(&p.inst_flags[0]), ld_u32(&p.inst_step[0]), ld_u32(&p.inst_slot_base[0]), s_species,
                   s_uni};
}

// Advance the record in slot i by one step: diffusion, reflection and the
// first successful first-order reaction (reaction_kernel.cuh:303-341: coins
// in list order, decay when the first product is absent, a second product
// becomes a birth).  kCount adds fired reactions to the event counters.
// The surface walk of a move from x0 to (x, y, z), a point the walls have
// already reflected into the box: the chord stays inside the box, so a panel
// that reaches a wall cannot be passed by way of the wall.  A reflection off
// a panel can leave the box, so the walls reflect the end once more.
// False = absorbed.
__device__ __forceinline__ bool surface_walk(const KParams& p, const DevInstance& I, uint32_t sp, const V3& x0,
                                             float& x, float& y, float& z) {
  V3 e{x, y, z};
  if (!surface_move(surf_view(p), sp, x0, e)) return false;
  x = reflect(e.x, I.lo[0], I.hi[0]);
  y = reflect(e.y, I.lo[1], I.hi[1]);
  z = reflect(e.z, I.lo[2], I.hi[2]);
  return true;
}

// kSurf = 1 walks each displacement (the diffusion step, product offsets)
// through the surface panels.  kSurf = 2 looks up the species mask of the
// cell where the step starts (cell_surf): a set bit means a panel the
// species sees lies within reach of the step or of the products it may
// place, and the record stops after its diffusion with o.n = -1 so that
// the caller queues it for a walk (k_bin_surface); other records finish
// here, and no panel could have changed their step.
template <bool kTable, bool kCount, bool kSingle, int kSurf = 0>
__device__ __forceinline__ void advance_rec(const KParams& p, const SingleCtx& ctx, const float4 rec, uint32_t i,
                                            Out2& o) {
  o.n = 0;
  const uint32_t w = rec_w(rec);
  if (w == kDead) return;
  const uint32_t inst = w >> 16, sp = w & kSpeciesMask;
  const DevInstance& I = inst_of<kSingle>(p, inst);
  const uint32_t flags = kSingle ? ctx.flags : p.inst_flags[inst];
  if (!advancing(flags)) {  // frozen or not active: kept where it is
    if (flags & kInstRemoved) return;
    o.r[0] = rec;
    o.key[0] = cell_key(I, rec.x, rec.y, rec.z);
    o.n = 1;
    return;
  }
  const uint32_t local = i - (kSingle ? ctx.slot_base : p.inst_slot_base[inst]);
  const uint32_t t = kSingle ? ctx.step : p.inst_step[inst];
  const uint32_t k0 = I.key_lo, k1 = I.key_hi;
  const DevSpecies S = kSingle ? ctx.species[sp] : p.species[I.block * p.S + sp];
  // the species mask of the cell the step starts in, loaded before the
  // arithmetic that hides its latency
  const uint32_t near = kSurf == 2 ? __ldg(&p.cell_surf[cell_key(I, rec.x, rec.y, rec.z)]) : 0u;

  const U4 rn = kSingle ? philox_keys(U4{local, t, kTagDiffuse, 0u}, p.keys0)
                        : philox(U4{local, t, kTagDiffuse, 0u}, k0, k1);
  float g0, g1, g2;
  normals3<kTable>(rn, p.gauss, g0, g1, g2);
  float x = __fmaf_rn(S.sigma, g0, rec.x), y = __fmaf_rn(S.sigma, g1, rec.y), z = __fmaf_rn(S.sigma, g2, rec.z);
  // one branch for the three axes
  if (!(x >= I.lo[0] && x <= I.hi[0] && y >= I.lo[1] && y <= I.hi[1] && z >= I.lo[2] && z <= I.hi[2])) {
    x = reflect(x, I.lo[0], I.hi[0]);
    y = reflect(y, I.lo[1], I.hi[1]);
    z = reflect(z, I.lo[2], I.hi[2]);
  }
  if (kSurf == 2 && ((near >> (sp < 7u ? sp : 7u)) & 1u)) {
    o.n = -1;
    return;
  }
  if (kSurf == 1 && !surface_walk(p, I, sp, V3{rec.x, rec.y, rec.z}, x, y, z)) return;  // absorbed
  uint32_t species = sp;
  int n = 1;

  // coin 0 is the diffusion block's spare word; coins 1.. come 4 per block
  U4 coins = rn;
  // most records of a one-instance handle leave by their first word
  const uint32_t n_uni = !kSingle || rn.w <= __float_as_uint(S.max_r) ? S.uni_count : 0u;
  for (uint32_t k = 0; k < n_uni; ++k) {
    if (k > 0 && ((k - 1) & 3u) == 0) coins = philox(U4{local, t, kTagUniCoin | ((k - 1) >> 2), 0u}, k0, k1);
    const DevUni& u = kSingle ? ctx.uni[S.uni_begin + k] : p.uni[I.block * p.U + S.uni_begin + k];
    if (u32_to_unit(k == 0 ? rn.w : word_of(coins, k - 1)) < u.prob) {
      if (kCount) atomicAdd(&p.pending[(size_t)inst * p.R + u.rxn], 1ull);
      if (u.prod0 < 0) return;  // decay: no record
      species = (uint32_t)u.prod0;
      if (u.prod1 >= 0) {
        float bx = x, by = y, bz = z;
        bool keep0 = true, keep1 = true;
        if (u.off0 != 0.0f || u.off1 != 0.0f) {
          float dx, dy, dz;
          unit_vector(local, t, kTagUniDir, 0u, k0, k1, dx, dy, dz);
          bx = reflect(__fmaf_rn(u.off1, dx, x), I.lo[0], I.hi[0]);
          by = reflect(__fmaf_rn(u.off1, dy, y), I.lo[1], I.hi[1]);
          bz = reflect(__fmaf_rn(u.off1, dz, z), I.lo[2], I.hi[2]);
          const V3 from{x, y, z};
          x = reflect(__fmaf_rn(u.off0, dx, x), I.lo[0], I.hi[0]);
          y = reflect(__fmaf_rn(u.off0, dy, y), I.lo[1], I.hi[1]);
          z = reflect(__fmaf_rn(u.off0, dz, z), I.lo[2], I.hi[2]);
          if (kSurf == 1) {
            // both products move from the reaction point
            keep1 = surface_walk(p, I, (uint32_t)u.prod1, from, bx, by, bz);
            keep0 = surface_walk(p, I, (uint32_t)u.prod0, from, x, y, z);
          }
        }
        const float4 born = make_float4(bx, by, bz, __uint_as_float(pack_w(inst, (uint32_t)u.prod1) | kNewborn));
        if (kSurf == 1 && !keep0) {  // the first product was absorbed: the birth takes its place
          if (!keep1) return;
          o.r[0] = born;
          o.key[0] = cell_key(I, bx, by, bz);
          o.n = 1;
          return;
        }
        o.r[1] = born;
        o.key[1] = cell_key(I, bx, by, bz);
        n = (kSurf == 1 && !keep1) ? 1 : 2;
      }
      break;
    }
  }
  o.r[0] = make_float4(x, y, z, __uint_as_float(pack_w(inst, species)));
  o.key[0] = cell_key(I, x, y, z);
  o.n = n;
}

// Zeroth-order birth number v of this step: uniform position in the box
// (reaction_cpu.cpp:44-60 with randPos, particleSystem.h:115-120).
template <bool kSingle>
__device__ __forceinline__ void advance_virtual(const KParams& p, const SingleCtx& ctx, uint32_t v, Out2& o) {
  const uint32_t nz = p.n_inst * p.Z;
  // entry e with zero_off[e] <= v < zero_off[e + 1]
  uint32_t lo = 0, hi = nz;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (p.zero_off[mid] <= v) lo = mid;
    else hi = mid;
  }
  const uint32_t inst = lo / p.Z, zr = lo % p.Z;
  const uint32_t k_local = v - p.zero_off[inst * p.Z];
  const DevInstance& I = inst_of<kSingle>(p, inst);
  const uint32_t t = kSingle ? ctx.step : p.inst_step[inst];
  const U4 r = philox(U4{k_local, t, kTagZeroPos, 0u}, I.key_lo, I.key_hi);
  const float x = fminf(__fmaf_rn(u24_to_unit(r.x), __fsub_rn(I.hi[0], I.lo[0]), I.lo[0]), I.hi[0]);
  const float y = fminf(__fmaf_rn(u24_to_unit(r.y), __fsub_rn(I.hi[1], I.lo[1]), I.lo[1]), I.hi[1]);
  const float z = fminf(__fmaf_rn(u24_to_unit(r.z), __fsub_rn(I.hi[2], I.lo[2]), I.lo[2]), I.hi[2]);
  const DevZero& Zr = p.zero[I.block * p.Z + zr];
  const uint32_t key = cell_key(I, x, y, z);
  o.r[0] = make_float4(x, y, z, __uint_as_float(pack_w(inst, (uint32_t)Zr.prod0) | kNewborn));
  o.key[0] = key;
  o.n = 1;
  if (Zr.prod1 >= 0) {
    o.r[1] = make_float4(x, y, z, __uint_as_float(pack_w(inst, (uint32_t)Zr.prod1) | kNewborn));
    o.key[1] = key;
    o.n = 2;
  }
}

// Lanes with equal keys add their count with one atomic.
__device__ __forceinline__ void warp_count(uint32_t* cnt, uint32_t key) {
  const uint32_t peers = __match_any_sync(kFull, key);
  if (key != kNoKey && lane_id() == (uint32_t)(__ffs(peers) - 1)) atomicAdd(&cnt[key], (uint32_t)__popc(peers));
}

// Lanes with equal keys take consecutive places of their cell with one
// atomic; the count goes back to zero as the cell fills.
__device__ __forceinline__ uint32_t warp_claim(uint32_t* cnt, uint32_t key) {
  const uint32_t peers = __match_any_sync(kFull, key);
  const int leader = __ffs(peers) - 1;
  const uint32_t rank = __popc(peers & ((1u << lane_id()) - 1u));
  uint32_t old = 0;
  if (key != kNoKey && lane_id() == (uint32_t)leader) old = atomicSub(&cnt[key], (uint32_t)__popc(peers));
  old = __shfl_sync(kFull, old, leader);
  return old - 1u - rank;
}

template <int kThreads>
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* total) {
  __shared__ uint32_t warp_sums[kThreads / 32];
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t n = __shfl_up_sync(kFull, incl, d);
    if (lane >= (uint32_t)d) incl += n;
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    uint32_t s = lane < kThreads / 32 ? warp_sums[lane] : 0u;
    uint32_t si = s;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t n = __shfl_up_sync(kFull, si, d);
      if (lane >= (uint32_t)d) si += n;
    }
    if (lane < kThreads / 32) warp_sums[lane] = si - s;
    const uint32_t tot = __shfl_sync(kFull, si, 31);
    if (lane == 0) *total = tot;
  }
  __syncthreads();
  const uint32_t r = warp_sums[warp] + incl - v;
  __syncthreads();
  return r;
}

// Fields of entry g (< 4) of KParams::zero0, read at fixed offsets.
__device__ __forceinline__ void zero0_entry(const KParams& p, uint32_t g, uint32_t& off, uint32_t& len,
                                            int32_t& kmin, uint32_t& rxn) {
  off = p.zero0[0].cdf_off, len = p.zero0[0].cdf_len, kmin = p.zero0[0].kmin, rxn = p.zero0[0].rxn;
#pragma unroll
  for (uint32_t z = 1; z < 4; ++z)
    if (g == z) off = p.zero0[z].cdf_off, len = p.zero0[z].cdf_len, kmin = p.zero0[z].kmin, rxn = p.zero0[z].rxn;
}

// Grid-wide barrier of a cooperative launch (every CTA resident) of fewer
// than 65,536 CTAs: thread 0 of each CTA arrives on a word that counts the
// arrivals in its low half and the barriers passed in its high half; the last
// to arrive takes the arrivals back and adds a barrier in one addition, for
// which the others poll.  (With the count and the generation in two words and
// a pause between polls, two more round trips to L2 and a part of a pause:
// k_scan at 2M particles took 11.5 us, now 9.9.)  The arrival releases the
// CTA's writes, the polls acquire the others'.  The wait is bounded: after
// kGridSpins polls the CTA raises kStatTimeout and the barrier returns false;
// the other CTAs then run out at the same barrier or the next, so every CTA
// returns, and the host clears the word.
constexpr uint32_t kGridSpins = 1u << 22;

__device__ bool grid_barrier(DevCtrl* c) {
  __shared__ uint32_t s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t at, now;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(at) : "l"(&c->bar_word) : "memory");
    bool ok = (at & 0xFFFFu) == gridDim.x - 1u;
    if (ok) {
      asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(&c->bar_word), "r"(0x10000u - gridDim.x)
                   : "memory");
    } else {
      for (uint32_t polls = 0; polls <= kGridSpins && !ok; ++polls) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(now) : "l"(&c->bar_word) : "memory");
        ok = (now ^ at) >> 16 != 0u;
      }
      if (!ok) raise(c, kStatTimeout);
    }
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0u;
}

// Bin layout.  A cell's places come in groups of kBinGroup, stored
// together, and group g of every cell forms one contiguous array:
// place off of a cell is bins[(g * n_cells + cell) * kBinGroup + off %
// kBinGroup], g = off / kBinGroup.  The records a warp bins belong to a
// few consecutive cells (the state is in cell order), so their stores fall
// on a few contiguous lines, and a cell's first records fill whole 32-byte
// sectors rather than half of one shared with a neighbour cell.  The pair
// kernel reads a cell's first kBinGroup places from one group.
__device__ __forceinline__ size_t bin_index(const KParams& p, uint32_t cell, uint32_t off) {
  // the group's number fits 32 bits (2^32 groups would be 256 GiB)
  return (size_t)((off / kBinGroup) * p.n_cells + cell) * kBinGroup + off % kBinGroup;
}

// A record waiting for its place in a bin: the warp's claim (atomicAdd on
// the cell count by the lane that leads the cell's peers) is issued when
// the record is made and consumed one record later, so the atomic's round
// trip to L2 overlaps the next record's arithmetic instead of stalling it.
struct PendingClaim {
  float4 r;
  uint32_t key;     // kNoKey: nothing pending in this lane
  uint32_t old;     // leader lane: count before the warp's claim
  uint32_t leader;  // lane holding `old` for this lane's cell
  uint32_t rank;    // this lane's place among its cell's peers
};

__device__ __forceinline__ PendingClaim claim_issue(uint32_t* cnt, uint32_t key, const float4& r) {
  PendingClaim c;
  c.r = r;
  c.key = key;
  const uint32_t peers = __match_any_sync(kFull, key);
  c.leader = (uint32_t)(__ffs(peers) - 1);
  c.rank = __popc(peers & ((1u << lane_id()) - 1u));
  c.old = 0;
  if (key != kNoKey && lane_id() == c.leader) c.old = atomicAdd(&cnt[key], (uint32_t)__popc(peers));
  return c;
}

__device__ __forceinline__ void claim_retire(const KParams& p, DevCtrl* c, const PendingClaim& pc) {
  const uint32_t off = __shfl_sync(kFull, pc.old, pc.leader) + pc.rank;
  if (pc.key == kNoKey) return;
  if (off < p.bin_cap) {
    p.bins[bin_index(p, pc.key, off)] = pc.r;
  } else {
    raise(c, kStatBins);
    atomicMax(&c->bin_need, off + 1u);
  }
}

// Binned path, pass 1 of 2: advance every record (as k_count) and write it
// into the next free place of its cell's bin.  Replaces k_count + k_scatter:
// the step's arithmetic runs once and nothing is recomputed.  First
// products keep the deferred claim above; the rare second products (births)
// claim and store at once.
// Slots a warp queues for k_bin_surface, written out 32 at a time with one
// atomicAdd on the queue count (a record per lane and atomic would all meet
// on that one word).
struct DeferBuffer {
  uint32_t slot[64];
};

__device__ __forceinline__ void defer_flush(const KParams& p, DevCtrl* c, DeferBuffer& b, uint32_t n) {
  __syncwarp();
  uint32_t base = 0;
  if (lane_id() == 0) base = atomicAdd(&c->n_surf, n);
  base = __shfl_sync(kFull, base, 0);
  if (lane_id() < n) {
    const uint32_t e = base + lane_id();
    if (e < p.capacity) p.surf_queue[e] = b.slot[lane_id()];
    else raise(c, kStatBounds);
  }
  __syncwarp();
}

template <bool kTable, bool kSingle, int kSurf, bool kSpread>
__device__ __forceinline__ void bin_records(const KParams& p, DevCtrl* c, const SingleCtx& ctx, DeferBuffer& defer_buf,
                                            const float4* __restrict__ st, uint32_t n_real, uint32_t* counts) {
  uint32_t n_defer = 0;  // slots in defer_buf (warp-uniform)
  PendingClaim pending;
  pending.key = kNoKey;
  pending.old = 0;
  pending.leader = 0;
  pending.rank = 0;
  stream_records<kSpread>(st, n_real, n_real, [&](uint32_t i, const float4& rec) {
    Out2 o;
    o.n = 0;
    if (i < n_real) advance_rec<kTable, true, kSingle, kSurf>(p, ctx, rec, i, o);
    if (kSurf == 2) {
      // records near a panel go to k_bin_surface
      const bool defer = o.n < 0;
      const uint32_t ball = __ballot_sync(kFull, defer);
      if (ball) {
        if (defer) {
          defer_buf.slot[n_defer + __popc(ball & ((1u << lane_id()) - 1u))] = i;
          o.n = 0;
        }
        n_defer += __popc(ball);
        if (n_defer >= 32u) {
          defer_flush(p, c, defer_buf, 32u);
          if (lane_id() + 32u < n_defer) defer_buf.slot[lane_id()] = defer_buf.slot[lane_id() + 32u];
          __syncwarp();
          n_defer -= 32u;
        }
      }
    }
    const PendingClaim next = claim_issue(counts, o.n > 0 ? o.key[0] : kNoKey, o.r[0]);
    if (__any_sync(kFull, o.n > 1)) claim_retire(p, c, claim_issue(counts, o.n > 1 ? o.key[1] : kNoKey, o.r[1]));
    claim_retire(p, c, pending);
    pending = next;
  });
  claim_retire(p, c, pending);
  if (kSurf == 2 && n_defer > 0) defer_flush(p, c, defer_buf, n_defer);
}

// Exclusive scan over the CTA's threads (whole warps); *total the sum, in
// every thread.
__device__ __forceinline__ uint32_t cta_scan(uint32_t v, uint32_t* total) {
  __shared__ uint32_t s_sum[32], s_total;
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t n = __shfl_up_sync(kFull, incl, d);
    if (lane >= (uint32_t)d) incl += n;
  }
  __syncthreads();  // s_sum and s_total of the last call are no longer read
  if (lane == 31) s_sum[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const uint32_t x = lane < (blockDim.x >> 5) ? s_sum[lane] : 0u;
    uint32_t y = x;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t n = __shfl_up_sync(kFull, y, d);
      if (lane >= (uint32_t)d) y += n;
    }
    s_sum[lane] = y - x;
    if (lane == 31) s_total = y;
  }
  __syncthreads();
  *total = s_total;
  return s_sum[warp] + incl - v;
}

// Zeroth-order births of the step, counted (inversion of the Poisson CDFs, as
// k_zeroth) and binned by one CTA while the others advance the records; a
// call, so that its registers are not the streaming loop's.
template <bool kSingle>
__device__ __noinline__ void zeroth_births(const KParams& p, DevCtrl* c, const SingleCtx& ctx, uint32_t* counts) {
  const uint32_t nz = p.n_inst * p.Z;
  uint32_t carry = 0;
  for (uint32_t base = 0; base < nz; base += blockDim.x) {
    const uint32_t e = base + threadIdx.x;
    uint32_t cnt = 0;
    if (e < nz) {
      const uint32_t inst = e / p.Z, zr = e % p.Z;
      const DevInstance& I = inst_of<kSingle>(p, inst);
      if (advancing(kSingle ? ctx.flags : p.inst_flags[inst])) {
        const DevZero& Zr = p.zero[I.block * p.Z + zr];
        const U4 r = philox(U4{zr, kSingle ? ctx.step : p.inst_step[inst], kTagZeroCount, 0u}, I.key_lo, I.key_hi);
        const double u = u53_to_unit(r.x, r.y);
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
    uint32_t total;
    const uint32_t ex = cta_scan(cnt, &total);
    if (e < nz) p.zero_off[e] = carry + ex;
    carry += total;
  }
  if (threadIdx.x == 0) p.zero_off[nz] = carry;
  __syncthreads();
  for (uint32_t v0 = threadIdx.x & ~31u; v0 < carry; v0 += blockDim.x) {  // whole warps
    const uint32_t v = v0 + lane_id();
    Out2 o;
    o.n = 0;
    if (v < carry) advance_virtual<kSingle>(p, ctx, v, o);
    claim_retire(p, c, claim_issue(counts, o.n > 0 ? o.key[0] : kNoKey, o.r[0]));
    if (__any_sync(kFull, o.n > 1)) claim_retire(p, c, claim_issue(counts, o.n > 1 ? o.key[1] : kNoKey, o.r[1]));
  }
}

// The records of one cell, m-th at base[(m / kBinGroup) * stride + m %
// kBinGroup]: a bin of the binned sort (stride = kBinGroup x the number of
// cells) or a range of the compact scatter buffer (stride kBinGroup, so
// the m-th record is base[m]).
struct CellView {
  const float4* base;
  size_t stride;
  __device__ __forceinline__ size_t at(uint32_t m) const { return (size_t)(m / kBinGroup) * stride + m % kBinGroup; }
  __device__ __forceinline__ float4 operator[](uint32_t m) const { return base[at(m)]; }
  __device__ __forceinline__ float4 ldg(uint32_t m) const { return ld_step(base + at(m)); }
  __device__ __forceinline__ float ldg_x(uint32_t m) const {
    return ld_step(reinterpret_cast<const float*>(base + at(m)));
  }
  __device__ __forceinline__ float2 ldg_xy(uint32_t m) const {
    return ld_step(reinterpret_cast<const float2*>(base + at(m)));
  }
};

// Position of record r among the records of its cell [s, e) in canonical
// order; ties between identical records go by slot.
template <class View>
__device__ __forceinline__ uint32_t canonical_rank(const View sc, uint32_t s, uint32_t e, uint32_t slot,
                                                   const float4& r) {
  uint32_t rank = 0;
  for (uint32_t m = s; m < e; ++m) {
    const float4 q = sc[m];
    rank += (rec_less(q, r) || (m < slot && rec_equal(q, r))) ? 1u : 0u;
  }
  return rank;
}

__device__ __forceinline__ float dist2(const float4& a, const float4& b) {
  const float dx = __fsub_rn(a.x, b.x), dy = __fsub_rn(a.y, b.y), dz = __fsub_rn(a.z, b.z);
  return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
}

// Append candidate pair (lo < hi, canonical slots) of local reaction b,
// after its coin when the reaction probability is below 1.
// starts: the step's cell starts.
__device__ __forceinline__ void emit_pair(const KParams& p, DevCtrl* c, const uint32_t* starts, uint32_t lo, uint32_t hi, int32_t b,
                                          float prob, uint32_t inst, const DevInstance& I) {
  if (prob < 1.0f) {
    const uint32_t base_new = ld_step(&starts[I.cell_base]);
    const U4 u = philox(U4{lo - base_new, ld_step(&p.inst_step[inst]), kTagBimCoin, hi - base_new}, I.key_lo,
                        I.key_hi);
    if (!(u32_to_unit(u.x) < prob)) return;
  }
  const uint32_t idx = atomicAdd(&c->n_pairs, 1u);
  flag_phase(kFlagPairs);
  if (idx < p.pair_cap) p.pairs[idx] = DevPair{lo, hi, (uint32_t)b | (inst << 16), 0u};
  else raise(c, kStatPairs);
}

constexpr uint32_t kBigChunk = 2048;  // records of a unit: sorted in one pass through shared memory (16 KiB of keys)
constexpr int kBigGrid = 304;  // most CTAs of the large-cell kernel (cells they take in turn)

// First record of a cell: its bin, or its range of the compact scatter buffer.
template <bool kBinned>
__device__ __forceinline__ CellView cell_records(const KParams& p, uint32_t cell, uint32_t cs) {
  if (kBinned) return CellView{p.bins + bin_index(p, cell, 0), (size_t)p.n_cells * kBinGroup};
  return CellView{p.scatter + cs, kBinGroup};
}

// A record looking for partners.
struct Seeker {
  float4 r;
  uint32_t inst, block;
  float max_r, r2max;
  float xlim;          // |dx| bound of every pair within its binding radii
  const int32_t* row;  // second-order table row of its species
};

// False when the record takes no part in this step's pair search: born in
// this step, instance not advancing, or a species without second-order
// reactions.
// s_maxr (one-instance kernels): the species' largest radii in shared
// memory, with adv0 the instance's advancing state, read once per kernel.
template <bool kSingle>
__device__ __forceinline__ bool seeker_init(const KParams& p, const float4& r, Seeker& k,
                                            const float* s_maxr = nullptr, bool adv0 = true) {
  const uint32_t w = rec_w(r);
  if (w & kNewborn) return false;
  k.r = r;
  k.inst = w >> 16;
  const uint32_t sa = w & kSpeciesMask;
  if (kSingle && s_maxr) {
    if (!adv0) return false;
    k.block = p.inst0.block;
    k.max_r = s_maxr[sa];
  } else {
    if (!advancing(ld_step(&p.inst_flags[k.inst]))) return false;
    k.block = inst_of<kSingle>(p, k.inst).block;
    k.max_r = __ldg(&p.species[k.block * p.S + sa].max_r);
  }
  // a bound on every squared radius of the species (float rounding of max_r^2)
  k.r2max = k.max_r * k.max_r * 1.0001f;
  // fl(dx^2) <= d2 <= r2max, so |dx| <= max_r * 1.00005
  k.xlim = k.max_r * 1.001f;
  k.row = p.bim_table + sa * p.S;
  return k.max_r > 0.0f;
}

// Local second-order reaction of k with record q when q lies within its
// binding radius, else -1.
__device__ __forceinline__ int32_t pair_reaction(const KParams& p, const Seeker& k, const float4& q) {
  if (fabsf(__fsub_rn(q.x, k.r.x)) > k.xlim) return -1;
  const uint32_t wq = rec_w(q);
  if (wq & kNewborn) return -1;
  const float d2 = dist2(k.r, q);
  if (d2 > k.r2max) return -1;
  const int32_t b = __ldg(&k.row[wq & kSpeciesMask]);
  if (b < 0 || d2 > __ldg(&p.bim[k.block * p.B + (uint32_t)b].r2)) return -1;
  return b;
}

template <bool kSingle>
__device__ __forceinline__ void emit(const KParams& p, DevCtrl* c, const uint32_t* starts, const Seeker& k, uint32_t ca, uint32_t cq,
                                     int32_t b) {
  emit_pair(p, c, starts, min(ca, cq), max(ca, cq), b, __ldg(&p.bim[k.block * p.B + (uint32_t)b].prob), k.inst,
            inst_of<kSingle>(p, k.inst));
}

// True when a record may lie within its largest binding radius (plus the
// pruning margin) of a +x, +y or +z face of its cell, i.e. when forward_mask
// may return a neighbour; false for most records, which lie deeper inside
// their cell.  inv, shift: of its instance (KParams::near_grid); lim: of its
// species.  The grid coordinates are shifted down by more than any rounding
// of them, so none rounds up past the face it is near, and the 1% slack of
// lim exceeds the rounding of forward_mask's face distances: it never rejects
// a record that forward_mask would give a neighbour.
__device__ __forceinline__ bool near_forward_face(const float4& r, const float4& lim, const float (&inv)[3],
                                                  const float (&shift)[3]) {
  const float gx = __fmaf_rn(r.x, inv[0], shift[0]);
  const float gy = __fmaf_rn(r.y, inv[1], shift[1]);
  const float gz = __fmaf_rn(r.z, inv[2], shift[2]);
  return gx - floorf(gx) >= lim.y || gy - floorf(gy) >= lim.z || gz - floorf(gz) >= lim.w;
}

// The forward neighbour cells (higher key) of record k that its largest
// binding radius reaches: the cells whose shared face, edge or corner lies
// within it.  Every cross-cell pair within range is found from its
// lower-key side only, so each is tested once.  Bit b of the result names
// neighbour b: 0 = (+1, 0, 0); 1..3 = (-1..+1, +1, 0); 4..12 = (-1..+1,
// -1..+1, +1) in (dx, dy, dz), dx fastest.  *key0 receives the record's own
// cell key.  The cell coordinates are recomputed from the position exactly
// as the sort computed the key (cell_coord), which avoids integer division.
template <bool kSingle>
__device__ __forceinline__ uint32_t forward_mask(const KParams& p, const Seeker& k, uint32_t* key0) {
  const DevInstance& I = inst_of<kSingle>(p, k.inst);
  const float cl0 = I.cell[0], cl1 = I.cell[1], cl2 = I.cell[2];
  const uint32_t d0 = I.dims[0], d1 = I.dims[1], d2 = I.dims[2];
  const float gx = __fmul_rn(__fsub_rn(k.r.x, I.lo[0]), I.inv[0]);
  const float gy = __fmul_rn(__fsub_rn(k.r.y, I.lo[1]), I.inv[1]);
  const float gz = __fmul_rn(__fsub_rn(k.r.z, I.lo[2]), I.inv[2]);
  const int cx = min(max((int)floorf(gx), 0), (int)d0 - 1);
  const int cy = min(max((int)floorf(gy), 0), (int)d1 - 1);
  const int cz = min(max((int)floorf(gz), 0), (int)d2 - 1);
  *key0 = I.cell_base + ((uint32_t)cz * d1 + (uint32_t)cy) * d0 + (uint32_t)cx;
  const float margin = p.prune_margin * fminf(cl0, fminf(cl1, cl2));
  const float need = k.max_r + margin;
  const float fx = __fsub_rn(gx, (float)cx), fy = __fsub_rn(gy, (float)cy), fz = __fsub_rn(gz, (float)cz);
  const float hix = (1.0f - fx) * cl0, hiy = (1.0f - fy) * cl1, hiz = (1.0f - fz) * cl2;
  // Every forward neighbour lies across the +x, +y or +z face.  Squared
  // distance to the -/+ face along each axis, infinite where no
  // cell lies beyond the face; a neighbour is marked when the sum over its
  // axes, added as (x + y) + z, is within need^2.  No branch: the warp
  // takes the records of a drain together, so every lane's marking used to
  // run the loops of the slowest.
  const float far = __int_as_float(0x7f800000);
  const float lox = fx * cl0, loy = fy * cl1;
  const float need2 = need * need;
  const float xm = cx > 0 ? lox * lox : far, xp = cx + 1 < (int)d0 ? hix * hix : far;
  const float ym = cy > 0 ? loy * loy : far, yp = cy + 1 < (int)d1 ? hiy * hiy : far;
  const float zp = cz + 1 < (int)d2 ? hiz * hiz : far;
  uint32_t mask = xp <= need2 ? 1u : 0u;  // (+1, 0, 0)
  mask |= (xm + yp <= need2 ? 1u : 0u) << 1;
  mask |= (yp <= need2 ? 1u : 0u) << 2;
  mask |= (xp + yp <= need2 ? 1u : 0u) << 3;
  const float ey[3] = {ym, 0.0f, yp}, ex[3] = {xm, 0.0f, xp};
#pragma unroll
  for (int dy = 0; dy < 3; ++dy) {
#pragma unroll
    for (int dx = 0; dx < 3; ++dx) mask |= ((ex[dx] + ey[dy]) + zp <= need2 ? 1u : 0u) << (4 + dy * 3 + dx);
  }
  return mask;
}

// Key of forward neighbour b (bit numbering of forward_mask) of cell key0.
__device__ __forceinline__ uint32_t forward_key(uint32_t key0, uint32_t b, uint32_t d0, uint32_t d1) {
  int dx, dy, dz;
  if (b == 0) {
    dx = 1, dy = 0, dz = 0;
  } else if (b < 4) {
    dx = (int)b - 2, dy = 1, dz = 0;
  } else {
    const int q = (int)b - 4;
    dx = q % 3 - 1, dy = q / 3 - 1, dz = 1;
  }
  return (uint32_t)((int)key0 + (dz * (int)d1 + dy) * (int)d0 + dx);
}

// Pairs of seeker k (canonical slot ca) with the records of neighbour cell
// nkey (first slot ns, nn records), found from k's side.
template <bool kBinned, bool kSingle>
__device__ __forceinline__ void visit_cell(const KParams& p, DevCtrl* c, const uint32_t* starts, const Seeker& k, uint32_t ca,
                                           uint32_t nkey, uint32_t ns, uint32_t nn) {
  if (nn > kBigCell) return;  // pairs with large cells are found by k_pairs_big
  const CellView nb = cell_records<kBinned>(p, nkey, ns);
  // x words of the first members together (overlapping latencies); a full
  // record only for members within the x window, taken from a bit mask
  // (places past the cell read as all-ones bits, a NaN |dx|).  The mask in
  // place of a branch per member: 0.248 against 0.261 ms on the 16M c3
  // step, although only the records near a +face come here.
  constexpr uint32_t kBatch = 8;
  float xs[kBatch];
#pragma unroll
  for (uint32_t m = 0; m < kBatch; ++m) xs[m] = m < nn ? nb.ldg_x(m) : __uint_as_float(0xFFFFFFFFu);
  uint32_t inx = 0;
#pragma unroll
  for (uint32_t m = 0; m < kBatch; ++m) inx |= (fabsf(__fsub_rn(xs[m], k.r.x)) <= k.xlim ? 1u : 0u) << m;
  while (inx) {
    const uint32_t m = (uint32_t)(__ffs(inx) - 1);
    inx &= inx - 1u;
    const float4 q = nb.ldg(m);
    const int32_t b = pair_reaction(p, k, q);
    if (b >= 0) emit<kSingle>(p, c, starts, k, ca, ns + canonical_rank(nb, 0, nn, m, q), b);
  }
  for (uint32_t m = kBatch; m < nn; ++m) {
    const float4 q = nb.ldg(m);
    const int32_t b = pair_reaction(p, k, q);
    if (b >= 0) emit<kSingle>(p, c, starts, k, ca, ns + canonical_rank(nb, 0, nn, m, q), b);
  }
}

// Canonical order + pair search.  A warp takes tasks of 32 consecutive
// cells, from the highest key down, and strings the tasks' records
// together into one stream: round r of the warp takes stream records
// 32r .. 32r+31, one per lane, whatever cells and tasks they come from, so
// only the warp's last round runs partly empty.  (Rounds that stopped at
// each task's end left 14% of the lanes idle on the 16M c3 step, whose
// tasks hold about 97 records.)  At most two tasks are open at a time:
// their non-empty cells sit in a per-warp ring, and a task is opened (its
// cell ranges read and scanned) when the stream runs short of the next
// round and the task before the last one has ended.  There are no CTA-wide
// barriers.  For its record a lane
//   * counts the records of its cell that precede it in canonical order,
//     reading only their x words (records whose x bits occur twice in the
//     cell are ranked again on all four words), and writes it to
//     cell_start[cell] + that rank in the next state;
//   * in the same loop marks the cell's later records (storage order)
//     whose x lies within its largest binding radius; only those are read
//     in full and tested, each in-cell pair once;
//   * tests, cheaply and with no branch, whether its record lies within
//     its largest binding radius of a +face of its cell (near_forward_face)
//     and queues those few records in the warp's shared queue; the warp
//     takes them 32 at a time, one per lane, marks their forward neighbour
//     cells (forward_mask) and visits them.  Marking the neighbours of
//     every record in line, and visiting them from the record's own lane,
//     held whole warps for the sake of one or two lanes.
// Canonical slots of partners are computed only for pairs within range.
// Cells above kBigCell records are queued for the large-cell kernels.  kBinned: the
// records come from the cell bins, whose counts are cleared here for the
// next step; otherwise from the compact scatter buffer.
//
// Bulk-copy staging of each task's first bin group was slower on the 16M c3
// step (0.325 against 0.272 ms): the staging buffers took the L1 space that
// the rank loads and neighbour visits hit in.
constexpr uint32_t kFaceQueue = 64;  // queued records per warp (< 32 between drains, + one round's push)
constexpr uint32_t kCellRing = 64;   // open cells per warp: two tasks of at most 32 non-empty cells

// Records near a +face queued by a warp.
struct FaceQueue {
  float4 rec[kFaceQueue];
  uint32_t ca[kFaceQueue];
};

// Take the first 32 queued records, one per lane (lane < n), move the rest
// (n - 32 < 32 entries) to the front, then mark and visit the forward
// neighbour cells of the lane's record.  Warp-uniform call.
template <bool kBinned, bool kSingle>
__device__ __forceinline__ void drain_faces(const KParams& p, DevCtrl* c, const uint32_t* starts, FaceQueue& q, uint32_t n,
                                            const float* s_maxr, bool adv0) {
  const uint32_t lane = lane_id();
  __syncwarp();
  const float4 r = q.rec[lane];
  const uint32_t ca = q.ca[lane];
  __syncwarp();
  if (lane + 32u < n) {
    q.rec[lane] = q.rec[lane + 32u];
    q.ca[lane] = q.ca[lane + 32u];
  }
  __syncwarp();
  if (lane >= n) return;
  Seeker k;
  if (!seeker_init<kSingle>(p, r, k, s_maxr, adv0)) return;
  uint32_t key0 = 0;
  uint32_t nbm = forward_mask<kSingle>(p, k, &key0);
  const DevInstance& I = inst_of<kSingle>(p, k.inst);
  while (nbm) {
    const uint32_t nkey = forward_key(key0, (uint32_t)(__ffs(nbm) - 1), I.dims[0], I.dims[1]);
    nbm &= nbm - 1u;
    const uint32_t ns = ld_step(&starts[nkey]);
    visit_cell<kBinned, kSingle>(p, c, starts, k, ca, nkey, ns, ld_step(&starts[nkey + 1]) - ns);
  }
}

// Per-species tables of a one-instance handle's pair search: the largest
// binding radius, and KParams::near_lim.
template <bool kSingle>
struct PairSpecies {
  float max_r[kSingle ? kCtxSpecies : 1];
  float4 lim[kSingle ? kCtxSpecies : 1];
};

// All threads of the CTA call it; one barrier.
template <bool kSingle>
__device__ __forceinline__ void pair_species(const KParams& p, PairSpecies<kSingle>& sp) {
  if constexpr (kSingle) {
    for (uint32_t t = threadIdx.x; t < p.S; t += blockDim.x) {
      sp.max_r[t] = p.species[p.inst0.block * p.S + t].max_r;
      sp.lim[t] = p.near_lim[t];
    }
    __syncthreads();
  }
}

// Per-warp working sets of the pair search (CTAs of kWarps warps): the ring of
// the open tasks' non-empty cells -- key, first slot, records, stream offset of
// the cell's first record -- and the records near a +face.
template <bool kHasBim, int kWarps>
struct PairShared {
  uint4 cell[kWarps][kCellRing];
  FaceQueue face[kHasBim ? kWarps : 1];
  uint32_t ticket;  // kOwn: tasks of the CTA's range taken
};

// kOwn: each CTA has a range of cells of its own, cut into tasks that its
// warps take from a counter (sh.ticket, 0 before the call): with a fixed share
// of cells per warp the fullest of 4,864 shares, 40% above the mean, held up
// the barrier behind the search.  Tasks hold a round's worth of records or
// more, and are small enough that a warp takes four.  Else the warps of the
// grid take tasks of 32 cells in turn.
// starts: the step's cell starts (copied to p.cell_start when they are a copy
// elsewhere); clear: the counts set to 0 for a later step.
constexpr uint32_t kOwnCells = 8;
template <bool kHasBim, bool kBinned, bool kSingle, bool kOwn, int kWarps>
__device__ __forceinline__ void pair_cells(const KParams& p, DevCtrl* c, float4* __restrict__ nx, bool adv0,
                                           PairShared<kHasBim, kWarps>& sh, const PairSpecies<kSingle>& sp,
                                           const uint32_t* starts, uint32_t* clear) {
  const uint32_t warp = threadIdx.x >> 5, lane = lane_id();
  const uint32_t nw = gridDim.x * (blockDim.x >> 5);
  const uint32_t tk0 = blockIdx.x * (blockDim.x >> 5) + warp;
  // the CTA's cells [own_lo, end) in tasks of own_cells, or every nw-th task
  // of the n_tasks
  const uint32_t own_lo = kOwn ? (uint32_t)((uint64_t)p.n_cells * blockIdx.x / gridDim.x) : 0u;
  const uint32_t end = kOwn ? (uint32_t)((uint64_t)p.n_cells * (blockIdx.x + 1u) / gridDim.x) : p.n_cells;
  const uint32_t own_cells = kOwn ? min(max((end - own_lo) / (4u * kWarps), kOwnCells), 32u) : 32u;
  const uint32_t n_tasks = (p.n_cells + 31u) >> 5;
  uint32_t my_tasks = kOwn ? ~0u : (tk0 < n_tasks ? (n_tasks - 1u - tk0) / nw + 1u : 0u);
  const uint32_t le_mask = lane == 31 ? kFull : ((2u << lane) - 1u);
  FaceQueue& fqueue = sh.face[kHasBim ? warp : 0];
  uint32_t fq = 0;  // queued records (warp-uniform)
  // First cell of the warp's i-th task.  Tasks taken in turn run from the highest key down: the
  // bins written last by k_bin (its records stream in ascending cell
  // order) are still in L2, and the next state's low slots, written last
  // here, are the first the next step's k_bin reads.
  auto first_cell = [&](uint32_t i) {
    if (!kOwn) return (n_tasks - 1u - (tk0 + i * nw)) * 32u;
    uint32_t t = 0;
    if (lane == 0) t = atomicAdd(&sh.ticket, 1u);
    return own_lo + __shfl_sync(kFull, t, 0) * own_cells;
  };
  // The two task slots (slot = task index & 1): the stream offset of the
  // lane's cell in each, ~0 for an empty cell.
  uint32_t o0 = ~0u, o1 = ~0u;
  uint32_t opened = 0;   // tasks opened
  uint32_t last = 0;     // stream offset of the last opened task (the end of the one before it)
  uint32_t loaded = 0;   // stream records of the opened tasks
  uint32_t entries = 0;  // ring entries written
  uint32_t before = 0;   // ring entries whose cells start before the round
  // A round takes stream records [rb, rb + 32); one that the open tasks
  // cannot fill (the last task before it still open, or no task left)
  // ends at `loaded`, where the next round starts.
  for (uint32_t rb = 0;;) {
    // Open tasks while the stream falls short of this round and the slot
    // to be reused holds a task that has ended.
    while (loaded < rb + 32u && opened < my_tasks && last <= rb) {
      const uint32_t sl = opened & 1u;
      const uint32_t first = first_cell(opened), cell = first + lane;
      if (kOwn && first >= end) {
        my_tasks = opened;
        break;
      }
      uint32_t cs = 0, n = 0;
      if (cell < end && (!kOwn || lane < own_cells)) {
        cs = ld_step(&starts[cell]);
        n = ld_step(&starts[cell + 1]) - cs;
        if (kBinned) clear[cell] = 0u;
        if (kOwn && starts != p.cell_start) p.cell_start[cell] = cs;
        if (n > kBigCell) {
          // its place in the queue and its first unit in one atomic, so
          // that the entries are in unit order
          const unsigned long long b =
              atomicAdd(&c->big_queue, (unsigned long long)((n + kBigChunk - 1u) / kBigChunk) << 32 | 1ull);
          atomicMax(&c->big_max, n);
          flag_phase(kFlagBig);
          if ((uint32_t)b < p.big_cap) p.big[(uint32_t)b] = make_uint2(cell, (uint32_t)(b >> 32));
          else raise(c, kStatBounds);
          n = 0;
        }
      }
      const uint32_t ball = __ballot_sync(kFull, n > 0);
      uint32_t incl = n;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, incl, d);
        if (lane >= (uint32_t)d) incl += t;
      }
      const uint32_t off = loaded + incl - n;
      __syncwarp();  // the ring entries about to be replaced are no longer read
      if (n > 0) {
        const uint32_t e = (entries + __popc(ball & ((1u << lane) - 1u))) & (kCellRing - 1u);
        sh.cell[warp][e] = make_uint4(cell, cs, n, off);
      }
      entries += __popc(ball);
      last = loaded;
      loaded += __shfl_sync(kFull, incl, 31);
      if (sl) o1 = n > 0 ? off : ~0u;
      else o0 = n > 0 ? off : ~0u;
      ++opened;
      __syncwarp();
    }
    if (rb >= loaded) break;  // every task opened and taken
    // lanes at which a cell starts in this round
    const uint32_t M = __reduce_or_sync(kFull, (o0 - rb < 32u ? 1u << (o0 - rb) : 0u) |
                                                   (o1 - rb < 32u ? 1u << (o1 - rb) : 0u));
    const uint32_t t = rb + lane;
    bool near = false;  // this lane's record may have partners in forward neighbour cells
    uint32_t ca = 0;
    float4 ra = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (t < loaded) {
      const uint32_t e = (before + __popc(M & le_mask) - 1u) & (kCellRing - 1u);
      const uint4 cc = sh.cell[warp][e];
      const uint32_t ocell = cc.x, ocs = cc.y, on = cc.z;
      const uint32_t j = t - cc.w;
      const CellView cb = cell_records<kBinned>(p, ocell, ocs);
      ra = kBinned ? ld_step(&p.bins[bin_index(p, ocell, j)]) : cb.ldg(j);
      // the record's bounds, in one load (two with its instance's flags); its
      // seeker is made only when it has candidates (k_pairs_cells 234 -> 221.5
      // us on the 16M c3 step, 190 -> 183 on 64 c4 instances, whose records
      // loaded 14 words of their instance and species before)
      float4 lim = make_float4(-1.0f, 2.0f, 2.0f, 2.0f);
      if (kHasBim && kSingle) {
        if (adv0 && !(rec_w(ra) & kNewborn)) lim = sp.lim[rec_w(ra) & kSpeciesMask];
      } else if (kHasBim) {
        const uint32_t w = rec_w(ra), inst = w >> 16;
        const bool adv = advancing(ld_step(&p.inst_flags[inst]));
        const float4 l = __ldg(&p.near_lim[inst * p.S + (w & kSpeciesMask)]);
        if (adv && !(w & kNewborn)) lim = l;
      }
      const float xlim = lim.x;
      const uint32_t rx = __float_as_uint(ra.x);
      // rank: members with smaller x bits; le also counts equal ones (the
      // record itself among them), so le - rank > 1 means a tie to break
      // on all four words.  cand: bit m = member m < 32 within xlim in both
      // x and y (a bound on |dx| and |dy| of any pair within range), so
      // only members near in two coordinates are read in full and tested:
      // 0.246 -> 0.242 ms on the 16M c3 step against x alone.  The first
      // kRankBatch members' x and y are loaded together (one 8-byte load
      // each), so their latencies overlap; larger cells continue one member
      // at a time on x.  The batch runs without a branch per member
      // (0.272 -> 0.261 ms): places past the cell read as all-ones x bits,
      // which count in neither rank nor le and give a NaN |dx| that is
      // never in range.
      constexpr uint32_t kRankBatch = 8;
      uint32_t rank = 0, le = 0, cand = 0;
      // members [0, 6) always, [6, 8) only when a lane of the warp has more
      // than six (0.2386 -> 0.2378 ms on the 16M c3 step)
      constexpr uint32_t kRankFirst = 6;
      float2 xs[kRankBatch];
      auto rank_members = [&](uint32_t m0, uint32_t m1) {
#pragma unroll
        for (uint32_t m = m0; m < m1; ++m) xs[m] = m < on ? cb.ldg_xy(m) : make_float2(__uint_as_float(0xFFFFFFFFu), 0.0f);
#pragma unroll
        for (uint32_t m = m0; m < m1; ++m) {
          const uint32_t qb = __float_as_uint(xs[m].x);
          rank += qb < rx ? 1u : 0u;
          le += qb <= rx ? 1u : 0u;
          cand |= (fabsf(__fsub_rn(xs[m].x, ra.x)) <= xlim && fabsf(__fsub_rn(xs[m].y, ra.y)) <= xlim ? 1u : 0u) << m;
        }
      };
      rank_members(0, kRankFirst);
      if (__any_sync(__activemask(), on > kRankFirst)) rank_members(kRankFirst, kRankBatch);
      for (uint32_t m = kRankBatch; m < on; ++m) {
        const float qx = cb.ldg_x(m);
        const uint32_t qb = __float_as_uint(qx);
        rank += qb < rx ? 1u : 0u;
        le += qb <= rx ? 1u : 0u;
        if (m < 32u && fabsf(__fsub_rn(qx, ra.x)) <= xlim) cand |= 1u << m;
      }
      cand &= j >= 31u ? 0u : ~((2u << j) - 1u);  // later members only
      if (le - rank > 1u) rank = canonical_rank(cb, 0, on, j, ra);
      ca = ocs + rank;
      if (ca < p.capacity) nx[ca] = make_float4(ra.x, ra.y, ra.z, __uint_as_float(rec_w(ra) & ~kNewborn));
      else raise(c, kStatBounds);
      if (kHasBim && (cand || (on > 32u && xlim >= 0.0f))) {
        Seeker k;
        seeker_init<kSingle>(p, ra, k, kSingle ? sp.max_r : nullptr, adv0);
        while (cand) {
          const uint32_t m = (uint32_t)(__ffs(cand) - 1);
          cand &= cand - 1u;
          const float4 qm = cb.ldg(m);
          const int32_t bb = pair_reaction(p, k, qm);
          if (bb >= 0) emit<kSingle>(p, c, starts, k, ca, ocs + canonical_rank(cb, 0, on, m, qm), bb);
        }
        for (uint32_t m = max(j + 1u, 32u); m < on; ++m) {  // cells of 33..kBigCell records
          const float4 qm = cb.ldg(m);
          const int32_t bb = pair_reaction(p, k, qm);
          if (bb >= 0) emit<kSingle>(p, c, starts, k, ca, ocs + canonical_rank(cb, 0, on, m, qm), bb);
        }
      }
      if (kHasBim && kSingle) {
        near = near_forward_face(ra, lim, p.inst0.inv, p.near_shift);
      } else if (kHasBim) {
        const float4* grid = &p.near_grid[2u * (rec_w(ra) >> 16)];
        const float4 a = __ldg(grid), b = __ldg(grid + 1);
        const float inv[3] = {a.x, a.y, a.z}, shift[3] = {b.x, b.y, b.z};
        near = near_forward_face(ra, lim, inv, shift);
      }
    }
    if (kHasBim) {
      // records near a +face into the warp's queue, visited 32 at a time
      const uint32_t ball = __ballot_sync(kFull, near);
      if (near) {
        const uint32_t pos = fq + __popc(ball & ((1u << lane) - 1u));
        fqueue.rec[pos] = ra;
        fqueue.ca[pos] = ca;
      }
      fq += __popc(ball);
      if (fq >= 32u) {
        drain_faces<kBinned, kSingle>(p, c, starts, fqueue, fq, kSingle ? sp.max_r : nullptr, adv0);
        fq -= 32u;
      }
    }
    before += __popc(M);
    rb = min(rb + 32u, loaded);
    __syncwarp();
  }
  if (kHasBim && fq > 0) drain_faces<kBinned, kSingle>(p, c, starts, fqueue, fq, kSingle ? sp.max_r : nullptr, adv0);
}

// ------------------------------------------------------------ large cells
// A cell of more than kBigCell records (particles released at one point, a
// collapse) is cut into units of kBigChunk records, and every phase spreads
// units, not cells, over the CTAs: with a CTA per cell, 20,000 particles
// released at a point kept one SM busy for 20 to 31 ms a step while 151
// idled; the same steps take 0.13 ms (half of it sorting, half pairs).
// What bounds the phases now is latency: the bitonic network's barriers,
// the dependent L2 loads of the rank searches, the grid barriers between
// phases.
constexpr uint32_t kBigWays = 32;     // sorted runs one merge pass joins
constexpr uint32_t kBigParts = 32;    // most CTAs that share a unit's pair search
constexpr uint32_t kBigSegments = 8;  // pieces of a seeker block's sweep when few units are queued

// Merge passes that turn a cell of n records, sorted unit by unit, into one
// run.
__device__ __forceinline__ uint32_t big_passes(uint32_t n) {
  uint32_t passes = 0;
  for (uint64_t w = kBigChunk; w < n; w *= kBigWays) ++passes;
  return passes;
}

// A queued cell and its records.
struct BigCell {
  uint32_t cell, cs, n;
  uint32_t first;  // first record of the unit asked for
};

// Queue entry of unit u: entries hold (cell, first unit) in unit order.
__device__ __forceinline__ BigCell big_unit(const KParams& p, uint32_t nbig, uint32_t u) {
  uint32_t lo = 0, hi = nbig;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldcg(&p.big[mid]).y <= u) lo = mid;
    else hi = mid;
  }
  const uint2 e = __ldcg(&p.big[lo]);
  BigCell b;
  b.cell = e.x;
  b.cs = p.cell_start[e.x];
  b.n = p.cell_start[e.x + 1] - b.cs;
  b.first = (u - e.y) * kBigChunk;
  return b;
}

// The two buffers the merge passes of a cell alternate between: its ranges
// of the two halves of big_scratch.  (The cell's own bin, free once its
// units are sorted, made a poor second buffer: the groups of a bin lie
// n_cells x 64 bytes apart, a page each for a crowded cell, and the
// searches of the pair phase ran on TLB misses.)
__device__ __forceinline__ float4* big_buffer(const KParams& p, uint32_t cs, uint32_t which) {
  return p.big_scratch + (which & 1u ? p.capacity : 0u) + cs;
}

// Sum over the runs of width w in [lo, hi) of the records that order before
// e (before or equal in runs ahead of e's own), e's own run excluded.  Eight
// searches at a time, so that their loads are in flight together.
__device__ __forceinline__ uint32_t runs_rank(const float4* v, uint32_t w, uint32_t lo, uint32_t hi, uint32_t own,
                                              const float4& e) {
  constexpr uint32_t kIlp = 8;
  const uint32_t runs = (hi - lo + w - 1u) / w;
  uint32_t rank = 0;
  for (uint32_t r = 0; r < runs; r += kIlp) {
    uint32_t at[kIlp], len[kIlp];
#pragma unroll
    for (uint32_t k = 0; k < kIlp; ++k) {
      const uint64_t b = lo + (uint64_t)(r + k) * w;
      at[k] = 0;
      len[k] = r + k != own && b < hi ? min(w, hi - (uint32_t)b) : 0u;
    }
    for (uint32_t step = w; step; step >>= 1) {
#pragma unroll
      for (uint32_t k = 0; k < kIlp; ++k) {
        if (at[k] + step > len[k]) continue;
        const float4 q = v[lo + (r + k) * w + at[k] + step - 1u];
        if (r + k < own ? !rec_less(e, q) : rec_less(q, e)) at[k] += step;
      }
    }
#pragma unroll
    for (uint32_t k = 0; k < kIlp; ++k) rank += at[k];
  }
  return rank;
}

// Bitonic network over the keys s_key[0, size), size a power of two, by the
// threads of the CTA.
template <class Less>
__device__ __forceinline__ void bitonic_network(unsigned long long* s_key, uint32_t size, Less&& less) {
  for (uint32_t k = 2; k <= size; k <<= 1) {
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      for (uint32_t t = threadIdx.x; t < size / 2; t += blockDim.x) {
        const uint32_t i = ((t & ~(j - 1u)) << 1) | (t & (j - 1u)), ixj = i | j;
        const unsigned long long q0 = s_key[i], q1 = s_key[ixj];
        const bool swap = less(q1, q0) == ((i & k) == 0);
        s_key[i] = swap ? q1 : q0;
        s_key[ixj] = swap ? q0 : q1;
      }
      __syncthreads();
    }
  }
}

// Records of a unit with the same x bits are put in order by counting over
// their stretch of equal keys, up to this many apart; a unit with a longer
// stretch goes through the network once more, by all four words (by index
// when identical).  2,000 immobile molecules with one x: 845 us a step when
// the stretch was counted over whatever its length, 82 so, 38 with distinct x
// (and 89 with a network over whole records, one CTA a cell).
constexpr uint32_t kTieStretch = 8;
__device__ __noinline__ void sort_tied_keys(unsigned long long* s_key, uint32_t size, uint32_t len, const CellView cb,
                                            uint32_t first) {
  bitonic_network(s_key, size, [&](unsigned long long a, unsigned long long b) {
    const uint32_t i = (uint32_t)a, j = (uint32_t)b;
    if (a >> 32 != b >> 32 || i >= len || j >= len) return a < b;  // past the unit: all ones
    const float4 q = cb[first + i], r = cb[first + j];
    return rec_less(q, r) || (i < j && rec_equal(q, r));
  });
}

// Canonical order of the queued cells.  Phase 1 sorts each unit in shared
// memory (a bitonic network over keys) into big_scratch;
// then each merge pass joins up to kBigWays runs into one: a record's place
// is its index in its own run plus its rank in the others.  After a cell's
// last pass its run lies in big_buffer(passes), newborn marks kept, where
// the pair search reads it, and in the next state without them.  False when
// a grid barrier ran out (the same answer in every CTA that returns).
template <bool kBinned>
__device__ bool big_sort(const KParams& p, DevCtrl* c, uint32_t nbig, uint32_t units,
                         unsigned long long* s_key) {
  __shared__ BigCell s_big;
  float4* nx = next_state(p, ld_u32(&c->cur));
  const uint32_t passes = big_passes(ld_u32(&c->big_max));
  for (uint32_t u = blockIdx.x; u < units; u += gridDim.x) {
    __syncthreads();  // s_big and s_key of the last unit are no longer read
    if (threadIdx.x == 0) s_big = big_unit(p, nbig, u);
    __syncthreads();
    const BigCell b = s_big;
    if ((uint64_t)b.cs + b.n > p.capacity || b.first >= b.n) {
      if (threadIdx.x == 0) raise(c, kStatBounds);
      continue;  // uniform over the CTA
    }
    const uint32_t len = min(kBigChunk, b.n - b.first);
    uint32_t size = 64;
    while (size < len) size <<= 1;
    const CellView cb = cell_records<kBinned>(p, b.cell, b.cs);
    // Keys (x bits, index) through the network instead of whole records:
    // half the shared-memory traffic and one comparison per exchange.
    for (uint32_t i = threadIdx.x; i < size; i += blockDim.x)
      s_key[i] = i < len ? (unsigned long long)__float_as_uint(cb[b.first + i].x) << 32 | i : ~0ull;
    __syncthreads();
    bitonic_network(s_key, size, [](unsigned long long a, unsigned long long b) { return a < b; });
    // molecules lined up in x (a lattice, a membrane, a release that does not
    // diffuse): stretches of equal keys too long to count over
    bool tied = false;
    for (uint32_t i = threadIdx.x; i + kTieStretch < len; i += blockDim.x)
      tied |= s_key[i] >> 32 == s_key[i + kTieStretch] >> 32;
    tied = __syncthreads_or(tied) != 0;
    if (tied) sort_tied_keys(s_key, size, len, cb, b.first);
    const bool done = b.n <= kBigChunk;
    float4* tmp = big_buffer(p, b.cs, 0) + b.first;
    for (uint32_t i = threadIdx.x; i < len; i += blockDim.x) {
      const unsigned long long key = s_key[i];
      const float4 r = cb[b.first + (uint32_t)key];
      // records with the same x bits are placed by all four words (by index
      // when identical), counted over their stretch of equal keys
      uint32_t at = i, lo = i, hi = i + 1u;
      const uint32_t xb = (uint32_t)(key >> 32);
      while (!tied && lo > 0 && (uint32_t)(s_key[lo - 1u] >> 32) == xb) --lo;
      while (!tied && hi < len && (uint32_t)(s_key[hi] >> 32) == xb) ++hi;
      if (hi - lo > 1u) {
        at = lo;
        for (uint32_t m = lo; m < hi; ++m) {
          const float4 q = cb[b.first + (uint32_t)s_key[m]];
          at += rec_less(q, r) || (m < i && rec_equal(q, r)) ? 1u : 0u;
        }
      }
      tmp[at] = r;
      if (done) nx[b.cs + b.first + at] = make_float4(r.x, r.y, r.z, __uint_as_float(rec_w(r) & ~kNewborn));
    }
  }
  // few units: several CTAs share one unit's records
  const uint32_t split = min(max(gridDim.x / units, 1u), kBigChunk / blockDim.x), piece = (kBigChunk + split - 1u) / split;
  uint32_t w = kBigChunk;
  for (uint32_t pass = 0; pass < passes; ++pass, w *= kBigWays) {
    if (!grid_barrier(c)) return false;
    for (uint32_t job = blockIdx.x; job < units * split; job += gridDim.x) {
      __syncthreads();
      if (threadIdx.x == 0) s_big = big_unit(p, nbig, job / split);
      __syncthreads();
      const BigCell b = s_big;
      if ((uint64_t)b.cs + b.n > p.capacity || b.n <= w) continue;
      const float4* src = big_buffer(p, b.cs, pass);
      float4* dst = big_buffer(p, b.cs, pass + 1u);
      const uint64_t span = (uint64_t)w * kBigWays;
      const bool last = span >= b.n;
      const uint32_t begin = b.first + (job % split) * piece;
      const uint32_t end = min(min(begin + piece, b.first + kBigChunk), b.n);
      for (uint32_t i = begin + threadIdx.x; i < end; i += blockDim.x) {
        const float4 e = src[i];
        const uint32_t lo = (uint32_t)(i / span * span), hi = (uint32_t)min((uint64_t)b.n, lo + span);
        const uint32_t own = (i - lo) / w;
        const uint32_t at = lo + (i - lo - own * w) + runs_rank(src, w, lo, hi, own, e);
        dst[at] = e;
        if (last) nx[b.cs + at] = make_float4(e.x, e.y, e.z, __uint_as_float(rec_w(e) & ~kNewborn));
      }
    }
  }
  return true;
}
// CTA-uniform status read (the large-cell kernel uses barriers).
__device__ __forceinline__ bool stop_block(const DevCtrl* c) {
  __shared__ uint32_t s_stop;
  if (threadIdx.x == 0) s_stop = ld_u32(&c->status);
  __syncthreads();
  const bool stop = s_stop != 0;
  __syncthreads();
  return stop;
}

// What the lanes of a warp look for in a list of records: their own
// seekers (lane on), the window on x that holds every partner of any of
// them, and the species any of them reacts with.
struct WarpSeekers {
  Seeker k;
  uint32_t ca;       // canonical slot of the lane's seeker
  uint32_t partners; // bit s: some lane's species reacts with species s (all ones when S > 32)
  float lo, hi;
};

__device__ __forceinline__ float warp_min(float v) {
#pragma unroll
  for (int d = 16; d; d >>= 1) v = fminf(v, __shfl_xor_sync(kFull, v, d));
  return v;
}

// The warp's seekers (lanes `on`) against records [m0, m1) of the list v.
// Each lane loads one record and drops it unless it lies in the warp's x
// window and is of a species some lane reacts with; the few that remain
// are passed around and tested by every lane, so records of species that
// do not react cost a thirty-second of a test.  kRun: v is the canonical
// run of a large cell (slots base + m), and only records past `after` (the
// lane's own index, or -1) count; else an ordinary cell of nn records.
template <bool kRun, class List>
__device__ void warp_sweep(const KParams& p, DevCtrl* c, const WarpSeekers& s, bool on, const List v,
                           uint32_t m0, uint32_t m1, uint32_t base, uint32_t nn, int64_t after) {
  constexpr uint32_t kBatch = 4;  // loads in flight per lane (k_pairs_big 350 -> 282 us on the release below)
  const uint32_t lane = lane_id();
  const float4 none = make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(kDead));
  for (uint32_t m = m0; m < m1; m += 32u * kBatch) {
    float4 q[kBatch];
#pragma unroll
    for (uint32_t u = 0; u < kBatch; ++u) q[u] = m1 - m > 32u * u + lane ? v[m + 32u * u + lane] : none;
#pragma unroll
    for (uint32_t u = 0; u < kBatch; ++u) {
      const uint32_t wq = rec_w(q[u]), sp = wq & kSpeciesMask;
      uint32_t ball = __ballot_sync(kFull, wq != kDead && !(wq & kNewborn) && q[u].x >= s.lo && q[u].x <= s.hi &&
                                               (p.S > 32u || ((s.partners >> sp) & 1u)));
      while (ball) {
        const uint32_t src = (uint32_t)(__ffs(ball) - 1), at = m + 32u * u + src;
        ball &= ball - 1u;
        float4 r;
        r.x = __shfl_sync(kFull, q[u].x, src);
        r.y = __shfl_sync(kFull, q[u].y, src);
        r.z = __shfl_sync(kFull, q[u].z, src);
        r.w = __shfl_sync(kFull, q[u].w, src);
        if (!on || (kRun && (int64_t)at <= after)) continue;
        // |dy| bounds the distance as |dx| does; the pair test decides
        if (fabsf(__fsub_rn(r.y, s.k.r.y)) > s.k.xlim) continue;
        const int32_t b = pair_reaction(p, s.k, r);
        if (b < 0) continue;
        emit<false>(p, c, p.cell_start, s.k, s.ca, base + (kRun ? at : canonical_rank(v, 0, nn, at, r)), b);
      }
    }
    __syncwarp();
  }
}

// The records of [lo, hi) of the run v whose |x| lies in [t0, t1], as
// [*a, *b); |x| rises over the range.  The whole warp searches both ends
// together, 16 probes each a round.
__device__ __forceinline__ void warp_range(const float4* v, uint32_t lo, uint32_t hi, float t0, float t1, uint32_t* a,
                                           uint32_t* b) {
  const uint32_t half = lane_id() >> 4, k = lane_id() & 15u;
  uint32_t l = lo, h = hi;  // the lane's half: 0 looks for the first >= t0, 1 for the first > t1
  while (__any_sync(kFull, l < h)) {
    const uint32_t n = h - l, step = (n + 15u) >> 4;
    bool below = false;
    if (n) {
      const float x = fabsf(v[l + min((k + 1u) * step, n) - 1u].x);  // last record of the lane's piece
      below = half ? x <= t1 : x < t0;
    }
    const uint32_t ball = __ballot_sync(kFull, below) >> (half * 16u) & 0xFFFFu;
    if (n) {
      const uint32_t skip = min((uint32_t)__popc(ball) * step, n);  // pieces passed over whole
      if (skip >= n) {
        l = h;
      } else {
        h = min(l + skip + step, h) - 1u;  // the piece's last record is not below
        l += skip;
      }
    }
  }
  *a = __shfl_sync(kFull, l, 0);
  *b = __shfl_sync(kFull, l, 16);
}

// The sweep of a canonical run [0, n) of a large cell, restricted to the
// warp's x window; segment `seg` of `nseg` takes its share of each of the
// two ranges (x >= 0 ascending, then x < 0 by rising |x|).  from: no record
// before it counts.
__device__ void run_sweep(const KParams& p, DevCtrl* c, const WarpSeekers& s, bool on, const float4* v, uint32_t n,
                          uint32_t base, uint32_t from, int64_t after, uint32_t seg, uint32_t nseg) {
  // first record with the sign bit set
  const float x0 = v[0].x, x1 = v[n - 1u].x;
  uint32_t npos = n;
  if (__float_as_uint(x0) & 0x80000000u) {
    npos = 0;
  } else if (__float_as_uint(x1) & 0x80000000u) {
    uint32_t lo = 0, hi = n;
    while (hi - lo > 0) {
      const uint32_t mid = (lo + hi) >> 1;
      if (__float_as_uint(v[mid].x) & 0x80000000u) hi = mid;
      else lo = mid + 1u;
    }
    npos = lo;
  }
  for (int part = 0; part < 2; ++part) {
    uint32_t a, b;
    if (part == 0) {
      if (npos == 0 || !(s.hi >= 0.0f)) continue;
      warp_range(v, 0, npos, fmaxf(s.lo, 0.0f), s.hi, &a, &b);
    } else {
      if (npos == n || !(s.lo <= 0.0f)) continue;
      warp_range(v, npos, n, fmaxf(-s.hi, 0.0f), -s.lo, &a, &b);
    }
    a = max(a, from);
    if (a >= b) continue;
    const uint32_t len = b - a;
    const uint32_t m0 = a + (uint32_t)((uint64_t)len * seg / nseg), m1 = a + (uint32_t)((uint64_t)len * (seg + 1u) / nseg);
    warp_sweep<true>(p, c, s, on, v, m0, m1, base, n, after);
  }
}

// The warp's seekers: x window (widened past the rounding of x +- xlim;
// xlim itself is 0.1% above the largest radius) and partner species.
__device__ __forceinline__ void warp_seekers(const KParams& p, WarpSeekers& s, bool on, const uint32_t* s_partners) {
  const float inf = __int_as_float(0x7f800000);
  const float wx = on ? 1.001f * s.k.xlim + 1e-6f * fabsf(s.k.r.x) : 0.0f;
  s.partners = __reduce_or_sync(kFull, on && p.S <= 32u ? s_partners[rec_w(s.k.r) & kSpeciesMask] : 0u);
  s.lo = warp_min(on ? s.k.r.x - wx : inf);
  s.hi = -warp_min(on ? -(s.k.r.x + wx) : inf);
}

// Neighbour cells that the largest binding radius of seeker k, in the cell
// (cx, cy, cz), reaches: bit (dz * 3 + dy) * 3 + dx, offsets 0..2 for -1..+1.
// An axis's distance counts only when it is within reach by itself (a record
// past its face by rounding has a negative distance).
__device__ __forceinline__ uint32_t big_mask(const KParams& p, const DevInstance& I, const Seeker& k, uint32_t cx,
                                             uint32_t cy, uint32_t cz) {
  const float inf = __int_as_float(0x7f800000);
  const float cl0 = I.cell[0], cl1 = I.cell[1], cl2 = I.cell[2];
  const float fx = __fsub_rn(__fmul_rn(__fsub_rn(k.r.x, I.lo[0]), I.inv[0]), (float)cx);
  const float fy = __fsub_rn(__fmul_rn(__fsub_rn(k.r.y, I.lo[1]), I.inv[1]), (float)cy);
  const float fz = __fsub_rn(__fmul_rn(__fsub_rn(k.r.z, I.lo[2]), I.inv[2]), (float)cz);
  const float need = k.max_r + p.prune_margin * fminf(cl0, fminf(cl1, cl2)), need2 = need * need;
  const float ex[3] = {cx > 0 ? fx * cl0 : inf, 0.0f, cx + 1u < I.dims[0] ? (1.0f - fx) * cl0 : inf};
  const float ey[3] = {cy > 0 ? fy * cl1 : inf, 0.0f, cy + 1u < I.dims[1] ? (1.0f - fy) * cl1 : inf};
  const float ez[3] = {cz > 0 ? fz * cl2 : inf, 0.0f, cz + 1u < I.dims[2] ? (1.0f - fz) * cl2 : inf};
  uint32_t mask = 0;
#pragma unroll
  for (int t = 0; t < 27; ++t) {
    const float dx = ex[t % 3], dy = ey[t / 3 % 3], dz = ez[t / 9];
    if (t != 13 && dx <= need && dy <= need && dz <= need && dx * dx + dy * dy + dz * dz <= need2) mask |= 1u << t;
  }
  return mask;
}

// Pairs of the large cells, on the canonical runs big_sort left.  Each pair
// that involves a large cell is tested once:
//   * inside the cell, against the later records of the run;
//   * with a large neighbour, from the lower-key cell of the two;
//   * with an ordinary neighbour, here, in either direction (k_pairs_cells
//     skips large forward neighbours).
// Warps take 32 seekers at a time, consecutive in x, so that their windows
// overlap.  Inside the cell these are 32 consecutive records.  For a
// neighbour cell the CTA first lists the unit's records within reach of it
// (a few per cent) and takes those 32 at a time: sweeping the neighbour for
// every block of 32 records on behalf of the one or two lanes near it took
// 160 of the kernel's 250 us.  With few units queued their work is spread
// over more CTAs and a sweep over several warps.
template <bool kBinned, uint32_t kThreads>
__device__ void big_pairs(const KParams& p, DevCtrl* c, uint32_t nbig, uint32_t units) {
  constexpr uint32_t kWarps = kThreads / 32u, kPer = kBigChunk / kThreads;  // records of a unit per thread
  static_assert(kPer * kWarps == 64u, "one warp scans the counts");
  __shared__ BigCell s_big;
  __shared__ uint32_t s_partners[32], s_union, s_count[kPer * kWarps + 1];
  __shared__ uint16_t s_list[kBigChunk];
  // species a species reacts with, as bits
  if (p.S <= 32u && threadIdx.x < p.S) {
    uint32_t m = 0;
    for (uint32_t t = 0; t < p.S; ++t) m |= (p.bim_table[threadIdx.x * p.S + t] >= 0 ? 1u : 0u) << t;
    s_partners[threadIdx.x] = m;
  }
  const uint32_t parts = min(max(2u * gridDim.x / units, 1u), kBigParts);
  const uint32_t nseg = parts > 1u ? kBigSegments : 1u;
  const uint32_t own = (parts + 1u) / 2u, turns = min((parts + 1u) / 2u, 13u);  // CTAs on the own cell, on neighbours
  const uint32_t warp = threadIdx.x >> 5, lane = lane_id();
  for (uint32_t job = blockIdx.x; job < units * (own + turns); job += gridDim.x) {
    __syncthreads();
    if (threadIdx.x == 0) {
      s_big = big_unit(p, nbig, job / (own + turns));
      s_union = 0;
    }
    __syncthreads();
    const BigCell bc = s_big;
    if ((uint64_t)bc.cs + bc.n > p.capacity || bc.first >= bc.n) continue;
    const float4* run = big_buffer(p, bc.cs, big_passes(bc.n));
    const uint32_t len = min(kBigChunk, bc.n - bc.first), part = job % (own + turns);
    WarpSeekers s;
    if (part < own) {
      for (uint32_t item = part * kWarps + warp; item < (len + 31u) / 32u * nseg; item += own * kWarps) {
        const uint32_t i0 = bc.first + item / nseg * 32u, i = i0 + lane;
        s.ca = bc.cs + i;
        const bool on = i < bc.n && seeker_init<false>(p, run[i], s.k);
        if (!__any_sync(kFull, on)) continue;
        warp_seekers(p, s, on, s_partners);
        run_sweep(p, c, s, on, run, bc.n, bc.cs, i0 + 1u, (int64_t)i, item % nseg, nseg);
      }
      continue;
    }
    // the records near each neighbour; every record of a cell has its instance
    const DevInstance& I = p.inst[rec_w(run[0]) >> 16];
    const uint32_t d0 = I.dims[0], d1 = I.dims[1], local = bc.cell - I.cell_base;
    const uint32_t cx = local % d0, cy = local / d0 % d1, cz = local / d0 / d1;
    uint32_t mask[kPer], any = 0;
#pragma unroll
    for (uint32_t e = 0; e < kPer; ++e) {
      const uint32_t i = e * kThreads + threadIdx.x;
      mask[e] = i < len && seeker_init<false>(p, run[bc.first + i], s.k) ? big_mask(p, I, s.k, cx, cy, cz) : 0u;
      any |= mask[e];
    }
    any = __reduce_or_sync(kFull, any);
    if (lane == 0 && any) atomicOr(&s_union, any);
    __syncthreads();
    uint32_t todo = s_union;
    for (uint32_t turn = 0; todo; ++turn) {  // the same in every thread of the CTA
      const uint32_t t = (uint32_t)(__ffs(todo) - 1);
      todo &= todo - 1u;
      if (turn % turns != part - own) continue;
      const uint32_t nkey =
          bc.cell + (uint32_t)(((int)(t / 9u) - 1) * (int)d1 + ((int)(t / 3u % 3u) - 1)) * d0 + t % 3u - 1u;
      const uint32_t ns = ld_step(&p.cell_start[nkey]), nn = ld_step(&p.cell_start[nkey + 1]) - ns;
      const bool large = nn > kBigCell;
      if (nn == 0 || (large && t < 13u)) continue;  // a large lower-key neighbour finds the pair itself
#pragma unroll
      for (uint32_t e = 0; e < kPer; ++e) {
        const uint32_t ball = __ballot_sync(kFull, (mask[e] >> t) & 1u);
        if (lane == 0) s_count[e * kWarps + warp] = __popc(ball);
      }
      __syncthreads();
      if (warp == 0) {  // exclusive scan of the 64 counts
        const uint32_t a = s_count[2u * lane], b = s_count[2u * lane + 1u];
        uint32_t incl = a + b;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const uint32_t v = __shfl_up_sync(kFull, incl, d);
          if (lane >= (uint32_t)d) incl += v;
        }
        s_count[2u * lane] = incl - a - b;
        s_count[2u * lane + 1u] = incl - b;
        if (lane == 31) s_count[kPer * kWarps] = incl;
      }
      __syncthreads();
#pragma unroll
      for (uint32_t e = 0; e < kPer; ++e) {
        const bool hit = (mask[e] >> t) & 1u;
        const uint32_t ball = __ballot_sync(kFull, hit);
        if (hit) s_list[s_count[e * kWarps + warp] + __popc(ball & ((1u << lane) - 1u))] = (uint16_t)(e * kThreads + threadIdx.x);
      }
      __syncthreads();
      const uint32_t m = s_count[kPer * kWarps], blocks = (m + 31u) / 32u;
      const uint32_t cut = large ? max(kWarps / blocks, 1u) : 1u;
      for (uint32_t item = warp; item < blocks * cut; item += kWarps) {
        const uint32_t j = item / cut * 32u + lane;
        const uint32_t i = bc.first + (j < m ? s_list[j] : 0u);
        s.ca = bc.cs + i;
        const bool on = j < m && seeker_init<false>(p, run[i], s.k);
        if (!__any_sync(kFull, on)) continue;
        warp_seekers(p, s, on, s_partners);
        if (large) run_sweep(p, c, s, on, big_buffer(p, ns, big_passes(nn)), nn, ns, 0u, -1, item % cut, cut);
        else warp_sweep<false>(p, c, s, on, cell_records<kBinned>(p, nkey, ns), 0u, nn, ns, nn, -1);
      }
      __syncthreads();  // s_count and s_list are no longer read
    }
  }
}

// Move the events of the committed step into the cumulative counters.
__device__ __forceinline__ void commit_events(const KParams& p) {
  const uint32_t n = p.n_inst * p.R;
  for (uint32_t e = threadIdx.x; e < n; e += blockDim.x) {
    const unsigned long long v = __ldcg(&p.pending[e]), before = __ldcg(&p.events[e]);
    if (v) {
      p.events[e] = before + v;
      p.pending[e] = 0;
    }
  }
}

// Candidate pairs above which the matching runs over the whole grid.
constexpr uint32_t kMatchOneCta = 8192;

// Rounds of locally dominant pairs over K candidates, by the threads of one
// CTA (kGrid false: __syncthreads, counters in shared memory) or of the
// whole cooperative grid (kGrid: grid barriers, counters in DevCtrl).
//
// In round r a pending pair (i, j) offers tag(r) | j to best[i] and
// tag(r) | i to best[j] (atomicMin); the pairs that are each other's
// minimum are matched (best = 0 at both ends), and a pending pair with a
// matched end is dropped.  tag(r) falls with r, so values of earlier rounds
// lose every minimum and best needs no reset between rounds: two passes and
// two barriers per round.  The pairs still pending are compacted, with
// their ends, into one of two lists for the next round.  Each round matches
// the smallest pending pair at least, so there are at most K rounds; the
// result is the greedy matching in (lower slot, upper slot) order.
// False when a grid barrier ran out (kStatTimeout is set).
template <bool kGrid>
__device__ bool match_rounds(const KParams& p, DevCtrl* c, uint32_t K, uint32_t* next) {
  DevPair* pr = p.pairs;
  unsigned long long* best = p.best;
  uint4* lists[2] = {p.match_list, p.match_list + p.pair_cap};
  const uint32_t tid = kGrid ? blockIdx.x * blockDim.x + threadIdx.x : threadIdx.x;
  const uint32_t nthr = kGrid ? gridDim.x * blockDim.x : blockDim.x;
  const uint32_t lane = lane_id();
  auto sync = [&]() -> bool {
    if (kGrid) return grid_barrier(c);
    __syncthreads();
    return true;
  };
  // Each thread takes kMatchIlp list entries at a time, so that their
  // loads (entry, then the two matcher words) are in flight together.
  constexpr uint32_t kMatchIlp = 4;
  uint32_t n_pend = K;
  for (uint32_t round = 0; n_pend > 0 && round <= K; ++round) {
    const uint4* in = round == 0 ? nullptr : lists[(round - 1) & 1];
    uint4* out = lists[round & 1];
    const unsigned long long tag = (unsigned long long)(0xFFFFFFFFu - round) << 32;
    const uint32_t span = nthr * kMatchIlp;
    // pass A: offers, except from pairs with an end matched in an earlier round
    for (uint32_t e0 = tid; e0 < n_pend; e0 += span) {
      uint4 ent[kMatchIlp];
      unsigned long long bi[kMatchIlp], bj[kMatchIlp];
#pragma unroll
      for (uint32_t u = 0; u < kMatchIlp; ++u) {
        const uint32_t e = e0 + u * nthr;
        if (e < n_pend) ent[u] = in ? in[e] : make_uint4(e, pr[e].i, pr[e].j, 0u);
      }
#pragma unroll
      for (uint32_t u = 0; u < kMatchIlp; ++u) {
        bi[u] = bj[u] = kFree64;
        if (round > 0 && e0 + u * nthr < n_pend) {
          bi[u] = __ldcg(&best[ent[u].y]);
          bj[u] = __ldcg(&best[ent[u].z]);
        }
      }
#pragma unroll
      for (uint32_t u = 0; u < kMatchIlp; ++u)
        if (e0 + u * nthr < n_pend && bi[u] != 0ull && bj[u] != 0ull) {
          atomicMin(&best[ent[u].y], tag | ent[u].z);
          atomicMin(&best[ent[u].z], tag | ent[u].y);
        }
    }
    if (!sync()) return false;
    // pass B: match mutual minima, drop pairs with a matched end, keep the
    // rest (the loop runs over whole warps: the ballot needs every lane)
    const uint32_t warp_first = tid - lane;
    for (uint32_t e0 = warp_first; e0 < n_pend; e0 += span) {
      uint4 ent[kMatchIlp];
      unsigned long long bi[kMatchIlp], bj[kMatchIlp];
#pragma unroll
      for (uint32_t u = 0; u < kMatchIlp; ++u) {
        const uint32_t e = e0 + u * nthr + lane;
        if (e < n_pend) ent[u] = in ? in[e] : make_uint4(e, pr[e].i, pr[e].j, 0u);
      }
#pragma unroll
      for (uint32_t u = 0; u < kMatchIlp; ++u)
        if (e0 + u * nthr + lane < n_pend) {
          bi[u] = __ldcg(&best[ent[u].y]);
          bj[u] = __ldcg(&best[ent[u].z]);
        }
#pragma unroll
      for (uint32_t u = 0; u < kMatchIlp; ++u) {
        bool keep = false;
        if (e0 + u * nthr + lane < n_pend) {
          if (bi[u] == (tag | ent[u].z) && bj[u] == (tag | ent[u].y)) {
            best[ent[u].y] = 0ull;
            best[ent[u].z] = 0ull;
            pr[ent[u].x].state = 1;
          } else if (bi[u] == 0ull || bj[u] == 0ull) {
            pr[ent[u].x].state = 2;
          } else {
            keep = true;
          }
        }
        // survivors to the next list, one atomic per warp
        const uint32_t ball = __ballot_sync(kFull, keep);
        uint32_t base = 0;
        if (ball && lane == 0) base = atomicAdd(&next[round & 1], (uint32_t)__popc(ball));
        base = __shfl_sync(kFull, base, 0);
        if (keep) out[base + __popc(ball & ((1u << lane) - 1u))] = ent[u];
      }
    }
    if (!sync()) return false;
    n_pend = kGrid ? *(volatile uint32_t*)&next[round & 1] : next[round & 1];
    // The other counter was last read before this round's first barrier,
    // and the next round appends to it only after its own first barrier;
    // this round's counter is reset only after the next round's second
    // barrier, when every thread has read it.  No third barrier is needed.
    if (tid == 0) next[(round + 1) & 1] = 0;
  }
  return true;
}

// Candidate pairs up to which one CTA decides the matching in shared memory.
constexpr uint32_t kMatchFew = 256;

// Shared words of the matcher.
struct MatchShared {
  uint32_t next[2], deaths;
  uint2 pair[kMatchFew];
  uint8_t state[kMatchFew];  // DevPair::state
};

// The greedy matching of K <= kMatchFew pairs, one per thread (thread k < K
// holds pair k), as rounds of locally dominant pairs; every thread of the
// CTA calls it.  Returns the state of the thread's pair.  Most steps of a
// dilute system have a handful of pairs and none in conflict, so one pass
// over the others settles them, without the matcher words in global memory
// and their round trips (k_match 14.3 -> 13.2 us on the 16M c3 step, where
// most of it is the launch).
__device__ __forceinline__ uint32_t match_few(uint32_t K, uint32_t i, uint32_t j, MatchShared& sh) {
  const uint32_t k = threadIdx.x;
  uint32_t state = k < K ? 0u : 2u;
  if (k < K) {
    sh.pair[k] = make_uint2(i, j);
    sh.state[k] = 0;
  }
  __syncthreads();
  for (uint32_t round = 0; round <= K; ++round) {
    // a pair is accepted when no undecided pair with a common end comes
    // before it in (lower slot, upper slot) order
    bool first = state == 0;
    if (first)
      for (uint32_t m = 0; m < K; ++m) {
        const uint2 q = sh.pair[m];
        if (m == k || !(q.x == i || q.y == i || q.x == j || q.y == j) || sh.state[m] != 0) continue;
        if (q.x < i || (q.x == i && q.y < j)) first = false;
      }
    __syncthreads();
    if (first) {
      state = 1;
      sh.state[k] = 1;
    }
    if (!__syncthreads_or(state == 0)) break;
    // pairs that lost an end are dropped
    if (state == 0)
      for (uint32_t m = 0; m < K; ++m) {
        const uint2 q = sh.pair[m];
        if (sh.state[m] == 1 && (q.x == i || q.y == i || q.x == j || q.y == j)) state = 2;
      }
    __syncthreads();
    if (k < K && state == 2) sh.state[k] = 2;
    if (!__syncthreads_or(state == 0)) break;
  }
  return state;
}

// Resolve the candidate pairs into a matching, apply the reactions and
// commit the step.  Each particle reacts at most once; the pairs accepted
// are those of the greedy scan in (lower slot, upper slot) order, found in
// parallel as rounds of locally dominant pairs (match_rounds).  Launched
// cooperatively over the grid: with at most kMatchOneCta candidates (most
// steps) one CTA does everything (grid false); with more, every CTA takes
// part in the rounds and the products, and CTA 0 commits.  False when a grid
// barrier ran out.  mine: match_pair(), asked for before K was known.
__device__ __forceinline__ DevPair match_pair(const KParams& p) {
  return threadIdx.x < min(kMatchFew, p.pair_cap) ? p.pairs[threadIdx.x] : DevPair{0u, 0u, 0u, 0u};
}

template <bool kSurf>
__device__ __forceinline__ bool match_commit(const KParams& p, DevCtrl* c, uint32_t K, const DevPair& mine, bool grid,
                                             MatchShared& sh) {
  // read before the barriers below; one thread advances it at the end
  const uint32_t step_now = (uint32_t)*(volatile uint64_t*)&c->step;
  const uint32_t cur = ld_u32(&c->cur);
  float4* __restrict__ nx = next_state(p, cur);
  DevPair* pr = p.pairs;
  unsigned long long* best = p.best;
  if (threadIdx.x < 2) sh.next[threadIdx.x] = 0;
  if (threadIdx.x == 0) sh.deaths = 0;

  // Products of an accepted pair: at the D-weighted reaction point,
  // displaced along a random direction when the reaction has an unbinding
  // radius.  br: the pair's reaction; ri, rj: the records in its slots.
  auto react = [&](const DevPair& q, DevBim br, const float4& ri, const float4& rj) {
    const uint32_t inst = q.b >> 16;
    const DevInstance& I = p.inst[inst];
    if (br.next >= 0) {
      // competing reactions of this pair: the one whose share of the
      // pair's summed rate holds the coin
      const uint32_t base_new = p.cell_start[I.cell_base];
      const U4 u = philox(U4{q.i - base_new, p.inst_step[inst], kTagBimChannel, q.j - base_new}, I.key_lo,
                          I.key_hi);
      const float coin = u24_to_unit(u.x);
      for (uint32_t hop = 0; hop < p.B && !(coin < br.thresh) && br.next >= 0; ++hop)
        br = p.bim[I.block * p.B + (uint32_t)br.next];
    }
    const bool i_first = (int32_t)(rec_w(ri) & kSpeciesMask) == br.react0;
    const uint32_t m1 = i_first ? q.i : q.j, m2 = i_first ? q.j : q.i;
    const float4 p1 = i_first ? ri : rj, p2 = i_first ? rj : ri;
    const float rx = __fmaf_rn(br.x, p1.x, __fmul_rn(br.omx, p2.x));
    const float ry = __fmaf_rn(br.x, p1.y, __fmul_rn(br.omx, p2.y));
    const float rz = __fmaf_rn(br.x, p1.z, __fmul_rn(br.omx, p2.z));
    float dx = 0.0f, dy = 0.0f, dz = 0.0f;
    if (br.off0 != 0.0f || br.off1 != 0.0f) {
      const uint32_t base_new = p.cell_start[I.cell_base];
      unit_vector(q.i - base_new, p.inst_step[inst], kTagBimDir, q.j - base_new, I.key_lo, I.key_hi, dx, dy,
                  dz);
    }
    uint32_t dead = 0;
    const float4 none = make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(kDead));
    float4 n1 = none, n2 = none;
    // each product moves from the reaction point by its offset, through the
    // surfaces when there are any, then the walls
    auto place = [&](int32_t prod, float off, float4& out) {
      if (prod < 0) {
        ++dead;
        return;
      }
      float ex = reflect(__fmaf_rn(off, dx, rx), I.lo[0], I.hi[0]);
      float ey = reflect(__fmaf_rn(off, dy, ry), I.lo[1], I.hi[1]);
      float ez = reflect(__fmaf_rn(off, dz, rz), I.lo[2], I.hi[2]);
      if (kSurf && off != 0.0f && !surface_walk(p, I, (uint32_t)prod, V3{rx, ry, rz}, ex, ey, ez)) {
        ++dead;
        return;
      }
      out = make_float4(ex, ey, ez, __uint_as_float(pack_w(inst, (uint32_t)prod)));
    };
    place(br.prod0, br.off0, n1);
    place(br.prod1, br.off1, n2);
    nx[m1] = n1;
    nx[m2] = n2;
    atomicAdd(&p.pending[(size_t)inst * p.R + br.rxn], 1ull);
    if (dead) atomicAdd(&sh.deaths, dead);
  };

  // the pair's reaction and records: asked for together, before they are
  // needed where that can be
  auto reaction_of = [&](const DevPair& q) {
    const uint32_t block = p.n_inst == 1u ? p.inst0.block : p.inst[q.b >> 16].block;
    return p.bim[block * p.B + (q.b & 0xFFFFu)];
  };
  uint32_t done = 0;  // pairs settled without the rounds in global memory
  if (!grid && K <= kMatchFew) {
    done = K;
    if (K > 0) {
      DevPair q{0u, 0u, 0u, 0u};
      DevBim br{};
      float4 ri = make_float4(0.0f, 0.0f, 0.0f, 0.0f), rj = ri;
      if (threadIdx.x < K) {
        q = mine;
        br = reaction_of(q);
        ri = nx[q.i];
        rj = nx[q.j];
      }
      const uint32_t state = match_few(K, q.i, q.j, sh);
      if (threadIdx.x < K) {
        pr[threadIdx.x].state = state;
        if (state == 1u) react(q, br, ri, rj);
      }
    }
  } else if (grid) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      c->match_next[0] = c->match_next[1] = 0;
      c->match_deaths = 0;
    }
    if (p.match_withhold && blockIdx.x == 0) return false;  // test switch: the other CTAs' waits run out
    if (!grid_barrier(c)) return false;
    if (!match_rounds<true>(p, c, K, c->match_next)) return false;
  } else {
    __syncthreads();
    match_rounds<false>(p, c, K, sh.next);
  }
  const uint32_t tid = grid ? blockIdx.x * blockDim.x + threadIdx.x : threadIdx.x;
  const uint32_t nthr = grid ? gridDim.x * blockDim.x : blockDim.x;
  for (uint32_t k = done + tid; k < K; k += nthr) {
    const DevPair q = pr[k];
    if (q.state == 1) react(q, reaction_of(q), nx[q.i], nx[q.j]);
  }
  for (uint32_t k = done + tid; k < K; k += nthr) {
    best[pr[k].i] = kFree64;
    best[pr[k].j] = kFree64;
  }
  __syncthreads();
  if (grid) {
    // every CTA's products and deaths are in before CTA 0 commits
    if (threadIdx.x == 0 && sh.deaths) atomicAdd(&c->match_deaths, sh.deaths);
    if (!grid_barrier(c)) return false;
    if (blockIdx.x != 0) return true;
    if (threadIdx.x == 0) sh.deaths = *(volatile uint32_t*)&c->match_deaths;
    __syncthreads();
  }
  // the commit: events from the first threads, instances from the last,
  // the control words from one between, so that their loads overlap
  commit_events(p);
  for (uint32_t inst = blockDim.x - 1u - threadIdx.x; inst < p.n_inst; inst += blockDim.x) {
    const uint32_t base = p.cell_start[p.inst[inst].cell_base];
    advance_instance_step(p, inst, step_now);
    p.inst_slot_base[inst] = base;
  }
  if (threadIdx.x == blockDim.x / 2u) {
    const uint32_t n_sorted = ld_u32(&c->n_sorted), steps_done = ld_u32(&c->steps_done);
    c->n_pairs_last = K;
    c->n_pairs = 0;
    c->big_queue = 0;
    c->big_max = 0;
    c->n_surf = 0;
    c->surf_ticket = 0;
    c->deaths_last = sh.deaths;
    c->n_slots = n_sorted;
    c->n_virtual = 0;
    c->cur = cur ^ 1u;
    *(volatile uint64_t*)&c->step = (*(volatile uint64_t*)&c->step) + 1u;
    c->steps_done = steps_done + 1u;
  }
  return true;
}

}  // namespace
}  // namespace bd
