// bd_resident.cu -- several timesteps of a small binned system in one launch.
//
// One step as a chain of kernels (k_bin, k_scan, k_pairs_cells, k_pairs_big,
// k_match) costs 21 us however small the system: launches, their ramps and the
// chains of dependent loads at the head of each kernel, not the work.  Here
// the whole step runs in one cooperative kernel that stays resident for many
// steps, and what bounds it is round trips to L2 (0.4 us each): a barrier of
// the grid is three of them.  c2 steps, chain and here, us: 1,000 particles
// 21.9 / 11.0, 10,000 22.7 / 12.7, 40,000 25.9 / 20.3, 80,000 27.3 / 27.5, on at
// most a quarter of the SMs (on all of them 17.0 at 40,000 and 23.6 at 100,000,
// but then nothing else runs beside it); 100,000 at 8 a cell 38.8 / 32.4, at 20
// 78.6 / 46.7, where the chain's warps take turns of 32 cells.  So a step has as few barriers as it can:
// two when it has no candidate pairs.
//   * The cell scan is not a phase: after binning every CTA scans all counts
//     for itself into shared memory (up to kSmallCells cells; above that the
//     CTAs scan a range each, at the price of two more barriers).
//   * Barriers carry what the phase met (candidate pairs, large cells, a
//     failure) in the arrival word, so nobody reads control words after one.
//   * With one instance, a step without candidates is committed by CTA 0
//     while the others are already binning the next: they know the next
//     step's state without reading it.
//   * The cell counts alternate between two arrays, so that one is cleared
//     while the other is read.
// The phases are the functions of bd_step.cuh, so the results are those of
// the kernel chain bit for bit.
//
// Every wait is bounded.  A CTA that fails, times out or finds a status bit
// says so in the arrival word and leaves; the others leave when they see it.
// They need not leave at the same barrier: the step in flight is not
// committed, and no CTA can reach the phase that overwrites the state the
// step started from before every CTA has passed the barrier after it.
#define BD_PHASES_IN_ONE_LAUNCH
#include "bd_step.cuh"

#include <algorithm>

namespace bd {
namespace {

// CTAs of 1024 threads, one per SM: a barrier of 608 CTAs of 256
// threads took about twice the time of one of 152.
constexpr int kThreads = 1024, kWarps = kThreads / 32;
// Cells whose starts every CTA keeps in shared memory (128 KiB beside the
// pair search's 74).
constexpr uint32_t kSmallCells = 32768;

// The arrival word: CTAs arrived since the launch (bits 0-17), then sums over
// the arrivals that brought candidate pairs (18-32), large cells (33-47) and
// a matching for the whole grid (48-55), and of those that failed (56-63).
// kResidentSteps steps of at most seven barriers of 255 CTAs fit.
constexpr uint32_t kPairsBit = 18, kBigBit = 33, kGridBit = 48, kFailedBit = 56;
constexpr unsigned long long kFailed = 1ull << kFailedBit;
static_assert(kResidentSteps * 7u * 255u < (1u << kPairsBit) && kResidentSteps * 255u < (1u << 15) &&
                  kResidentSteps < 256u,
              "arrival word fields");

// What a barrier reports: the fields of the arrival word to look at.  A CTA
// that polls late may already see arrivals at the next barrier, so a field
// is looked at only at barriers after which no CTA can add to it before
// every CTA has gone on.
enum Report : unsigned long long {
  kNothing = 0,
  kPhaseReport = ((1ull << kGridBit) - 1ull) & ~((1ull << kPairsBit) - 1ull),
  kGridReport = (1ull << kFailedBit) - (1ull << kGridBit),
};
enum Met : uint32_t { kMetPairs = 1, kMetBig = 2, kMetGrid = 4, kMetFailure = 8 };

struct Barrier {
  unsigned long long* word;
  unsigned long long seen;  // the reported fields as of their last report (thread 0)
  uint32_t target;          // arrivals that complete the next barrier (thread 0)
};

// Barrier of the grid.  Returns what any CTA met in the phase it ends, the
// same in every CTA but for kMetFailure (see above), on which the caller
// leaves.  The arrival releases the CTA's writes, the polls acquire the
// others'.
__device__ __forceinline__ uint32_t phase_barrier(DevCtrl* c, Barrier& b, Report report) {
  __shared__ uint32_t s_met;
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile uint32_t* flags = phase_flags();
    unsigned long long add = 1ull;
    if (flags[kFlagPairs]) add += 1ull << kPairsBit;
    if (flags[kFlagBig]) add += 1ull << kBigBit;
    if (flags[kFlagGrid]) add += 1ull << kGridBit;
    if (flags[kFlagStop]) add += kFailed;
    flags[kFlagPairs] = flags[kFlagBig] = flags[kFlagGrid] = 0u;
    unsigned long long w = 0;
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(b.word), "l"(add) : "memory");
    uint32_t met = kMetFailure;
    for (uint32_t polls = 0; polls <= kGridSpins; ++polls) {
      asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(b.word) : "memory");
      if (w >= kFailed) break;
      if ((uint32_t)w % (1u << kPairsBit) >= b.target) {
        met = 0;
        break;
      }
    }
    if (met && w < kFailed) {  // the wait ran out
      atomicOr(&c->status, kStatTimeout);
      asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(b.word), "l"(kFailed) : "memory");
    }
    const unsigned long long news = (w ^ b.seen) & report;
    if (news >> kPairsBit & 0x7FFFu) met |= kMetPairs;
    if (news >> kBigBit & 0x7FFFu) met |= kMetBig;
    if (news >> kGridBit & 0xFFu) met |= kMetGrid;
    b.seen ^= news;
    b.target += gridDim.x;
    s_met = met;
  }
  __syncthreads();
  return s_met;  // written again only after the next barrier's first __syncthreads
}

// The last CTA to leave resets the arrival word for the next launch.
__device__ __forceinline__ void leave(DevCtrl* c) {
  __syncthreads();
  if (threadIdx.x != 0) return;
  __threadfence();
  if (atomicAdd(&c->res_left, 1u) == gridDim.x - 1u) {
    c->res_word = 0ull;
    c->res_left = 0u;
  }
}

// Counts [lo, hi) (lo a multiple of 4, hi - lo <= kSmallCells) scanned by the
// CTA into s[0, hi - lo]: s[i] = the counts of the first i cells.  Returns
// their sum.  Loads are 16 bytes a thread and all in flight together; each
// thread then scans a run of its own in shared memory, of odd length so that
// the runs start in different banks.
__device__ __forceinline__ uint32_t scan_counts(const uint32_t* counts, uint32_t lo, uint32_t hi, uint32_t* s) {
  const uint32_t n = hi - lo;
#pragma unroll 4
  for (uint32_t i = threadIdx.x * 4u; i < n; i += kThreads * 4u)
    *reinterpret_cast<uint4*>(s + i) = __ldcg(reinterpret_cast<const uint4*>(counts + lo + i));
  __syncthreads();
  const uint32_t q = ((n + kThreads - 1u) / kThreads) | 1u;
  const uint32_t a = min(threadIdx.x * q, n), b = min(a + q, n);
  uint32_t sum = 0;
  for (uint32_t i = a; i < b; ++i) sum += s[i];
  uint32_t total;
  uint32_t run = cta_scan(sum, &total);
  for (uint32_t i = a; i < b; ++i) {
    const uint32_t v = s[i];
    s[i] = run;
    run += v;
  }
  if (threadIdx.x == kThreads - 1u) s[n] = total;
  __syncthreads();
  return total;
}

// The parts that few steps reach, or that one CTA runs, are calls: inlined,
// their registers made the streaming phases spill more.  (At the 64 registers
// of 1,024 threads every variant spills some: 204 to 328 bytes of stores.)
template <bool kHasBim>
__device__ __noinline__ bool big_cells(const KParams& p, DevCtrl* c, unsigned long long* s_key) {
  const unsigned long long queued = __ldcg(&c->big_queue);
  const uint32_t nbig = min((uint32_t)queued, p.big_cap), units = (uint32_t)(queued >> 32);
  if (p.big_scratch_cap < 2ull * p.capacity) {
    if (threadIdx.x == 0) raise(c, kStatScratch);
    return true;  // the next barrier ends the step
  }
  if (!big_sort<true>(p, c, nbig, units, s_key)) return false;
  if (!kHasBim) return true;
  if (!grid_barrier(c)) return false;
  big_pairs<true, kThreads>(p, c, nbig, units);
  return true;
}

__device__ __noinline__ bool match_step(const KParams& p, DevCtrl* c, uint32_t K, const DevPair& mine, bool grid,
                                        MatchShared& sh) {
  return match_commit<false>(p, c, K, mine, grid, sh);
}

template <bool kTable, bool kHasBim, bool kSingle>
__global__ void __launch_bounds__(kThreads, 1) k_resident(const __grid_constant__ KParams p, uint32_t nsteps) {
  __shared__ DevSpecies s_species[kSingle ? kCtxSpecies : 1];
  __shared__ DevUni s_uni[kSingle ? kCtxUni : 1];
  __shared__ PairSpecies<kSingle> s_pair_species;
  __shared__ MatchShared s_match;
  __shared__ unsigned long long s_events[kSingle ? kResidentReactions : 1];
  __shared__ uint32_t s_before;
  __shared__ DeferBuffer s_defer;  // not used: no surfaces here
  // the pair search's working sets or the large-cell sort's keys, then the
  // cell starts
  extern __shared__ __align__(16) unsigned char s_phase[];
  uint32_t* s_start = reinterpret_cast<uint32_t*>(
      s_phase + (sizeof(PairShared<kHasBim, kWarps>) > kBigChunk * 8u ? sizeof(PairShared<kHasBim, kWarps>)
                                                                      : kBigChunk * 8u));
  // The parameters for the functions that are called: by reference to the
  // kernel's own they would be loads that miss L1 after every barrier.
  __shared__ KParams s_params;
  for (uint32_t i = threadIdx.x; i < sizeof(KParams) / 4u; i += kThreads)
    reinterpret_cast<uint32_t*>(&s_params)[i] = reinterpret_cast<const uint32_t*>(&p)[i];
  PairShared<kHasBim, kWarps>& s_pair = *reinterpret_cast<PairShared<kHasBim, kWarps>*>(s_phase);
  DevCtrl* c = p.ctrl;
  uint32_t cur = ld_u32(&c->cur), n_real = ld_u32(&c->n_slots);
  uint64_t step = *(volatile uint64_t*)&c->step;
  if (threadIdx.x < kPhaseFlags) phase_flags()[threadIdx.x] = 0u;
  SingleCtx ctx{};
  if (kSingle) ctx = single_ctx(p, s_species, s_uni);
  const uint32_t target = ld_u32(&p.inst_target[0]);  // one instance
  pair_species<kSingle>(p, s_pair_species);
  Barrier bar{&c->res_word, 0ull, gridDim.x};
  // A step before this launch failed: nothing to do.  (If another CTA of this
  // launch has just set the bit, the others learn of it at the barrier.)
  if (threadIdx.x == 0 && ld_u32(&c->status)) flag_phase(kFlagStop);
  __syncthreads();
  if (*(volatile uint32_t*)(phase_flags() + kFlagStop)) nsteps = 0;
  const bool small = p.n_cells <= kSmallCells;
  for (uint32_t k = 0; k < nsteps; ++k) {
    uint32_t* counts = p.cell_count + (step & 1u) * (size_t)p.count_stride;
    uint32_t* other = p.cell_count + (~step & 1u) * (size_t)p.count_stride;
    bin_records<kTable, kSingle, 0, true>(p, c, ctx, s_defer, cur_state(p, cur), n_real, counts);
    if (p.Z && blockIdx.x == gridDim.x - 1u) zeroth_births<kSingle>(s_params, c, ctx, counts);
    if (p.scan_withhold && blockIdx.x == 0) {  // test switch: CTA 0 never arrives
      if (gridDim.x == 1 && threadIdx.x == 0) atomicOr(&c->status, kStatTimeout);
      return;
    }
    if (threadIdx.x == 0) s_pair.ticket = 0u;
    if (phase_barrier(c, bar, kNothing) & kMetFailure) break;
    uint32_t total = 0;
    if (small) {
      total = scan_counts(counts, 0, p.n_cells, s_start);
    } else {
      // each CTA scans a range and shifts it once all ranges' sums are
      // known; then every start is in p.cell_start
      const uint32_t per = ((p.n_cells + gridDim.x - 1u) / gridDim.x + 3u) & ~3u;
      const uint32_t lo = min(blockIdx.x * per, p.n_cells), hi = min(lo + per, p.n_cells);
      const uint32_t own = scan_counts(counts, lo, hi, s_start);
      if (threadIdx.x == 0) p.tile_sums[blockIdx.x] = own;
      if (phase_barrier(c, bar, kNothing) & kMetFailure) break;
      const uint32_t t = threadIdx.x < gridDim.x ? __ldcg(&p.tile_sums[threadIdx.x]) : 0u;
      const uint32_t ex = cta_scan(t, &total);
      if (threadIdx.x == blockIdx.x) s_before = ex;
      __syncthreads();
      const uint32_t before = s_before;
      for (uint32_t i = lo + threadIdx.x; i < hi; i += kThreads) p.cell_start[i] = s_start[i - lo] + before;
      if (hi == p.n_cells && threadIdx.x == 0) p.cell_start[p.n_cells] = total;
      if (phase_barrier(c, bar, kNothing) & kMetFailure) break;
    }
    if (blockIdx.x == 0) {
      if (threadIdx.x == 0) {
        c->n_sorted = total;
        if (small) p.cell_start[p.n_cells] = total;
        if (total > p.capacity) raise(c, kStatCapacity);
      }
      // first- and zeroth-order events of the step, final since the last
      // barrier; they count when the step commits
      if (kSingle && threadIdx.x < p.R) {
        s_events[threadIdx.x] = __ldcg(&p.pending[threadIdx.x]);
        p.pending[threadIdx.x] = 0ull;
      }
    }
    if (total > p.capacity) break;  // the same in every CTA
    pair_cells<kHasBim, true, kSingle, true, kWarps>(p, c, next_state(p, cur), kSingle ? advancing(ctx.flags) : true,
                                                     s_pair,
                                                     s_pair_species, small ? s_start : p.cell_start, other);
    uint32_t met = phase_barrier(c, bar, kPhaseReport);
    if (met & kMetFailure) break;
    if (met & kMetBig) {
      if (!big_cells<kHasBim>(s_params, c, reinterpret_cast<unsigned long long*>(s_phase))) return;
      if (phase_barrier(c, bar, kPhaseReport) & kMetFailure) break;
    }
    if (kSingle && !(met & (kMetPairs | kMetBig))) {
      // no candidates: CTA 0 commits, the others go on
      if (blockIdx.x == 0) {
        if (threadIdx.x < p.R && s_events[threadIdx.x])
          p.events[threadIdx.x] = __ldcg(&p.events[threadIdx.x]) + s_events[threadIdx.x];
        if (threadIdx.x == 0) {
          c->n_pairs_last = 0;
          c->deaths_last = 0;
          c->n_slots = total;
          c->n_virtual = 0;
          c->cur = cur ^ 1u;
          *(volatile uint64_t*)&c->step = step + 1u;
          c->steps_done = ld_u32(&c->steps_done) + 1u;
          if (advancing(ctx.flags)) {
            p.inst_step[0] = ctx.step + 1u;
            if (ctx.step + 1u >= target) {
              p.inst_flags[0] = ctx.flags | kInstFrozen;
              p.inst_frozen[0] = (uint32_t)step;
            }
          }
          p.inst_slot_base[0] = 0u;
        }
      }
    } else {
      // CTA 0 matches and commits while the others wait, unless so many
      // candidates came up that every CTA has to take part.  The step's first-
      // and zeroth-order events count with the commit, before the barrier that
      // may report another CTA's failure in the next step: a committed step is
      // not taken again.
      auto count_events = [&]() {
        if (kSingle && threadIdx.x < p.R && s_events[threadIdx.x])
          p.events[threadIdx.x] = __ldcg(&p.events[threadIdx.x]) + s_events[threadIdx.x];
      };
      uint32_t K = 0;
      if (blockIdx.x == 0) {
        K = ld_u32(&c->n_pairs);
        const DevPair mine = match_pair(p);
        if (K > p.pair_cap) {
          if (threadIdx.x == 0) raise(c, kStatPairs);
        } else if (K > kMatchOneCta && gridDim.x > 1) {
          flag_phase(kFlagGrid);
        } else {
          match_step(s_params, c, K, mine, false, s_match);
          count_events();
        }
      }
      met = phase_barrier(c, bar, kGridReport);
      if (met & kMetFailure) break;
      if (met & kMetGrid) {
        if (!match_step(s_params, c, ld_u32(&c->n_pairs), DevPair{}, true, s_match)) return;
        if (blockIdx.x == 0) count_events();
        if (phase_barrier(c, bar, kNothing) & kMetFailure) break;
      }
    }
    // the next step's state
    cur ^= 1u;
    n_real = total;
    step += 1u;
    if (kSingle) {
      if (advancing(ctx.flags)) {
        ctx.step += 1u;
        if (ctx.step >= target) ctx.flags |= kInstFrozen;
      }
      ctx.slot_base = 0u;
    }
  }
  if (nsteps == 0) phase_barrier(c, bar, kNothing);
  leave(c);
}

template <bool kHasBim>
size_t phase_bytes(uint32_t n_cells) {
  const size_t phase = std::max(sizeof(PairShared<kHasBim, kWarps>), (size_t)kBigChunk * 8u);
  // the starts, and room for the four counts of a load past the last one
  return phase + ((size_t)std::min(n_cells, kSmallCells) + 8u) * sizeof(uint32_t);
}

template <bool kTable, bool kHasBim, bool kSingle>
void launch(const KParams& p, uint32_t nsteps, unsigned grid, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = phase_bytes<kHasBim>(p.n_cells);
  cfg.stream = s;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeCooperative;
  attr.val.cooperative = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = grid > 1 ? 1 : 0;
  cudaLaunchKernelEx(&cfg, k_resident<kTable, kHasBim, kSingle>, p, nsteps);
}

// CTAs per SM (0 or 1) with the largest dynamic shared memory.
template <bool kTable, bool kHasBim, bool kSingle>
int resident_ctas() {
  int a = 0;
  const auto kernel = k_resident<kTable, kHasBim, kSingle>;
  const int bytes = (int)phase_bytes<kHasBim>(kSmallCells);
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, kernel, kThreads, bytes) != cudaSuccess)
    return 0;
  return std::min(a, 1);
}

}  // namespace

int resident_grid(int n_sm) {
  const int a = std::min({resident_ctas<true, true, true>(), resident_ctas<true, true, false>(),
                          resident_ctas<true, false, true>(), resident_ctas<true, false, false>(),
                          resident_ctas<false, true, true>(), resident_ctas<false, true, false>(),
                          resident_ctas<false, false, true>(), resident_ctas<false, false, false>()});
  const int grid = std::min(a * n_sm, 255);  // the arrival word's failure field
  // a quarter of them has to hold the starts of the largest grid (150,000
  // cells) between them
  return grid / 4 < 5 ? 0 : grid;
}

void enqueue_resident(const KParams& p, bool table, bool has_bim, uint32_t nsteps, uint64_t n_slots,
                      const LaunchShape& shape, cudaStream_t s) {
  // 8 warps of records per CTA while there are SMs for it: fewer CTAs meet
  // sooner, more SMs work faster.  A CTA's range of cells has to fit its
  // shared memory (kSmallCells) however few the records.  A quarter of the SMs
  // at most, half for larger sparse grids: a launch holds its SMs for
  // up to 64 steps, and with all of them other streams' work waited for it.
  // Handles of 40,000 particles side by side, us a step of each, all SMs /
  // a quarter / the chain of kernels: one 17 / 20 / 26, two 33 / 21 / 30, four
  // 65 / 21 / 35, eight 130 / 41 / 50, sixteen - / 82 / 98.
  const uint64_t want = std::max<uint64_t>({(n_slots + 255u) / 256u, (p.n_cells + 4095u) / 4096u, 1u});
  const int share = p.n_cells <= kResidentDense || n_slots <= kResidentSparse ? 4 : 2;
  const unsigned grid = (unsigned)std::min<uint64_t>(want, (uint64_t)std::max(shape.grid_resident / share, 1));
  const bool single = p.n_inst == 1 && p.S <= kCtxSpecies && p.U <= kCtxUni && p.R <= kResidentReactions;
#define BD_RESIDENT(T, B, S) launch<T, B, S>(p, nsteps, grid, s)
  if (table) {
    if (has_bim) single ? BD_RESIDENT(true, true, true) : BD_RESIDENT(true, true, false);
    else single ? BD_RESIDENT(true, false, true) : BD_RESIDENT(true, false, false);
  } else {
    if (has_bim) single ? BD_RESIDENT(false, true, true) : BD_RESIDENT(false, true, false);
    else single ? BD_RESIDENT(false, false, true) : BD_RESIDENT(false, false, false);
  }
#undef BD_RESIDENT
}

}  // namespace bd
