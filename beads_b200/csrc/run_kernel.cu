// run_kernel.cu -- whole MD steps in one persistent kernel.
//
// A step launched kernel by kernel costs about 20 us before any work: five
// kernels at ~0.6 us each inside a captured graph, their own latencies, and
// the conditional node that holds the rebuild chain (8 us when it is not
// taken, 17 us when it is, on top of its kernels).  k_run takes a stretch of
// steps instead: one cooperative launch of at most one wave of blocks, a
// barrier over its blocks (1.1 us at up to 296 blocks, 1.3 us at 592) between
// the stages, and the rebuild chain behind a flag every block reads after the
// drift.  A step without a rebuild holds two barriers (three with bonded
// terms), so it is bound by the latency of its own loads until the pair
// forces fill the GPU.
//
// Every stage is the device function that the one-stage kernels call
// (step_device.cuh), and the totals are integers, so a run gives the same
// bits either way.  Blocks read positions and lists through the coherent path,
// since the same kernel writes them.
#include "kernels.cuh"
#include "step_device.cuh"

#include <algorithm>
#include <map>
#include <mutex>
#include <stdexcept>
#include <string>
#include <utility>

namespace bb {
namespace {

// One barrier over all blocks of the launch; `target` counts the arrivals of
// this launch.  The wait is bounded: when the other blocks do not arrive
// within rv.wait_limit reads (some seconds) it marks *status and returns false,
// and the caller leaves the kernel.
__device__ __forceinline__ bool grid_barrier(const RunView& rv, unsigned* status,
                                             uint32_t& target) {
  RunControl* ctl = rv.ctl;
  __shared__ bool ok;
  target += gridDim.x;
  __syncthreads();
  if (threadIdx.x == 0) {
    // Release: the block's writes (ordered before this by the barrier above)
    // are visible to whoever acquires the count.
    uint32_t seen;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;"
                 : "=r"(seen) : "l"(&ctl->arrive) : "memory");
    bool done = static_cast<int32_t>(seen + 1u - target) >= 0;
    for (uint32_t tries = 0; !done && tries < rv.wait_limit; ++tries) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(&ctl->arrive) : "memory");
      done = static_cast<int32_t>(seen - target) >= 0;
    }
    if (!done) atomicOr(status, kStatusStalled);
    ok = done;
  }
  __syncthreads();
  return ok;
}

union RunShared {
  uint32_t sort_keys[kBlock / 32][kSortRankMax];
  BuildShared build[kBuildWarps];
};

// Kinetic energy of replica r from its buckets (one full warp; lane 0 holds
// the sum, like every other lane).
__device__ __forceinline__ double bucket_kinetic(const long long* ke_part, uint32_t r,
                                                 uint32_t lane) {
  long long a = 0, c = 0;
  const longlong2* bucket = reinterpret_cast<const longlong2*>(ke_part) + (size_t)r * kKeBuckets;
#pragma unroll
  for (uint32_t k = 0; k < kKeBuckets / 32u; ++k) {
    const longlong2 q = __ldcg(&bucket[k * 32u + lane]);
    a += q.x;
    c += q.y;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(kFull, a, o);
    c += __shfl_xor_sync(kFull, c, o);
  }
  return from_fixed(a, c);
}

// Runs F(v, b) for the listed slot blocks of the rebuilding replicas.
template <typename F>
__device__ __forceinline__ void for_listed_blocks(const DeviceView& v, F&& f) {
  const uint32_t total = v.chain_block_start[v.n_replicas];
  for (uint32_t w = blockIdx.x; w < total; w += gridDim.x) {
    uint32_t lo = 0, hi = v.n_replicas;  // start[lo] <= w < start[hi]
    while (hi - lo > 1u) {
      const uint32_t mid = (lo + hi) >> 1;
      if (v.chain_block_start[mid] <= w) lo = mid; else hi = mid;
    }
    f(v.rp[lo].block_begin + (w - v.chain_block_start[lo]));
  }
}

constexpr uint32_t kMinGrid = 296;
// Threads per particle of the pair forces: a small system has threads to
// spare, and its steps take as long as a thread's share of a list.
constexpr int kRunTpa = 4;
// Contexts whose pair forces fit two blocks per SM in one pass keep eight list
// entries in flight per thread instead of four, at the registers of four
// blocks per SM.
constexpr int kSmallBlocksPerSm = 4;
constexpr uint32_t kSmallItems = 2u * 148u;
constexpr uint32_t kRunScanPer = 4;                        // consecutive cells per thread
constexpr uint32_t kRunScanChunk = kBlock * kRunScanPer;  // work items per block of the scan
// Replicas of up to this many cells are scanned by one block each.
constexpr uint32_t kRunScanCells = 4u * kRunScanChunk;

// Steps since + 1 .. step - 1 of the launch moved no slot far enough; their
// checks are counted here.
__device__ __forceinline__ void count_checks(const ReplicaParams& p, ReplicaState* st,
                                             uint32_t since, uint32_t step) {
  if (p.skin == 0.0f || step <= since) return;
  const unsigned long long lo = st->step + since, hi = st->step + step;
  st->checks_since_build += p.check_every == 1u
                                ? step - since
                                : (uint32_t)(hi / p.check_every - lo / p.check_every);
}

// Cell starts of large replicas, the work items in chunks of kRunScanChunk:
// chunk totals, then each chunk adds the totals before it.  Every particle of
// a rebuilding replica is counted once, so the running total of a replica's
// first cell is work_atoms.  False after a barrier that ran out.
__device__ __forceinline__ bool run_scan(const DeviceView& v, const RunView& rv, uint32_t items,
                                         uint32_t& target) {
  const uint32_t chunks = (items + kRunScanChunk - 1u) / kRunScanChunk;
  for (uint32_t ch = blockIdx.x; ch < chunks; ch += gridDim.x) {
    uint32_t s = 0;
#pragma unroll
    for (uint32_t k = 0; k < kRunScanPer; ++k) {
      const uint32_t w = ch * kRunScanChunk + k * kBlock + threadIdx.x;
      if (w < items) {
        const uint32_t r = work_replica(v, w);
        s += __ldcg(&v.cell_count[v.rp[r].cell_begin + (w - v.work_start[r])]);
      }
    }
    uint32_t total;
    block_exclusive_scan<kBlock>(s, total);
    if (threadIdx.x == 0) rv.chunk_sum[ch] = total;
  }
  if (!grid_barrier(rv, &v.rs->status, target)) return false;
  for (uint32_t ch = blockIdx.x; ch < chunks; ch += gridDim.x) {
    uint32_t before = 0;
    for (uint32_t k = threadIdx.x; k < ch; k += kBlock) before += rv.chunk_sum[k];
    uint32_t prefix;
    block_exclusive_scan<kBlock>(before, prefix);
    uint32_t cnt[kRunScanPer], s = 0;
    const uint32_t w0 = ch * kRunScanChunk + threadIdx.x * kRunScanPer;
#pragma unroll
    for (uint32_t k = 0; k < kRunScanPer; ++k) {
      cnt[k] = 0u;
      if (w0 + k < items) {
        const uint32_t r = work_replica(v, w0 + k);
        cnt[k] = __ldcg(&v.cell_count[v.rp[r].cell_begin + (w0 + k - v.work_start[r])]);
      }
      s += cnt[k];
    }
    uint32_t total;
    uint32_t run = prefix + block_exclusive_scan<kBlock>(s, total);
#pragma unroll
    for (uint32_t k = 0; k < kRunScanPer; ++k) {
      if (w0 + k < items) {
        const uint32_t r = work_replica(v, w0 + k);
        const ReplicaParams& p = v.rp[r];
        const uint32_t c = w0 + k - v.work_start[r];
        const uint32_t at = p.atom_begin + run - rv.work_atoms[r];
        v.cell_start[p.start_base + c] = at;
        v.cell_cursor[p.cell_begin + c] = at;
        v.cell_count[p.cell_begin + c] = 0u;
        if (c + 1u == p.n_cells) v.cell_start[p.start_base + c + 1u] = p.atom_begin + p.n_atoms;
      }
      run += cnt[k];
    }
  }
  return grid_barrier(rv, &v.rs->status, target);
}

// The work lists of the replicas that rebuild in this step (the last block):
// work_start / chain_block_start / work_atoms hold the cells, slot blocks and
// particles of the rebuilding replicas before each replica.  The replicas'
// state is left alone: other blocks read it meanwhile.
template <int kPre>
__device__ void run_plan(const DeviceView& v, const RunView& rv, const RunRecord& rec,
                         uint32_t step) {
  uint32_t cells = 0, blocks = 0, atoms = 0;
  bool reorder = false, wide = false;
  for (uint32_t base = 0; base < v.n_replicas; base += kBlock) {
    const uint32_t r = base + threadIdx.x;
    uint32_t c = 0, b = 0, n = 0;
    if (r < v.n_replicas) {
      const ReplicaParams& p = v.rp[r];
      const ReplicaState* st = &v.rs[r];
      if (needs_rebuild<kPre>(p, st, st->step + step + 1ull)) {
        c = p.n_cells;
        b = p.n_pad / kBlock;
        n = p.n_atoms;
        reorder |= p.sort_every > 0u && (st->builds + 1ull) % p.sort_every == 0ull;
        wide |= c > kRunScanCells;
        if (rec.flags) rec.flags[(size_t)(rec.k0 + step + 1u) * v.n_replicas + r] = 1u;
      }
    }
    uint32_t tc = c, tb = b, tn = n, ec = 0, eb = 0, en = 0;
    if (v.n_replicas > 1u) {
      ec = block_exclusive_scan<kBlock>(c, tc);
      eb = block_exclusive_scan<kBlock>(b, tb);
      en = block_exclusive_scan<kBlock>(n, tn);
    }
    if (r < v.n_replicas) {
      v.work_start[r] = cells + ec;
      v.chain_block_start[r] = blocks + eb;
      rv.work_atoms[r] = atoms + en;
    }
    cells += tc;
    blocks += tb;
    atoms += tn;
  }
  reorder = __syncthreads_or(reorder);
  wide = __syncthreads_or(wide);
  if (threadIdx.x == 0) {
    v.work_start[v.n_replicas] = cells;
    v.chain_block_start[v.n_replicas] = blocks;
    rv.work_atoms[v.n_replicas] = atoms;
    rv.ctl->reorder = reorder ? 1u : 0u;
    rv.ctl->wide = wide ? 1u : 0u;
    rv.ctl->next = 0u;  // (last read before the barrier that ended the build before)
    if (cells != 0u) *v.chain_launches += 1ull;
  }
}

// The rebuild chain after a drift in which some slot moved half the skin;
// blocks bin, scatter and reorder the slot blocks [b0, b1) they drift.  False
// after a barrier that ran out.  A barrier and the loads behind it cost 2-3 us,
// so the stages are few: the plan is made while the slots are binned, and the
// replicas' state advances while the cells are scanned.
template <int kPre>
__device__ __forceinline__ bool run_rebuild(const DeviceView& v, const RunView& rv,
                                            const RunRecord& rec, RunShared& sh, uint32_t b0,
                                            uint32_t b1, uint32_t since, uint32_t step,
                                            uint32_t& target) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  if (blockIdx.x == gridDim.x - 1u) run_plan<kPre>(v, rv, rec, step);
  for (uint32_t b = b0; b < b1; ++b) {
    const uint32_t r = v.block_replica[b];
    const ReplicaState* st = &v.rs[r];
    if (needs_rebuild<kPre>(v.rp[r], st, st->step + step + 1ull)) bin_slots(v, v.rp[r], b);
  }
  if (!grid_barrier(rv, &v.rs->status, target)) return false;
  const uint32_t items = v.work_start[v.n_replicas];
  const bool reorder = rv.ctl->reorder != 0u;
  const bool wide = rv.ctl->wide != 0u;
  for (uint32_t r = (gridDim.x - 1u - blockIdx.x) * kBlock + threadIdx.x; r < v.n_replicas;
       r += gridDim.x * kBlock) {
    ReplicaState* st = &v.rs[r];
    if (kPre == kPreEval) {
      force_rebuild(v.rp[r], st, true);
    } else {
      if (kPre == kPreVerlet) count_checks(v.rp[r], st, since, step);
      decide_replica<kPre>(v.rp[r], st, st->step + step + 1ull);
    }
  }
  if (items == 0u) return grid_barrier(rv, &v.rs->status, target);  // launch-uniform
  if (!wide) {
    // Cell starts, a block per rebuilding replica.
    for (uint32_t r = blockIdx.x; r < v.n_replicas; r += gridDim.x) {
      if (v.work_start[r] == v.work_start[r + 1u]) continue;  // block-uniform
      const ReplicaParams& p = v.rp[r];
      uint32_t* count = v.cell_count + p.cell_begin;
      uint32_t* start = v.cell_start + p.start_base;
      uint32_t* cursor = v.cell_cursor + p.cell_begin;
      uint32_t run = p.atom_begin;
      const uint32_t n_cells = p.n_cells;
      for (uint32_t base = 0; base < n_cells; base += kRunScanChunk) {
        const uint32_t c0 = base + threadIdx.x * kRunScanPer;
        uint32_t cnt[kRunScanPer], s = 0;
#pragma unroll
        for (uint32_t k = 0; k < kRunScanPer; ++k) {
          cnt[k] = c0 + k < n_cells ? __ldcg(&count[c0 + k]) : 0u;
          s += cnt[k];
        }
        uint32_t total;
        uint32_t at = run + block_exclusive_scan<kBlock>(s, total);
#pragma unroll
        for (uint32_t k = 0; k < kRunScanPer; ++k) {
          if (c0 + k < n_cells) {
            start[c0 + k] = at;
            cursor[c0 + k] = at;
            count[c0 + k] = 0u;
          }
          at += cnt[k];
        }
        run += total;
      }
      if (threadIdx.x == 0) start[n_cells] = run;
    }
    if (!grid_barrier(rv, &v.rs->status, target)) return false;
  } else if (!run_scan(v, rv, items, target)) {
    return false;
  }
  for (uint32_t b = b0; b < b1; ++b) scatter_block(v, b);
  if (!grid_barrier(rv, &v.rs->status, target)) return false;
  if (rv.any_sparse) {
    // A thread per cell; the few cells too big for one are taken by its whole
    // warp at once.  (A warp walking every cell of 2,000 beads in 1.2 million
    // cells found nothing to do for most of a step.)
    for (uint32_t w0 = (blockIdx.x * kBuildWarps + warp) * 32u; w0 < items;
         w0 += gridDim.x * kBlock) {
      const uint32_t w = w0 + lane;
      const bool left = w < items && !sort_cell_sparse(v, w) && v.rp[work_replica(v, w)].sparse;
      uint32_t todo = __ballot_sync(kFull, left);
      for (; todo != 0u; todo &= todo - 1u) {  // warp-uniform
        const uint32_t wb = w0 + (uint32_t)__ffs(todo) - 1u;
        const uint32_t r = work_replica(v, wb);
        sort_cell(v, v.rp[r], wb - v.work_start[r], lane, sh.sort_keys[warp]);
        __syncwarp();
      }
    }
  }
  if (rv.any_dense) {
    for (uint32_t w = blockIdx.x * kBuildWarps + warp; w < items; w += gridDim.x * kBuildWarps) {
      const uint32_t r = work_replica(v, w);
      if (v.rp[r].sparse) continue;  // warp-uniform
      sort_cell(v, v.rp[r], w - v.work_start[r], lane, sh.sort_keys[warp]);
      __syncwarp();
    }
  }
  if (!grid_barrier(rv, &v.rs->status, target)) return false;
  if (reorder) {
    for (uint32_t b = b0; b < b1; ++b) reorder_gather_block(v, b);
    if (!grid_barrier(rv, &v.rs->status, target)) return false;
    for (uint32_t b = b0; b < b1; ++b) reorder_commit_block(v, b);
    if (!grid_barrier(rv, &v.rs->status, target)) return false;
    if (v.excl_cap > 0u) {
      for (uint32_t b = b0; b < b1; ++b) project_exclusions_block(v, b, false);
      if (!grid_barrier(rv, &v.rs->status, target)) return false;
    }
  }
  // A thread per particle only where sparse cells alone fill the GPU several
  // times over: below that its serial walk of 27 cells (~60 us) is what the
  // stage takes, and a warp per cell does the same lists in a fraction.
  const uint32_t warps = gridDim.x * kBuildWarps;
  const bool by_thread = rv.any_sparse && items > 24u * warps;
  if (by_thread) {
    // (slot rows: the stage layout is not touched)
    for_listed_blocks(v, [&](uint32_t b) {
      build_sparse_block<true, false>(v, b, sh.build[0].lay);
    });
  }
  if (rv.any_dense || !by_thread) {
    // A cell per warp, or a share of one.  A warp walks its cell's candidates
    // in a few chunks (~1.5 us each) and its particles one by one within
    // each (~0.25 us), so the share is chosen for the fewest such steps over
    // the warps' rounds.  A warp's first share is its own, further ones come off
    // a counter: dealt in fixed rounds, every warp waited for those with a share
    // in the last, part-filled one (100,003 LJ beads 58.3 -> 54.7 us a step).
    const uint32_t homes = rv.work_atoms[v.n_replicas] / items + 1u;
    uint32_t parts = 1u, best = 0xffffffffu;
    for (uint32_t t = 1u; t <= min(homes, 16u); ++t) {
      const uint32_t rounds = (items * t + warps - 1u) / warps;
      const uint32_t cost = rounds * (6u + (homes + t - 1u) / t);
      if (cost < best) best = cost, parts = t;
    }
    const uint32_t shares = items * parts;
    uint32_t k = blockIdx.x * kBuildWarps + warp;
    auto following = [&]() -> uint32_t {
      if (shares <= warps) return shares;
      uint32_t n = 0;
      if (lane == 0u) n = atomicAdd(&rv.ctl->next, 1u);
      return warps + __shfl_sync(kFull, n, 0);
    };
    for (; k < shares; k = following()) {  // warp-uniform
      const uint32_t w = k / parts;
      const uint32_t r = work_replica(v, w);
      const ReplicaParams& p = v.rp[r];
      if (by_thread && p.sparse) continue;
      build_cell<true, false>(v, p, &v.rs[r], p.cell_begin + (w - v.work_start[r]), lane,
                              sh.build[warp], k - w * parts, parts);
    }
  }
  return grid_barrier(rv, &v.rs->status, target);
}

// kPre: velocity Verlet (drift, rebuild, forces and second half-kick per step)
// or the capped descent (forces, move, rebuild per iteration), or one
// evaluation (rebuild, forces, totals).  kObs: energies and virial of every
// step.
template <int kPre, bool kObs, int kNt, bool kSmall>
__global__ void __launch_bounds__(kBlock, kSmall ? kSmallBlocksPerSm : kRunBlocksPerSm)
k_run(DeviceView v, RunView rv, RunRecord rec, uint32_t n_steps, float sd_dmax, float sd_fref) {
  constexpr bool kVerlet = kPre == kPreVerlet;
  constexpr bool kEval = kPre == kPreEval;
  __shared__ RunShared sh;
  // The parameters and the LJ table of the replica at hand: after a barrier
  // they would come from L2 again.
  __shared__ ReplicaParams p;
  __shared__ LjCoeff table[kNt == 0 ? kMaxTypes * kMaxTypes : kNt * kNt];
  __shared__ float lam_s;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t gthread = blockIdx.x * kBlock + threadIdx.x;
  const bool kinetic = kEval || (kVerlet && (kObs || rv.need_kinetic != 0));
  const bool bonded = v.has_bonded != 0;
  // A launch queued behind one whose barrier ran out finds the counts in
  // disorder (the host takes no further call on such a context).
  if (__ldcg(&v.rs->status) & kStatusStalled) return;
  uint32_t target = 0, cur = 0xffffffffu;
  // Consecutive slot blocks and pair-force items per block: an item's
  // neighbours are mostly those of the item before it.
  const uint32_t b0 = (uint32_t)((uint64_t)v.n_blocks * blockIdx.x / gridDim.x);
  const uint32_t b1 = (uint32_t)((uint64_t)v.n_blocks * (blockIdx.x + 1u) / gridDim.x);
  const uint32_t n_items = v.n_blocks * kRunTpa;
  const uint32_t i0 = (uint32_t)((uint64_t)n_items * blockIdx.x / gridDim.x);
  const uint32_t i1 = (uint32_t)((uint64_t)n_items * (blockIdx.x + 1u) / gridDim.x);

  auto enter = [&](uint32_t r) {  // block-uniform
    if (r == cur) return;
    cur = r;
    __syncthreads();
    const uint32_t* src = reinterpret_cast<const uint32_t*>(&v.rp[r]);
    for (uint32_t k = threadIdx.x; k < sizeof(ReplicaParams) / 4u; k += kBlock) {
      reinterpret_cast<uint32_t*>(&p)[k] = src[k];
    }
    __syncthreads();
    for (int t = threadIdx.x; t < p.n_types * p.n_types; t += kBlock) {
      table[t] = v.lj[p.lj_offset + t];
    }
    __syncthreads();
  };
  auto replica_of = [&](uint32_t b) -> uint32_t {
    return v.n_replicas == 1u ? 0u : v.block_replica[b];
  };

  auto forces = [&](long long* ke, float4* vel) -> bool {
    for (uint32_t item = i0; item < i1; ++item) {
      enter(replica_of(item / kRunTpa));
      lj_block<kObs, kPre == kPreDescent, kRunTpa, kSmall ? 8 : 4, true, kNt, true>(v, p, cur, item, table,
                                                         kVerlet && !bonded, kinetic, ke, vel);
    }
    if (bonded) {
      const uint32_t terms = v.n_bond_terms + v.n_angle_terms + v.n_dihedral_terms;
      for (uint32_t t = gthread; t < terms; t += gridDim.x * kBlock) bonded_term<kObs>(v, t);
      if (!grid_barrier(rv, &v.rs->status, target)) return false;
      for (uint32_t b = b0; b < b1; ++b) {
        enter(replica_of(b));
        bonded_block<kObs>(v, p, cur, b, kVerlet, kinetic, ke, vel);
      }
    }
    return true;
  };

  // What step s left, replica by replica (a warp each), once its buckets are
  // complete: observables and recorded scale and kinetic energy.
  auto epilogue = [&](uint32_t s, const long long* ke) {
    for (uint32_t r = blockIdx.x * kBuildWarps + warp; r < v.n_replicas;
         r += gridDim.x * kBuildWarps) {
      const double kin = kinetic ? bucket_kinetic(ke, r, lane) : 0.0;
      if (lane != 0u) continue;
      const double l = kVerlet && kinetic ? berendsen_lambda(v.rp[r], kin) : 1.0;
      if (rec.lam) {
        rec.lam[(size_t)(rec.k0 + s + 1u) * v.n_replicas + r] = l;
        rec.kin[(size_t)(rec.k0 + s + 1u) * v.n_replicas + r] = kin;
      }
      if (kObs) {
        const ReplicaObs o = take_observables(&v.rs[r], v.rs[r].step + (kEval ? 0u : s + 1u), kin,
                                                l);
        if (rec.obs) rec.obs[(size_t)s * v.n_replicas + r] = o;
        if (s + 1u == n_steps) v.obs[r] = o;
      }
    }
  };

  uint32_t since = 0;  // steps whose checks are counted
  if (kEval) {
    // Own velocities: the pending scale, and their kinetic energy.
    for (uint32_t b = b0; b < b1; ++b) {
      const uint32_t r = replica_of(b);
      enter(r);
      const uint32_t i = b * kBlock + threadIdx.x;
      const bool real = (i - p.atom_begin) < p.n_atoms;
      const float lam = (float)v.rs[r].lambda;
      float4 u = real ? v.vel[i] : make_float4(0.f, 0.f, 0.f, 1.f);
      if (real && lam != 1.0f) {
        u.x = __fmul_rn(u.x, lam);
        u.y = __fmul_rn(u.y, lam);
        u.z = __fmul_rn(u.z, lam);
        v.vel[i] = u;
      }
      post_partial(v.ke_part, &v.rs[r], r, real,
                   post_slot_vm(v, p, &v.rs[r], i, real, false, true, u, 0.f, 0.f, 0.f));
    }
    if (!run_rebuild<kPre>(v, rv, rec, sh, b0, b1, 0u, 0u, target)) return;
    if (!forces(nullptr, nullptr)) return;
    if (!grid_barrier(rv, &v.rs->status, target)) return;
  }
  for (uint32_t s = 0; !kEval && s < n_steps; ++s) {
    long long* ke = (s & 1u) ? rv.ke_odd : v.ke_part;
    long long* ke_other = (s & 1u) ? v.ke_part : rv.ke_odd;
    if (!kVerlet) {
      if (!forces(nullptr, nullptr)) return;
      if (!grid_barrier(rv, &v.rs->status, target)) return;
    }
    const size_t record = (size_t)(rec.k0 + s + 1u) * v.n_slots;
    if (kVerlet && s > 0u && (kObs || rec.lam)) epilogue(s - 1u, ke_other);
    uint32_t scaled = 0xffffffffu;
    float lam = 1.0f;
    for (uint32_t b = b0; b < b1; ++b) {
      const uint32_t r = replica_of(b);
      enter(r);
      if (kVerlet && r != scaled && (s == 0u || (kinetic && p.thermostat == 1))) {
        // The pending scale: the state's before the first step, then from
        // the kinetic energy of the step before.
        __syncthreads();
        if (warp == 0) {
          const double l =
              s == 0u ? v.rs[r].lambda : berendsen_lambda(p, bucket_kinetic(ke_other, r, lane));
          if (lane == 0u) lam_s = (float)l;
        }
        __syncthreads();
        lam = lam_s;
      } else if (r != scaled) {
        lam = 1.0f;
      }
      scaled = r;
      pre_block<kPre>(v, p, &v.rs[r], b, p.check_every == 1u ? 0ull : v.rs[r].step + s + 1ull, lam,
                      sd_dmax, sd_fref, &rv.ctl->any[s & 1u],
                      kVerlet && rec.pos ? rec.pos + record : nullptr);
      if (kVerlet && p.skin == 0.0f && threadIdx.x == 0) rv.ctl->any[s & 1u] = 1u;
    }
    if (!grid_barrier(rv, &v.rs->status, target)) return;
    if (__ldcg(&rv.ctl->any[s & 1u]) != 0u) {  // launch-uniform
      if (!run_rebuild<kPre>(v, rv, rec, sh, b0, b1, since, s, target)) return;
      since = s + 1u;
      if (kVerlet && rec.snap_nbr && v.work_start[v.n_replicas] != 0u) {
        for_listed_blocks(v, [&](uint32_t b) {
          snapshot_block(v, b, rec.snap_nbr + record * v.nbr_stride, rec.snap_cnt + record);
        });
      }
    }
    // What follows is not read before the next barrier.
    if (gthread == 0u) rv.ctl->any[(s + 1u) & 1u] = 0u;
    if (kVerlet) {
      if (kinetic) {
        longlong2* z = reinterpret_cast<longlong2*>(ke_other);
        for (uint32_t k = gthread; k < v.n_replicas * kKeBuckets; k += gridDim.x * kBlock) {
          z[k] = make_longlong2(0, 0);
        }
      }
      if (!forces(ke, rec.vel ? rec.vel + record : nullptr)) return;
      if (!grid_barrier(rv, &v.rs->status, target)) return;
    }
  }
  if (kVerlet || kEval) {
    long long* ke = (n_steps & 1u) ? v.ke_part : rv.ke_odd;  // of the last step
    if (kObs || rec.lam) epilogue(n_steps - 1u, ke);
    for (uint32_t r = blockIdx.x * kBuildWarps + warp; r < v.n_replicas;
         r += gridDim.x * kBuildWarps) {
      double kin = 0.0;
      if (kinetic) {
        kin = bucket_kinetic(ke, r, lane);
        __syncwarp();
        longlong2* z = reinterpret_cast<longlong2*>(ke) + (size_t)r * kKeBuckets;
        for (uint32_t k = lane; k < kKeBuckets; k += 32u) z[k] = make_longlong2(0, 0);
      }
      if (lane == 0u) {
        ReplicaState* st = &v.rs[r];
        if (kVerlet && since < n_steps) {
          count_checks(v.rp[r], st, since, n_steps);
          st->need_rebuild = 0u;
          st->reorder_now = 0u;
        }
        st->lambda = kVerlet && kinetic ? berendsen_lambda(v.rp[r], kin) : 1.0;
        if (kVerlet) st->step += n_steps;
        if (kinetic) st->last_kinetic = kin;
      }
    }
  }
  if (threadIdx.x == 0) {
    if (blockIdx.x == 0) rv.ctl->any[0] = rv.ctl->any[1] = 0u;
    __threadfence();
    // The last block to leave rearms the barrier for the next launch.
    if (atomicAdd(&rv.ctl->left, 1u) == gridDim.x - 1u) {
      rv.ctl->arrive = 0u;
      rv.ctl->left = 0u;
    }
  }
}

void check(cudaError_t e) {
  if (e != cudaSuccess) {
    throw std::runtime_error(std::string("CUDA launch of run failed: ") + cudaGetErrorString(e));
  }
}

// Blocks of one wave of `kernel` on the current device (kept per kernel and
// device).
uint32_t wave_of(const void* kernel) {
  static std::mutex mutex;
  static std::map<std::pair<int, const void*>, uint32_t> waves;
  int device = 0, sms = 0, per_sm = 0;
  check(cudaGetDevice(&device));
  const std::lock_guard<std::mutex> lock(mutex);
  uint32_t& wave = waves[{device, kernel}];
  if (wave == 0u) {
    check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kBlock, 0));
    wave = (uint32_t)(sms * per_sm);
  }
  return wave;
}

template <int kPre, bool kObs, int kNt, bool kSmall>
void launch_as(const StepLaunch& l, RunView& rv, const RunRecord& rec, uint32_t n_steps) {
  auto* kernel = k_run<kPre, kObs, kNt, kSmall>;
  // One wave at most.  Pair-force items of a small system leave blocks idle,
  // but a rebuild shares its cells over every warp, and barriers take the same
  // time up to about two blocks per SM.
  const uint32_t most =
      rv.max_blocks != 0u ? rv.max_blocks : wave_of(reinterpret_cast<const void*>(kernel));
  uint32_t blocks = std::min(most, std::max(kMinGrid, l.v.n_blocks * (uint32_t)kRunTpa));
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kBlock);
  cfg.stream = l.stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  // A process that has part of the SMs may be refused a wave of all of them: any
  // number of blocks takes the same steps, so half as many are tried, and kept
  // for the context.
  for (;;) {
    cfg.gridDim = dim3(blocks);
    const cudaError_t e =
        cudaLaunchKernelEx(&cfg, kernel, l.v, rv, rec, n_steps, l.sd_dmax, l.sd_fref);
    if (e != cudaErrorCooperativeLaunchTooLarge || blocks <= 1u) {
      check(e);
      return;
    }
    (void)cudaGetLastError();
    blocks = (blocks + 1u) / 2u;
    rv.max_blocks = blocks;
  }
}

template <int kPre, bool kObs, int kNt>
void launch_one(const StepLaunch& l, RunView& rv, const RunRecord& rec, uint32_t n_steps) {
  if (l.v.n_blocks * (uint32_t)kRunTpa <= kSmallItems) {
    launch_as<kPre, kObs, kNt, true>(l, rv, rec, n_steps);
  } else {
    launch_as<kPre, kObs, kNt, false>(l, rv, rec, n_steps);
  }
}

// The LJ table specialisation of the batch: its coefficients in registers for
// one or two types.
template <int kPre, bool kObs>
void launch_types(const StepLaunch& l, RunView& rv, const RunRecord& rec, uint32_t n_steps) {
  switch (l.lj_types) {
    case 1: launch_one<kPre, kObs, 1>(l, rv, rec, n_steps); break;
    case 2: launch_one<kPre, kObs, 2>(l, rv, rec, n_steps); break;
    default: launch_one<kPre, kObs, 0>(l, rv, rec, n_steps); break;
  }
}

}  // namespace

void launch_run(const StepLaunch& l, RunView& rv, uint32_t n_steps, bool observables,
                const RunRecord& rec) {
  if (observables) {
    launch_types<kPreVerlet, true>(l, rv, rec, n_steps);
  } else {
    launch_types<kPreVerlet, false>(l, rv, rec, n_steps);
  }
}

void launch_descent(const StepLaunch& l, RunView& rv, uint32_t n_steps) {
  launch_types<kPreDescent, false>(l, rv, RunRecord{}, n_steps);
}

void launch_eval(const StepLaunch& l, RunView& rv) {
  launch_one<kPreEval, true, 0>(l, rv, RunRecord{}, 1);
}

uint32_t run_scan_chunks(uint32_t total_cells) {
  return (total_cells + kRunScanChunk - 1u) / kRunScanChunk;
}

}  // namespace bb
