// kernels.cu -- sm_100a kernels of the BEADS per-step hot path.
//
// Reference behaviour followed (paths inside the reference project):
//   cell id             native/src/simulation/neighbor/cell_list_build.cu:110-166
//   neighbour inclusion native/src/simulation/neighbor/full/full_neighbor_path_common.cuh:49-94
//   stencils            full/regular_cell_neighbor_builder.cu:40-113,
//                       full/small_dimension_neighbor_builder.cu:56-142
//   rebuild policy      native/src/simulation/neighbor/neighbor_system.cpp:79-216
//   displacement check  native/src/simulation/neighbor/rebuild_tracker.cu:50-94
//   LJ pair             native/src/forcefield/pair/pair_lj.cu:21-192
//   harmonic bond       native/src/forcefield/bond/bond_harmonic.cu:24-99
//   harmonic angle      native/src/forcefield/angle/angle_harmonic.cu:23-178
//   harmonic dihedral   native/src/forcefield/dihedral/dihedral_harmonic.cu:22-227
//   velocity Verlet     native/src/dynamics/integrator/velocity_verlet.cu:59-111
//   Berendsen           native/src/dynamics/thermostat/berendsen_thermostat.cu:104-163
//
// Design (not a translation): every kernel runs over all replicas of a batch
// at once; a block never straddles two replicas; the rebuild decision is taken
// on the device so a captured step loop needs no host round trip; totals are
// reduced in 64-bit fixed point so they do not depend on block scheduling;
// bonded terms are evaluated once each and their members' forces gathered per
// particle, so no force atomics exist anywhere.
#include "kernels.cuh"
#include "device_util.cuh"
#include "step_device.cuh"

#include <algorithm>
#include <cstdio>
#include <map>
#include <mutex>
#include <stdexcept>
#include <string>

namespace bb {
namespace {

template <int kMode>
__global__ void __launch_bounds__(kBlock)
k_pre(DeviceView v, float sd_dmax, float sd_fref) {
  wait_prior_grid();
  const uint32_t r = v.block_replica[blockIdx.x];
  ReplicaState* st = &v.rs[r];
  pre_block<kMode>(v, v.rp[r], st, blockIdx.x, st->step + 1ull,
                   (kMode == kPreVerlet) ? (float)st->lambda : 1.0f, sd_dmax, sd_fref, nullptr, nullptr);
}

// pre, second part: one thread per replica takes the rebuild decision of
// this step from the displacement flag k_pre's blocks set (a separate launch
// instead of a last-block handshake: no fence and no same-address atomic in
// each of k_pre's blocks).
template <int kMode>
__global__ void k_decide(DeviceView v, cudaGraphConditionalHandle cond, int use_cond) {
  wait_prior_grid();
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= v.n_replicas) return;
  ReplicaState* st = &v.rs[r];
  const unsigned need = decide_replica<kMode>(v.rp[r], st, st->step + 1ull);
  // Inside a captured step the rebuild chain is the body of a conditional
  // graph node: any replica that rebuilds switches it on for this step.
  if (need && use_cond) cudaGraphSetConditional(cond, 1u);
  if (kMode == kPreVerlet) st->lambda = 1.0;
}

// Marks every replica for a rebuild (initial build / explicit eval).
__global__ void k_force_rebuild_flags(DeviceView v, int count_build) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= v.n_replicas) return;
  force_rebuild(v.rp[r], &v.rs[r], count_build != 0);
}

// rebuild 2: exclusive scan of the cell counts (the cell starts), in three
// kernels so that a replica with many cells is scanned by many blocks:
// k_scan_sum (one block per chunk of kScanChunk cells: the chunk's total),
// k_scan (one block per replica: the work list of the per-cell kernels and
// the exclusive prefix of the replica's chunk totals) and k_scan_cells (one
// block per chunk: the starts and cursors of its cells; the counts are reset
// for the next build).  When every replica fits one chunk, k_scan_single
// does all three in one launch.
constexpr int kScanThreads = 1024;
constexpr int kScanWarps = kScanThreads / 32;
constexpr uint32_t kScanPer = kScanChunk / kScanThreads;  // consecutive cells per thread

// ---------------------------------------------------------------------------
// The per-slot kernels of the rebuild chain (bin, scatter, reorder) touch
// only the replicas that rebuild.  In a batch, where a step typically
// rebuilds a fifth of the replicas, they walk a list of those replicas'
// 128-slot blocks with a grid of about one wave, instead of launching one
// block per slot block of the batch that mostly returns at once.  Block item
// w is block w - chain_block_start[q] of the rebuilding replica q with
// chain_block_start[q] <= w < chain_block_start[q + 1]; k_chain_blocks (one
// block) lays the list out at the head of the chain.
__global__ void __launch_bounds__(kScanThreads) k_chain_blocks(DeviceView v) {
  uint32_t run = 0;
  for (uint32_t base = 0; base < v.n_replicas; base += kScanThreads) {
    const uint32_t q = base + threadIdx.x;
    const uint32_t x = (q < v.n_replicas && v.rs[q].need_rebuild) ? v.rp[q].n_pad / kBlock : 0u;
    uint32_t total;
    const uint32_t ex = block_exclusive_scan<kScanThreads>(x, total);
    if (q < v.n_replicas) v.chain_block_start[q] = run + ex;
    run += total;
  }
  if (threadIdx.x == 0) v.chain_block_start[v.n_replicas] = run;
}

// Runs F(v, b) for every slot block b this launch covers: the listed blocks
// of the rebuilding replicas (grid-stride over the list) or, without the
// list, block blockIdx.x of the batch.  F returns early for blocks of
// replicas that do not rebuild; it holds no barrier.
template <void (*F)(const DeviceView&, uint32_t)>
__device__ __forceinline__ void for_chain_blocks(const DeviceView& v) {
  if (v.chain_block_list) {
    const uint32_t* start = v.chain_block_start;
    const uint32_t total = start[v.n_replicas];
    for (uint32_t w = blockIdx.x; w < total; w += gridDim.x) {
      uint32_t lo = 0, hi = v.n_replicas;  // start[lo] <= w < start[hi]
      while (hi - lo > 1u) {
        const uint32_t mid = (lo + hi) >> 1;
        if (start[mid] <= w) lo = mid; else hi = mid;
      }
      F(v, v.rp[lo].block_begin + (w - start[lo]));
    }
  } else {
    F(v, blockIdx.x);
  }
}

__global__ void __launch_bounds__(kBlock) k_bin(DeviceView v) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *v.chain_launches += 1ull;  // launches of the chain
    *v.big_cells = 0u;
  }
  for_chain_blocks<bin_block>(v);
}

__global__ void __launch_bounds__(kScanThreads) k_scan_sum(DeviceView v) {
  const uint32_t b = blockIdx.x;
  const uint32_t r = v.scan_chunk_replica[b];
  if (!v.rs[r].need_rebuild) return;
  const ReplicaParams& p = v.rp[r];
  const uint32_t c0 = (b - v.scan_chunk_first[r]) * kScanChunk;
  const uint32_t* count = v.cell_count + p.cell_begin;
  uint32_t s = 0;
#pragma unroll
  for (uint32_t k = 0; k < kScanPer; ++k) {
    const uint32_t c = c0 + k * kScanThreads + threadIdx.x;
    if (c < p.n_cells) s += count[c];
  }
  s = __reduce_add_sync(kFull, s);
  __shared__ uint32_t part[kScanWarps];
  if ((threadIdx.x & 31u) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int w = 0; w < kScanWarps; ++w) t += part[w];
    v.scan_chunk_sum[b] = t;
  }
}

// Work list of the per-cell kernels (cell sort, list build): work item w is
// cell w - work_start[q] of the rebuilding replica q with work_start[q] <= w
// < work_start[q + 1].  Block r (one per replica) writes entry r (the cells
// of the rebuilding replicas before it), block 0 also the total.
__device__ __forceinline__ void write_work_start(const DeviceView& v, uint32_t r) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  {
    uint32_t before = 0, all = 0;
    for (uint32_t q = threadIdx.x; q < v.n_replicas; q += kScanThreads) {
      const uint32_t c = v.rs[q].need_rebuild ? v.rp[q].n_cells : 0u;
      all += c;
      before += q < r ? c : 0u;
    }
    before = __reduce_add_sync(kFull, before);
    all = __reduce_add_sync(kFull, all);
    __shared__ uint32_t part[2][kScanWarps];
    if (lane == 0) {
      part[0][warp] = before;
      part[1][warp] = all;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t sb = 0, sa = 0;
      for (int w = 0; w < kScanWarps; ++w) {
        sb += part[0][w];
        sa += part[1][w];
      }
      v.work_start[r] = sb;
      if (r == 0) v.work_start[v.n_replicas] = sa;
    }
  }
}

__global__ void __launch_bounds__(kScanThreads) k_scan(DeviceView v) {
  const uint32_t r = blockIdx.x;
  write_work_start(v, r);
  if (!v.rs[r].need_rebuild) return;  // block-uniform
  const ReplicaParams& p = v.rp[r];
  // Exclusive prefix of the replica's chunk totals, in place.
  const uint32_t f0 = v.scan_chunk_first[r], f1 = v.scan_chunk_first[r + 1];
  uint32_t run = 0;
  for (uint32_t base = f0; base < f1; base += kScanThreads) {
    const uint32_t at = base + threadIdx.x;
    const uint32_t x = at < f1 ? v.scan_chunk_sum[at] : 0u;
    uint32_t total;
    const uint32_t ex = block_exclusive_scan<kScanThreads>(x, total);
    if (at < f1) v.scan_chunk_sum[at] = run + ex;
    run += total;
  }
  if (threadIdx.x == 0) v.cell_start[p.start_base + p.n_cells] = p.atom_begin + p.n_atoms;
}

// Starts and cursors of the cells of chunk `chunk` of replica p (the counts
// are reset for the next build); `prefix` is the count total of the
// replica's chunks before it.
__device__ __forceinline__ void scan_chunk_cells(const DeviceView& v, const ReplicaParams& p,
                                                 uint32_t chunk, uint32_t prefix) {
  const uint32_t c0 = chunk * kScanChunk + threadIdx.x * kScanPer;
  uint32_t* count = v.cell_count + p.cell_begin;
  uint32_t cnt[kScanPer];
  uint32_t s = 0;
#pragma unroll
  for (uint32_t k = 0; k < kScanPer; ++k) {
    cnt[k] = c0 + k < p.n_cells ? count[c0 + k] : 0u;
    s += cnt[k];
  }
  uint32_t total;
  uint32_t run = p.atom_begin + prefix + block_exclusive_scan<kScanThreads>(s, total);
  uint32_t* start = v.cell_start + p.start_base;
  uint32_t* cursor = v.cell_cursor + p.cell_begin;
#pragma unroll
  for (uint32_t k = 0; k < kScanPer; ++k) {
    const uint32_t c = c0 + k;
    if (c < p.n_cells) {
      start[c] = run;
      cursor[c] = run;
      count[c] = 0u;
    }
    run += cnt[k];
  }
}

__global__ void __launch_bounds__(kScanThreads) k_scan_cells(DeviceView v) {
  const uint32_t b = blockIdx.x;
  const uint32_t r = v.scan_chunk_replica[b];
  if (!v.rs[r].need_rebuild) return;
  scan_chunk_cells(v, v.rp[r], b - v.scan_chunk_first[r], v.scan_chunk_sum[b]);
}

// The same scan when every replica's cells fit one chunk (a batch of small
// replicas): the work list, then the replica's starts and cursors with a
// zero chunk prefix, in one launch instead of three.
__global__ void __launch_bounds__(kScanThreads) k_scan_single(DeviceView v) {
  const uint32_t r = blockIdx.x;
  write_work_start(v, r);
  if (!v.rs[r].need_rebuild) return;  // block-uniform
  const ReplicaParams& p = v.rp[r];
  scan_chunk_cells(v, p, 0u, 0u);
  if (threadIdx.x == 0) v.cell_start[p.start_base + p.n_cells] = p.atom_begin + p.n_atoms;
}

__global__ void __launch_bounds__(kBlock) k_scatter(DeviceView v) {
  for_chain_blocks<scatter_block>(v);
}

__global__ void __launch_bounds__(kBlock) k_cellsort_sparse(DeviceView v) {
  const uint32_t w = blockIdx.x * kBlock + threadIdx.x;
  // The cells left over are listed for k_cellsort (the cursors are free once
  // the slots are scattered).
  if (w < v.work_start[v.n_replicas] && !sort_cell_sparse(v, w)) {
    v.cell_cursor[atomicAdd(v.big_cells, 1u)] = w;
  }
}

// Warp w sorts work item w (k_scan): the warps past the cells of the
// rebuilding replicas return after one load.  listed: every replica is sparse,
// and a few blocks walk the cells k_cellsort_sparse listed instead (a warp per
// cell that finds nothing to do took ~12 us of a 200,000-bead melt's rebuild).
__global__ void __launch_bounds__(kBlock) k_cellsort(DeviceView v, int listed) {
  __shared__ uint32_t sort_keys[kBlock / 32][kSortRankMax];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t first = blockIdx.x * (kBlock / 32) + warp;
  const uint32_t n = listed ? *v.big_cells : v.work_start[v.n_replicas];
  const uint32_t step = listed ? gridDim.x * (kBlock / 32) : n;
  for (uint32_t k = first; k < n; k += step) {  // warp-uniform
    const uint32_t w = listed ? v.cell_cursor[k] : k;
    const uint32_t r = work_replica(v, w);
    sort_cell(v, v.rp[r], w - v.work_start[r], lane, sort_keys[warp]);
    __syncwarp();
  }
}

__global__ void __launch_bounds__(kBlock) k_reorder_gather(DeviceView v) {
  for_chain_blocks<reorder_gather_block>(v);
}

__global__ void __launch_bounds__(kBlock) k_reorder_commit(DeviceView v) {
  for_chain_blocks<reorder_commit_block>(v);
}

__global__ void __launch_bounds__(kBlock)
k_project_exclusions(DeviceView v, int force_all) {
  project_exclusions_block(v, blockIdx.x, force_all != 0);
}

// Warps w parts .. w parts + parts - 1 build the lists of work item w (k_scan),
// a share of its cell's particles each: the warps past the cells of the
// rebuilding replicas return after one load.
template <bool kExcl, bool kByQ>
__global__ void __launch_bounds__(kBlock, 7) k_build(DeviceView v, uint32_t parts) {
  __shared__ BuildShared sh[kBuildWarps];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t k = blockIdx.x * kBuildWarps + warp;
  const uint32_t w = k / parts;
  if (w >= v.work_start[v.n_replicas]) return;  // warp-uniform
  const uint32_t r = work_replica(v, w);
  const ReplicaParams& p = v.rp[r];
  if (p.sparse) return;  // built by k_build_sparse
  build_cell<kExcl, kByQ>(v, p, &v.rs[r], p.cell_begin + (w - v.work_start[r]), lane, sh[warp],
                           k - w * parts, parts);
}

template <bool kExcl, bool kByQ>
__global__ void __launch_bounds__(kBlock, kByQ ? 1 : 12) k_build_sparse(DeviceView v) {
  __shared__ StageLayout lay;
  build_sparse_block<kExcl, kByQ>(v, blockIdx.x, lay);
}

// Same, one bucket add per block (k_post: a short streaming kernel where the
// block barrier costs little and fewer adds contend for the buckets).
template <bool kKinetic>
__device__ __forceinline__ void post_partial_block(const DeviceView& v, ReplicaState* st,
                                                   uint32_t r, bool real, double ke) {
  if (!kKinetic) return;
  __shared__ long long part[2][kBlock / 32];
  const Fixed f = real ? to_fixed(ke, &st->status) : Fixed{0, 0};
  long long a = f.whole, c = f.frac;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_down_sync(kFull, a, o);
    c += __shfl_down_sync(kFull, c, o);
  }
  if ((threadIdx.x & 31) == 0) {
    part[0][threadIdx.x >> 5] = a;
    part[1][threadIdx.x >> 5] = c;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    long long sa = 0, sc = 0;
    for (int w = 0; w < kBlock / 32; ++w) {
      sa += part[0][w];
      sc += part[1][w];
    }
    unsigned long long* bucket = reinterpret_cast<unsigned long long*>(v.ke_part) +
                                 2 * ((size_t)r * kKeBuckets + blockIdx.x % kKeBuckets);
    if (sa != 0) atomicAdd(bucket, static_cast<unsigned long long>(sa));
    if (sc != 0) atomicAdd(bucket + 1, static_cast<unsigned long long>(sc));
  }
}

constexpr int kFinishThreads = 128;
static_assert(kKeBuckets <= (uint32_t)kFinishThreads, "one finish thread per bucket");

template <bool kKick, bool kObs, bool kKinetic>
__global__ void __launch_bounds__(kFinishThreads) k_post_finish(DeviceView v) {
  wait_prior_grid();
  const uint32_t r = blockIdx.x;
  const ReplicaParams& p = v.rp[r];
  ReplicaState* st = &v.rs[r];
  __shared__ long long part[2][kFinishThreads / 32];
  long long a = 0, c = 0;
  if (kKinetic) {
    if (threadIdx.x < kKeBuckets) {
      longlong2* bucket = reinterpret_cast<longlong2*>(v.ke_part) + (size_t)r * kKeBuckets +
                          threadIdx.x;
      const longlong2 q = *bucket;
      *bucket = make_longlong2(0, 0);
      a = q.x;
      c = q.y;
    }
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_down_sync(kFull, a, o);
      c += __shfl_down_sync(kFull, c, o);
    }
    if ((threadIdx.x & 31) == 0) {
      part[0][threadIdx.x >> 5] = a;
      part[1][threadIdx.x >> 5] = c;
    }
    __syncthreads();
  }
  if (threadIdx.x != 0) return;
  double kin = 0.0;
  if (kKinetic) {
    long long sa = 0, sc = 0;
    for (int w = 0; w < kFinishThreads / 32; ++w) {
      sa += part[0][w];
      sc += part[1][w];
    }
    kin = from_fixed(sa, sc);
  }
  finish_replica<kObs>(v, r, kKick, kKinetic, kin);
}

template <bool kObs, int kMode, int kTpa, int kUnroll, bool kNoL1, int kNt>
__global__ void __launch_bounds__(kBlock, (!kObs && kMode == kForcePlain && kUnroll == 4) ? 8 : 1)
k_lj(DeviceView v) {
  __shared__ LjCoeff table[kMaxTypes * kMaxTypes];
  const uint32_t r = v.block_replica[blockIdx.x / kTpa];
  const ReplicaParams& p = v.rp[r];
  for (int t = threadIdx.x; t < p.n_types * p.n_types; t += kBlock) table[t] = v.lj[p.lj_offset + t];
  __syncthreads();
  constexpr bool kPost = kMode >= kForcePost;
  lj_block<kObs, kMode == kForceClamp, kTpa, kUnroll, kNoL1, kNt, false>(
      v, p, r, blockIdx.x, table, kPost, kMode == kForcePostKinetic || (kPost && kObs), v.ke_part);
}

// LJ pair forces of a staged context: block g handles the 128 particles of
// cell-order rows [128 g, 128 g + 128) (kTpa threads each).  Its first warp
// derives the group's stage layout (stage_layout, the same function the list
// build used), the block copies the stage -- pos[cell_atoms[q]] for every q
// of every window, one window per warp at a time -- into shared memory, and
// every neighbour position of the pair loop is then a shared-memory load
// instead of an L1/L2 gather.  A group whose layout fell back to slot
// entries reads global positions, as k_lj does.  The arithmetic, the list
// order and the canonical summation order are k_lj's, so the forces, energies
// and virial are bit-identical to k_lj's for the same list.
// Four entries in flight and the general table whatever the schedule and the
// types: 200,000 beads at four threads per particle take 113 us a step, 137 with
// eight entries and one type's coefficients in registers; the 200,000-bead
// mixture at two threads 78, 82 with two types' in registers (20,011 beads 31.5
// and 30.9).
template <bool kObs, int kMode, int kTpa>
__global__ void __launch_bounds__(kBlock* kTpa) k_lj_staged(DeviceView v) {
  constexpr int kUnroll = 4, kNt = 0;
  constexpr bool kNoL1 = true;
  constexpr int kThreads = kBlock * kTpa;
  constexpr bool kClamp = kMode == kForceClamp;
  constexpr bool kPost = kMode >= kForcePost;
  constexpr bool kKinetic = kMode == kForcePostKinetic || (kPost && kObs);
  extern __shared__ float4 stage[];  // v.stage_cap + 1 entries
  __shared__ StageLayout lay;
  __shared__ LjCoeff table[kMaxTypes * kMaxTypes];
  const uint32_t g = blockIdx.x;
  const uint32_t r = v.block_replica[g];
  const ReplicaParams& p = v.rp[r];
  const int nt = p.n_types;
  for (int t = threadIdx.x; t < nt * nt; t += kThreads) table[t] = v.lj[p.lj_offset + t];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  if (warp == 0) stage_layout(v, p, g, lane, v.stage_cap, lay);
  __syncthreads();
  const bool staged = lay.n_win != 0u;
  if (staged) {
    const uint32_t n_win = lay.n_win;
    for (uint32_t w = warp; w < n_win; w += kThreads / 32) {
      const uint32_t q0 = lay.qbeg[w], b = lay.base[w];
      const uint32_t len = (w + 1u < n_win ? lay.base[w + 1u] : lay.size) - b;
      for (uint32_t t = lane; t < len; t += 32u) stage[b + t] = v.pos[v.cell_atoms[q0 + t]];
    }
    if (threadIdx.x == 0) stage[lay.size] = v.pos[v.n_slots];  // the far particle
    __syncthreads();
  }

  const uint32_t sub = threadIdx.x % kTpa;
  const uint32_t q = g * kBlock + threadIdx.x / kTpa;
  const bool real = q >= lay.q_first && q < lay.q_end;
  // Padding rows are padding slots (inert, never written).
  const uint32_t i = real ? v.cell_atoms[q] : q;
  LjAcc<kTpa> ax, ay, az, ae, aw;
  float4 vm_kick = make_float4(0.f, 0.f, 0.f, 1.f);
  ax.zero();
  ay.zero();
  az.zero();
  ae.zero();
  aw.zero();
  {
    const float4 xi = v.pos[i];
    if (kPost) vm_kick = (real && sub == 0u) ? v.vel[i] : make_float4(0.f, 0.f, 0.f, 1.f);
    CoeffRow<kNt> coeff;
    coeff.init(table + __float_as_int(xi.w) * nt);
    const uint32_t n = real ? v.nbr_count[q] : 0u;
    const uint32_t n_warp = __reduce_max_sync(kFull, n);
    const float rc2 = p.force_cut_sq;
    const float hmin = fminf(p.half[0], fminf(p.half[1], p.half[2]));
    const float half_min_sq = hmin * hmin;
    const float rcm = 1.001f * sqrtf(rc2) + 1e-6f * fmaxf(p.len[0], fmaxf(p.len[1], p.len[2]));
    const bool inside = !real ||
        (xi.x - p.lo[0] >= rcm && p.lo[0] + p.len[0] - xi.x > rcm &&
         xi.y - p.lo[1] >= rcm && p.lo[1] + p.len[1] - xi.y > rcm &&
         xi.z - p.lo[2] >= rcm && p.lo[2] + p.len[2] - xi.z > rcm);
    const bool all_inside = __all_sync(kFull, inside);
    if (staged) {
      if (all_inside) {
        lj_pairs<kObs, kClamp, kTpa, kUnroll, kNoL1, false, kNt, true>(
            v, p, coeff, xi, q, stage, lay.size, sub, n, n_warp, rc2, half_min_sq, ax, ay, az,
            ae, aw);
      } else {
        lj_pairs<kObs, kClamp, kTpa, kUnroll, kNoL1, true, kNt, true>(
            v, p, coeff, xi, q, stage, lay.size, sub, n, n_warp, rc2, half_min_sq, ax, ay, az,
            ae, aw);
      }
    } else {
      if (all_inside) {
        lj_pairs<kObs, kClamp, kTpa, kUnroll, kNoL1, false, kNt>(
            v, p, coeff, xi, q, v.pos, v.n_slots, sub, n, n_warp, rc2, half_min_sq, ax, ay, az,
            ae, aw);
      } else {
        lj_pairs<kObs, kClamp, kTpa, kUnroll, kNoL1, true, kNt>(
            v, p, coeff, xi, q, v.pos, v.n_slots, sub, n, n_warp, rc2, half_min_sq, ax, ay, az,
            ae, aw);
      }
    }
  }
  const float fx = ax.total(), fy = ay.total(), fz = az.total();
  const bool owner = real && sub == 0u;
  if (owner) v.force[i] = make_float4(fx, fy, fz, 0.f);
  ReplicaState* st = &v.rs[r];
  double ke = 0.0;
  if (kPost) ke = post_slot_vm(v, p, st, i, owner, true, kKinetic, vm_kick, fx, fy, fz);
  if (kObs) {
    const float e = ae.total(), w = -aw.total();
    block_add_lane<kThreads>(owner, 0.5 * (double)e, st, kAccPair);
    block_add_lane<kThreads>(owner, 0.5 * (double)w, st, kAccVirial);
  }
  if (kPost && kKinetic) post_partial(v.ke_part, st, r, owner, ke);
}

// Slot-indexed copy of a staged context's list (debug views): out_count[slot]
// and out[slot * cap + k] = neighbour slot, decoding stage indices through the
// group's layout.  One block of 128 threads per group.
__global__ void __launch_bounds__(kBlock) k_list_to_slots(DeviceView v, uint32_t cap,
                                                          uint32_t* out_count, uint32_t* out) {
  __shared__ StageLayout lay;
  const uint32_t g = blockIdx.x;
  const ReplicaParams& p = v.rp[v.block_replica[g]];
  if (threadIdx.x < 32) stage_layout(v, p, g, threadIdx.x, v.stage_cap, lay);
  __syncthreads();
  const uint32_t q = g * kBlock + threadIdx.x;
  if (q < lay.q_first || q >= lay.q_end) return;
  const uint32_t i = v.cell_atoms[q];
  const uint32_t n = v.nbr_count[q];
  out_count[i] = n;
  const uint32_t* list = v.nbr + nbr_index(q, 0, v.nbr_stride);
  for (uint32_t k = 0; k < n && k < cap; ++k) {
    uint32_t e = list[(size_t)k * kGroup];
    if (lay.n_win != 0u) {
      uint32_t w = 0;  // last window whose base <= e
      while (w + 1u < lay.n_win && lay.base[w + 1u] <= e) ++w;
      e = v.cell_atoms[lay.qbeg[w] + (e - lay.base[w])];
    }
    out[(size_t)i * cap + k] = e;
  }
}

template <bool kObs>
__global__ void __launch_bounds__(kBlock) k_bonded_terms(DeviceView v) {
  const uint32_t t = blockIdx.x * kBlock + threadIdx.x;
  if (t < v.n_bond_terms + v.n_angle_terms + v.n_dihedral_terms) bonded_term<kObs>(v, t);
}

template <bool kObs, int kMode>
__global__ void __launch_bounds__(kBlock) k_bonded(DeviceView v) {
  constexpr bool kPost = kMode >= kForcePost;
  const uint32_t r = v.block_replica[blockIdx.x];
  bonded_block<kObs>(v, v.rp[r], r, blockIdx.x, kPost, kMode == kForcePostKinetic || (kPost && kObs),
                     v.ke_part);
}

// ---------------------------------------------------------------------------
// post: second half-kick and kinetic energy (FP64 per slot, one fixed-point
// bucket add per block); k_post_finish then does the per-replica epilogue
// (observables, Berendsen lambda for the next step, applied lazily by pre,
// step counter).  The same per-slot work runs inside the last force kernel
// when the schedule fuses the kick.

template <bool kKick, bool kObs, bool kKinetic>
__global__ void __launch_bounds__(kBlock) k_post(DeviceView v) {
  wait_prior_grid();
  const uint32_t b = blockIdx.x;
  const uint32_t r = v.block_replica[b];
  const ReplicaParams& p = v.rp[r];
  ReplicaState* st = &v.rs[r];
  const uint32_t i = b * kBlock + threadIdx.x;
  const bool real = (i - p.atom_begin) < p.n_atoms;
  float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
  if (kKick && real) f = v.force[i];
  const double ke = post_slot(v, p, st, i, real, kKick, kKinetic || kObs, f.x, f.y, f.z);
  post_partial_block<kKinetic || kObs>(v, st, r, real, ke);
}

// Applies the pending Berendsen scale so host reads see the scaled velocities.
__global__ void k_apply_lambda(DeviceView v) {
  const uint32_t b = blockIdx.x;
  const uint32_t r = v.block_replica[b];
  const ReplicaParams& p = v.rp[r];
  ReplicaState* st = &v.rs[r];
  const uint32_t i = b * kBlock + threadIdx.x;
  const float lam = (float)st->lambda;
  if ((i - p.atom_begin) < p.n_atoms && lam != 1.0f) {
    float4 u = v.vel[i];
    u.x = __fmul_rn(u.x, lam);
    u.y = __fmul_rn(u.y, lam);
    u.z = __fmul_rn(u.z, lam);
    v.vel[i] = u;
  }
  if (arrive_last(&st->done_pre, p.n_pad / kBlock) && threadIdx.x == 0) {
    st->lambda = 1.0;
    st->done_pre = 0u;
  }
}

__global__ void k_scatter_state(DeviceView v, const float* pos_tag,
                                const float* vel_tag, uint32_t n_tags) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_tags) return;
  const uint32_t s = v.slot_of_tag[t];
  if (pos_tag) {
    float4 x = v.pos[s];
    x.x = pos_tag[3 * (size_t)t];
    x.y = pos_tag[3 * (size_t)t + 1];
    x.z = pos_tag[3 * (size_t)t + 2];
    v.pos[s] = x;
  }
  if (vel_tag) {
    float4 u = v.vel[s];
    u.x = vel_tag[3 * (size_t)t];
    u.y = vel_tag[3 * (size_t)t + 1];
    u.z = vel_tag[3 * (size_t)t + 2];
    v.vel[s] = u;
  }
}

__global__ void k_gather_state(DeviceView v, float* pos_tag, float* vel_tag,
                               uint32_t n_tags) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_tags) return;
  const uint32_t s = v.slot_of_tag[t];
  if (pos_tag) {
    const float4 x = v.pos[s];
    pos_tag[3 * (size_t)t] = x.x;
    pos_tag[3 * (size_t)t + 1] = x.y;
    pos_tag[3 * (size_t)t + 2] = x.z;
  }
  if (vel_tag) {
    const float4 u = v.vel[s];
    vel_tag[3 * (size_t)t] = u.x;
    vel_tag[3 * (size_t)t + 1] = u.y;
    vel_tag[3 * (size_t)t + 2] = u.z;
  }
}

void check_launch(const char* what) {
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    throw std::runtime_error(std::string("CUDA launch of ") + what +
                             " failed: " + cudaGetErrorString(e));
  }
}

// Launches a kernel as a programmatic dependent of the previous work in the
// stream (also inside a stream capture): its blocks may be scheduled while
// that work drains, hiding the launch gap, and wait in wait_prior_grid()
// before touching its results.  Used for the short per-step kernels that
// follow another kernel directly.
template <typename... P, typename... A>
void launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t stream,
                      const char* what, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = 0;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
  if (e != cudaSuccess) {
    throw std::runtime_error(std::string("CUDA launch of ") + what +
                             " failed: " + cudaGetErrorString(e));
  }
}

}  // namespace

void launch_pre(const StepLaunch& l, int mode, cudaGraphConditionalHandle cond, bool use_cond) {
  const uint32_t dg = (l.v.n_replicas + 127) / 128;
  if (mode == kPreDescent) {
    launch_dependent(k_pre<kPreDescent>, dim3(l.v.n_blocks), dim3(kBlock), l.stream, "pre", l.v,
                     l.sd_dmax, l.sd_fref);
    launch_dependent(k_decide<kPreDescent>, dim3(dg), dim3(128), l.stream, "decide", l.v, cond,
                     use_cond ? 1 : 0);
  } else {
    launch_dependent(k_pre<kPreVerlet>, dim3(l.v.n_blocks), dim3(kBlock), l.stream, "pre", l.v,
                     0.f, 0.f);
    launch_dependent(k_decide<kPreVerlet>, dim3(dg), dim3(128), l.stream, "decide", l.v, cond,
                     use_cond ? 1 : 0);
  }
  check_launch("decide");
}

void launch_project_exclusions(const StepLaunch& l, bool force_all) {
  if (l.excl_cap == 0) return;
  k_project_exclusions<<<l.v.n_blocks, kBlock, 0, l.stream>>>(l.v, force_all ? 1 : 0);
  check_launch("project_exclusions");
}

void launch_rebuild(const StepLaunch& l, bool force_all, bool count_build) {
  if (force_all) {
    k_force_rebuild_flags<<<(l.v.n_replicas + 127) / 128, 128, 0, l.stream>>>(
        l.v, count_build ? 1 : 0);
    check_launch("force_rebuild_flags");
  }
  // With the block list, the per-slot kernels of the chain walk the
  // rebuilding replicas' blocks with a grid of chain_grid blocks.
  const uint32_t sg = l.v.chain_block_list ? l.chain_grid : l.v.n_blocks;
  if (l.v.chain_block_list) {
    k_chain_blocks<<<1, kScanThreads, 0, l.stream>>>(l.v);
    check_launch("chain blocks");
  }
  k_bin<<<sg, kBlock, 0, l.stream>>>(l.v);
  check_launch("bin");
  if (l.v.n_scan_chunks == l.v.n_replicas) {  // every replica fits one chunk
    k_scan_single<<<l.v.n_replicas, kScanThreads, 0, l.stream>>>(l.v);
    check_launch("scan");
  } else {
    k_scan_sum<<<l.v.n_scan_chunks, kScanThreads, 0, l.stream>>>(l.v);
    check_launch("scan sum");
    k_scan<<<l.v.n_replicas, kScanThreads, 0, l.stream>>>(l.v);
    check_launch("scan");
    k_scan_cells<<<l.v.n_scan_chunks, kScanThreads, 0, l.stream>>>(l.v);
    check_launch("scan cells");
  }
  k_scatter<<<sg, kBlock, 0, l.stream>>>(l.v);
  check_launch("scatter");
  if (l.any_sparse) {
    k_cellsort_sparse<<<(l.v.total_cells + kBlock - 1) / kBlock, kBlock, 0, l.stream>>>(l.v);
    check_launch("cellsort sparse");
  }
  const uint32_t sort_blocks = (l.v.total_cells + kBlock / 32 - 1) / (kBlock / 32);
  if (l.any_dense) {
    k_cellsort<<<sort_blocks, kBlock, 0, l.stream>>>(l.v, 0);
  } else {
    k_cellsort<<<std::min(sort_blocks, 148u), kBlock, 0, l.stream>>>(l.v, 1);
  }
  check_launch("cellsort");
  k_reorder_gather<<<sg, kBlock, 0, l.stream>>>(l.v);
  check_launch("reorder_gather");
  k_reorder_commit<<<sg, kBlock, 0, l.stream>>>(l.v);
  check_launch("reorder_commit");
  if (l.excl_cap > 0) {
    k_project_exclusions<<<l.v.n_blocks, kBlock, 0, l.stream>>>(l.v, 0);
    check_launch("project_exclusions");
  }
  const uint32_t parts = l.build_parts;
  const uint32_t bg = (l.v.total_cells * parts + kBuildWarps - 1) / kBuildWarps;
#define BB_BUILD(excl, q)                                                                  \
  do {                                                                                     \
    if (l.any_dense) k_build<excl, q><<<bg, kBlock, 0, l.stream>>>(l.v, parts);                   \
    if (l.any_sparse) k_build_sparse<excl, q><<<l.v.n_blocks, kBlock, 0, l.stream>>>(l.v); \
  } while (0)
  if (l.excl_cap > 0) {
    if (l.v.list_by_q) BB_BUILD(true, true); else BB_BUILD(true, false);
  } else {
    if (l.v.list_by_q) BB_BUILD(false, true); else BB_BUILD(false, false);
  }
#undef BB_BUILD
  check_launch("build");
}

// Steps that need observables (thermo rows, eval) use the general-table
// kernel at depth 4 with the tuned threads per particle; every variant sums
// forces in the same order, so the choice never shows in the results.
template <int kTpa>
void launch_lj_obs(const StepLaunch& l, int mode) {
  const dim3 grid(l.v.n_blocks * kTpa);
  if (mode == kForcePlain) {
    k_lj<true, kForcePlain, kTpa, 4, true, 0><<<grid, kBlock, 0, l.stream>>>(l.v);
  } else {  // the kinetic total is part of the observables
    k_lj<true, kForcePost, kTpa, 4, true, 0><<<grid, kBlock, 0, l.stream>>>(l.v);
  }
}

template <int kTpa, int kUnroll, bool kNoL1, int kNt>
void launch_lj_tpa(const StepLaunch& l, int mode) {
  const dim3 grid(l.v.n_blocks * kTpa);
#define BB_LJ(m) k_lj<false, m, kTpa, kUnroll, kNoL1, kNt><<<grid, kBlock, 0, l.stream>>>(l.v)
  switch (mode) {
    case kForcePlain: BB_LJ(kForcePlain); break;
    case kForcePost: BB_LJ(kForcePost); break;
    default: BB_LJ(kForcePostKinetic); break;
  }
#undef BB_LJ
}

template <int kTpa, int kUnroll, bool kNoL1>
void launch_lj_nt(const StepLaunch& l, int mode) {
  switch (l.lj_types) {
    case 1: launch_lj_tpa<kTpa, kUnroll, kNoL1, 1>(l, mode); break;
    case 2: launch_lj_tpa<kTpa, kUnroll, kNoL1, 2>(l, mode); break;
    default: launch_lj_tpa<kTpa, kUnroll, kNoL1, 0>(l, mode); break;
  }
}

namespace {

// Staged contexts: every pair-force launch goes to k_lj_staged (the list
// rows are cell-order rows there), with (stage_cap + 1) float4 of dynamic
// shared memory.
size_t staged_smem(const StepLaunch& l) { return (size_t)(l.v.stage_cap + 1u) * sizeof(float4); }

template <bool kObs, int kMode, int kTpa>
void staged_one(const StepLaunch& l) {
  k_lj_staged<kObs, kMode, kTpa><<<l.v.n_blocks, kBlock * kTpa, staged_smem(l), l.stream>>>(l.v);
}

template <bool kObs, int kMode, int kTpa>
void staged_attr(size_t smem) {
  const cudaError_t e = cudaFuncSetAttribute(k_lj_staged<kObs, kMode, kTpa>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) {
    throw std::runtime_error(std::string("staged pair kernel shared memory: ") +
                             cudaGetErrorString(e));
  }
}

template <int kTpa>
void staged_attrs(size_t smem) {
  staged_attr<true, kForcePlain, kTpa>(smem);
  staged_attr<true, kForcePost, kTpa>(smem);
  staged_attr<false, kForcePlain, kTpa>(smem);
  staged_attr<false, kForcePost, kTpa>(smem);
  staged_attr<false, kForcePostKinetic, kTpa>(smem);
}

template <int kTpa>
void launch_staged(const StepLaunch& l, bool observables, int mode) {
  if (observables) {
    if (mode == kForcePlain) staged_one<true, kForcePlain, kTpa>(l);
    else staged_one<true, kForcePost, kTpa>(l);
  } else {
    switch (mode) {
      case kForcePlain: staged_one<false, kForcePlain, kTpa>(l); break;
      case kForcePost: staged_one<false, kForcePost, kTpa>(l); break;
      default: staged_one<false, kForcePostKinetic, kTpa>(l); break;
    }
  }
}

void launch_forces_staged(const StepLaunch& l, bool observables, bool clamp, int mode) {
  if (clamp) {
    staged_one<false, kForceClamp, 2>(l);
  } else {
    switch (l.lj_tpa) {
      case 2: launch_staged<2>(l, observables, mode); break;
      case 4: launch_staged<4>(l, observables, mode); break;
      default: launch_staged<1>(l, observables, mode); break;
    }
  }
  check_launch("lj_staged");
}

}  // namespace

// Raises the dynamic shared-memory limit of every staged pair-force variant to
// at least `smem` bytes (once per context, outside any stream capture).  The
// limit belongs to the kernels on a device, so it is never lowered: another
// context may need the larger one.
void prepare_staged_kernels(size_t smem) {
  static std::mutex mutex;
  static std::map<int, size_t> limits;
  const std::lock_guard<std::mutex> lock(mutex);
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess) throw std::runtime_error("no CUDA device");
  size_t& limit = limits[device];
  if (smem <= limit) return;
  staged_attr<false, kForceClamp, 2>(smem);
  staged_attrs<1>(smem);
  staged_attrs<2>(smem);
  staged_attrs<4>(smem);
  limit = smem;
}

void launch_list_to_slots(const StepLaunch& l, uint32_t cap, uint32_t* out_count, uint32_t* out) {
  k_list_to_slots<<<l.v.n_blocks, kBlock, 0, l.stream>>>(l.v, cap, out_count, out);
  check_launch("list_to_slots");
}

void launch_forces(const StepLaunch& l, bool observables, bool clamp, bool post, int parts) {
  const bool fuse = post && l.fuse_post != 0;
  const int fin = !fuse ? kForcePlain : (l.need_kinetic ? kForcePostKinetic : kForcePost);
  const bool bonded = l.v.has_bonded != 0 && (parts & kForceBonded) != 0;
  if ((parts & kForcePair) == 0) {
    // bonded terms alone (profiling)
  } else if (l.v.list_by_q) {
    launch_forces_staged(l, observables, clamp, bonded ? kForcePlain : fin);
  } else if (clamp) {
    k_lj<false, kForceClamp, 1, 8, false, 0><<<l.v.n_blocks, kBlock, 0, l.stream>>>(l.v);
  } else if (observables) {
    const int mode = bonded ? kForcePlain : fin;
    switch (l.lj_tpa) {
      case 2: launch_lj_obs<2>(l, mode); break;
      case 4: launch_lj_obs<4>(l, mode); break;
      default: launch_lj_obs<1>(l, mode); break;
    }
  } else {
    const int mode = bonded ? kForcePlain : fin;
    // (threads per particle, batch depth, list load policy) -> one instantiation
    const int key = l.lj_tpa * 100 + l.lj_unroll * 10 + (l.lj_no_l1 ? 1 : 0);
    switch (key) {
#define BB_CASE(t, u, pf) \
  case t * 100 + u * 10 + pf: launch_lj_nt<t, u, pf != 0>(l, mode); break;
      BB_CASE(1, 8, 0) BB_CASE(1, 8, 1) BB_CASE(1, 4, 0) BB_CASE(1, 4, 1)
      BB_CASE(2, 8, 0) BB_CASE(2, 8, 1) BB_CASE(2, 4, 0) BB_CASE(2, 4, 1)
      BB_CASE(4, 8, 0) BB_CASE(4, 8, 1) BB_CASE(4, 4, 0) BB_CASE(4, 4, 1)
#undef BB_CASE
      default: throw std::runtime_error("unsupported pair-force schedule");
    }
  }
  if (parts & kForcePair) check_launch("lj");
  if (bonded) {
    const uint32_t n_terms = l.v.n_bond_terms + l.v.n_angle_terms + l.v.n_dihedral_terms;
    const uint32_t tg = (n_terms + kBlock - 1) / kBlock;
    if (tg > 0) {
      if (observables) {
        k_bonded_terms<true><<<tg, kBlock, 0, l.stream>>>(l.v);
      } else {
        k_bonded_terms<false><<<tg, kBlock, 0, l.stream>>>(l.v);
      }
      check_launch("bonded terms");
    }
#define BB_BONDED(obs, mode) k_bonded<obs, mode><<<l.v.n_blocks, kBlock, 0, l.stream>>>(l.v)
    if (observables) {
      if (fin == kForcePlain) BB_BONDED(true, kForcePlain);
      else BB_BONDED(true, kForcePost);
    } else {
      switch (fin) {
        case kForcePlain: BB_BONDED(false, kForcePlain); break;
        case kForcePost: BB_BONDED(false, kForcePost); break;
        default: BB_BONDED(false, kForcePostKinetic); break;
      }
    }
#undef BB_BONDED
    check_launch("bonded");
  }
  if (fuse) {
    const bool kin = fin == kForcePostKinetic || observables;
    const dim3 fg(l.v.n_replicas), ft(kFinishThreads);
    if (observables) {
      launch_dependent(k_post_finish<true, true, true>, fg, ft, l.stream, "post finish", l.v);
    } else if (kin) {
      launch_dependent(k_post_finish<true, false, true>, fg, ft, l.stream, "post finish", l.v);
    } else {
      launch_dependent(k_post_finish<true, false, false>, fg, ft, l.stream, "post finish", l.v);
    }
    check_launch("post finish");
  }
  if (post && !fuse) launch_post(l, true, observables);
}

void launch_post(const StepLaunch& l, bool kick, bool observables) {
  const bool kin = l.need_kinetic != 0;
  const dim3 fg(l.v.n_replicas);
  if (kick) {
    if (observables) {
      launch_dependent(k_post<true, true, true>, dim3(l.v.n_blocks), dim3(kBlock), l.stream,
                       "post", l.v);
      launch_dependent(k_post_finish<true, true, true>, dim3(fg), dim3(kFinishThreads), l.stream,
                       "post finish", l.v);
    } else if (kin) {
      launch_dependent(k_post<true, false, true>, dim3(l.v.n_blocks), dim3(kBlock), l.stream,
                       "post", l.v);
      launch_dependent(k_post_finish<true, false, true>, dim3(fg), dim3(kFinishThreads), l.stream,
                       "post finish", l.v);
    } else {
      launch_dependent(k_post<true, false, false>, dim3(l.v.n_blocks), dim3(kBlock), l.stream,
                       "post", l.v);
      launch_dependent(k_post_finish<true, false, false>, dim3(fg), dim3(kFinishThreads), l.stream,
                       "post finish", l.v);
    }
  } else {
    launch_dependent(k_post<false, true, true>, dim3(l.v.n_blocks), dim3(kBlock), l.stream,
                     "post", l.v);
    launch_dependent(k_post_finish<false, true, true>, dim3(fg), dim3(kFinishThreads), l.stream,
                     "post finish", l.v);
  }
  check_launch("post");
}

void launch_apply_lambda(const StepLaunch& l) {
  k_apply_lambda<<<l.v.n_blocks, kBlock, 0, l.stream>>>(l.v);
  check_launch("apply_lambda");
}

void launch_scatter_state(const StepLaunch& l, const float* pos_tag,
                          const float* vel_tag, uint32_t n_tags_total) {
  k_scatter_state<<<(n_tags_total + 255) / 256, 256, 0, l.stream>>>(
      l.v, pos_tag, vel_tag, n_tags_total);
  check_launch("scatter_state");
}

void launch_gather_state(const StepLaunch& l, float* pos_tag, float* vel_tag,
                         uint32_t n_tags_total) {
  k_gather_state<<<(n_tags_total + 255) / 256, 256, 0, l.stream>>>(
      l.v, pos_tag, vel_tag, n_tags_total);
  check_launch("gather_state");
}

}  // namespace bb
