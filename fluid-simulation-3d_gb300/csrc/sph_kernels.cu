// SPH substep kernels for GB300 (sm_103a).
//
// One substep (engine/physics/physicsWorld.cc:39-111) is:
//   k_predict_hash   gravity + prediction + cell index + key, counting-sort
//                    histogram (warp-aggregated atomics)    :42-48, :473-482
//   k_scan_*         exclusive prefix of the key histogram = start table
//   k_scatter        bucket each particle at start[key] + arrival rank
//   k_reorder        deterministic order inside each bucket and gather of
//                    the state into SoA float4                :484-496
//   k_cell_table     per cell, its neighbour runs (the bucket walk of
//                    :331-346 resolved once per cell instead of per particle)
//   k_density_*      density / near density and neighbour lists :304-365
//   k_pressure       pressure + near pressure over the list   :367-422
//   k_visc_integrate Jacobi viscosity over the list, integrate, box
//                    collision, next substep's prediction    :424-464, :81-108
// and, when a substep is captured for export, k_ref_* rebuild the
// reference's own spatial lookup (HashCell keys, (key, index) order and
// startIndices, :466-496) from the same predicted positions.
//
// The neighbour kernels come in forms for small launches (k_density_rows,
// k_pressure_coop, k_visc_coop, k_cell_table_rows), the general ones, and ones
// with another register cap (k_visc_dense); they give the same bits, and the
// rules beside the launchers choose by the launch's tiles.
//
// The sort key is the internal cell index (sph_device.cuh), modulo the scene
// size where the grid is too large for a table of its own; inside a key bucket
// particles are ordered by (cell index, particle index), so every cell is a
// contiguous run of slots and the three cells of an x-row usually one run.
// Every kernel is a segmented launch: warps stride over a tile table of
// (scene, first slot) runs of up to 32 particles of one scene, so one launch
// serves any number of scenes of uneven sizes.
#include "sph_kernels.h"

#include <algorithm>
#include <array>

namespace sph {

namespace {

constexpr uint32_t kFull = 0xffffffffu;

__device__ __forceinline__ uint32_t warp_id_global() {
  return blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
}
__device__ __forceinline__ uint32_t warps_total() {
  return gridDim.x * (blockDim.x >> 5);
}
__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31; }

// glm dot(v, v) of physicsWorld.cc:355: three rounded products summed left to
// right (no FMA contraction), so boundary pairs classify as in the reference.
__device__ __forceinline__ float dist2(float dx, float dy, float dz) {
  return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)),
                   __fmul_rn(dz, dz));
}
// Fast estimate of the same value (within a few ulp of dist2).
__device__ __forceinline__ float dist2_fast(float dx, float dy, float dz) {
  return fmaf(dz, dz, fmaf(dy, dy, dx * dx));
}
// Hardware square root estimate (0 -> 0). The form that flushes denormals is
// faster (walk 172 -> 164 us at 1M, 1204 -> 1140 us at 8.4M) and changes no
// density: the result is only used as r - sqrt(d2), a denormal d2 has sqrt(d2) <
// 1.1e-19, and r - 1.1e-19 rounds to r for every radius whose 1/r^5 kernel scale
// is finite.
__device__ __forceinline__ float sqrt_approx(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void flag(uint32_t* status, uint32_t f) {
  atomicOr(status, f);
}

// Entry k of slot i's neighbour list. Groups of 32 slots own kNbrCap rows of
// 32 entries (8 KB), so a warp's appends and loads of one entry are contiguous
// and all its rows lie side by side. A row per entry number over all slots
// (the lists' rows a whole capacity apart) made each warp touch some 30 pages
// at once: at 8.4M particles (33 MB between rows) the density walk took
// 1526 us against 1204 us with this layout, the pass of two substeps 6.32
// against 5.67 ms; at 1M 820 against 812 us. 64-bit: slots * kNbrCap passes
// 2^32 for capacities above 2^26.
__device__ __forceinline__ uint64_t nbr_index(uint32_t i, uint32_t k) {
  return static_cast<uint64_t>(i & ~31u) * kNbrCap + k * 32u + (i & 31u);
}

// The viscosity pass's particle records, (predicted position, post-pressure
// velocity), six floats. The plain force kernels keep them as a float4 (x, y,
// z, vx) and a float2 (vy, vz): their gathers are bound by the L1 data pipe,
// which 24 B a neighbour load less than one padded 32-byte record (one
// 256-bit load): viscosity at 1M 91 -> 83 us, at 8.4M 599 -> 585 us. The
// latency forms, which wait on loads and not on the pipe, take the 32-byte
// record and half the loads (16,384 particles: 2 us a substep).
__device__ __forceinline__ void load_state(const float4* __restrict__ rec,
                                           const float2* __restrict__ rec_b, uint32_t j,
                                           float4& a, float4& b) {
  const float4 x = __ldg(rec + j);
  const float2 y = __ldg(rec_b + j);
  a = make_float4(x.x, x.y, x.z, 0.0f);
  b = make_float4(x.w, y.x, y.y, 0.0f);
}
__device__ __forceinline__ void store_state(float4* __restrict__ rec, float2* __restrict__ rec_b,
                                            uint32_t i, float4 a, float4 b) {
  rec[i] = make_float4(a.x, a.y, a.z, b.x);
  rec_b[i] = make_float2(b.y, b.z);
}
__device__ __forceinline__ void load_rec(const float4* __restrict__ rec,
                                         uint32_t j, float4& a, float4& b) {
  asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y),
                 "=f"(b.z), "=f"(b.w)
               : "l"(rec + 2ull * j)
               : "memory");
}
__device__ __forceinline__ void store_rec(float4* __restrict__ rec, uint32_t i,
                                          float4 a, float4 b) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               :
               : "l"(rec + 2ull * i), "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w),
                 "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
               : "memory");
}

// kGather consecutive entries of slot i's list from entry k0, those below
// cnt (<= the list capacity) only: a batch of 3 that starts near the end of
// a full list would otherwise read past the list rows. Each entry is read
// once per pass, so the loads carry the streaming (evict-first) hint and
// leave the cache to the neighbours' gathered state.
// With kStep = 2 (two lanes per particle) a lane reads every other entry:
// k0, k0 + 2, ...
template <int kGather, int kStep = 1>
__device__ __forceinline__ void load_nbr_batch(const uint32_t* __restrict__ nbr,
                                               uint32_t i, uint32_t k0, uint32_t cnt,
                                               uint32_t (&j)[kGather]) {
  const uint32_t* p = nbr + nbr_index(i, k0);
#pragma unroll
  for (int u = 0; u < kGather; ++u)
    j[u] = k0 + kStep * u < cnt ? __ldcs(p + kStep * u * 32) : 0u;
}

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t x) {
  const uint32_t lane = lane_id();
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, x, d);
    if (lane >= static_cast<uint32_t>(d)) x += y;
  }
  return x;
}

// Rank among the lanes of the warp that share `key`, and one atomicAdd per
// distinct key (particles stored in the previous sorted order share cells
// with their warp neighbours). All 32 lanes must call; inactive lanes pass
// active = false and get 0.
__device__ __forceinline__ uint32_t aggregated_rank(uint32_t* count,
                                                    uint32_t key,
                                                    bool active) {
  const uint32_t am = __ballot_sync(kFull, active);
  if (!active) return 0u;
  const uint32_t lane = lane_id();
  const uint32_t peers = __match_any_sync(am, key);
  const int leader = __ffs(peers) - 1;
  uint32_t base = 0;
  if (static_cast<int>(lane) == leader) base = atomicAdd(count + key, __popc(peers));
  base = __shfl_sync(peers, base, leader);
  return base + __popc(peers & ((1u << lane) - 1u));
}

// Row w (dy = w/3 - 1, dz = w%3 - 1) of a cell of a direct key table: its
// three x-neighbour cells are consecutive table entries, so the row is one
// run from two start-table reads. k0 = tbase + cell - gwy - gwz, the entry of
// row 0's middle cell.
__device__ __forceinline__ uint2 direct_row(const SceneDev& S,
                                            const uint32_t* __restrict__ start,
                                            uint32_t k0, int w) {
  const uint32_t k = k0 + static_cast<uint32_t>(w / 3) * S.gwy +
                     static_cast<uint32_t>(w % 3) * S.gwz;
  const uint32_t f = __ldg(start + k - 1);
  return make_uint2(f, (__ldg(start + k + 2) - f) | kRunMerged);
}

// Neighbour walk of a particle: the particles of its cell's 27 neighbour
// cells -- every candidate the reference's bucket loops would accept within
// the cutoff -- row by row, a merged row as one run. A direct key table
// gives each row from the start table (cell = the particle's cell index);
// otherwise the rows come from the cell's table built by k_cell_table (cf =
// the cell's first slot). Both visit the same particles in the same order.
template <int kTables, class F>
__device__ __forceinline__ void walk_runs(const SceneDev& S,
                                          const uint32_t* __restrict__ start,
                                          const uint2* __restrict__ cell_tab,
                                          uint32_t cf, uint32_t cell,
                                          const float4* __restrict__ pred,
                                          F&& visit) {
  const bool direct = kTables == kTablesDirect    ? true
                    : kTables == kTablesBuckets ? false
                                                : S.direct != 0u;
  if (direct) {
    // rows (dy, dz) in the cell table's order (dz fastest); k = the row's
    // middle cell
    uint32_t k = S.tbase + cell - S.gwy - S.gwz;
    int dz = 0;
#pragma unroll 1
    for (int w = 0; w < 9; ++w) {
      const uint32_t e = __ldg(start + k + 2);
#pragma unroll 1
      for (uint32_t j = __ldg(start + k - 1); j < e; ++j) visit(j, __ldg(pred + j));
      if (++dz == 3) { dz = 0; k += S.gwy - 2u * S.gwz; } else { k += S.gwz; }
    }
    return;
  }
  const uint2* row = cell_tab + static_cast<uint64_t>(cf) * 27u;
#pragma unroll 1
  for (int w = 0; w < 9; ++w, row += 3) {
    const uint2 m = __ldg(row);
    if (m.y & kRunMerged) {
      const uint32_t e = m.x + (m.y & ~kRunMerged);
#pragma unroll 1
      for (uint32_t j = m.x; j < e; ++j) visit(j, __ldg(pred + j));
    } else {
#pragma unroll 1
      for (int k = 0; k < 3; ++k) {
        const uint2 run = k ? __ldg(row + k) : m;
#pragma unroll 1
        for (uint32_t j = run.x; j < run.x + run.y; ++j) visit(j, __ldg(pred + j));
      }
    }
  }
}

// One row of the same walk for the latency forms, visit(j, q, true) for its
// particles in the same order, kBatch candidates in flight (one at a time, a
// candidate costs an L2 round trip; the last batch repeats the run's last
// particle with false). k: the table entry of the row's middle cell in a
// direct table; tab: the row's entries in the cell table. A run is walked if
// enter(its length) says so.
template <int kTables, uint32_t kBatch, class Enter, class F>
__device__ __forceinline__ void walk_row(bool direct, const uint32_t* __restrict__ start,
                                         uint32_t k, const uint2* __restrict__ tab,
                                         const float4* __restrict__ pred, Enter&& enter,
                                         F&& visit) {
  auto run = [&](uint32_t j, uint32_t e) {
    if (!enter(e - j)) return;
    for (; j < e; j += kBatch) {
      float4 q[kBatch];
#pragma unroll
      for (uint32_t u = 0; u < kBatch; ++u) q[u] = __ldg(pred + min(j + u, e - 1u));
#pragma unroll
      for (uint32_t u = 0; u < kBatch; ++u) visit(j + u, q[u], j + u < e);
    }
  };
  if (kTables == kTablesDirect || (kTables == kTablesMixed && direct)) {
    run(__ldg(start + k - 1), __ldg(start + k + 2));
    return;
  }
  const uint2 m = __ldg(tab);
  if (m.y & kRunMerged) {
    run(m.x, m.x + (m.y & ~kRunMerged));
    return;
  }
#pragma unroll 1
  for (int c = 0; c < 3; ++c) {
    const uint2 x = c ? __ldg(tab + c) : m;
    run(x.x, x.x + x.y);
  }
}

// walk_runs by walk_row.
template <int kTables, uint32_t kBatch, class F>
__device__ __forceinline__ void walk_rows(const SceneDev& S, const uint32_t* __restrict__ start,
                                          const uint2* __restrict__ cell_tab, uint32_t cf,
                                          uint32_t cell, const float4* __restrict__ pred,
                                          F&& visit) {
#pragma unroll 1
  for (uint32_t w = 0; w < 9u; ++w)
    walk_row<kTables, kBatch>(S.direct != 0u, start,
                              S.tbase + cell + (w / 3u - 1u) * S.gwy + (w % 3u - 1u) * S.gwz,
                              cell_tab + static_cast<uint64_t>(cf) * 27u + 3u * w, pred,
                              [](uint32_t) { return true; }, visit);
}

// --------------------------------------------------------- scenes and tiles
// Part of the scene table as a kernel parameter (up to the parameters' 4 KB,
// and 32 KB for large batches): it needs no staging memory and no wait, and is
// copied when the launch is made.
template <int N> struct SceneChunk {
  SceneDev s[N];
};
constexpr int kFewScenes = 4000 / sizeof(SceneDev);
constexpr int kManyScenes = 32000 / sizeof(SceneDev);

template <int N>
__global__ void k_scenes(const __grid_constant__ SceneChunk<N> chunk, uint32_t words,
                         uint32_t* __restrict__ table) {
  pdl_launch();
  const uint32_t* w = reinterpret_cast<const uint32_t*>(&chunk);
  for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) table[i] = w[i];
}

// Tile tables after a change of the layout, a thread a tile: its scene is the
// last one whose first tile is not past it (a scene without particles shares
// its first tile with the next). 16 B a tile, so bound by the launch.
__global__ void k_tiles(const SceneDev* __restrict__ scene_table, uint32_t scenes, uint32_t ntiles,
                        uint2* __restrict__ tiles_old, uint2* __restrict__ tiles_new) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ntiles) return;
  uint32_t lo = 0, hi = pdl_wait(scenes);  // tile0 of lo is <= t, of hi (if any) > t
  while (hi - lo > 1u) {
    const uint32_t mid = lo + (hi - lo) / 2u;
    if (scene_table[mid].tile0 <= t) lo = mid; else hi = mid;
  }
  const SceneDev& S = scene_table[lo];
  const uint32_t f = (t - S.tile0) * kTile, len = min(static_cast<uint32_t>(kTile), S.n - f);
  tiles_old[t] = make_tile(lo, S.old_base + f, len);
  tiles_new[t] = make_tile(lo, S.base + f, len);
}

// ----------------------------------------------------------------- predict
__device__ __forceinline__ void predict_key(const SceneDev& S, float4 p,
                                            float4 v, uint32_t& key,
                                            uint32_t& cell) {
  float3 vn, pr;
  predict(S, p, v, vn, pr);
  cell = cell_index(S, pr);
  key = table_key(S, cell);
}

__global__ void k_predict_hash(const uint2* __restrict__ tiles, uint32_t ntiles,
                               const SceneDev* __restrict__ scenes,
                               const float4* __restrict__ pos,
                               const float4* __restrict__ vel,
                               uint32_t* __restrict__ count,
                               uint4* __restrict__ keyrank) {
  pdl_launch();
  const uint32_t lane = lane_id();
  for (uint32_t t = warp_id_global(); t < ntiles; t += warps_total()) {
    const uint2 tile = tiles[t];
    const SceneDev S = scenes[tile_scene(tile)];  // registers, not reloads
    const uint32_t s = pdl_wait(tile.y) + lane;
    const bool live = lane < tile_len(tile);
    uint32_t key = 0, cell = 0, id = 0;
    if (live) {
      const float4 p = pos[s];
      predict_key(S, p, vel[s], key, cell);
      id = __float_as_uint(p.w);
    }
    const uint32_t r = aggregated_rank(count, key, live);
    if (live) keyrank[s] = make_uint4(key, r, cell, id);
  }
}

// -------------------------------------------------------------------- scan
constexpr int kScanThreads = 512;
constexpr int kScanItems = 4;
constexpr int kScanBlock = kScanThreads * kScanItems;
constexpr uint32_t kScanFoldBlocks = 4096;  // fold the partials scan up to here

// Block-wide exclusive scan of one value per thread; returns the block total
// through *total.
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t x,
                                                    uint32_t* total) {
  __shared__ uint32_t warp_sums[32];
  const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
  const uint32_t incl = warp_incl_scan(x);
  if (lane == 31) warp_sums[w] = incl;
  __syncthreads();
  if (w == 0) {
    const uint32_t nw = blockDim.x >> 5;
    uint32_t v = lane < nw ? warp_sums[lane] : 0u;
    v = warp_incl_scan(v);
    warp_sums[lane] = v;
  }
  __syncthreads();
  const uint32_t before = w > 0 ? warp_sums[w - 1] : 0u;
  *total = warp_sums[(blockDim.x >> 5) - 1];
  __syncthreads();
  return before + incl - x;
}

// The kScanItems (= 4) consecutive counts of a thread: one 16-byte load
// inside the table, element loads at its ragged end.
__device__ __forceinline__ uint4 load_counts(const uint32_t* __restrict__ count, uint32_t b0,
                                             uint32_t len) {
  if (b0 + 4u <= len) return *reinterpret_cast<const uint4*>(count + b0);
  uint4 v = make_uint4(0u, 0u, 0u, 0u);
  if (b0 < len) v.x = count[b0];
  if (b0 + 1u < len) v.y = count[b0 + 1u];
  if (b0 + 2u < len) v.z = count[b0 + 2u];
  return v;
}

__global__ void __launch_bounds__(kScanThreads)
k_scan_reduce(const uint32_t* __restrict__ count, uint32_t len,
              uint32_t* __restrict__ partial) {
  static_assert(kScanItems == 4, "one uint4 of counts per thread");
  const uint32_t b0 = pdl_enter(blockIdx.x * kScanBlock + threadIdx.x * kScanItems);
  const uint4 v = load_counts(count, b0, len);
  uint32_t total;
  block_excl_scan(v.x + v.y + v.z + v.w, &total);
  if (threadIdx.x == 0) partial[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads)
k_scan_partials(uint32_t* __restrict__ partial, uint32_t nb,
                uint32_t* __restrict__ start, uint32_t len) {
  const uint32_t thread = pdl_enter(threadIdx.x);
  uint32_t carry = 0;
  for (uint32_t c = 0; c < nb; c += kScanThreads) {
    const uint32_t i = c + thread;
    const uint32_t v = i < nb ? partial[i] : 0u;
    uint32_t total;
    const uint32_t ex = block_excl_scan(v, &total);
    if (i < nb) partial[i] = carry + ex;
    carry += total;
  }
  if (threadIdx.x == 0) start[len] = carry;
}

// Down-sweep. With `fold` the block totals in `partial` are raw (no
// k_scan_partials): each block sums the totals before it itself -- O(nb^2)
// reads in all, so the launcher folds only up to kScanFoldBlocks blocks --
// and the last block writes the grand total start[len]. The block's own
// counts are loaded first, so their latency overlaps the fold's reads, and
// one block pass both scans the counts and sums the fold.
__global__ void __launch_bounds__(kScanThreads)
k_scan_down(uint32_t* __restrict__ count, uint32_t len,
            const uint32_t* __restrict__ partial, uint32_t nb, int fold,
            uint32_t* __restrict__ start) {
  __shared__ uint32_t warp_scan[kScanThreads / 32], warp_fold[kScanThreads / 32];
  const uint32_t block = pdl_enter(blockIdx.x);
  const uint32_t b0 = block * kScanBlock + threadIdx.x * kScanItems;
  const uint4 v = load_counts(count, b0, len);
  uint32_t f = 0;
  if (fold) {
    for (uint32_t c = threadIdx.x; c < block; c += kScanThreads) f += partial[c];
  }
  const uint32_t s = v.x + v.y + v.z + v.w;
  const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
  const uint32_t incl = warp_incl_scan(s);
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) f += __shfl_xor_sync(kFull, f, d);
  if (lane == 31) warp_scan[w] = incl;
  if (lane == 0) warp_fold[w] = f;
  __syncthreads();
  constexpr uint32_t kWarps = kScanThreads / 32;
  uint32_t before = 0, block_total = 0, base = 0;
#pragma unroll
  for (uint32_t u = 0; u < kWarps; ++u) {  // smem broadcasts: every lane reads the same word
    const uint32_t ws = warp_scan[u];
    before += u < w ? ws : 0u;
    block_total += ws;
    base += warp_fold[u];
  }
  if (!fold) base = partial[block];
  uint32_t run = base + before + incl - s;
  if (b0 + 4u <= len) {
    uint4 o;
    o.x = run;
    o.y = o.x + v.x;
    o.z = o.y + v.y;
    o.w = o.z + v.z;
    *reinterpret_cast<uint4*>(start + b0) = o;
    *reinterpret_cast<uint4*>(count + b0) = make_uint4(0u, 0u, 0u, 0u);  // next histogram
  } else {
    const uint32_t vv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
      if (b0 + k < len) {
        start[b0 + k] = run;
        count[b0 + k] = 0u;
      }
      run += vv[k];
    }
  }
  if (fold && block + 1 == nb && threadIdx.x == 0) start[len] = base + block_total;
}

// ----------------------------------------------------------------- scatter
__global__ void k_scatter(const uint2* __restrict__ tiles, uint32_t ntiles,
                          const uint4* __restrict__ keyrank,
                          const uint32_t* __restrict__ start, uint32_t total,
                          uint2* __restrict__ tmp_hi,
                          uint32_t* __restrict__ tmp_src, uint32_t* status) {
  pdl_launch();
  const uint32_t lane = lane_id();
  for (uint32_t t = warp_id_global(); t < ntiles; t += warps_total()) {
    const uint2 tile = tiles[t];
    const uint32_t s = pdl_wait(tile.y) + lane;
    if (lane >= tile_len(tile)) continue;
    const uint4 kr = keyrank[s];
    const uint32_t dst = start[kr.x] + kr.y;
    if (dst >= total) { flag(status, kStatusRange); continue; }
    tmp_hi[dst] = make_uint2(kr.z, kr.w);
    tmp_src[dst] = s;
  }
}

// ----------------------------------------------------------------- reorder
// Thread per bucketed slot: rank the particle inside its bucket by
// (cell index, particle index), recompute its gravity/prediction exactly as
// k_predict_hash did, and write the state to its final slot. kCells: also its
// cell index and the first slot of its cell (its run of equal cell index), which
// the cell table and the cell-tile density read; where every table is a grid a
// bucket is one cell, and nothing reads the two (8 of 104 B a particle: 8.4M
// 231 -> 217 us for the whole sort).
template <bool kCells>
__global__ void k_reorder(const uint2* __restrict__ tiles, uint32_t ntiles,
                          const SceneDev* __restrict__ scenes,
                          const uint2* __restrict__ tmp_hi,
                          const uint32_t* __restrict__ tmp_src,
                          const uint32_t* __restrict__ start,
                          const float4* __restrict__ pos_in,
                          const float4* __restrict__ vel_in,
                          float4* __restrict__ pos_out,
                          float4* __restrict__ vel_out,
                          float4* __restrict__ pred,
                          uint32_t* __restrict__ hash_s,
                          uint32_t* __restrict__ cell_first,
                          uint32_t src_limit, uint32_t* status) {
  pdl_launch();
  const uint32_t lane = lane_id();
  for (uint32_t t = warp_id_global(); t < ntiles; t += warps_total()) {
    const uint2 tile = tiles[t];
    const SceneDev S = scenes[tile_scene(tile)];  // registers, not reloads
    const uint32_t slot = pdl_wait(tile.y) + lane;
    if (lane >= tile_len(tile)) continue;
    const uint2 me = tmp_hi[slot];
    const uint32_t src = tmp_src[slot];
    if (src >= src_limit) { flag(status, kStatusRange); continue; }
    const float4 p = pos_in[src];
    const float4 v = vel_in[src];
    float3 vn, pr;
    predict(S, p, v, vn, pr);
    // the cell index travelled with the entry: k_predict_hash (or the fused
    // prediction) computed it from this same prediction
    const uint32_t cell = me.x;
    const uint32_t key = table_key(S, cell);
    const uint32_t b0 = start[key], b1 = start[key + 1];
    if (slot < b0 || slot >= b1) {
      flag(status, kStatusRange);
      continue;
    }
    uint32_t rank = 0, below = 0;
    for (uint32_t u = b0; u < b1; ++u) {
      const uint2 o = tmp_hi[u];
      if (kCells) {
        below += (o.x < me.x) ? 1u : 0u;
        rank += (o.x < me.x || (o.x == me.x && o.y < me.y)) ? 1u : 0u;
      } else {
        rank += o.y < me.y ? 1u : 0u;
      }
    }
    const uint32_t f = b0 + rank;
    pos_out[f] = p;
    vel_out[f] = make_float4(vn.x, vn.y, vn.z, 0.0f);
    pred[f] = make_float4(pr.x, pr.y, pr.z, __uint_as_float(cell));
    if (kCells) {
      hash_s[f] = cell;
      cell_first[f] = b0 + below;
    }
  }
}

// -------------------------------------------------------------- cell table
// The run of cell index `cell` in its key bucket [b0, b1). A bucket is
// sorted by cell index, so the cell's particles are one run and entries of
// other cells that share the bucket are left out, as the reference's
// float(hash) test leaves them out (:346); a bucket holding a single cell is
// the common case and is recognised from its first and last entries.
__device__ __forceinline__ uint2 bucket_run(uint32_t cell, uint32_t b0,
                                            uint32_t b1,
                                            const uint32_t* __restrict__ hash_s) {
  uint32_t first = b0, len = 0;
  if (b1 > b0) {
    const uint32_t h0 = __ldg(hash_s + b0), h1 = __ldg(hash_s + b1 - 1);
    if (h0 == cell && h1 == cell) {
      len = b1 - b0;
    } else if (h0 <= cell && cell <= h1) {
      for (uint32_t u = b0; u < b1; ++u) {
        const bool eq = __ldg(hash_s + u) == cell;
        if (eq && len == 0) first = u;
        len += eq ? 1u : 0u;
      }
    }
  }
  return make_uint2(first, len);
}

// For each cell (its first slot) of a scene with a bucket key table, the
// runs of its 27 neighbour cells as 9 rows (dy, dz) of three x-runs. The
// x-neighbours of a row have consecutive cell indices, hence consecutive
// keys; when their runs are adjacent in the layout (their buckets hold no
// other cell -- the usual case inside the box) the row is stored as one run
// flagged kRunMerged in its first entry (its other two entries are left
// unwritten: a third of the table's stores, which the readers skip).
// cell_row: row w of the cell whose first slot is `slot`.
__device__ __forceinline__ void cell_row(const SceneDev& S, uint32_t slot, uint32_t w, uint32_t kmax,
                                         const uint32_t* __restrict__ hash_s,
                                         const uint32_t* __restrict__ start,
                                         uint2* __restrict__ cell_tab) {
  const uint32_t dy = w / 3u - 1u, dz = w % 3u - 1u;  // mod 2^32
  const uint32_t mid = __ldg(hash_s + slot) + dy * S.gwy + dz * S.gwz;
  uint2* out = cell_tab + static_cast<uint64_t>(slot) * 27u + 3u * w;
  // keys of mid - 1, mid, mid + 1: neighbours of mid's key modulo n,
  // except across the 2^32 wrap of the index
  const uint32_t km = fastmod(mid, S.fm, S.n);
  const uint32_t kl = mid == 0u ? kmax : (km == 0u ? S.n - 1u : km - 1u);
  const uint32_t kh = mid == 0xffffffffu ? 0u : (km + 1u == S.n ? 0u : km + 1u);
  const uint32_t* st = start + S.tbase;
  const uint32_t l0 = __ldg(st + kl), l1 = __ldg(st + kl + 1);
  const uint32_t m0 = kl + 1u == km ? l1 : __ldg(st + km);
  const uint32_t m1 = __ldg(st + km + 1);
  const uint32_t h0 = kh == km + 1u ? m1 : __ldg(st + kh);
  const uint32_t h1 = __ldg(st + kh + 1);
  uint2 run[3];
  run[0] = bucket_run(mid - 1u, l0, l1, hash_s);
  run[1] = bucket_run(mid, m0, m1, hash_s);
  run[2] = bucket_run(mid + 1u, h0, h1, hash_s);
  uint32_t f = 0, e = 0;
  bool any = false, adjacent = true;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (run[k].y == 0) continue;
    if (!any) {
      f = run[k].x;
      e = f + run[k].y;
      any = true;
    } else if (run[k].x == e) {
      e += run[k].y;
    } else {
      adjacent = false;
    }
  }
  if (adjacent) {
    out[0] = make_uint2(f, (e - f) | kRunMerged);
  } else {
    out[0] = run[0];
    out[1] = run[1];
    out[2] = run[2];
  }
}

// Lanes take (cell, row) pairs of the warp's tile in parallel; the warp's
// cell leaders are listed in shared memory (kCellTableBlock threads per block).
constexpr int kCellTableBlock = 256;

__global__ void __launch_bounds__(kCellTableBlock)
k_cell_table(const uint2* __restrict__ tiles, uint32_t ntiles,
             const SceneDev* __restrict__ scenes,
             const uint32_t* __restrict__ hash_s,
             const uint32_t* __restrict__ cell_first,
             const uint32_t* __restrict__ start, uint2* __restrict__ cell_tab) {
  pdl_launch();
  __shared__ uint8_t s_lead[kCellTableBlock / 32][32];
  uint8_t* lead = s_lead[threadIdx.x >> 5];
  const uint32_t lane = lane_id();
  for (uint32_t t = warp_id_global(); t < ntiles; t += warps_total()) {
    const uint2 tile = tiles[t];
    const SceneDev S = scenes[tile_scene(tile)];  // registers, not reloads
    const uint32_t first = pdl_wait(tile.y);
    if (S.direct) continue;  // its rows come from the start table
    const uint32_t i = first + lane;
    const bool live = lane < tile_len(tile);
    const bool leader = live && cell_first[i] == i;
    const uint32_t lmask = __ballot_sync(kFull, leader);
    if (leader) lead[__popc(lmask & ((1u << lane) - 1u))] = static_cast<uint8_t>(lane);
    __syncwarp();
    const uint32_t pairs = __popc(lmask) * 9u;
    const uint32_t kmax = fastmod(0xffffffffu, S.fm, S.n);  // key of 2^32 - 1
    for (uint32_t q = lane; q < pairs; q += 32) {
      const uint32_t c = q / 9u, w = q - c * 9u;
      cell_row(S, first + lead[c], w, kmax, hash_s, start, cell_tab);
    }
    __syncwarp();  // the next tile rewrites the leader list
  }
}

// Latency form for small launches: nine warps a tile, a row each, the lanes
// that lead a cell at work (k_cell_table gives a warp up to nine such passes
// one after another: 1,000 particles 11 us).
__global__ void __launch_bounds__(288)
k_cell_table_rows(const uint2* __restrict__ tiles, uint32_t ntiles,
                  const SceneDev* __restrict__ scenes, const uint32_t* __restrict__ hash_s,
                  const uint32_t* __restrict__ cell_first, const uint32_t* __restrict__ start,
                  uint2* __restrict__ cell_tab) {
  pdl_launch();
  const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
  for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const uint2 tile = tiles[t];
    const SceneDev S = scenes[tile_scene(tile)];
    const uint32_t i = pdl_wait(tile.y) + lane;
    if (S.direct) continue;  // its rows come from the start table
    if (lane < tile_len(tile) && cell_first[i] == i)
      cell_row(S, i, w, fastmod(0xffffffffu, S.fm, S.n), hash_s, start, cell_tab);
  }
}

// ----------------------------------------------------------------- density
// CalculateDensity (:325-365) for one particle (self included) and its
// neighbour list (dist <= r, self excluded) for the force passes. The walk forms
// classify every candidate on the reference's exact d2 and sum as they go; the
// cell-tile form lists by an estimate first (k_density). Contributions vanish at
// the cutoff ((r-dist)^2), so the hardware square root serves the kernel value.
// The self pair contributes (r, r).
// One pair's share of the density sums, w = r - dist.
__device__ __forceinline__ void density_sum(float w, float& s2, float& s3) {
  const float w2 = w * w;
  s2 += w2;
  s3 = fmaf(w2, w, s3);
}

__device__ __forceinline__ void density_pair(const SceneDev& S, float d2,
                                             float& s2, float& s3) {
  density_sum(S.r - sqrt_approx(d2), s2, s3);
}

__device__ __forceinline__ void density_store(const SceneDev& S, uint32_t i,
                                              float s2, float s3, uint32_t cnt,
                                              float2* __restrict__ dens_a,
                                              float4* __restrict__ dens_b,
                                              uint32_t* __restrict__ ncount) {
  const float rho = s2 * S.vol2, rhon = s3 * S.vol3;
  dens_a[i] = make_float2(rho, rhon);
  const float ir = 1.0f / rho, irn = 1.0f / rhon;
  const float P = (rho - S.rho0) * S.k, Pn = rhon * S.kn;
  dens_b[i] = make_float4(ir, P * ir, irn, Pn * irn);
  ncount[i] = cnt;
}

// Thread-per-particle form in one pass: each lane walks its cell's runs,
// classifies every candidate on the reference's exact d2 and accumulates the
// density and its list as it goes. Lanes of one cell walk identical runs, so
// their loads coincide; a lane keeps kBatch candidates in flight (the loads of a
// run's last batch may pass its end by kPredPad slots, whose pairs are
// dropped). At large sizes it fills 78% of the issue slots and 70% of the L1 data
// pipe (26 warp instructions a candidate, of which the hit path takes a third;
// four wavefronts a 16-byte load), below ~300k particles it waits on its loads. Against one candidate at a
// time at 32 registers: 131k particles 37 -> 30 us (a step of three substeps
// 298 -> 248), 500k 93 -> 84, 1M 166 -> 157, 4M 581 -> 567, 8.4M 1149 -> 1161.
// Batches of 2, 3, 5, 6, 8 and caps of 32, 36, 40 registers (spills) were slower.
// Batches of tiny scenes keep one candidate at 32 registers (tiny_scenes).
constexpr uint32_t kWalkBatch = 4;
static_assert(kWalkBatch - 1u <= kPredPad, "candidate loads past the last slot");

template <int kTables, int kRegs, uint32_t kBatch>
__global__ void __maxnreg__(kRegs)
k_density_walk(const uint2* __restrict__ tiles, uint32_t ntiles,
                const SceneDev* __restrict__ scenes, const float4* __restrict__ pred,
                const uint32_t* __restrict__ start, const uint32_t* __restrict__ cell_first,
                const uint2* __restrict__ cell_tab, float2* __restrict__ dens_a,
                float4* __restrict__ dens_b, uint32_t* __restrict__ nbr,
                uint32_t* __restrict__ ncount, uint32_t nbr_step, uint32_t nbr_cap) {
  pdl_launch();
  const uint32_t lane = lane_id();
  for (uint32_t t = warp_id_global(); t < ntiles; t += warps_total()) {
    const uint2 tile = tiles[t];
    const SceneDev& S = scenes[tile_scene(tile)];
    const bool direct = kTables == kTablesDirect    ? true
                      : kTables == kTablesBuckets ? false
                                                  : S.direct != 0u;
    const float cut = S.cut_le, r = S.r;
    const uint32_t i = pdl_wait(tile.y) + lane;
    if (lane >= tile_len(tile)) continue;
    const float4 me = pred[i];
    const float2 npxy = make_float2(-me.x, -me.y);
    float s2 = S.r2, s3 = S.r2 * r;  // self: w = r
    uint32_t cnt = 0;
    // next list entry: a bumped pointer is the cheapest append in the hit
    // path. The step and the capacity are run-time values: with constants in
    // their place the kernel takes 195 instead of 172 us at 1M
    uint32_t* wp = nbr + nbr_index(i, 0);
    auto run = [&](uint32_t j, uint32_t e) {
#pragma unroll 1
      for (; j < e; j += kBatch) {
        float4 q[kBatch];
#pragma unroll
        for (uint32_t u = 0; u < kBatch; ++u) q[u] = __ldg(pred + j + u);
#pragma unroll
        for (uint32_t u = 0; u < kBatch; ++u) {
          // dist2 with (dx, dy) as one packed FP32x2 pair (x and y are
          // adjacent in the record), every component rounded as the scalar
          // code rounds it
          const float2 dxy = __fadd2_rn(make_float2(q[u].x, q[u].y), npxy);
          const float2 sxy = __fmul2_rn(dxy, dxy);
          const float dz = q[u].z - me.z;
          const float d2 = __fadd_rn(__fadd_rn(sxy.x, sxy.y), __fmul_rn(dz, dz));
          // Pairs with dist <= r (d2 <= cut_le) enter the list; the density
          // takes (r - dist)^2 and (r - dist)^3 of the same pairs: those with
          // dist == r exactly, which the reference leaves out, add
          // (r - sqrt(d2))^2, the square of a rounding error.
          if (j + u < e && d2 <= cut && j + u != i) {
            if (cnt < nbr_cap) {
              *wp = j + u;
              wp += nbr_step;
            }
            ++cnt;
            density_sum(r - sqrt_approx(d2), s2, s3);
          }
        }
      }
    };
    if (direct) {
      // rows (dy, dz) in the cell table's order (dz fastest); k = the row's
      // middle cell
      uint32_t k = S.tbase + __float_as_uint(me.w) - S.gwy - S.gwz;
      uint32_t b = __ldg(start + k - 1), e = __ldg(start + k + 2);
      int dz = 0;
#pragma unroll 1
      for (int w = 0; w < 9; ++w) {
        if (++dz == 3) { dz = 0; k += S.gwy - 2u * S.gwz; } else { k += S.gwz; }
        uint32_t nb = 0, ne = 0;
        if (w < 8) {  // the next row's run
          nb = __ldg(start + k - 1);
          ne = __ldg(start + k + 2);
        }
        run(b, e);
        b = nb;
        e = ne;
      }
    } else {
      const uint2* row = cell_tab + static_cast<uint64_t>(cell_first[i]) * 27u;
#pragma unroll 1
      for (int w = 0; w < 9; ++w, row += 3) {
        const uint2 m = __ldg(row);
        const uint32_t runs = (m.y & kRunMerged) ? 1u : 3u;
#pragma unroll 1
        for (uint32_t k = 0; k < runs; ++k) {
          const uint2 x = k ? __ldg(row + k) : m;
          run(x.x, x.x + (x.y & ~kRunMerged));
        }
      }
    }
    density_store(S, i, s2, s3, cnt, dens_a, dens_b, ncount);
  }
}

// Latency form for small launches (kRowsTiles): nine warps (a block) share a
// tile, lane = particle, one row of the walk a warp. A pair within the cutoff
// goes (distance squared, slot) to the lane's queue in shared memory; after a
// barrier every warp moves its entries to their place in the particle's list --
// rows in walk order, so the list is k_density_walk's -- and leaves r - dist
// of each there for the first warp to sum in that order. The sums are therefore
// the walk's bit for bit, while the chain a particle waits for is one row of
// ~16 candidates instead of ~140 (measured: 16,384 particles 32 -> 11 us, 1,000
// 39 -> 11 us). The 46 KB a block take the SM's occupancy, so large launches
// lose (1M: 165 -> 292 us).
//
// Where a row has more hits than its queue holds, or the list overflows, the
// warps walk their rows once more, now that the place of every hit is known, and
// leave r - dist there themselves, past a list's length in the lane's queues. Only
// a particle with more than kRowSums neighbours is walked by the first warp
// alone. (Were it every such particle, one candidate at a time, a cloud of 60,000
// particles took, density of a substep, us: at 45 / 100 / 200 / 400 neighbours 162 /
// 310 / 584 / 1133, all particles at one point 51 ms; now 45 / 82 / 140 / 550, 13.4 ms;
// k_density_walk with one candidate at a time 64 / 110 / 191 / 380, 9.6 ms.)
constexpr int kRowWarps = 9;
constexpr uint32_t kRowCap = 16;  // hits a queue holds
constexpr uint32_t kRowSums = kNbrCap + 2u * kRowWarps * kRowCap;  // r - dist a lane has room for
constexpr uint32_t kRowLong = 1024;  // a run of more candidates goes uncounted: more hits than that

template <int kTables>
__global__ void __launch_bounds__(32 * kRowWarps, 4)  // the blocks an SM's shared memory holds
k_density_rows(const uint2* __restrict__ tiles, uint32_t ntiles,
               const SceneDev* __restrict__ scenes, const float4* __restrict__ pred,
               const uint32_t* __restrict__ start, const uint32_t* __restrict__ cell_first,
               const uint2* __restrict__ cell_tab, float2* __restrict__ dens_a,
               float4* __restrict__ dens_b, uint32_t* __restrict__ nbr,
               uint32_t* __restrict__ ncount) {
  __shared__ float2 s_hit[kRowWarps][kRowCap][32];
  __shared__ float s_w[kNbrCap][32];
  __shared__ uint32_t s_cnt[kRowWarps][32];
  pdl_launch();
  const uint32_t lane = lane_id(), s = threadIdx.x >> 5;
  for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const uint2 tile = tiles[t];
    const SceneDev& S = scenes[tile_scene(tile)];
    const float cut = S.cut_le, r = S.r;
    const uint32_t row0 = S.tbase + (s / 3u - 1u) * S.gwy + (s % 3u - 1u) * S.gwz;
    const bool direct = kTables == kTablesDirect    ? true
                      : kTables == kTablesBuckets ? false
                                                  : S.direct != 0u;
    const bool live = lane < tile_len(tile);
    const uint32_t i = pdl_wait(tile.y) + (live ? lane : 0u);
    const float4 me = pred[i];
    const uint32_t cell = __float_as_uint(me.w);
    const uint32_t cf = kTables == kTablesDirect ? 0u : cell_first[i];
    const float2 npxy = make_float2(-me.x, -me.y);
    // the row's particles within the cutoff: hit(slot, distance squared)
    auto row = [&](auto&& enter, auto&& hit) {
      walk_row<kTables, 4>(direct, start, row0 + cell,
                        cell_tab + static_cast<uint64_t>(cf) * 27u + s * 3u, pred, enter,
                        [&](uint32_t j, float4 q, bool in) {
        const float2 dxy = __fadd2_rn(make_float2(q.x, q.y), npxy);
        const float2 sxy = __fmul2_rn(dxy, dxy);
        const float dz = q.z - me.z;
        const float d2 = __fadd_rn(__fadd_rn(sxy.x, sxy.y), __fmul_rn(dz, dz));
        if (in && d2 <= cut && j != i) hit(j, d2);
      });
    };
    uint32_t cnt = 0;
    if (live)
      row([&](uint32_t len) {
        if (len <= kRowLong) return true;
        cnt = kRowSums + 1u;
        return false;
      }, [&](uint32_t j, float d2) {
        if (cnt < kRowCap) s_hit[s][cnt][lane] = make_float2(d2, __uint_as_float(j));
        ++cnt;
      });
    s_cnt[s][lane] = cnt;
    __syncthreads();
    uint32_t before = 0, total = 0;
#pragma unroll
    for (uint32_t u = 0; u < kRowWarps; ++u) {
      const uint32_t c = s_cnt[u][lane];
      before += u < s ? c : 0u;
      total += c;
    }
    uint32_t* const list = nbr + nbr_index(i, 0);
    // a term of the sums past a list's length: in the lane's queues, which
    // nothing reads any more then
    auto wide = [&](uint32_t k) -> float& {
      const uint32_t q = k - kNbrCap;
      return reinterpret_cast<float*>(&s_hit[0][0][lane])[q / 2u * 64u + q % 2u];
    };
    if (cnt <= kRowCap && total <= kNbrCap) {
      for (uint32_t k = 0; k < cnt; ++k) {
        const float2 h = s_hit[s][k][lane];
        s_w[before + k][lane] = r - sqrt_approx(h.x);
        list[(before + k) * 32u] = __float_as_uint(h.y);
      }
    } else if (total <= kRowSums) {
      uint32_t k = before;
      row([](uint32_t) { return true; }, [&](uint32_t j, float d2) {
        const float w = r - sqrt_approx(d2);
        if (k < kNbrCap) {
          s_w[k][lane] = w;
          list[k * 32u] = j;
        } else {
          wide(k) = w;
        }
        ++k;
      });
    }
    __syncthreads();
    if (s == 0 && live) {
      float s2 = S.r2, s3 = S.r2 * r;  // self: w = r
      if (total <= kRowSums) {
#pragma unroll 4
        for (uint32_t k = 0; k < min(total, kNbrCap); ++k) density_sum(s_w[k][lane], s2, s3);
#pragma unroll 4
        for (uint32_t k = kNbrCap; k < total; ++k) density_sum(wide(k), s2, s3);
      } else {
        uint32_t k = 0;
        walk_rows<kTables, 4>(S, start, cell_tab, cf, cell, pred, [&](uint32_t j, float4 q, bool in) {
          const float d2 = dist2(q.x - me.x, q.y - me.y, q.z - me.z);
          const bool hit = in && d2 <= cut && j != i;
          if (hit && k < kNbrCap) list[k * 32u] = j;
          k += hit;
          density_sum(hit ? r - sqrt_approx(d2) : 0.0f, s2, s3);  // + 0: no branch to wait in
        });
        total = k;
      }
      density_store(S, i, s2, s3, total, dens_a, dens_b, ncount);
    }
    __syncthreads();  // the next tile rewrites the queues
  }
}

// Eight particles a warp in the latency forms of the force kernels.
constexpr int kCoopPer = 8;
constexpr int kCoopSub = kTile / kCoopPer;  // warps a tile
constexpr int kCoopBlock = 128;
constexpr int kCoopWarps = kCoopBlock / 32;

// Cell-tile form, in two phases. Phase 1 lists the candidates within cut_hi, a
// 2e-6 superset of the cutoff, by the FMA estimate of d2; phase 2 re-reads the
// listed pairs, classifies each on the exact d2 and sums.
// Phase 1 is warp-cooperative over the cells of the warp's 32 slots: for
// each cell, lanes 0..26 fetch its 27 runs, a warp scan gives their offsets
// in the cell's flat candidate sequence, and each lane holds kChunks of those
// candidates in registers (its slot found by a shuffle binary search over
// the run offsets) -- a cell tile of kChunks*32 candidates. Every particle of
// the cell is then tested against the whole tile at once: one ballot per 32
// pairs appends the hits to that particle's list. Longer candidate sequences
// are processed tile by tile.
template <int kChunks>
__global__ void k_density(const uint2* __restrict__ tiles, uint32_t ntiles,
                          const SceneDev* __restrict__ scenes,
                          const float4* __restrict__ pred,
                          const uint32_t* __restrict__ start,
                          const uint32_t* __restrict__ cell_first,
                          const uint2* __restrict__ cell_tab,
                          float2* __restrict__ dens_a,
                          float4* __restrict__ dens_b,
                          uint32_t* __restrict__ nbr,
                          uint32_t* __restrict__ ncount) {
  const uint32_t warp = pdl_enter(warp_id_global());
  const uint32_t lane = lane_id();
  const uint32_t lt_mask = (1u << lane) - 1u;
  for (uint32_t t = warp; t < ntiles; t += warps_total()) {
    const uint2 tile = tiles[t];
    const SceneDev S = scenes[tile_scene(tile)];  // registers, not reloads
    const uint32_t i = tile.y + lane;
    const bool live = lane < tile_len(tile);
    const float4 me = live ? pred[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const uint32_t cf = live ? cell_first[i] : 0xffffffffu;
    const uint32_t cf_prev = __shfl_up_sync(kFull, cf, 1);
    const uint32_t lead = __ballot_sync(kFull, live && (lane == 0 || cf != cf_prev));
    const uint32_t live_end = tile_len(tile);
    // phase 1: candidate lists (FMA estimate of d2 within cut_hi)
    uint32_t cnt = 0;  // list length of this lane's particle
    for (uint32_t cells = lead; cells != 0;) {
      const int c0 = __ffs(cells) - 1;
      cells &= cells - 1;
      const int c1 = cells ? __ffs(cells) - 1 : static_cast<int>(live_end);
      const uint32_t cfc = __shfl_sync(kFull, cf, c0);
      const uint32_t cellc = __shfl_sync(kFull, __float_as_uint(me.w), c0);
      uint2 run = make_uint2(0u, 0u);
      if (S.direct) {
        if (lane < 27u && lane % 3u == 0u)
          run = direct_row(S, start, S.tbase + cellc - S.gwy - S.gwz, static_cast<int>(lane / 3u));
      } else if (lane < 27) {
        run = __ldg(cell_tab + static_cast<uint64_t>(cfc) * 27u + lane);
      }
      // a merged row keeps its run in its first entry; the other two are unused
      const uint32_t heads =
          __ballot_sync(kFull, lane < 27u && lane % 3u == 0u && (run.y & kRunMerged));
      if (lane < 27u && lane % 3u != 0u && ((heads >> (lane - lane % 3u)) & 1u)) run.y = 0u;
      run.y &= ~kRunMerged;
      const uint32_t incl = warp_incl_scan(run.y);
      const uint32_t excl = incl - run.y;
      const uint32_t total = __shfl_sync(kFull, incl, 31);
      for (uint32_t seg = 0; seg < total; seg += kChunks * 32u) {
        float4 q[kChunks];
        uint32_t js[kChunks];
#pragma unroll
        for (int c = 0; c < kChunks; ++c) {
          const uint32_t e = seg + c * 32u + lane;
          // o = number of runs ending at or before e (incl is ascending)
          uint32_t o = 0;
#pragma unroll
          for (uint32_t step = 16; step >= 1; step >>= 1) {
            const uint32_t probe = o + step - 1u;
            const uint32_t v = __shfl_sync(kFull, incl, probe < 27u ? probe : 26u);
            if (probe < 27u && v <= e) o += step;
          }
          const uint32_t src = o < 27u ? o : 26u;
          const uint32_t rx = __shfl_sync(kFull, run.x, src);
          const uint32_t rex = __shfl_sync(kFull, excl, src);
          js[c] = rx + (e - rex);
          q[c] = e < total ? __ldg(pred + js[c])
                           : make_float4(__int_as_float(0x7f800000), 0.f, 0.f, 0.f);
        }
        for (int pp = c0; pp < c1; ++pp) {
          const float px = __shfl_sync(kFull, me.x, pp);
          const float py = __shfl_sync(kFull, me.y, pp);
          const float pz = __shfl_sync(kFull, me.z, pp);
          const uint32_t ip = tile.y + static_cast<uint32_t>(pp);
          uint32_t base = __shfl_sync(kFull, cnt, pp);
#pragma unroll
          for (int c = 0; c < kChunks; ++c) {
            if (seg + c * 32u >= total) break;
            const float d2f = dist2_fast(q[c].x - px, q[c].y - py, q[c].z - pz);
            const bool hit = d2f <= S.cut_hi && js[c] != ip;
            const uint32_t hm = __ballot_sync(kFull, hit);
            if (hit) {
              const uint32_t k = base + __popc(hm & lt_mask);
              if (k < kNbrCap) nbr[nbr_index(ip, k)] = js[c];
            }
            base += __popc(hm);
          }
          if (lane == static_cast<uint32_t>(pp)) cnt = base;
        }
      }
    }
    if (!live) continue;
    const float3 p = make_float3(me.x, me.y, me.z);
    // phase 2: exact classification and the density sums
    float s2 = S.r2, s3 = S.r2 * S.r;  // self: w = r
    if (cnt <= kNbrCap) {
      uint32_t kept = 0;
      for (uint32_t k = 0; k < cnt; ++k) {
        const uint32_t j = nbr[nbr_index(i, k)];
        const float4 q = __ldg(pred + j);
        const float d2 = dist2(q.x - p.x, q.y - p.y, q.z - p.z);
        if (d2 <= S.cut_lt) density_pair(S, d2, s2, s3);
        if (d2 <= S.cut_le) {
          if (kept != k) nbr[nbr_index(i, kept)] = j;
          ++kept;
        }
      }
      cnt = kept;
    } else {
      // list overflow: sum directly; the force passes walk the runs too
      walk_runs<kTablesMixed>(S, start, cell_tab, cf, __float_as_uint(me.w), pred,
                              [&](uint32_t j, float4 q) {
        const float d2 = dist2(q.x - p.x, q.y - p.y, q.z - p.z);
        if (j != i && d2 <= S.cut_lt) density_pair(S, d2, s2, s3);
      });
    }
    density_store(S, i, s2, s3, cnt, dens_a, dens_b, ncount);
  }
}

// ---------------------------------------------------------------- pressure
// CalculatePressureForce (:367-422) over the particle's neighbour list (self
// excluded, dist <= r). shared/rho_j = 0.5*(Pi*(1/rho_j) + Pj/rho_j); the 0.5
// is folded into ds2h/ds3h. The list is read kGather (2, 3, 4 or 8, tuned)
// entries at a time so their neighbours' gathers are in flight together, the
// next batch's entries loading meanwhile. A list that overflowed
// falls back to the walk of the cell's runs.
__device__ __forceinline__ float pressure_term(const SceneDev& S, float d2, float Pi, float Pni,
                                               float4 b) {
  const float dist = __fsqrt_rn(d2);
  const float w = S.r - dist;
  const float a2 = S.ds2h * fmaf(Pi, b.x, b.y);
  const float a3 = S.ds3h * w * fmaf(Pni, b.z, b.w);
  return -w * (a2 + a3);
}

__device__ __forceinline__ void pressure_pair(const SceneDev& S, float3 p,
                                              float Pi, float Pni, float4 q,
                                              float4 b, float3& f) {
  const float dx = q.x - p.x, dy = q.y - p.y, dz = q.z - p.z;
  const float d2 = dist2(dx, dy, dz);
  const float tsum = pressure_term(S, d2, Pi, Pni, b);
  if (d2 > 0.0f) {
    const float s = tsum * rsqrtf(d2);
    f.x = fmaf(dx, s, f.x);
    f.y = fmaf(dy, s, f.y);
    f.z = fmaf(dz, s, f.z);
  } else {
    f.y += tsum;  // dir = (0,1,0) for coincident particles (:414)
  }
}

// kLanes lanes per particle (tuning.particles_per_warp = 32 / kLanes): a
// warp takes its tile's 32 particles in kLanes passes of 32 / kLanes; lane
// pair (l, l + 16) shares a particle, each summing every other list entry,
// and one shuffle combines the halves. The sums then run in another order
// than with one lane, so the two forms agree to rounding, not bit for bit.
template <int kGather, int kTables, int kLanes>
__global__ void k_pressure(const uint2* __restrict__ tiles, uint32_t ntiles,
                           const SceneDev* __restrict__ scenes,
                           const float4* __restrict__ pred,
                           const uint32_t* __restrict__ start,
                           const uint32_t* __restrict__ cell_first,
                           const uint2* __restrict__ cell_tab,
                           const float2* __restrict__ dens_a,
                           const float4* __restrict__ dens_b,
                           const uint32_t* __restrict__ nbr,
                           const uint32_t* __restrict__ ncount,
                           const float4* __restrict__ vel,
                           float4* __restrict__ rec_v, float2* __restrict__ rec_b,
                           float4* __restrict__ dbg_accp,
                           float4* __restrict__ dbg_velp) {
  static_assert(kLanes == 1 || kLanes == 2, "one or two lanes per particle");
  pdl_launch();
  const uint32_t lane = lane_id();
  constexpr uint32_t kPer = 32 / kLanes;  // particles per pass
  const uint32_t sub = lane / kPer;       // this lane's share of the list
  for (uint32_t t = warp_id_global(); t < ntiles; t += warps_total()) {
    const uint2 tile = tiles[t];
    const SceneDev S = scenes[tile_scene(tile)];  // registers, not reloads
    const uint32_t first = pdl_wait(tile.y);
#pragma unroll 1
    for (uint32_t h = 0; h < kLanes; ++h) {
      const uint32_t li = h * kPer + lane % kPer;
      if (kLanes == 1 && li >= tile_len(tile)) break;
      const bool live = li < tile_len(tile);
      const uint32_t i = first + (live ? li : 0u);
      const float4 pi = pred[i];
      const float3 p = make_float3(pi.x, pi.y, pi.z);
      const float2 di = dens_a[i];
      const float Pi = (di.x - S.rho0) * S.k, Pni = di.y * S.kn;
      float3 f = make_float3(0.0f, 0.0f, 0.0f);
      const uint32_t cnt = live ? ncount[i] : 0u;
      if (cnt <= kNbrCap) {
        uint32_t jn[kGather];
        if (sub < cnt) load_nbr_batch<kGather, kLanes>(nbr, i, sub, cnt, jn);
        for (uint32_t k0 = sub; k0 < cnt; k0 += kLanes * kGather) {
          uint32_t j[kGather];
          float4 q[kGather], b[kGather];
#pragma unroll
          for (int u = 0; u < kGather; ++u) j[u] = (k0 + kLanes * u < cnt) ? jn[u] : i;
          // the next batch's entries load while this batch's gathers fly
          if (k0 + kLanes * kGather < cnt)
            load_nbr_batch<kGather, kLanes>(nbr, i, k0 + kLanes * kGather, cnt, jn);
#pragma unroll
          for (int u = 0; u < kGather; ++u) {
            q[u] = __ldg(pred + j[u]);
            b[u] = __ldg(dens_b + j[u]);
          }
#pragma unroll
          for (int u = 0; u < kGather; ++u)
            if (k0 + kLanes * u < cnt) pressure_pair(S, p, Pi, Pni, q[u], b[u], f);
        }
      } else if (sub == 0) {
        walk_runs<kTables>(S, start, cell_tab, cell_first[i], __float_as_uint(pi.w), pred,
                           [&](uint32_t j, float4 q) {
          if (j == i) return;
          const float dx = q.x - p.x, dy = q.y - p.y, dz = q.z - p.z;
          if (dist2(dx, dy, dz) <= S.cut_le)
            pressure_pair(S, p, Pi, Pni, q, __ldg(dens_b + j), f);
        });
      }
      if (kLanes == 2) {
        f.x += __shfl_xor_sync(kFull, f.x, 16);
        f.y += __shfl_xor_sync(kFull, f.y, 16);
        f.z += __shfl_xor_sync(kFull, f.z, 16);
      }
      if (!live || sub != 0) continue;
      const float inv_rho = 1.0f / di.x;
      const float ax = f.x * inv_rho, ay = f.y * inv_rho, az = f.z * inv_rho;
      const float4 v = vel[i];
      const float4 vp = make_float4(v.x + ax * S.dt, v.y + ay * S.dt, v.z + az * S.dt, 0.f);
      store_state(rec_v, rec_b, i, pi, vp);
      if (dbg_accp) {
        dbg_accp[i] = make_float4(ax, ay, az, 0.0f);
        dbg_velp[i] = vp;
      }
    }
  }
}

// Latency form for small launches (kCoopTiles): eight particles a warp,
// four lanes a particle evaluate every fourth list entry each and leave (direction,
// magnitude) in shared memory; one lane a component sums them in list order,
// with the operations of pressure_pair, so the result is k_pressure's bit for bit
// (16,384 particles 14 -> 10 us; with 8 instead of 32 particles a warp and the
// terms staged it takes 2.3 times the plain form's instructions, which large
// launches pay: 1M 93 -> 210 us). A list that overflowed goes by walk_rows, two
// candidates in flight here (four spill) and four in the viscosity pass (a cloud
// of 28,000 particles of 200 neighbours, pressure / viscosity, us: one in flight
// 372 / 408, now 340 / 289, the plain forms 300 / 287).
constexpr int kCoopTerms = kNbrCap + 1;  // float4 rows, shifted a bank group each
constexpr int kCoopGather = 8;           // entries a lane has in flight (4: 16k-particle step 3 us longer)

// Component `comp` of the ordered sum of fma(direction, magnitude) over a row.
__device__ __forceinline__ float coop_sum(const float4* row, uint32_t comp, uint32_t cnt) {
  const float* p = reinterpret_cast<const float*>(row);
  float f = 0.0f;
#pragma unroll 4
  for (uint32_t k = 0; k < cnt; ++k) f = fmaf(p[4u * k + comp], p[4u * k + 3u], f);
  return f;
}

template <int kTables>
__global__ void __launch_bounds__(kCoopBlock)
k_pressure_coop(const uint2* __restrict__ tiles, uint32_t ntiles,
                const SceneDev* __restrict__ scenes, const float4* __restrict__ pred,
                const uint32_t* __restrict__ start, const uint32_t* __restrict__ cell_first,
                const uint2* __restrict__ cell_tab, const float2* __restrict__ dens_a,
                const float4* __restrict__ dens_b, const uint32_t* __restrict__ nbr,
                const uint32_t* __restrict__ ncount, const float4* __restrict__ vel,
                float4* __restrict__ rec_v, float4* __restrict__ dbg_accp,
                float4* __restrict__ dbg_velp) {
  __shared__ float4 s_t[kCoopWarps][kCoopPer][kCoopTerms];
  pdl_launch();
  const uint32_t lane = lane_id();
  const uint32_t pp = lane % kCoopPer, part = lane / kCoopPer;
  float4* const row = s_t[threadIdx.x >> 5][pp];
  for (uint32_t v = warp_id_global(); v < ntiles * kCoopSub; v += warps_total()) {
    const uint2 tile = tiles[v / kCoopSub];
    const uint32_t sub = v % kCoopSub * kCoopPer, len = tile_len(tile);
    if (sub >= len) continue;
    const SceneDev S = scenes[tile_scene(tile)];
    const bool live = sub + pp < len;
    const uint32_t i = pdl_wait(tile.y) + min(sub + pp, len - 1u);
    const float4 pi = pred[i];
    const float3 p = make_float3(pi.x, pi.y, pi.z);
    const float2 di = dens_a[i];
    const float4 vi = vel[i];
    const float Pi = (di.x - S.rho0) * S.k, Pni = di.y * S.kn;
    const uint32_t cnt = live ? ncount[i] : 0u;
    float3 f = make_float3(0.0f, 0.0f, 0.0f);
    if (cnt <= kNbrCap) {
      for (uint32_t k0 = part; k0 < cnt; k0 += 4u * kCoopGather) {
        uint32_t j[kCoopGather];
        float4 q[kCoopGather], b[kCoopGather];
        load_nbr_batch<kCoopGather, 4>(nbr, i, k0, cnt, j);
#pragma unroll
        for (int u = 0; u < kCoopGather; ++u) {
          if (k0 + 4u * u < cnt) {
            q[u] = __ldg(pred + j[u]);
            b[u] = __ldg(dens_b + j[u]);
          }
        }
#pragma unroll
        for (int u = 0; u < kCoopGather; ++u) {
          if (k0 + 4u * u < cnt) {
            const float dx = q[u].x - p.x, dy = q[u].y - p.y, dz = q[u].z - p.z;
            const float d2 = dist2(dx, dy, dz);
            const float tsum = pressure_term(S, d2, Pi, Pni, b[u]);
            // (a coincident pair's term is tsum, along y: -0 * 1 leaves x and z
            // what they are also where tsum is infinite)
            row[k0 + 4u * u] = d2 > 0.0f ? make_float4(dx, dy, dz, tsum * rsqrtf(d2))
                                         : make_float4(-0.0f, tsum, -0.0f, 1.0f);
          }
        }
      }
    } else if (part == 0) {
      walk_rows<kTables, 2>(S, start, cell_tab, cell_first[i], __float_as_uint(pi.w), pred,
                         [&](uint32_t j, float4 q, bool in) {
        if (!in || j == i) return;
        const float dx = q.x - p.x, dy = q.y - p.y, dz = q.z - p.z;
        if (dist2(dx, dy, dz) <= S.cut_le)
          pressure_pair(S, p, Pi, Pni, q, __ldg(dens_b + j), f);
      });
    }
    __syncwarp();
    const float fc = coop_sum(row, min(part, 2u), cnt <= kNbrCap ? cnt : 0u);
    const float fx = __shfl_sync(kFull, fc, pp), fy = __shfl_sync(kFull, fc, kCoopPer + pp),
                fz = __shfl_sync(kFull, fc, 2 * kCoopPer + pp);
    if (cnt <= kNbrCap) f = make_float3(fx, fy, fz);
    __syncwarp();  // the next slots rewrite the rows
    if (!live || part != 0) continue;
    const float inv_rho = 1.0f / di.x;
    const float ax = f.x * inv_rho, ay = f.y * inv_rho, az = f.z * inv_rho;
    const float4 vp = make_float4(vi.x + ax * S.dt, vi.y + ay * S.dt, vi.z + az * S.dt, 0.f);
    store_rec(rec_v, i, pi, vp);
    if (dbg_accp) {
      dbg_accp[i] = make_float4(ax, ay, az, 0.0f);
      dbg_velp[i] = vp;
    }
  }
}

// ------------------------------------------------ viscosity + integrate
// CalculateViscosityForce (:424-464) over the neighbour list reading the
// post-pressure snapshot (Jacobi); poly6 = (r^2 - d^2)^3 for dist < r. Then
// pos += v*dt and the box collision (:81-108). With fuse_next the next
// substep's prediction / cell index / histogram (k_predict_hash) runs here on the
// new state.
__device__ __forceinline__ void visc_pair(const SceneDev& S, float3 p,
                                          float4 vi, float4 q, float4 vj,
                                          float3& f) {
  const float dx = q.x - p.x, dy = q.y - p.y, dz = q.z - p.z;
  const float d2 = dist2(dx, dy, dz);
  if (d2 <= S.cut_lt) {
    const float w = S.r2 - d2;
    const float w3 = w * w * w;
    f.x = fmaf(vj.x - vi.x, w3, f.x);
    f.y = fmaf(vj.y - vi.y, w3, f.y);
    f.z = fmaf(vj.z - vi.z, w3, f.z);
  }
}

// The viscosity increment f of slot i, then the integration and the box
// collision; with fuse_next also the key of the new state's prediction (S_next
// is the same scene: its grid constants are read there, not kept in registers
// through the sum).
__device__ __forceinline__ void integrate(const SceneDev& S, const SceneDev& S_next, uint32_t i,
                                          float4 vi, float3 f, float4* __restrict__ pos,
                                          float4* __restrict__ vel, float4* __restrict__ out4,
                                          int fuse_next, float4* __restrict__ dbg_velv,
                                          uint32_t& key, uint32_t& cell, uint32_t& id, bool& bad) {
  const float c = S.vscale * S.mu * S.dt;
  float3 v = make_float3(vi.x + f.x * c, vi.y + f.y * c, vi.z + f.z * c);
  if (dbg_velv) dbg_velv[i] = make_float4(v.x, v.y, v.z, 0.0f);
  float4 x = pos[i];
  x.x = __fadd_rn(x.x, __fmul_rn(v.x, S.dt));
  x.y = __fadd_rn(x.y, __fmul_rn(v.y, S.dt));
  x.z = __fadd_rn(x.z, __fmul_rn(v.z, S.dt));
  // edgeDst = halfSize - |pos|; if <= 0 clamp to the wall and reflect.
  if (S.hx - fabsf(x.x) <= 0.0f) { x.x = S.hx * copysign_or_zero(x.x); v.x *= S.ndamp; }
  if (S.hy - fabsf(x.y) <= 0.0f) { x.y = S.hy * copysign_or_zero(x.y); v.y *= S.ndamp; }
  if (S.hz - fabsf(x.z) <= 0.0f) { x.z = S.hz * copysign_or_zero(x.z); v.z *= S.ndamp; }
  pos[i] = x;
  const float4 v4 = make_float4(v.x, v.y, v.z, 0.0f);
  vel[i] = v4;
  bad = !(isfinite(x.x) && isfinite(x.y) && isfinite(x.z) &&
          isfinite(v.x) && isfinite(v.y) && isfinite(v.z));
  id = __float_as_uint(x.w);
  if (out4) {
    if (id < S.n) out4[S.base + id] = make_float4(x.x, x.y, x.z, 0.34f);
    else bad = true;
  }
  if (fuse_next) predict_key(S_next, x, v4, key, cell);
}

// kLanes lanes per particle as in k_pressure.
template <int kGather, int kTables, int kLanes>
__device__ __forceinline__ void visc_tiles(
    const uint2* __restrict__ tiles, uint32_t ntiles,
    const SceneDev* __restrict__ scenes, const float4* __restrict__ pred,
    const uint32_t* __restrict__ start,
    const uint32_t* __restrict__ cell_first, const uint2* __restrict__ cell_tab,
    const uint32_t* __restrict__ nbr, const uint32_t* __restrict__ ncount, const float4* __restrict__ rec_v,
    const float2* __restrict__ rec_b,
    float4* __restrict__ pos, float4* __restrict__ vel,
    float4* __restrict__ out4, int fuse_next, uint32_t* __restrict__ count,
    uint4* __restrict__ keyrank, float4* __restrict__ dbg_velv,
    uint32_t* status) {
  static_assert(kLanes == 1 || kLanes == 2, "one or two lanes per particle");
  // (the early table read costs this kernel registers: 8.4M 599 -> 627 us)
  const uint32_t warp = pdl_enter(warp_id_global());
  const uint32_t lane = lane_id();
  constexpr uint32_t kPer = 32 / kLanes;  // particles per pass
  const uint32_t sub = lane / kPer;       // this lane's share of the list
  for (uint32_t t = warp; t < ntiles; t += warps_total()) {
    const uint2 tile = tiles[t];
    const SceneDev S = scenes[tile_scene(tile)];  // registers, not reloads
#pragma unroll 1
    for (uint32_t h = 0; h < kLanes; ++h) {
      const uint32_t li = h * kPer + lane % kPer;
      const bool in_tile = li < tile_len(tile);
      const bool live = in_tile && sub == 0;  // the lane that owns the particle
      const uint32_t i = tile.y + (in_tile ? li : 0u);
      bool bad = false;
      uint32_t key = 0, cell = 0, id = 0;
      float4 pi, vi;
      float3 f = make_float3(0.0f, 0.0f, 0.0f);
      if (in_tile) {
        load_state(rec_v, rec_b, i, pi, vi);
        const float3 p = make_float3(pi.x, pi.y, pi.z);
        const uint32_t cnt = ncount[i];
        if (cnt <= kNbrCap) {
          uint32_t jn[kGather];
          if (sub < cnt) load_nbr_batch<kGather, kLanes>(nbr, i, sub, cnt, jn);
          for (uint32_t k0 = sub; k0 < cnt; k0 += kLanes * kGather) {
            uint32_t j[kGather];
            float4 q[kGather], vj[kGather];
#pragma unroll
            for (int u = 0; u < kGather; ++u) j[u] = (k0 + kLanes * u < cnt) ? jn[u] : i;
            if (k0 + kLanes * kGather < cnt)
              load_nbr_batch<kGather, kLanes>(nbr, i, k0 + kLanes * kGather, cnt, jn);
#pragma unroll
            for (int u = 0; u < kGather; ++u) load_state(rec_v, rec_b, j[u], q[u], vj[u]);
#pragma unroll
            for (int u = 0; u < kGather; ++u)
              if (k0 + kLanes * u < cnt) visc_pair(S, p, vi, q[u], vj[u], f);
          }
        } else if (sub == 0) {
          walk_runs<kTables>(S, start, cell_tab, cell_first[i], __float_as_uint(pred[i].w), pred,
                             [&](uint32_t j, float4 q) {
            if (j == i) return;
            float4 a, b;
            load_state(rec_v, rec_b, j, a, b);
            visc_pair(S, p, vi, q, b, f);
          });
        }
      }
      if (kLanes == 2) {
        f.x += __shfl_xor_sync(kFull, f.x, 16);
        f.y += __shfl_xor_sync(kFull, f.y, 16);
        f.z += __shfl_xor_sync(kFull, f.z, 16);
      }
      if (live) {
        integrate(S, scenes[tile_scene(tile)], i, vi, f, pos, vel, out4, fuse_next, dbg_velv, key,
                  cell, id, bad);
      }
      if (fuse_next) {
        const uint32_t r = aggregated_rank(count, key, live);
        if (live) keyrank[i] = make_uint4(key, r, cell, id);
      }
      if (__any_sync(kFull, bad) && lane == 0) flag(status, kStatusNonFinite);
    }
  }
}

template <int kGather, int kTables, int kLanes>
__global__ void k_visc_integrate(
    const uint2* __restrict__ tiles, uint32_t ntiles,
    const SceneDev* __restrict__ scenes, const float4* __restrict__ pred,
    const uint32_t* __restrict__ start,
    const uint32_t* __restrict__ cell_first, const uint2* __restrict__ cell_tab,
    const uint32_t* __restrict__ nbr, const uint32_t* __restrict__ ncount, const float4* __restrict__ rec_v,
    const float2* __restrict__ rec_b,
    float4* __restrict__ pos, float4* __restrict__ vel,
    float4* __restrict__ out4, int fuse_next, uint32_t* __restrict__ count,
    uint4* __restrict__ keyrank, float4* __restrict__ dbg_velv,
    uint32_t* status) {
  visc_tiles<kGather, kTables, kLanes>(tiles, ntiles, scenes, pred, start, cell_first, cell_tab, nbr, ncount, rec_v,
                                       rec_b, pos, vel, out4, fuse_next, count, keyrank, dbg_velv, status);
}

// The default form for launches of many waves (dense_form): 40 registers, 48
// instead of 40 warps an SM, at 16 B of spills outside the loop.
template <int kTables>
__global__ void __maxnreg__(40) k_visc_dense(
    const uint2* __restrict__ tiles, uint32_t ntiles,
    const SceneDev* __restrict__ scenes, const float4* __restrict__ pred,
    const uint32_t* __restrict__ start,
    const uint32_t* __restrict__ cell_first, const uint2* __restrict__ cell_tab,
    const uint32_t* __restrict__ nbr, const uint32_t* __restrict__ ncount, const float4* __restrict__ rec_v,
    const float2* __restrict__ rec_b,
    float4* __restrict__ pos, float4* __restrict__ vel,
    float4* __restrict__ out4, int fuse_next, uint32_t* __restrict__ count,
    uint4* __restrict__ keyrank, float4* __restrict__ dbg_velv,
    uint32_t* status) {
  visc_tiles<2, kTables, 1>(tiles, ntiles, scenes, pred, start, cell_first, cell_tab, nbr, ncount, rec_v,
                            rec_b, pos, vel, out4, fuse_next, count, keyrank, dbg_velv, status);
}

// Latency form for small launches, as k_pressure_coop: the terms of visc_pair
// by four lanes a particle, summed in list order.
template <int kTables>
__global__ void __launch_bounds__(kCoopBlock) k_visc_coop(
    const uint2* __restrict__ tiles, uint32_t ntiles, const SceneDev* __restrict__ scenes,
    const float4* __restrict__ pred, const uint32_t* __restrict__ start,
    const uint32_t* __restrict__ cell_first, const uint2* __restrict__ cell_tab,
    const uint32_t* __restrict__ nbr, const uint32_t* __restrict__ ncount,
    const float4* __restrict__ rec_v, float4* __restrict__ pos, float4* __restrict__ vel,
    float4* __restrict__ out4, int fuse_next, uint32_t* __restrict__ count,
    uint4* __restrict__ keyrank, float4* __restrict__ dbg_velv, uint32_t* status) {
  __shared__ float4 s_t[kCoopWarps][kCoopPer][kCoopTerms];
  pdl_launch();
  const uint32_t lane = lane_id();
  const uint32_t pp = lane % kCoopPer, part = lane / kCoopPer;
  float4* const row = s_t[threadIdx.x >> 5][pp];
  for (uint32_t v = warp_id_global(); v < ntiles * kCoopSub; v += warps_total()) {
    const uint2 tile = tiles[v / kCoopSub];
    const uint32_t sub = v % kCoopSub * kCoopPer, len = tile_len(tile);
    if (sub >= len) continue;
    const SceneDev S = scenes[tile_scene(tile)];
    const bool in_tile = sub + pp < len;
    const uint32_t i = pdl_wait(tile.y) + min(sub + pp, len - 1u);
    float4 pi, vi;
    load_rec(rec_v, i, pi, vi);
    const float3 p = make_float3(pi.x, pi.y, pi.z);
    const uint32_t cnt = in_tile ? ncount[i] : 0u;
    float3 f = make_float3(0.0f, 0.0f, 0.0f);
    if (cnt <= kNbrCap) {
      for (uint32_t k0 = part; k0 < cnt; k0 += 4u * kCoopGather) {
        uint32_t j[kCoopGather];
        float4 q[kCoopGather], vj[kCoopGather];
        load_nbr_batch<kCoopGather, 4>(nbr, i, k0, cnt, j);
#pragma unroll
        for (int u = 0; u < kCoopGather; ++u)
          if (k0 + 4u * u < cnt) load_rec(rec_v, j[u], q[u], vj[u]);
#pragma unroll
        for (int u = 0; u < kCoopGather; ++u) {
          if (k0 + 4u * u < cnt) {
            const float dx = q[u].x - p.x, dy = q[u].y - p.y, dz = q[u].z - p.z;
            const float d2 = dist2(dx, dy, dz);
            const float w = S.r2 - d2;
            row[k0 + 4u * u] = d2 <= S.cut_lt
                                   ? make_float4(vj[u].x - vi.x, vj[u].y - vi.y, vj[u].z - vi.z,
                                                 w * w * w)
                                   : make_float4(-0.0f, -0.0f, -0.0f, 1.0f);  // no change
          }
        }
      }
    } else if (part == 0) {
      walk_rows<kTables, 4>(S, start, cell_tab, cell_first[i], __float_as_uint(pi.w), pred,
                         [&](uint32_t j, float4 q, bool in) {
        if (in && j != i) visc_pair(S, p, vi, q, __ldg(rec_v + 2ull * j + 1), f);
      });
    }
    __syncwarp();
    const float fc = coop_sum(row, min(part, 2u), cnt <= kNbrCap ? cnt : 0u);
    const float fx = __shfl_sync(kFull, fc, pp), fy = __shfl_sync(kFull, fc, kCoopPer + pp),
                fz = __shfl_sync(kFull, fc, 2 * kCoopPer + pp);
    if (cnt <= kNbrCap) f = make_float3(fx, fy, fz);
    __syncwarp();  // the next slots rewrite the rows
    const bool live = in_tile && part == 0u;
    bool bad = false;
    uint32_t key = 0, cell = 0, id = 0;
    if (live) integrate(S, S, i, vi, f, pos, vel, out4, fuse_next, dbg_velv, key, cell, id, bad);
    if (fuse_next) {
      const uint32_t r = aggregated_rank(count, key, live);
      if (live) keyrank[i] = make_uint4(key, r, cell, id);
    }
    if (__any_sync(kFull, bad) && lane == 0) flag(status, kStatusNonFinite);
  }
}

// ------------------------------------------------------------ readback
// Gather a scene's slot-ordered arrays into the caller's particle order.
__global__ void k_export(uint32_t first, uint32_t n,
                         const float4* __restrict__ pos,
                         const float4* __restrict__ vel,
                         const float2* __restrict__ dens,
                         float* __restrict__ opos, float* __restrict__ ovel,
                         float* __restrict__ odens,
                         uint32_t* __restrict__ oids) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const uint32_t s = first + k;
  const float4 p = pos[s];
  const uint32_t id = __float_as_uint(p.w);
  if (oids) oids[k] = id;
  if (id >= n) return;
  if (opos) { opos[3 * id] = p.x; opos[3 * id + 1] = p.y; opos[3 * id + 2] = p.z; }
  if (ovel) {
    const float4 v = vel[s];
    ovel[3 * id] = v.x; ovel[3 * id + 1] = v.y; ovel[3 * id + 2] = v.z;
  }
  if (odens) {
    const float2 d = dens[s];
    odens[2 * id] = d.x; odens[2 * id + 1] = d.y;
  }
}

// Caller index -> slot for scene slots [first, first + n): the inverse of
// the ids the slots carry. k_export_rows starts while it runs and waits for it:
// a download of 1k to 131k particles takes 2 us less than in sequence (8,193
// particles 16.6 -> 14.4, 131k 37.4 -> 35.1).
__global__ void k_slot_map(uint32_t first, uint32_t n, const float4* __restrict__ pos,
                           uint32_t* __restrict__ slot_of) {
  pdl_launch();
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const uint32_t id = __float_as_uint(pos[first + k].w);
  if (id < n) slot_of[id] = first + k;
}

// This lane's W floats of row i0 + lane (lane < rows) into the warp's staging
// row buffer, then the warp's rows out as 16-byte words: 32 full rows are
// 8W aligned words (out is 16-byte aligned and i0 a multiple of 32); a
// partial last group goes out word by word.
template <int W>
__device__ __forceinline__ void store_rows(float* buf, float* __restrict__ out, uint32_t i0,
                                           uint32_t rows, uint32_t lane, const float* v) {
  if (lane < rows) {
#pragma unroll
    for (int c = 0; c < W; ++c) buf[W * lane + c] = v[c];
  }
  __syncwarp();
  float* dst = out + static_cast<uint64_t>(W) * i0;
  if (rows == 32u) {
    if (lane < 8u * W)
      reinterpret_cast<float4*>(dst)[lane] = reinterpret_cast<const float4*>(buf)[lane];
  } else {
    for (uint32_t f = lane; f < W * rows; f += 32u) dst[f] = buf[f];
  }
  __syncwarp();
}

// Caller-order rows written straight into host memory the device maps
// (pinned, 16-byte aligned), a warp per 32 consecutive caller indices: the
// warp gathers its rows' slots through slot_of and stores whole aligned
// 16-byte words, so the host link carries full lines (scattered 12-byte row
// stores over the link run at a tenth of its rate). A caller index whose
// slot_of entry is not a slot of the scene (ids that are no permutation: the
// status flags report the lost slot) gets a zero row.
__global__ void __launch_bounds__(256) k_export_rows(uint32_t first, uint32_t n,
                                                     const uint32_t* __restrict__ slot_of,
                                                     const float4* __restrict__ pos,
                                                     const float4* __restrict__ vel,
                                                     const float2* __restrict__ dens,
                                                     float* __restrict__ opos,
                                                     float* __restrict__ ovel,
                                                     float* __restrict__ odens) {
  __shared__ __align__(16) float buf[8][96];
  const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  const uint32_t i0 = pdl_wait((blockIdx.x * 8u + w) * 32u);
  if (i0 >= n) return;
  const uint32_t rows = min(32u, n - i0);
  const uint32_t s = lane < rows ? slot_of[i0 + lane] : first;
  const bool ok = lane < rows && s - first < n;
  if (opos) {
    const float4 p = ok ? pos[s] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float v[3] = {p.x, p.y, p.z};
    store_rows<3>(buf[w], opos, i0, rows, lane, v);
  }
  if (ovel) {
    const float4 q = ok ? vel[s] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float v[3] = {q.x, q.y, q.z};
    store_rows<3>(buf[w], ovel, i0, rows, lane, v);
  }
  if (odens) {
    const float2 d = ok ? dens[s] : make_float2(0.f, 0.f);
    const float v[2] = {d.x, d.y};
    store_rows<2>(buf[w], odens, i0, rows, lane, v);
  }
}

// ------------------------------------------------------ reference lookup
// The reference's spatial lookup of a captured substep (UpdateSpatialLookup,
// physicsWorld.cc:466-496) from the predicted positions of the sorted
// layout, by a counting sort of its own: HashCell and key = hash % n of every
// particle (written by particle index), entries in (key, particle index)
// order, and the start of every key.
__global__ void k_ref_hash(const uint2* __restrict__ tiles, uint32_t ntiles,
                           const SceneDev* __restrict__ scenes,
                           const float4* __restrict__ pred,
                           const float4* __restrict__ pos,
                           uint32_t* __restrict__ count,
                           uint2* __restrict__ keyrank,
                           uint32_t* __restrict__ ohash,
                           uint32_t* __restrict__ okey, uint32_t* status) {
  const uint32_t warp = pdl_enter(warp_id_global());
  const uint32_t lane = lane_id();
  for (uint32_t t = warp; t < ntiles; t += warps_total()) {
    const uint2 tile = tiles[t];
    const SceneDev S = scenes[tile_scene(tile)];
    const uint32_t s = tile.y + lane;
    const bool live = lane < tile_len(tile);
    uint32_t key = 0, hash = 0, id = 0;
    if (live) {
      const float4 q = pred[s];
      hash = hash_of(S, make_float3(q.x, q.y, q.z));
      key = S.base + fastmod(hash, S.fm, S.n);
      id = __float_as_uint(pos[s].w);
    }
    const uint32_t r = aggregated_rank(count, key, live);
    if (!live) continue;
    keyrank[s] = make_uint2(key, r);
    if (id < S.n) {
      ohash[S.base + id] = hash;
      okey[S.base + id] = key - S.base;
    } else {
      flag(status, kStatusRange);
    }
  }
}

// Bucket every particle index at start[key] + arrival rank.
__global__ void k_ref_scatter(const uint2* __restrict__ tiles, uint32_t ntiles,
                              const float4* __restrict__ pos,
                              const uint2* __restrict__ keyrank,
                              const uint32_t* __restrict__ start,
                              uint32_t total, uint32_t* __restrict__ tmp,
                              uint32_t* status) {
  const uint32_t warp = pdl_enter(warp_id_global());
  const uint32_t lane = lane_id();
  for (uint32_t t = warp; t < ntiles; t += warps_total()) {
    const uint2 tile = tiles[t];
    const uint32_t s = tile.y + lane;
    if (lane >= tile_len(tile)) continue;
    const uint2 kr = keyrank[s];
    const uint32_t dst = start[kr.x] + kr.y;
    if (dst >= total) { flag(status, kStatusRange); continue; }
    tmp[dst] = __float_as_uint(pos[s].w);
  }
}

// Order every bucket by particle index: the canonical (key, index) order.
__global__ void k_ref_order(const uint2* __restrict__ tiles, uint32_t ntiles,
                            const float4* __restrict__ pos,
                            const uint2* __restrict__ keyrank,
                            const uint32_t* __restrict__ start,
                            const uint32_t* __restrict__ tmp,
                            uint32_t* __restrict__ sorted) {
  const uint32_t warp = pdl_enter(warp_id_global());
  const uint32_t lane = lane_id();
  for (uint32_t t = warp; t < ntiles; t += warps_total()) {
    const uint2 tile = tiles[t];
    const uint32_t s = tile.y + lane;
    if (lane >= tile_len(tile)) continue;
    const uint32_t key = keyrank[s].x;
    const uint32_t id = __float_as_uint(pos[s].w);
    const uint32_t b0 = start[key], b1 = start[key + 1];
    uint32_t rank = 0;
    for (uint32_t u = b0; u < b1; ++u) rank += tmp[u] < id ? 1u : 0u;
    if (b0 + rank < b1) sorted[b0 + rank] = id;
  }
}

// Per-slot debug intermediates of one scene to caller order.
__global__ void k_export_debug(uint32_t first, uint32_t n,
                               const float4* __restrict__ pos,
                               const float4* __restrict__ accp,
                               const float4* __restrict__ velp,
                               const float4* __restrict__ velv,
                               float* __restrict__ oaccp,
                               float* __restrict__ ovelp,
                               float* __restrict__ ovelv) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const uint32_t s = first + k;
  const uint32_t id = __float_as_uint(pos[s].w);
  if (id >= n) return;
  const float4 a = accp[s], b = velp[s], c = velv[s];
  oaccp[3 * id] = a.x; oaccp[3 * id + 1] = a.y; oaccp[3 * id + 2] = a.z;
  ovelp[3 * id] = b.x; ovelp[3 * id + 1] = b.y; ovelp[3 * id + 2] = b.z;
  ovelv[3 * id] = c.x; ovelv[3 * id + 1] = c.y; ovelv[3 * id + 2] = c.z;
}

// The timed sort's own layout of a captured substep, per slot of one scene:
// the particle at each slot (slot_ids, slot order), and per particle (caller
// order) its internal cell index (pred.w, written by k_reorder) and its
// entry in the scene's key table.
__global__ void k_export_layout(uint32_t first, uint32_t n,
                                const SceneDev* __restrict__ scene,
                                const float4* __restrict__ pos,
                                const float4* __restrict__ pred,
                                uint32_t* __restrict__ ocell,
                                uint32_t* __restrict__ okey,
                                uint32_t* __restrict__ oslot) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const uint32_t s = first + k;
  const uint32_t id = __float_as_uint(pos[s].w);
  const uint32_t cell = __float_as_uint(pred[s].w);
  oslot[k] = id;
  if (id >= n) return;
  const SceneDev& S = *scene;
  ocell[id] = cell;
  okey[id] = table_key(S, cell) - S.tbase;
}

// Load caller-order AoS arrays into a scene's slots (identity layout).
// The densities start at zero (unknown until the next step).
__global__ void k_import(uint32_t first, uint32_t n,
                         const float* __restrict__ ipos,
                         const float* __restrict__ ivel,
                         float4* __restrict__ pos, float4* __restrict__ vel,
                         float2* __restrict__ dens) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  dens[first + k] = make_float2(0.0f, 0.0f);
  pos[first + k] = ipos ? make_float4(ipos[3 * k], ipos[3 * k + 1],
                                      ipos[3 * k + 2], __uint_as_float(k))
                       : make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(k));
  vel[first + k] = ivel ? make_float4(ivel[3 * k], ivel[3 * k + 1],
                                      ivel[3 * k + 2], 0.0f)
                        : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}

// Upload from rows the device addresses directly: its own memory, or pinned
// host buffers read over the CPU link. The caller-order float3 rows of 32
// consecutive particles are 384 contiguous bytes, 24 float4. Each warp reads its
// chunk as aligned float4 (the link's transactions stay full) and transposes it
// through shared memory; a partial last chunk goes by scalar loads, so
// nothing outside the 3n floats is touched. The arrays must be 16-byte
// aligned (checked by the launcher's caller).
constexpr int kXferBlock = 256;
constexpr int kXferWarps = kXferBlock / 32;

// The histogram of a prediction that went unused, zeroed before an import
// writes its own: a kernel instead of a memset so that the import's loads and
// stores run beside it (launched programmatically, it waits before its first
// atomic). Passes of one upload, step and download, us, memset / this: a
// lattice of 2,000 particles 48.6 / 46.5, 8,000 54.8 / 53.0, 50,000 69.9 / 67.8, a
// dam of 16,384 in 3 substeps 93.3 / 91.5; at 1,000, where the host's launches
// bound the pass, 41.9 / 42.7: kClearRows.
constexpr uint32_t kClearRows = 1024;
__global__ void k_clear(uint4* __restrict__ words, uint32_t n) {
  pdl_launch();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) words[i] = make_uint4(0u, 0u, 0u, 0u);
}

// With `scene` the kernel also predicts the next step's first substep for
// the imported state exactly as k_predict_hash would (key, arrival rank,
// cell, caller index, and the histogram), so that step can skip it: device
// uploads did that, the import and the zeroing of the densities in three
// launches (1M: 8 + 3 + 20 us; a pass of one upload and step 800 -> 790 us,
// 1,000 particles 50 -> 44, 8.4M 5.54 -> 5.46 ms).
__global__ void __launch_bounds__(kXferBlock)
k_import_rows(uint32_t first, uint32_t n, const float* __restrict__ ipos,
              const float* __restrict__ ivel, float4* __restrict__ pos,
              float4* __restrict__ vel, float2* __restrict__ dens,
              const SceneDev* __restrict__ scene, uint32_t* __restrict__ count,
              uint4* __restrict__ keyrank) {
  __shared__ __align__(16) float s_rows[kXferWarps][2][96];
  const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
  const uint32_t k0 = (blockIdx.x * kXferWarps + w) * 32u;
  if (k0 >= n) return;  // whole warp
  const uint32_t cnt = min(32u, n - k0);
  float* sp = s_rows[w][0];
  float* sv = s_rows[w][1];
  const uint64_t f0 = 3ull * k0;
  if (cnt == 32u) {
    if (lane < 24u) {
      reinterpret_cast<float4*>(sp)[lane] =
          __ldcs(reinterpret_cast<const float4*>(ipos + f0) + lane);
      if (ivel)
        reinterpret_cast<float4*>(sv)[lane] =
            __ldcs(reinterpret_cast<const float4*>(ivel + f0) + lane);
    }
  } else {
    for (uint32_t e = lane; e < 3u * cnt; e += 32u) {
      sp[e] = ipos[f0 + e];
      if (ivel) sv[e] = ivel[f0 + e];
    }
  }
  __syncwarp();
  const bool live = lane < cnt;
  const uint32_t k = k0 + lane;
  float4 p4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), v4 = p4;
  if (live) {
    p4 = make_float4(sp[3 * lane], sp[3 * lane + 1], sp[3 * lane + 2], __uint_as_float(k));
    if (ivel) v4 = make_float4(sv[3 * lane], sv[3 * lane + 1], sv[3 * lane + 2], 0.0f);
    pos[first + k] = p4;
    vel[first + k] = v4;
    dens[first + k] = make_float2(0.0f, 0.0f);
  }
  if (scene) {  // every lane of the warp takes part (warp-aggregated atomics)
    const SceneDev S = *scene;
    uint32_t key = 0, cell = 0;
    if (live) predict_key(S, p4, v4, key, cell);
    key = pdl_wait(key);  // for k_clear
    const uint32_t r = aggregated_rank(count, key, live);
    if (live) keyrank[first + k] = make_uint4(key, r, cell, k);
  }
}

}  // namespace

// ------------------------------------------------------------- launchers
template <int N>
cudaError_t launch_scene_chunk(SceneDev* table, const SceneDev* host, uint32_t count,
                               cudaStream_t st) {
  SceneChunk<N> chunk;
  std::copy(host, host + count, chunk.s);
  return launch_pdl(false, k_scenes<N>, 1, 256, st, chunk,
                    count * static_cast<uint32_t>(sizeof(SceneDev) / 4),
                    reinterpret_cast<uint32_t*>(table));
}

cudaError_t launch_scenes(SceneDev* scene_table, const SceneDev* host, uint32_t scenes,
                          cudaStream_t st) {
  cudaError_t e = cudaSuccess;
  for (uint32_t s = 0; s < scenes && e == cudaSuccess;) {
    const uint32_t left = scenes - s;
    const uint32_t n = std::min<uint32_t>(left, left <= kFewScenes ? kFewScenes : kManyScenes);
    e = left <= kFewScenes ? launch_scene_chunk<kFewScenes>(scene_table + s, host + s, n, st)
                           : launch_scene_chunk<kManyScenes>(scene_table + s, host + s, n, st);
    s += n;
  }
  return e;
}

cudaError_t launch_tiles(const SceneDev* scene_table, uint32_t scenes, uint32_t ntiles,
                         uint2* tiles_old, uint2* tiles_new, cudaStream_t st) {
  if (ntiles == 0) return cudaSuccess;
  return launch_pdl(true, k_tiles, (ntiles + 255) / 256, 256, st, scene_table, scenes, ntiles,
                    tiles_old, tiles_new);
}

cudaError_t launch_predict_hash(const LaunchCtx& c, const Tiles& old_tiles,
                                cudaStream_t st) {
  if (old_tiles.n == 0) return cudaSuccess;
  return launch_pdl(c.pdl, k_predict_hash, grid_for(old_tiles.n, c.block_misc, c.max_blocks),
                    c.block_misc, st, old_tiles.d, old_tiles.n, c.scenes, c.pos,
                    c.vel, c.count, c.keyrank);
}

cudaError_t launch_scan(const LaunchCtx& c, uint32_t len, cudaStream_t st) {
  const uint32_t nb = (len + kScanBlock - 1) / kScanBlock;
  if (nb == 0) return cudaSuccess;
  const int fold = nb <= kScanFoldBlocks ? 1 : 0;
  cudaError_t e = launch_pdl(c.pdl, k_scan_reduce, nb, kScanThreads, st, c.count, len, c.partial);
  if (e == cudaSuccess && !fold)
    e = launch_pdl(c.pdl, k_scan_partials, 1, kScanThreads, st, c.partial, nb, c.start, len);
  if (e == cudaSuccess)
    e = launch_pdl(c.pdl, k_scan_down, nb, kScanThreads, st, c.count, len, c.partial, nb,
                   fold, c.start);
  return e;
}

int kernels_per_substep(uint32_t keys, int tables) {
  const uint32_t nb = (keys + kScanBlock - 1) / kScanBlock;
  return (nb <= kScanFoldBlocks ? 8 : 9) - (tables == kTablesDirect ? 1 : 0);
}

uint32_t scan_partials_needed(uint64_t len) {
  return static_cast<uint32_t>((len + kScanBlock - 1) / kScanBlock) + 1;
}

// Launches that take the latency forms (the walk and the lane-a-particle
// force kernels wait on serial chains while most of the GPU idles). Measured
// per substep, us, plain / latency form:
//   density  16k 32 / 11, 37k 35 / 16, 65k 36 / 25 (a settled pool 21 / 19),
//            90k 37 / 31 (pool 21 / 24), 131k 38 / 41
//   pressure 16k 14 / 10, 28k 14 / 11, 33k 12 / 13, 45k 14 / 14, 65k 14 / 19
//   viscosity alike
// The results are the plain forms' bit for bit, so a scene steps alike in a
// batch of any size. Tunings that choose another arithmetic (two lanes a
// particle, the cell tile) keep their own kernels.
constexpr uint32_t kRowsTiles = 2048;  // 65,536 particles
constexpr uint32_t kCoopTiles = 900;   // 28,800 particles

// Batches of tiny scenes: a tile each, mostly empty, whose walks are over after a
// few candidates. There the number of tiles at work counts: the latency forms
// hold four an SM and are kept to one wave of those, and the walk runs at 32
// registers (64 tiles an SM), a candidate at a time. Substeps of scenes x
// particles, us, by the other launches' forms / by these: 2,048 x 1 27.0 / 20.7,
// 2,000 x 9 34.1 / 31.0, 2,000 x 16 39.1 / 38.0, 16,000 x 3 54.7 / 49.3, 30,000 x 2
// 74.9 / 67.8, 16,000 x 10 79.7 / 74.4; but 2,000 x 24 43.3 / 45.0, 1,000 x 33
// 50.0 / 59.6.
constexpr uint32_t kTinyScene = 20;    // particles, on average
constexpr uint32_t kLatencyTiles = 4;  // tiles an SM holds in the latency forms
bool tiny_scenes(const LaunchCtx& c) { return c.particles < uint64_t{kTinyScene} * c.live; }
bool latency_wave(const LaunchCtx& c, uint32_t ntiles) {
  return !tiny_scenes(c) || ntiles <= kLatencyTiles * c.sms;
}
bool rows_table(const LaunchCtx& c, uint32_t ntiles) {
  return ntiles <= kRowsTiles && latency_wave(c, ntiles);
}
bool rows_form(const LaunchCtx& c, uint32_t ntiles) {
  return c.cell_tile <= 1 && rows_table(c, ntiles);
}
bool coop_form(const LaunchCtx& c, uint32_t ntiles) {
  return c.lanes == 1 && ntiles <= kCoopTiles && latency_wave(c, ntiles);
}

// Launches whose plain neighbour kernels fit the GPU in about one wave (48
// registers: 40 warps an SM) go out without the programmatic attribute. A
// kernel started early is placed around its predecessor's resident blocks,
// and with a single wave that uneven placement stays (more waves even it out):
// passes of three substeps, us, with it / without: 67k particles 187 / 171, 90k
// 218 / 180, 130k 245 / 205, 150k 252 / 219, 180k 257 / 252, 195k 266 / 268,
// 260k 360 / 364; a settled pool of 130k 160 / 142. (The latency forms gain
// from it: 37k 139 / 141.)
//
// Between 40 and 48 warps an SM the density and viscosity passes run at 40
// registers (some spills), which keeps them to one wave; the pressure pass
// would spill in its loop and stays at 48. Passes of three substeps, us, two
// waves / one: 200k particles 279 / 278, 210k 313 / 295, 220k 328 / 302, 232k 342
// / 315; a settled pool of 220k 207 / 199.
constexpr uint32_t kWaveWarps = 40;
constexpr uint32_t kDenseWarps = 48;  // at 40 registers
uint32_t waves(const LaunchCtx& c, uint32_t ntiles, uint32_t warps) {
  return (ntiles + warps * c.sms - 1) / (warps * c.sms);
}
bool dense_wave(const LaunchCtx& c, uint32_t ntiles) {
  return c.lanes == 1 && c.gather == 2 && c.cell_tile <= 1 && ntiles > kWaveWarps * c.sms &&
         ntiles <= kDenseWarps * c.sms;
}
bool one_wave(const LaunchCtx& c, uint32_t ntiles) {
  return ntiles > kRowsTiles && (ntiles <= kWaveWarps * c.sms || dense_wave(c, ntiles));
}

// Launches whose viscosity pass runs at 48 instead of 40 warps an SM: where that
// saves a wave, and those of more than three waves (else the last wave costs
// more than the occupancy gives). Viscosity per substep, us, 40 / 48 warps: 262k
// particles 28.7 / 30.2, 420k (three waves / two) 38.6 / 36.8, 500k 43.6 / 45.9,
// 700k 57.8 / 54.5, 1M 82.2 / 79.1 (a settled pool 54.0 / 52.3), 2M 149.7 / 140.3,
// 8.4M 583 / 539. The pressure pass needs 48 registers: at 40 it spills in its
// loop (1M 91 / 104).
constexpr uint32_t kDenseWaves = 3;
bool dense_form(const LaunchCtx& c, uint32_t ntiles) {
  return c.lanes == 1 && c.gather == 2 &&
         (ntiles > kDenseWaves * kWaveWarps * c.sms ||
          (ntiles > kRowsTiles && waves(c, ntiles, kDenseWarps) < waves(c, ntiles, kWaveWarps)));
}

// List entries a lane of the plain force kernels gathers at once: at least 8,
// then 4, where too few warps hide the loads (the results do not depend on
// it). Passes of three substeps, us, by 2 / 4 / 8 entries: 32k particles 134 / 124
// / 120, 37k 137 / 126 / 123, 50k 156 / 146 / 152, 67k 173 / 168 / 171, 90k 178 /
// 178 / 200. Three, at 59 registers and 32 warps an SM, where those make no more
// waves than the 40 warps of two: 236k 346 / 335 (two / three entries), 284k 375 /
// 361, 308k 387 / 375, 428k 517 / 504; settled pools 215 / 211, 229 / 227, 239 /
// 237, 317 / 314; but 332k 405 / 410, 380k 441 / 462, 500k 565 / 565.
constexpr uint32_t kGather8Tiles = 1200;
constexpr uint32_t kGather3Warps = 32;
constexpr int kGatherBlock = 512;  // larger ones gather what the tuning asks for, if it fits
int force_gather(const LaunchCtx& c, uint32_t ntiles) {
  if (c.block_force > kGatherBlock) return c.gather;
  const bool three = c.lanes == 1 && ntiles > kDenseWarps * c.sms &&
                     ntiles <= kDenseWaves * kWaveWarps * c.sms &&
                     waves(c, ntiles, kGather3Warps) == waves(c, ntiles, kWaveWarps);
  return std::max(c.gather, ntiles <= kGather8Tiles ? 8 : ntiles <= kRowsTiles ? 4 : three ? 3 : 2);
}

std::array<int, 8> launch_forms(const LaunchCtx& c, uint32_t ntiles) {
  const bool rows = rows_form(c, ntiles), coop = coop_form(c, ntiles);
  return {c.cell_tile,
          rows ? 0 : c.block_nbr,
          rows ? 0 : dense_wave(c, ntiles),
          coop ? 0 : c.lanes,
          coop ? 0 : c.block_force,
          coop ? 0 : force_gather(c, ntiles),
          coop ? 0 : dense_form(c, ntiles),
          one_wave(c, ntiles)};
}

cudaError_t launch_sort_reorder(const LaunchCtx& c, const Tiles& old_tiles,
                                const Tiles& new_tiles, uint32_t total,
                                cudaStream_t st) {
  cudaError_t e = cudaSuccess;
  if (old_tiles.n)
    e = launch_pdl(c.pdl, k_scatter, grid_for(old_tiles.n, c.block_misc, c.max_blocks),
                   c.block_misc, st, old_tiles.d, old_tiles.n, c.keyrank, c.start,
                   total, c.tmp_hi, c.tmp_src, c.status);
  if (new_tiles.n && e == cudaSuccess) {
    e = launch_pdl(c.pdl,
                   c.tables == kTablesDirect && c.cell_tile <= 1 ? k_reorder<false>
                                                                 : k_reorder<true>,
                   grid_for(new_tiles.n, c.block_misc, c.max_blocks),
                   c.block_misc, st, new_tiles.d, new_tiles.n, c.scenes, c.tmp_hi,
                   c.tmp_src, c.start, c.pos, c.vel, c.pos2, c.vel2, c.pred,
                   c.hash_s, c.cell_first, c.src_limit, c.status);
    if (e == cudaSuccess && c.tables != kTablesDirect)
      e = rows_table(c, new_tiles.n)
              ? launch_pdl(c.pdl, k_cell_table_rows, new_tiles.n, 32 * kRowWarps, st, new_tiles.d,
                           new_tiles.n, c.scenes, c.hash_s, c.cell_first, c.start, c.cell_tab)
              : launch_pdl(c.pdl, k_cell_table,
                           grid_for(new_tiles.n, kCellTableBlock, c.max_blocks), kCellTableBlock,
                           st, new_tiles.d, new_tiles.n, c.scenes, c.hash_s, c.cell_first, c.start,
                           c.cell_tab);
  }
  return e;
}

template <int kRegs, uint32_t kBatch> auto density_kernel(int tables) {
  return tables == kTablesDirect    ? k_density_walk<kTablesDirect, kRegs, kBatch>
         : tables == kTablesBuckets ? k_density_walk<kTablesBuckets, kRegs, kBatch>
                                    : k_density_walk<kTablesMixed, kRegs, kBatch>;
}

cudaError_t launch_density(const LaunchCtx& c, const Tiles& tiles,
                           cudaStream_t st) {
  if (tiles.n == 0) return cudaSuccess;
  if (rows_form(c, tiles.n))
    return launch_pdl(c.pdl,
                      c.tables == kTablesDirect    ? k_density_rows<kTablesDirect>
                      : c.tables == kTablesBuckets ? k_density_rows<kTablesBuckets>
                                                   : k_density_rows<kTablesMixed>,
                      tiles.n, 32 * kRowWarps, st, tiles.d, tiles.n, c.scenes, c.pred, c.start,
                      c.cell_first, c.cell_tab, c.dens_a, c.dens_b, c.nbr, c.ncount);
  const int b = c.block_nbr;
  const uint32_t g = grid_for(tiles.n, b, c.max_blocks);
  if (c.cell_tile <= 1)
    return launch_pdl(c.pdl && !one_wave(c, tiles.n),
                      tiny_scenes(c)           ? density_kernel<32, 1>(c.tables)
                      : dense_wave(c, tiles.n) ? density_kernel<40, kWalkBatch>(c.tables)
                                               : density_kernel<48, kWalkBatch>(c.tables),
                      g, b, st, tiles.d, tiles.n, c.scenes, c.pred,
                      c.start, c.cell_first, c.cell_tab, c.dens_a, c.dens_b, c.nbr,
                      c.ncount, 32u, kNbrCap);
  auto kern = c.cell_tile <= 64    ? k_density<2>
              : c.cell_tile <= 128 ? k_density<4>
              : c.cell_tile <= 192 ? k_density<6>
                                   : k_density<8>;
  return launch_pdl(c.pdl, kern, g, b, st, tiles.d, tiles.n, c.scenes, c.pred,
                    c.start, c.cell_first, c.cell_tab, c.dens_a, c.dens_b, c.nbr,
                    c.ncount);
}

// The instantiations for a gather batch (2, 3, 4 or 8) and the launch's
// table forms.
template <int kTables, int kLanes>
auto pressure_kernel(int gather) {
  return gather == 2   ? k_pressure<2, kTables, kLanes>
         : gather == 3 ? k_pressure<3, kTables, kLanes>
         : gather == 8 ? k_pressure<8, kTables, kLanes>
                       : k_pressure<4, kTables, kLanes>;
}

template <int kTables>
auto pressure_kernel(int gather, int lanes) {
  return lanes == 2 ? pressure_kernel<kTables, 2>(gather) : pressure_kernel<kTables, 1>(gather);
}

template <int kTables, int kLanes>
auto visc_kernel(int gather) {
  return gather == 2   ? k_visc_integrate<2, kTables, kLanes>
         : gather == 3 ? k_visc_integrate<3, kTables, kLanes>
         : gather == 8 ? k_visc_integrate<8, kTables, kLanes>
                       : k_visc_integrate<4, kTables, kLanes>;
}

template <int kTables>
auto visc_kernel(int gather, int lanes) {
  return lanes == 2 ? visc_kernel<kTables, 2>(gather) : visc_kernel<kTables, 1>(gather);
}

// pick(gather), or the kernel of the next smaller batch that a block of `block`
// threads has the registers for: 4 entries take up to 77 a thread, 8 up to 127,
// where 1,024 threads leave 64 (two take 62 at most). 256 threads fit whatever
// a kernel takes and need no question. The results do not depend on the batch.
template <class Pick> auto fitting_kernel(Pick pick, int gather, int block) {
  for (;;) {
    const auto kern = pick(gather);
    cudaFuncAttributes a{};
    if (gather == 2 || block <= 256 ||
        (cudaFuncGetAttributes(&a, kern) == cudaSuccess && a.maxThreadsPerBlock >= block))
      return kern;
    gather = gather == 8 ? 4 : gather - 1;
  }
}

cudaError_t launch_pressure(const LaunchCtx& c, const Tiles& tiles,
                            cudaStream_t st) {
  if (tiles.n == 0) return cudaSuccess;
  if (coop_form(c, tiles.n))
    return launch_pdl(c.pdl,
                      c.tables == kTablesDirect    ? k_pressure_coop<kTablesDirect>
                      : c.tables == kTablesBuckets ? k_pressure_coop<kTablesBuckets>
                                                   : k_pressure_coop<kTablesMixed>,
                      grid_for(tiles.n * kCoopSub, kCoopBlock, c.max_blocks), kCoopBlock, st,
                      tiles.d, tiles.n, c.scenes, c.pred, c.start, c.cell_first, c.cell_tab,
                      c.dens_a, c.dens_b, c.nbr, c.ncount, c.vel2, c.rec_v, c.dbg_accp,
                      c.dbg_velp);
  const int b = c.block_force;
  auto kern = fitting_kernel([&](int gather) {
    return c.tables == kTablesDirect    ? pressure_kernel<kTablesDirect>(gather, c.lanes)
           : c.tables == kTablesBuckets ? pressure_kernel<kTablesBuckets>(gather, c.lanes)
                                        : pressure_kernel<kTablesMixed>(gather, c.lanes);
  }, force_gather(c, tiles.n), b);
  // Started early beside k_density_rows' blocks this kernel would run with the
  // L1 their shared memory leaves it (37k particles: 9 us a substep).
  return launch_pdl(c.pdl && !rows_form(c, tiles.n) && !one_wave(c, tiles.n), kern,
                    grid_for(tiles.n, b, c.max_blocks), b, st, tiles.d, tiles.n, c.scenes, c.pred, c.start, c.cell_first, c.cell_tab,
                    c.dens_a, c.dens_b, c.nbr, c.ncount,
                    c.vel2, c.rec_v, c.rec_b, c.dbg_accp, c.dbg_velp);
}

cudaError_t launch_visc_integrate(const LaunchCtx& c, const Tiles& tiles,
                                  int fuse_next, int write_out,
                                  cudaStream_t st) {
  if (tiles.n == 0) return cudaSuccess;
  if (coop_form(c, tiles.n))
    return launch_pdl(c.pdl,
                      c.tables == kTablesDirect    ? k_visc_coop<kTablesDirect>
                      : c.tables == kTablesBuckets ? k_visc_coop<kTablesBuckets>
                                                   : k_visc_coop<kTablesMixed>,
                      grid_for(tiles.n * kCoopSub, kCoopBlock, c.max_blocks), kCoopBlock, st,
                      tiles.d, tiles.n, c.scenes, c.pred, c.start, c.cell_first, c.cell_tab, c.nbr,
                      c.ncount, c.rec_v, c.pos2, c.vel2, write_out ? c.out4 : nullptr, fuse_next,
                      c.count, c.keyrank, c.dbg_velv, c.status);
  const int b = c.block_force;
  auto kern = dense_form(c, tiles.n)
                  ? (c.tables == kTablesDirect    ? k_visc_dense<kTablesDirect>
                     : c.tables == kTablesBuckets ? k_visc_dense<kTablesBuckets>
                                                  : k_visc_dense<kTablesMixed>)
                  : fitting_kernel([&](int gather) {
    return c.tables == kTablesDirect    ? visc_kernel<kTablesDirect>(gather, c.lanes)
           : c.tables == kTablesBuckets ? visc_kernel<kTablesBuckets>(gather, c.lanes)
                                        : visc_kernel<kTablesMixed>(gather, c.lanes);
  }, force_gather(c, tiles.n), b);
  return launch_pdl(c.pdl && !one_wave(c, tiles.n), kern, grid_for(tiles.n, b, c.max_blocks), b,
                    st, tiles.d, tiles.n, c.scenes, c.pred, c.start, c.cell_first, c.cell_tab, c.nbr,
                    c.ncount, c.rec_v, c.rec_b, c.pos2, c.vel2,
                    write_out ? c.out4 : nullptr, fuse_next, c.count, c.keyrank,
                    c.dbg_velv, c.status);
}

cudaError_t launch_export(uint32_t first, uint32_t n, const float4* pos,
                          const float4* vel, const float2* dens, float* opos,
                          float* ovel, float* odens, uint32_t* oids,
                          cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  return launch_pdl(false, k_export, (n + 255) / 256, 256, st, first, n, pos, vel, dens, opos,
                    ovel, odens, oids);
}

cudaError_t launch_export_rows(uint32_t first, uint32_t n, const float4* pos,
                              const float4* vel, const float2* dens, uint32_t* slot_of,
                              float* opos, float* ovel, float* odens, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const cudaError_t e =
      launch_pdl(false, k_slot_map, (n + 255) / 256, 256, st, first, n, pos, slot_of);
  if (e != cudaSuccess) return e;
  return launch_pdl(true, k_export_rows, (n + 255) / 256, 256, st, first, n, slot_of, pos, vel,
                    dens, opos, ovel, odens);
}

cudaError_t launch_export_debug(uint32_t first, uint32_t n, const float4* pos,
                                const float4* accp, const float4* velp,
                                const float4* velv, float* oaccp, float* ovelp,
                                float* ovelv, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  return launch_pdl(false, k_export_debug, (n + 255) / 256, 256, st, first, n, pos, accp, velp,
                    velv, oaccp, ovelp, ovelv);
}

cudaError_t launch_export_layout(uint32_t first, uint32_t n, const SceneDev* scene,
                                 const float4* pos, const float4* pred, uint32_t* ocell,
                                 uint32_t* okey, uint32_t* oslot, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  return launch_pdl(false, k_export_layout, (n + 255) / 256, 256, st, first, n, scene, pos, pred,
                    ocell, okey, oslot);
}

cudaError_t launch_ref_lookup(const LaunchCtx& c, const Tiles& new_tiles,
                              uint32_t total, cudaStream_t st) {
  if (new_tiles.n == 0) return cudaSuccess;
  const uint32_t g = grid_for(new_tiles.n, c.block_misc, c.max_blocks);
  cudaError_t e = launch_pdl(c.pdl, k_ref_hash, g, c.block_misc, st, new_tiles.d,
                             new_tiles.n, c.scenes, c.pred, c.pos2, c.dbg_count,
                             c.dbg_keyrank, c.dbg_hash, c.dbg_key, c.status);
  LaunchCtx d = c;  // the scan over the lookup's own histogram
  d.count = c.dbg_count;
  d.start = c.dbg_start;
  d.partial = c.dbg_partial;
  if (e == cudaSuccess) e = launch_scan(d, total, st);
  if (e == cudaSuccess)
    e = launch_pdl(c.pdl, k_ref_scatter, g, c.block_misc, st, new_tiles.d, new_tiles.n,
                   c.pos2, c.dbg_keyrank, c.dbg_start, total, c.dbg_tmp, c.status);
  if (e == cudaSuccess)
    e = launch_pdl(c.pdl, k_ref_order, g, c.block_misc, st, new_tiles.d, new_tiles.n,
                   c.pos2, c.dbg_keyrank, c.dbg_start, c.dbg_tmp, c.dbg_sorted);
  return e;
}

cudaError_t launch_import(uint32_t first, uint32_t n, const float* ipos,
                          const float* ivel, float4* pos, float4* vel, float2* dens,
                          cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  return launch_pdl(false, k_import, (n + 255) / 256, 256, st, first, n, ipos, ivel, pos, vel,
                    dens);
}

cudaError_t launch_import_rows(uint32_t first, uint32_t n, const float* ipos,
                               const float* ivel, float4* pos, float4* vel, float2* dens,
                               const SceneDev* scene, uint32_t* count, uint32_t clear,
                               uint4* keyrank, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const uint32_t words = (clear + 3) / 4;  // (the tables end on a 16-byte word)
  const bool beside = words && n > kClearRows;
  cudaError_t e = cudaSuccess;
  if (beside) {
    e = launch_pdl(false, k_clear, (words + 255) / 256, 256, st, reinterpret_cast<uint4*>(count),
                   words);
  } else if (words) {
    e = cudaMemsetAsync(count, 0, sizeof(uint4) * words, st);
  }
  if (e != cudaSuccess) return e;
  const uint32_t warps = (n + 31) / 32;
  return launch_pdl(beside, k_import_rows, (warps + kXferWarps - 1) / kXferWarps, kXferBlock,
                    st, first, n, ipos, ivel, pos, vel, dens, scene, count, keyrank);
}

}  // namespace sph
