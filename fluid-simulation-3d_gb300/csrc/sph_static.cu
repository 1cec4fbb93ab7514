// Spatial lookup that allocates no device memory.
//
// Some callers cannot allocate device memory: an interactive render loop
// (like the reference's GL app) must not call cudaMalloc/cudaFree mid-frame
// because they synchronise the whole device and stall the frame; engines that
// own a fixed memory budget or a pool forbid allocations from plug-ins.
// sph_spatial_lookup_static serves them: the caller passes its own device
// buffers for inputs and outputs, and the working memory (the entries between
// the two sorting passes) is the file-scope array below, 8 B per particle for
// up to SPH_STATIC_LOOKUP_MAX particles -- 512 KiB that every GPU loading this
// library keeps until the process exits.
//
// The entry point has no counterpart in the reference; it builds the same
// lookup as the main path's sort (hash, key = hash % n, the canonical
// (key, index) order, the start table with 0x7fffffff for empty keys), in one
// kernel of one eight-block cluster whose work is linear in n whatever the
// keys: a stable radix sort of the 16-bit keys in two passes of 8 bits, so a
// scene whose particles all share one key costs what any other scene of its
// size does. (Up to 512 particles one block ranks every entry among the others,
// without the working memory; that cost depends on n alone, too.)
#include <cstdint>
#include <mutex>
#include <string>

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "../../include/sph_gb300.h"
#include "sph_device.cuh"

namespace sph {

namespace {

constexpr uint32_t kMax = SPH_STATIC_LOOKUP_MAX;
constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
constexpr int kBlocks = 8;  // one cluster
constexpr int kRounds = kMax / (kBlocks * kThreads);  // entries a thread holds at most
constexpr int kMaxDevices = 64;

static_assert(kMax <= 65536, "an entry packs a 16-bit key and a 16-bit index");

// Packed (key, index) entries after the first and the second pass.
__device__ __align__(256) uint32_t g_lookup_scratch[2 * kMax];

std::mutex g_mu;
uint32_t* g_scratch_addr[kMaxDevices] = {};
std::string g_static_error;

struct RadixSmem {
  uint32_t warp_digits[kWarps][256];  // per warp: entries of each digit, then their prefix
  uint32_t block_digits[2][256];      // per pass: the block's entries of each digit
  uint32_t first[256];                // first position of the block's entries of each digit
  uint32_t sums[8];
};

// One stable pass over the cluster's entries by the 8 bits at `shift`. Warp
// gw of the cluster holds the entries [32 gw rounds, 32 (gw + 1) rounds), 32
// consecutive ones a round, so order of warps, rounds and lanes is the order
// of the entries. The rank of an entry among those of its digit is its rank
// in the warp (lanes with equal digits, after the earlier rounds') plus the
// counts of the warps and blocks before; blocks read each other's counts from
// distributed shared memory.
__device__ __forceinline__ void radix_pass(cooperative_groups::cluster_group& cluster,
                                           RadixSmem& sm, int pass, const uint32_t (&v)[kRounds],
                                           uint32_t first, uint32_t rounds, uint32_t n,
                                           uint32_t* __restrict__ out) {
  const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  const uint32_t shift = 16u + 8u * pass;
  uint32_t* const digits = sm.warp_digits[w];
  for (uint32_t d = lane; d < 256u; d += 32u) digits[d] = 0u;
  __syncwarp();
  uint32_t rank[kRounds];
#pragma unroll
  for (uint32_t k = 0; k < kRounds; ++k) {
    rank[k] = 0;
    if (k >= rounds) continue;  // uniform
    const bool valid = first + 32u * k + lane < n;
    const uint32_t am = __ballot_sync(0xffffffffu, valid);
    if (valid) {
      const uint32_t d = (v[k] >> shift) & 255u;
      const uint32_t peers = __match_any_sync(am, d);
      const uint32_t mine = __popc(peers & ((1u << lane) - 1u));
      const uint32_t b = digits[d];
      rank[k] = b + mine;
      __syncwarp(am);
      if (mine == 0u) digits[d] = b + __popc(peers);
    }
    __syncwarp();
  }
  __syncthreads();
  if (threadIdx.x < 256u) {
    uint32_t run = 0;
#pragma unroll 8
    for (int u = 0; u < kWarps; ++u) {
      const uint32_t c = sm.warp_digits[u][threadIdx.x];
      sm.warp_digits[u][threadIdx.x] = run;
      run += c;
    }
    sm.block_digits[pass][threadIdx.x] = run;
  }
  cluster.sync();
  uint32_t before = 0, total = 0;
  if (threadIdx.x < 256u) {
#pragma unroll
    for (uint32_t b = 0; b < kBlocks; ++b) {
      const uint32_t c = *cluster.map_shared_rank(&sm.block_digits[pass][threadIdx.x], b);
      before += b < cluster.block_rank() ? c : 0u;
      total += c;
    }
  }
  uint32_t incl = total;  // inclusive prefix over the digits: eight warps
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= static_cast<uint32_t>(d)) incl += y;
  }
  if (w < 8u && lane == 31u) sm.sums[w] = incl;
  __syncthreads();
  if (threadIdx.x < 256u) {
    uint32_t base = incl - total + before;
#pragma unroll
    for (uint32_t u = 0; u < 8; ++u) base += u < w ? sm.sums[u] : 0u;
    sm.first[threadIdx.x] = base;
  }
  __syncthreads();
#pragma unroll
  for (uint32_t k = 0; k < kRounds; ++k) {
    if (k < rounds && first + 32u * k + lane < n) {
      const uint32_t d = (v[k] >> shift) & 255u;
      out[sm.first[d] + digits[d] + rank[k]] = v[k];
    }
  }
  cluster.sync();  // the entries are in place for every block
}

// Latency-bound: two passes of a few cluster barriers each. 50,000 particles
// take 27 us, 1048 us when one block ordered the entries with its first warp,
// 32 at a time.
__global__ void __cluster_dims__(kBlocks, 1, 1) __launch_bounds__(kThreads)
k_lookup_static(const float* __restrict__ pred3, uint32_t n, float r,
                uint64_t fm, uint32_t* __restrict__ scratch,
                uint32_t* __restrict__ ohash, uint32_t* __restrict__ okey,
                uint32_t* __restrict__ osorted, uint32_t* __restrict__ ostart) {
  __shared__ RadixSmem sm;
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t gw = cluster.block_rank() * kWarps + (threadIdx.x >> 5);
  const uint32_t rounds = (n + kBlocks * kThreads - 1u) / (kBlocks * kThreads);
  const uint32_t first = gw * 32u * rounds;
  uint32_t v[kRounds];
  // HashCell(PositionToCellCoord(pred)), key = hash % n
  // (physicsWorld.cc:499-516).
#pragma unroll
  for (uint32_t k = 0; k < kRounds; ++k) {
    const uint32_t i = first + 32u * k + lane;
    v[k] = 0u;
    if (k < rounds && i < n) {
      const float3 p = make_float3(pred3[3 * i], pred3[3 * i + 1], pred3[3 * i + 2]);
      const uint32_t h = hash_cell(cell_of(p.x, r), cell_of(p.y, r), cell_of(p.z, r));
      const uint32_t key = fastmod(h, fm, n);
      ohash[i] = h;
      okey[i] = key;
      ostart[i] = 0x7fffffffu;
      v[k] = key << 16 | i;
    }
  }
  radix_pass(cluster, sm, 0, v, first, rounds, n, scratch);
#pragma unroll
  for (uint32_t k = 0; k < kRounds; ++k) {
    const uint32_t i = first + 32u * k + lane;
    if (k < rounds && i < n) v[k] = __ldcg(scratch + i);
  }
  radix_pass(cluster, sm, 1, v, first, rounds, n, scratch + kMax);
  // sorted ids, and the start of each key: the entry whose predecessor has
  // another key
#pragma unroll
  for (uint32_t k = 0; k < kRounds; ++k) {
    const uint32_t i = first + 32u * k + lane;
    if (k < rounds && i < n) {
      const uint32_t e = __ldcg(scratch + kMax + i);
      const uint32_t key = e >> 16;
      osorted[i] = e & 0xffffu;
      if (i == 0u || __ldcg(scratch + kMax + i - 1u) >> 16 != key) ostart[key] = i;
    }
  }
}

// The smallest calls: one block of a thread a particle, which ranks its entry
// among all of them. A cluster's launch and barriers would be most of such a call.
// us a call, the cluster / this: 32 particles 8.4 / 4.3, 100 8.4 / 4.2, 256 10.0 /
// 4.3, 400 10.4 / 6.4, 512 10.4 / 8.4; the ranking grows with n^2, so the line is
// drawn there.
constexpr uint32_t kSmall = 512;
__global__ void __launch_bounds__(kSmall)
k_lookup_small(const float* __restrict__ pred3, uint32_t n, float r, uint64_t fm,
               uint32_t* __restrict__ ohash, uint32_t* __restrict__ okey,
               uint32_t* __restrict__ osorted, uint32_t* __restrict__ ostart) {
  __shared__ __align__(16) uint32_t s_entry[kSmall];
  __shared__ uint32_t s_sorted[kSmall];
  const uint32_t i = threadIdx.x;  // (the block is n rounded up to whole warps)
  uint32_t mine = 0xffffffffu;
  if (i < n) {
    const float3 p = make_float3(pred3[3 * i], pred3[3 * i + 1], pred3[3 * i + 2]);
    const uint32_t h = hash_cell(cell_of(p.x, r), cell_of(p.y, r), cell_of(p.z, r));
    const uint32_t key = fastmod(h, fm, n);
    ohash[i] = h;
    okey[i] = key;
    ostart[i] = 0x7fffffffu;
    mine = key << 16 | i;
  }
  s_entry[i] = mine;
  __syncthreads();
  uint32_t rank = 0;
#pragma unroll 4
  for (uint32_t k = 0; k < n; k += 4u) {
    const uint4 e = *reinterpret_cast<const uint4*>(s_entry + k);
    rank += (e.x < mine) + (e.y < mine) + (e.z < mine) + (e.w < mine);
  }
  if (i < n) s_sorted[rank] = mine;
  __syncthreads();
  if (i < n) {
    const uint32_t e = s_sorted[i], key = e >> 16;
    osorted[i] = e & 0xffffu;
    if (i == 0u || s_sorted[i - 1u] >> 16 != key) ostart[key] = i;
  }
}

}  // namespace

}  // namespace sph

extern "C" const char* sph_static_error(void) {
  std::lock_guard<std::mutex> lock(sph::g_mu);
  return sph::g_static_error.c_str();
}

extern "C" int sph_spatial_lookup_static(const float* dpred3, uint32_t n,
                                         float radius, uint32_t* dhash,
                                         uint32_t* dkey, uint32_t* dsorted_ids,
                                         uint32_t* dstart, void* stream) {
  using namespace sph;
  auto fail = [](int code, const std::string& msg) {
    std::lock_guard<std::mutex> lock(g_mu);
    g_static_error = msg;
    return code;
  };
  if (n == 0 || n > kMax)
    return fail(SPH_ERR_INVALID,
                "sph_spatial_lookup_static: n must be in [1, " +
                    std::to_string(kMax) + "], got " + std::to_string(n));
  if (!dpred3 || !dhash || !dkey || !dsorted_ids || !dstart)
    return fail(SPH_ERR_INVALID, "sph_spatial_lookup_static: null buffer");
  if (!(radius > 0.0f))
    return fail(SPH_ERR_INVALID, "sph_spatial_lookup_static: radius must be > 0");
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess)
    return fail(SPH_ERR_CUDA, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
  if (dev < 0 || dev >= kMaxDevices)
    return fail(SPH_ERR_INVALID, "sph_spatial_lookup_static: device index too large");
  uint32_t* scratch = nullptr;
  {
    // First call on a device: resolve the array's device address with that
    // device current (a host-side use of the symbol is not a device address).
    std::lock_guard<std::mutex> lock(g_mu);
    if (!g_scratch_addr[dev]) {
      void* p = nullptr;
      e = cudaGetSymbolAddress(&p, g_lookup_scratch);
      if (e != cudaSuccess) {
        g_static_error = std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e);
        return SPH_ERR_CUDA;
      }
      g_scratch_addr[dev] = static_cast<uint32_t*>(p);
    }
    scratch = g_scratch_addr[dev];
  }
  const uint64_t fm = (~static_cast<uint64_t>(0)) / n + 1;
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  e = n <= kSmall
          ? launch_pdl(false, k_lookup_small, 1, static_cast<int>((n + 31u) / 32u * 32u), st,
                       dpred3, n, radius, fm, dhash, dkey, dsorted_ids, dstart)
          : launch_pdl(false, k_lookup_static, kBlocks, kThreads, st, dpred3, n, radius, fm,
                       scratch, dhash, dkey, dsorted_ids, dstart);
  if (e != cudaSuccess)
    return fail(SPH_ERR_CUDA, std::string("lookup kernel: ") + cudaGetErrorString(e));
  return SPH_OK;
}
