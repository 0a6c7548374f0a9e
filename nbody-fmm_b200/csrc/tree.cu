// Tree build on the GPU, bit-exact with Tree::init_tree (tree.cpp:15-91).
//
// The reference rebins every particle into a hash map once per iteration of
// its depth loop (tree.cpp:43-69).  Here each particle's key is computed once
// at the maximum depth D (16 in 3D, 32 in 2D, tree.cpp:38): the reference's
// leaf coordinate at depth d, (unsigned)((x - a) / ((b - a) / 2^d)), equals
// floor(2^d * q) with q = (x - a) / (b - a) in FP64, because dividing by a
// power of two commutes with IEEE rounding; so the key at depth d is the key
// at D shifted right by dim*(D-d).  One radix sort of the D-keys then holds
// the cells of every depth as runs: particle i starts a cell at each depth
// above the number of levels its key shares with the key before it.  One
// pass over the sorted keys counts the cells and the largest cell of every
// depth, so that the depth loop and the sizes of all levels need one read of
// the host, and one more writes the cells of all levels.  The reference's
// leaves with their particles in input order (tree.cpp:62-66) are the leaf
// runs with each run put back in input order (a rank count inside the leaf),
// or for leaves of more than 512 particles a second stable sort of the
// depth-d keys in input order.
#include <algorithm>
#include <cstddef>
#include <vector>

#include "common.cuh"
#include "tree.cuh"

namespace fmm {

// ------------------------------------------------------------------ scan
static constexpr int SCAN_BLOCK = 256;
static constexpr int SCAN_ITEMS = 8;
static constexpr int SCAN_TILE = SCAN_BLOCK * SCAN_ITEMS;

__device__ inline uint32_t block_excl_scan(uint32_t v, uint32_t *s_warp, uint32_t &total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < (SCAN_BLOCK / 32) ? s_warp[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < SCAN_BLOCK / 32) s_warp[lane] = w;
  }
  __syncthreads();
  uint32_t base = warp ? s_warp[warp - 1] : 0;
  total = s_warp[SCAN_BLOCK / 32 - 1];
  __syncthreads();
  return base + x - v;
}

__global__ void k_scan_reduce(const uint32_t *in, int64_t n, uint32_t *block_sums) {
  __shared__ uint32_t s_warp[SCAN_BLOCK / 32];
  int64_t base = (int64_t)blockIdx.x * SCAN_TILE;
  uint32_t s = 0;
  for (int i = 0; i < SCAN_ITEMS; ++i) {
    int64_t k = base + (int64_t)i * SCAN_BLOCK + threadIdx.x;
    if (k < n) s += in[k];
  }
  uint32_t total;
  block_excl_scan(s, s_warp, total);
  if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}

__global__ void k_scan_blocks(uint32_t *sums, int nb, uint32_t *total_out) {
  __shared__ uint32_t s_warp[SCAN_BLOCK / 32];
  uint32_t carry = 0;
  for (int b0 = 0; b0 < nb; b0 += SCAN_BLOCK) {
    int k = b0 + threadIdx.x;
    uint32_t v = k < nb ? sums[k] : 0, tot;
    uint32_t e = block_excl_scan(v, s_warp, tot);
    if (k < nb) sums[k] = carry + e;
    carry += tot;
  }
  if (threadIdx.x == 0 && total_out) *total_out = carry;
}

// Without block offsets (block_offs null) every block adds up the sums of the
// blocks before it itself, and the last one writes the total.
__global__ void k_scan_apply(const uint32_t *in, uint32_t *out, int64_t n, const uint32_t *block_offs,
                             const uint32_t *sums, uint32_t *total_out) {
  __shared__ uint32_t s_warp[SCAN_BLOCK / 32];
  int64_t base = (int64_t)blockIdx.x * SCAN_TILE + (int64_t)threadIdx.x * SCAN_ITEMS;
  uint32_t off, total;
  if (block_offs) {
    off = block_offs[blockIdx.x];
  } else {
    uint32_t t = 0;
    for (int k = threadIdx.x; k < (int)blockIdx.x; k += SCAN_BLOCK) t += sums[k];
    block_excl_scan(t, s_warp, off);
  }
  uint32_t v[SCAN_ITEMS], s = 0;
  for (int i = 0; i < SCAN_ITEMS; ++i) {
    int64_t k = base + i;
    v[i] = k < n ? in[k] : 0;
    s += v[i];
  }
  uint32_t e = block_excl_scan(s, s_warp, total) + off;
  for (int i = 0; i < SCAN_ITEMS; ++i) {
    int64_t k = base + i;
    if (k < n) out[k] = e;
    e += v[i];
  }
  if (!block_offs && total_out && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *total_out = off + total;
}

// Exclusive prefix sum of n uint32 (in may alias out); *total_dev = sum.
void exclusive_scan(Workspace &ws, const uint32_t *in, uint32_t *out, int64_t n, uint32_t *total_dev,
                    cudaStream_t st) {
  int nb = (int)std::max<int64_t>(1, (n + SCAN_TILE - 1) / SCAN_TILE);
  uint32_t *sums = ws.scan_tmp(nb);
  if (!ws.ok) return;  // out of memory: the caller looks at ws.ok
  // k_scan_reduce uses a strided tile layout and k_scan_apply a blocked one;
  // both cover the same SCAN_TILE elements per block, so the sums agree.
  // Up to 2048 blocks (4M elements) adding the sums up in every block is
  // cheaper than a launch for it.
  const bool two = nb <= 2048;
  k_scan_reduce<<<nb, SCAN_BLOCK, 0, st>>>(in, n, sums);
  if (!two) k_scan_blocks<<<1, SCAN_BLOCK, 0, st>>>(sums, nb, total_dev);
  k_scan_apply<<<nb, SCAN_BLOCK, 0, st>>>(in, out, n, two ? nullptr : sums, sums, total_dev);
  ws.launches += two ? 2 : 3;
}

// ------------------------------------------------------------ radix sort
static constexpr int RS_BLOCK = 256;
static constexpr int RS_ROUNDS = 8;
static constexpr int RS_TILE = RS_BLOCK * RS_ROUNDS;
// Largest leaf whose order k_leaf_order redoes in place (each particle counts
// the smaller input indices of its leaf); larger leaves take the full sort.
static constexpr int LEAF_ORDER_MAX = 512;
// Up to this many tiles (65,536 items) the scatter adds up the tiles'
// histograms itself, two launches per digit instead of four.
static constexpr int RS_FUSED_TILES = 32;

// hist: [digit][tile], or [tile][256] (by_tile).
__global__ void k_radix_hist(const uint64_t *keys, int64_t n, int shift, uint32_t *hist, int nb, bool by_tile) {
  __shared__ uint32_t h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  int64_t base = (int64_t)blockIdx.x * RS_TILE;
  for (int r = 0; r < RS_ROUNDS; ++r) {
    int64_t i = base + (int64_t)r * RS_BLOCK + threadIdx.x;
    if (i < n) atomicAdd(&h[(keys[i] >> shift) & 255u], 1u);
  }
  __syncthreads();
  if (by_tile) hist[(int64_t)blockIdx.x * 256 + threadIdx.x] = h[threadIdx.x];
  else hist[(int64_t)threadIdx.x * nb + blockIdx.x] = h[threadIdx.x];
}

// Stable scatter of one tile of RS_TILE items: items are ranked in (round,
// warp, lane) order, which is their input order inside the tile, and placed
// in shared memory in digit order; then consecutive threads write each
// digit's run to its consecutive places in the output (coalesced stores).
// offs: the exclusive scan of the [digit][tile] histograms, or with by_tile
// the [tile][256] histograms themselves, which thread d adds up for digit d.
__global__ void __launch_bounds__(RS_BLOCK) k_radix_scatter(const uint64_t *kin, const uint32_t *vin, uint64_t *kout,
                                                            uint32_t *vout, int64_t n, int shift, const uint32_t *offs,
                                                            int nb, bool by_tile) {
  __shared__ uint64_t s_key[RS_TILE];
  __shared__ uint32_t s_val[RS_TILE];
  __shared__ uint32_t s_goff[256], s_tstart[256], s_run[256], s_warp[RS_BLOCK / 32];
  __shared__ uint32_t s_cnt[RS_BLOCK / 32][256];
  __shared__ uint32_t s_pre[RS_BLOCK / 32][256];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t base = (int64_t)blockIdx.x * RS_TILE;
  const int tile_n = (int)min((int64_t)RS_TILE, n - base);
  if (by_tile) {
    uint32_t all = 0, before = 0, total;
    for (int b = 0; b < nb; ++b) {
      const uint32_t v = offs[(int64_t)b * 256 + tid];
      if (b == (int)blockIdx.x) before = all;
      all += v;
    }
    s_goff[tid] = block_excl_scan(all, s_warp, total) + before;
  } else {
    s_goff[tid] = offs[(int64_t)tid * nb + blockIdx.x];  // the digit's first place in the output
  }
  s_run[tid] = 0;
  s_tstart[tid] = 0;  // the tile's digit histogram first
  __syncthreads();
  uint64_t key[RS_ROUNDS];
  uint32_t val[RS_ROUNDS], dig[RS_ROUNDS];
#pragma unroll
  for (int r = 0; r < RS_ROUNDS; ++r) {
    const int k = r * RS_BLOCK + tid;
    const bool valid = k < tile_n;
    key[r] = valid ? kin[base + k] : 0ull;
    val[r] = valid ? vin[base + k] : 0u;
    dig[r] = valid ? (uint32_t)((key[r] >> shift) & 255u) : 256u + lane;  // invalid lanes: distinct, unused
    if (valid) atomicAdd(&s_tstart[dig[r]], 1u);
  }
  __syncthreads();
  uint32_t total;
  const uint32_t ex = block_excl_scan(s_tstart[tid], s_warp, total);  // syncs after every thread read its count
  s_tstart[tid] = ex;  // the digit's first place in the tile's digit order
  const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
  for (int r = 0; r < RS_ROUNDS; ++r) {
    for (int w = 0; w < RS_BLOCK / 32; ++w) s_cnt[w][tid] = 0;
    __syncthreads();
    const uint32_t d = dig[r];
    const bool valid = d < 256u;
    const uint32_t peers = __match_any_sync(0xffffffffu, d);
    const uint32_t rank = __popc(peers & lt);
    if (valid && rank == 0) s_cnt[warp][d] = __popc(peers);
    __syncthreads();
    uint32_t run = 0;
    for (int w = 0; w < RS_BLOCK / 32; ++w) {
      const uint32_t c = s_cnt[w][tid];
      s_pre[w][tid] = run;
      run += c;
    }
    __syncthreads();
    if (valid) {
      const uint32_t lp = s_tstart[d] + s_run[d] + s_pre[warp][d] + rank;
      s_key[lp] = key[r];
      s_val[lp] = val[r];
    }
    __syncthreads();
    s_run[tid] += run;
  }
  __syncthreads();
  for (int k = tid; k < tile_n; k += RS_BLOCK) {
    const uint64_t kk = s_key[k];
    const uint32_t d = (uint32_t)((kk >> shift) & 255u);
    const uint32_t pos = s_goff[d] + ((uint32_t)k - s_tstart[d]);
    kout[pos] = kk;
    vout[pos] = s_val[k];
  }
}

// The whole sort of up to 32,768 items in one launch: a cluster of up to 8
// CTAs, one tile of 256 RR items each, goes through the digits with two
// cluster barriers per digit (histograms out, items moved) instead of two
// launches; the tiles' histograms and the ping-pong buffers are in global
// memory (L2).  A warp takes 32 RR consecutive items: one count of its items
// per digit, then their places round by round; the rounds are a chain, so RR
// is the smallest that eight CTAs hold the items with.
static constexpr int RC_MAX_CLUSTER = 8;

__device__ inline void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int RC_ROUNDS>
__global__ void __launch_bounds__(RS_BLOCK) k_sort_cluster(uint64_t *ka, uint32_t *va, uint64_t *kb, uint32_t *vb, int n,
                                                           int bits, uint32_t *hist) {
  __shared__ uint32_t s_warp[RS_BLOCK / 32];
  __shared__ uint32_t s_cnt[RS_BLOCK / 32][256];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nb = gridDim.x;
  const int base = blockIdx.x * RS_BLOCK * RC_ROUNDS + warp * 32 * RC_ROUNDS;
  for (int shift = 0; shift < bits; shift += 8) {
    uint64_t key[RC_ROUNDS];
    uint32_t val[RC_ROUNDS];
    for (int b = lane; b < 256; b += 32) s_cnt[warp][b] = 0;
    __syncwarp();
#pragma unroll
    for (int r = 0; r < RC_ROUNDS; ++r) {
      const int i = base + r * 32 + lane;
      key[r] = i < n ? __ldcg(ka + i) : 0ull;  // (written by other SMs in the digit before)
      val[r] = i < n ? __ldcg(va + i) : 0u;
    }
    // items past the end take digit 256 + lane (no peers, counted nowhere)
#pragma unroll
    for (int r = 0; r < RC_ROUNDS; ++r) {
      const bool in = base + r * 32 + lane < n;
      const uint32_t d = in ? (uint32_t)(key[r] >> shift) & 255u : 256u + lane;
      const uint32_t peers = __match_any_sync(0xffffffffu, d);
      if (in && lane == __ffs(peers) - 1) s_cnt[warp][d] += (uint32_t)__popc(peers);
      __syncwarp();
    }
    __syncthreads();
    uint32_t mine = 0;
    for (int w = 0; w < RS_BLOCK / 32; ++w) mine += s_cnt[w][tid];
    __stcg(hist + blockIdx.x * 256 + tid, mine);
    cluster_sync();
    uint32_t all = 0, before = 0, total;
    for (int b = 0; b < nb; ++b) {
      const uint32_t v = __ldcg(hist + b * 256 + tid);
      if (b < (int)blockIdx.x) before += v;
      all += v;
    }
    uint32_t run = block_excl_scan(all, s_warp, total) + before;
    for (int w = 0; w < RS_BLOCK / 32; ++w) {
      const uint32_t c = s_cnt[w][tid];
      s_cnt[w][tid] = run;  // where the warp's items of this digit start
      run += c;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RC_ROUNDS; ++r) {
      const bool in = base + r * 32 + lane < n;
      const uint32_t d = in ? (uint32_t)(key[r] >> shift) & 255u : 256u + lane;
      const uint32_t peers = __match_any_sync(0xffffffffu, d);
      const uint32_t at = in ? s_cnt[warp][d] : 0u;
      __syncwarp();
      if (in) {
        const uint32_t pos = at + __popc(peers & ((1u << lane) - 1u));
        __stcg(kb + pos, key[r]);
        __stcg(vb + pos, val[r]);
        if (lane == __ffs(peers) - 1) s_cnt[warp][d] = at + (uint32_t)__popc(peers);
      }
      __syncwarp();
    }
    cluster_sync();
    uint64_t *kt = ka;
    ka = kb;
    kb = kt;
    uint32_t *vt = va;
    va = vb;
    vb = vt;
  }
}

// Sorts (keys, vals) by the low `bits` bits of the key, stably; the result
// ends in (keys, vals) (the buffers are ping-ponged with the alternates).
// A cluster launch can be refused for want of resources: nothing may then go
// on, since the unsorted values would be used as indices.
int radix_sort(Workspace &ws, uint64_t *&keys, uint32_t *&vals, uint64_t *&keys_alt, uint32_t *&vals_alt, int64_t n,
               int bits, cudaStream_t st) {
  if (n <= 1 || bits <= 0) return FMM_OK;
  if (n <= (int64_t)RS_BLOCK * 16 * RC_MAX_CLUSTER) {
    int rounds = 2, nc = 1;
    while ((int64_t)RS_BLOCK * rounds * RC_MAX_CLUSTER < n) rounds *= 2;
    while ((int64_t)RS_BLOCK * rounds * nc < n) nc *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)nc);
    cfg.blockDim = dim3(RS_BLOCK);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)nc;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    uint32_t *chist = ws.radix_hist(nc);
    if (!ws.ok) return FMM_ERR_OUT_OF_MEMORY;
    auto kern = rounds == 2 ? k_sort_cluster<2> : rounds == 4 ? k_sort_cluster<4> : rounds == 8 ? k_sort_cluster<8>
                                                                                              : k_sort_cluster<16>;
    CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, keys, vals, keys_alt, vals_alt, (int)n, bits, chist));
    ws.launches += 1;
    if (((bits + 7) / 8) & 1) {
      std::swap(keys, keys_alt);
      std::swap(vals, vals_alt);
    }
    return FMM_OK;
  }
  int nb = (int)((n + RS_TILE - 1) / RS_TILE);
  uint32_t *hist = ws.radix_hist(nb);
  if (!ws.ok) return FMM_ERR_OUT_OF_MEMORY;
  const bool by_tile = nb <= RS_FUSED_TILES;
  for (int shift = 0; shift < bits; shift += 8) {
    k_radix_hist<<<nb, RS_BLOCK, 0, st>>>(keys, n, shift, hist, nb, by_tile);
    if (!by_tile) exclusive_scan(ws, hist, hist, (int64_t)256 * nb, nullptr, st);
    if (!ws.ok) return FMM_ERR_OUT_OF_MEMORY;
    k_radix_scatter<<<nb, RS_BLOCK, 0, st>>>(keys, vals, keys_alt, vals_alt, n, shift, hist, nb, by_tile);
    ws.launches += 2;
    std::swap(keys, keys_alt);
    std::swap(vals, vals_alt);
  }
  return FMM_OK;
}

// ------------------------------------------------------------ bucket lists
// List y's block sums: items per (bucket, tile); key 255 is in no bucket.
__global__ void __launch_bounds__(RS_BLOCK) k_bucket_hist(const uint8_t *keys, int64_t n, uint32_t *hist, int nb,
                                                          bool by_tile, uint32_t *counts) {
  __shared__ uint32_t h[256];
  const int y = blockIdx.y, tid = threadIdx.x;
  h[tid] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * RS_TILE;
  for (int r = 0; r < RS_ROUNDS; ++r) {
    const int64_t i = base + (int64_t)r * RS_BLOCK + tid;
    const uint32_t d = i < n ? keys[(int64_t)y * n + i] : 255u;
    const uint32_t peers = __match_any_sync(0xffffffffu, d);
    if (d != 255u && (tid & 31) == __ffs(peers) - 1) atomicAdd(&h[d], (uint32_t)__popc(peers));
  }
  __syncthreads();
  if (by_tile) hist[((int64_t)y * nb + blockIdx.x) * 256 + tid] = h[tid];
  else hist[((int64_t)y * 256 + tid) * nb + blockIdx.x] = h[tid];
  if (h[tid]) atomicAdd(&counts[y * 256 + tid], h[tid]);
}

// Stable scatter: the items of each tile in input order to their bucket's
// places, ranked by (round, warp, lane).  offs: the exclusive scan of the
// [list][bucket][tile] sums, or with by_tile the [list][tile][256] sums.
__global__ void __launch_bounds__(RS_BLOCK) k_bucket_scatter(const uint8_t *keys, int64_t n, const uint32_t *offs,
                                                             int nb, bool by_tile, int first, int *out) {
  __shared__ uint32_t s_at[256], s_warp[RS_BLOCK / 32];
  __shared__ uint32_t s_cnt[RS_BLOCK / 32][256];
  const int y = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (by_tile) {
    uint32_t all = 0, before = 0, total;
    for (int b = 0; b < nb; ++b) {
      const uint32_t v = offs[((int64_t)y * nb + b) * 256 + tid];
      if (b == (int)blockIdx.x) before = all;
      all += v;
    }
    s_at[tid] = block_excl_scan(all, s_warp, total) + before;
  } else {
    s_at[tid] = offs[((int64_t)y * 256 + tid) * nb + blockIdx.x] - offs[(int64_t)y * 256 * nb];
  }
  out += (int64_t)y * n;
  // a warp takes 32 RS_ROUNDS consecutive items: one count of its items per
  // bucket, then the places of its rounds one after another
  const int64_t base = (int64_t)blockIdx.x * RS_TILE + (int64_t)warp * 32 * RS_ROUNDS;
  uint32_t dig[RS_ROUNDS];
  uint32_t any = 0;
  for (int b = lane; b < 256; b += 32) s_cnt[warp][b] = 0;
  __syncwarp();
#pragma unroll
  for (int r = 0; r < RS_ROUNDS; ++r) {
    const int64_t i = base + r * 32 + lane;
    dig[r] = i < n ? keys[(int64_t)y * n + i] : 255u;
    any |= dig[r] != 255u;
    const uint32_t peers = __match_any_sync(0xffffffffu, dig[r]);
    if (dig[r] != 255u && lane == __ffs(peers) - 1) s_cnt[warp][dig[r]] += (uint32_t)__popc(peers);
    __syncwarp();
  }
  if (!__syncthreads_or((int)any)) return;
  uint32_t run = s_at[tid];
  for (int w = 0; w < RS_BLOCK / 32; ++w) {
    const uint32_t c = s_cnt[w][tid];
    s_cnt[w][tid] = run;  // where the warp's items of this bucket start
    run += c;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < RS_ROUNDS; ++r) {
    const uint32_t d = dig[r];
    const uint32_t peers = __match_any_sync(0xffffffffu, d);
    const uint32_t at = d != 255u ? s_cnt[warp][d] : 0u;
    __syncwarp();
    if (d != 255u) {
      out[at + __popc(peers & ((1u << lane) - 1u))] = first + (int)(base + r * 32 + lane);
      if (lane == __ffs(peers) - 1) s_cnt[warp][d] = at + (uint32_t)__popc(peers);
    }
    __syncwarp();
  }
}

// Lists of the cells first .. first + n by their 8-bit key, nlist lists from
// nlist x n keys: list y is out[y n ..), bucket after bucket (255 left out),
// ascending inside a bucket; counts[y * 256 + b] (zeroed by the caller) the
// size of its bucket b.  The keys are bytes and most cells are in no bucket,
// so this reads a byte per cell where a sort of (key, cell) pairs moved 32.
void bucket_lists(Workspace &ws, const uint8_t *keys, int nlist, int64_t n, int first, int *out, uint32_t *counts,
                  cudaStream_t st) {
  const int nb = (int)std::max<int64_t>(1, (n + RS_TILE - 1) / RS_TILE);
  const bool by_tile = nb <= RS_FUSED_TILES;
  uint32_t *hist = ws.radix_hist(nlist * nb);
  if (!ws.ok) return;
  const dim3 grid(nb, nlist);
  k_bucket_hist<<<grid, RS_BLOCK, 0, st>>>(keys, n, hist, nb, by_tile, counts);
  if (!by_tile) exclusive_scan(ws, hist, hist, (int64_t)256 * nb * nlist, nullptr, st);
  if (!ws.ok) return;
  k_bucket_scatter<<<grid, RS_BLOCK, 0, st>>>(keys, n, hist, nb, by_tile, first, out);
  ws.launches += 2;
}

// ------------------------------------------------------------- split items
// Parts of at most `chunk` particles of cell first + i, 0 past the end and for
// a cell without bit 0 of its flag (flag null: every cell).
__device__ inline uint32_t cell_parts(const uint8_t *flag, int cell0, int first, int64_t i, int64_t count,
                                      const int *pbeg, const int *pend, int chunk) {
  const int64_t g = first + i;
  if (i >= count || (flag && !(flag[g - cell0] & 1))) return 0;
  return (uint32_t)((pend[g] - pbeg[g] + (int64_t)chunk - 1) / chunk);
}

__global__ void k_split_reduce(const uint8_t *flag, int cell0, int first, int64_t count, const int *pbeg,
                               const int *pend, int chunk, uint32_t *sums) {
  __shared__ uint32_t s_warp[SCAN_BLOCK / 32];
  uint32_t s = 0, total;
  for (int q = 0; q < SCAN_ITEMS; ++q)
    s += cell_parts(flag, cell0, first, (int64_t)blockIdx.x * SCAN_TILE + q * SCAN_BLOCK + threadIdx.x, count, pbeg,
                    pend, chunk);
  block_excl_scan(s, s_warp, total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// A thread takes SCAN_ITEMS consecutive cells; cells of more than two parts
// are written by the whole warp.
__global__ void k_split_fill(const uint8_t *flag, int cell0, int first, int64_t count, const int *pbeg,
                             const int *pend, int chunk, const uint32_t *sums, int2 *items, uint32_t *nitems) {
  __shared__ uint32_t s_warp[SCAN_BLOCK / 32];
  const int lane = threadIdx.x & 31;
  uint32_t t = 0, before, total, v[SCAN_ITEMS], s = 0;
  for (int k = threadIdx.x; k < (int)blockIdx.x; k += SCAN_BLOCK) t += sums[k];
  block_excl_scan(t, s_warp, before);
  const int64_t i0 = (int64_t)blockIdx.x * SCAN_TILE + (int64_t)threadIdx.x * SCAN_ITEMS;
#pragma unroll
  for (int q = 0; q < SCAN_ITEMS; ++q) s += v[q] = cell_parts(flag, cell0, first, i0 + q, count, pbeg, pend, chunk);
  uint32_t at = block_excl_scan(s, s_warp, total) + before;
#pragma unroll
  for (int q = 0; q < SCAN_ITEMS; ++q) {
    const int g = (int)(first + i0 + q);
    if (v[q] >= 1 && v[q] <= 2) items[at] = make_int2(g, 0);
    if (v[q] == 2) items[at + 1] = make_int2(g, 1);
    for (unsigned m = __ballot_sync(0xffffffffu, v[q] > 2); m; m &= m - 1) {
      const int b = __ffs(m) - 1, gb = __shfl_sync(0xffffffffu, g, b);
      const uint32_t cb = __shfl_sync(0xffffffffu, v[q], b), ab = __shfl_sync(0xffffffffu, at, b);
      for (uint32_t k = lane; k < cb; k += 32) items[ab + k] = make_int2(gb, (int)k);
    }
    at += v[q];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *nitems = before + total;
}

// The list of (cell, part) of the cells [first, first + count), parts of at
// most `chunk` particles, in the order of the cells; *nitems its length.  The
// counts are formed again for the second launch instead of stored, and up to
// 2048 cells take one launch: small systems are bound by launches.
void split_items(Workspace &ws, const uint8_t *flag, int cell0, int first, int64_t count, int chunk, int2 *items,
                 uint32_t *nitems, cudaStream_t st) {
  const int nb = (int)std::max<int64_t>(1, (count + SCAN_TILE - 1) / SCAN_TILE);
  uint32_t *sums = ws.scan_tmp(nb);
  if (!ws.ok) return;
  if (nb > 1)
    k_split_reduce<<<nb, SCAN_BLOCK, 0, st>>>(flag, cell0, first, count, ws.cell_pbeg, ws.cell_pend, chunk, sums);
  k_split_fill<<<nb, SCAN_BLOCK, 0, st>>>(flag, cell0, first, count, ws.cell_pbeg, ws.cell_pend, chunk, sums, items,
                                          nitems);
  ws.launches += nb > 1 ? 2 : 1;
}

// ------------------------------------------------------------ tree kernels
// AABB (tree.cpp:20-30) plus a finiteness check of positions and masses.
// Every block writes its box to part[block][6]; the last one to finish (a
// ticket per block; *ticket returns to zero) reduces them into geom = {min,
// max}.  (Atomic minima and maxima of every warp on the same six words took
// 50 us on 2^20 particles, most of a 25 MB read's 5 us.)
__global__ void __launch_bounds__(256) k_aabb(const double *pos, const double *mass, int64_t n, int dim,
                                              unsigned long long *part, unsigned int *ticket, double *geom,
                                              unsigned int *err) {
  __shared__ unsigned long long s_box[8][6];
  __shared__ bool s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long v[6] = {~0ull, ~0ull, ~0ull, 0ull, 0ull, 0ull};
  bool bad = false;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if (d >= dim) break;
      const double x = pos[i * dim + d];
      bad |= !isfinite(x);
      const unsigned long long u = dbl_to_ordered(x);
      v[d] = u < v[d] ? u : v[d];
      v[3 + d] = u > v[3 + d] ? u : v[3 + d];
    }
    bad |= !isfinite(mass[i]);
  }
  if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(err, FMM_DEV_ERR_NONFINITE_INPUT);
  // the block's box: thread d < 6 ends with component d
  auto reduce = [&]() {
#pragma unroll
    for (int d = 0; d < 6; ++d) {
#pragma unroll
      for (int o = 16; o; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(0xffffffffu, v[d], o);
        v[d] = d < 3 ? (t < v[d] ? t : v[d]) : (t > v[d] ? t : v[d]);
      }
      if (lane == 0) s_box[warp][d] = v[d];
    }
    __syncthreads();
    unsigned long long r = 0;
    if (threadIdx.x < 6) {
      const int d = threadIdx.x;
      r = s_box[0][d];
      for (int w = 1; w < 8; ++w) r = d < 3 ? min(r, s_box[w][d]) : max(r, s_box[w][d]);
    }
    return r;
  };
  unsigned long long r = reduce();
  if (threadIdx.x < 6) part[(size_t)blockIdx.x * 6 + threadIdx.x] = r;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
#pragma unroll
  for (int d = 0; d < 6; ++d) v[d] = d < 3 ? ~0ull : 0ull;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x)
#pragma unroll
    for (int d = 0; d < 6; ++d) {
      const unsigned long long t = __ldcg(part + (size_t)b * 6 + d);
      v[d] = d < 3 ? min(v[d], t) : max(v[d], t);
    }
  r = reduce();
  if (threadIdx.x < 6) geom[threadIdx.x] = threadIdx.x % 3 < dim ? ordered_to_dbl(r) : 0.0;
  if (threadIdx.x == 0) *ticket = 0;
}

// Key of each particle at the maximum depth Dmax; values = input index.
__global__ void k_keys(const double *pos, int64_t n, int dim, int Dmax, const double *geom, uint64_t *keys,
                       uint32_t *vals) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t c[3] = {0, 0, 0};
  const uint64_t cmax = (Dmax >= 32) ? 0xffffffffull : ((1ull << Dmax) - 1);
  const double scale = ldexp(1.0, Dmax);
  for (int d = 0; d < dim; ++d) {
    double a = geom[d], b = geom[3 + d];
    if (b == a) continue;  // zero extent: the reference's 0/0 -> coordinate 0
    double q = (pos[i * dim + d] - a) / (b - a);
    uint64_t v = (uint64_t)(q * scale);
    c[d] = (uint32_t)(v > cmax ? cmax : v);
  }
  keys[i] = morton_encode(dim, c[0], c[1], c[2]);
  vals[i] = (uint32_t)i;
}

// Leaf key at depth D of each particle, in input order.
__global__ void k_leafkeys_input(const double *pos, int64_t n, int dim, int Dmax, int D, const double *geom,
                                 uint64_t *lk, uint32_t *vals) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t c[3] = {0, 0, 0};
  const uint64_t cmax = (Dmax >= 32) ? 0xffffffffull : ((1ull << Dmax) - 1);
  const double scale = ldexp(1.0, Dmax);
  for (int d = 0; d < dim; ++d) {
    double a = geom[d], b = geom[3 + d];
    if (b == a) continue;
    double q = (pos[i * dim + d] - a) / (b - a);
    uint64_t v = (uint64_t)(q * scale);
    c[d] = (uint32_t)(v > cmax ? cmax : v) >> (Dmax - D);
  }
  lk[i] = morton_encode(dim, c[0], c[1], c[2]);
  vals[i] = (uint32_t)i;
}

// Levels 0 .. cp on which sorted keys a <= b share their cell (cp = Dmax: the
// same key): level d compares the keys shifted right by dim (Dmax - d).
__device__ inline int common_level(uint64_t a, uint64_t b, int dim, int Dmax) {
  const uint64_t x = a ^ b;
  return x ? Dmax - 1 - (63 - __clzll((long long)x)) / dim : Dmax;
}

static constexpr int LV_BLOCK = 256, LV_ROUNDS = 4, LV_TILE = LV_BLOCK * LV_ROUNDS, LV_MAX = FMM_MAX_DEPTH + 1;

// One pass over the sorted Dmax keys for all depths at once.  Particle i
// starts a cell on every level d > cp(i - 1, i) (all levels for i = 0).
//   blockcnt[d * nb + tile]: cells of level d that start in the tile;
//   lev[d]: their sum, lev[LV_MAX + d]: the largest cell of level d (zeroed
//   by the caller).
// The cell that particle i starts on level d ends where the key differs on
// level d; from the deepest level up its end only moves on, so one walk
// (doubling steps, then halving) gives the sizes on all levels.  Levels on
// which the next particle starts a cell too have size 1.  Where a level takes
// more than 32 particles further, the warp searches for that lane's ends
// together, 32 places at a time: the first particles of coarse cells walked
// alone for most of the kernel (77 us on 2^20 keys).
__global__ void __launch_bounds__(LV_BLOCK) k_levels(const uint64_t *keys, int64_t n, int dim, int Dmax, int nb,
                                                     uint32_t *blockcnt, uint32_t *lev) {
  __shared__ uint32_t s_cnt[LV_MAX + 1], s_max[LV_MAX];
  for (int d = threadIdx.x; d <= LV_MAX; d += LV_BLOCK) {
    s_cnt[d] = 0;
    if (d < LV_MAX) s_max[d] = 1;
  }
  __syncthreads();
  for (int r = 0; r < LV_ROUNDS; ++r) {
    const int64_t i = (int64_t)blockIdx.x * LV_TILE + r * LV_BLOCK + threadIdx.x;
    const uint64_t k = i < n ? keys[i] : 0;
    // the particle starts a cell on the levels first .. Dmax (first = Dmax + 1: on none)
    const int first = i >= n ? Dmax + 1 : i == 0 ? 0 : common_level(keys[i - 1], k, dim, Dmax) + 1;
    const unsigned peers = __match_any_sync(0xffffffffu, first);
    if ((threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&s_cnt[first], (uint32_t)__popc(peers));
    int64_t j = i + 1;  // the keys in [i, j) share level d
    int d = j < n ? common_level(k, keys[j], dim, Dmax) : -1;
    for (; d >= first; --d) {
      const int sh = dim * (Dmax - d);
      auto same = [&](int64_t q) { return q < n && (sh >= 64 || (keys[q] >> sh) == (k >> sh)); };
      int64_t step = 1;
      while (step <= 32 && same(j + step - 1)) {
        j += step;
        step *= 2;
      }
      if (step > 32) break;  // a long run
      for (step /= 2; step > 0; step /= 2)
        if (same(j + step - 1)) j += step;
      const uint32_t len = (uint32_t)(j - i);
      if (len > s_max[d]) atomicMax(&s_max[d], len);
    }
    // the long runs, lane by lane
    const int lane = threadIdx.x & 31;
    for (unsigned todo = __ballot_sync(0xffffffffu, d >= first); todo; todo &= todo - 1) {
      const int b = __ffs(todo) - 1;
      const uint64_t kk = __shfl_sync(0xffffffffu, k, b);
      const int64_t ii = i - lane + b;
      int64_t e = __shfl_sync(0xffffffffu, j, b);  // the keys in [ii, e) share level dd
      const int low = __shfl_sync(0xffffffffu, first, b);
      for (int dd = __shfl_sync(0xffffffffu, d, b); dd >= low; --dd) {
        const int sh = dim * (Dmax - dd);
        // the keys are sorted: of 32 places a stride apart the first c are in the run
        auto places = [&](int64_t stride, int64_t end) {
          const int64_t q = e + (lane + 1) * stride - 1;
          return __popc(__ballot_sync(0xffffffffu, q < end && (sh >= 64 || (keys[q] >> sh) == (kk >> sh))));
        };
        int64_t stride = 32;
        int c;
        while (e += (c = places(stride, n)) * stride, c == 32) stride *= 32;
        int64_t width = min(stride - 1, n - e);  // the end is in [e, e + width]
        while (width > 0) {
          stride = (width + 31) / 32;
          c = places(stride, e + width);
          e += c * stride;
          width = min(stride - 1, width - c * stride);
        }
        if (lane == 0) atomicMax(&s_max[dd], (uint32_t)(e - ii));
      }
    }
  }
  __syncthreads();
  if (threadIdx.x <= Dmax) {
    const int d = threadIdx.x;
    uint32_t c = 0;
    for (int f = 0; f <= d; ++f) c += s_cnt[f];
    blockcnt[(size_t)d * nb + blockIdx.x] = c;
    if (c) atomicAdd(&lev[d], c);
    // (a word read a moment early only costs an atomic that changes nothing)
    if (s_max[d] > *(volatile uint32_t *)&lev[LV_MAX + d]) atomicMax(&lev[LV_MAX + d], s_max[d]);
  }
}

// Exclusive scan of each level's tile counts, in place: one block per level.
__global__ void __launch_bounds__(SCAN_BLOCK) k_level_scan(uint32_t *blockcnt, int nb) {
  __shared__ uint32_t s_warp[SCAN_BLOCK / 32];
  uint32_t *row = blockcnt + (size_t)blockIdx.x * nb;
  uint32_t carry = 0;
  for (int b0 = 0; b0 < nb; b0 += SCAN_TILE) {
    uint32_t v[SCAN_ITEMS], s = 0, tot;
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; ++i) {
      const int k = b0 + (int)threadIdx.x * SCAN_ITEMS + i;
      v[i] = k < nb ? row[k] : 0;
      s += v[i];
    }
    uint32_t e = carry + block_excl_scan(s, s_warp, tot);
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; ++i) {
      const int k = b0 + (int)threadIdx.x * SCAN_ITEMS + i;
      if (k < nb) row[k] = e;
      e += v[i];
    }
    carry += tot;
  }
}

// The cells of all levels 0 .. D from the sorted Dmax keys and the scanned
// tile counts: cell r of a level is the r-th particle that starts one there
// (a ballot per level and 32 particles).  Writes keys, particle ranges,
// parents and children (filled with -1 before) and every particle's leaf.
__global__ void __launch_bounds__(LV_BLOCK) k_make_cells(const uint64_t *keys, int64_t n, int dim, int Dmax, int D,
                                                         int nb, const uint32_t *blockoff, LevelOffsets lo,
                                                         uint64_t *ckey, int *cpbeg, int *cpend, int *cparent,
                                                         int *cchild, int *ccoll, int *leaf_of) {
  __shared__ uint32_t s_wc[LV_MAX][LV_BLOCK / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // a warp takes 32 LV_ROUNDS consecutive particles
  const int64_t base = (int64_t)blockIdx.x * LV_TILE + warp * 32 * LV_ROUNDS;
  uint64_t key[LV_ROUNDS];
  int first[LV_ROUNDS];
#pragma unroll
  for (int r = 0; r < LV_ROUNDS; ++r) {
    const int64_t i = base + r * 32 + lane;
    key[r] = i < n ? keys[i] : 0;
    first[r] = i >= n ? LV_MAX + 1 : i == 0 ? 0 : common_level(keys[i - 1], key[r], dim, Dmax) + 1;
  }
  for (int d = 0; d <= D; ++d) {
    int c = 0;
#pragma unroll
    for (int r = 0; r < LV_ROUNDS; ++r) c += __popc(__ballot_sync(0xffffffffu, first[r] <= d));
    if (lane == 0) s_wc[d][warp] = (uint32_t)c;
  }
  __syncthreads();
  const int ns = dim == 3 ? 27 : 9;
  if (blockIdx.x == 0 && (int)threadIdx.x < ns)  // the root's only colleague is itself
    ccoll[(int64_t)lo.off[0] * ns + threadIdx.x] = (int)threadIdx.x == ns / 2 ? lo.off[0] : -1;
  int up[LV_ROUNDS];  // the particle's cell one level up
#pragma unroll
  for (int r = 0; r < LV_ROUNDS; ++r) up[r] = -1;
  for (int d = 0; d <= D; ++d) {
    int c = lo.off[d] + (int)blockoff[(size_t)d * nb + blockIdx.x] - 1;
    for (int w = 0; w < warp; ++w) c += (int)s_wc[d][w];
    const int sh = dim * (Dmax - d);
#pragma unroll
    for (int r = 0; r < LV_ROUNDS; ++r) {
      const int64_t i = base + r * 32 + lane;
      const bool head = first[r] <= d;
      const unsigned m = __ballot_sync(0xffffffffu, head);
      const int cell = c + __popc(m & (0xffffffffu >> (31 - lane)));
      c += __popc(m);
      if (head) {
        const uint64_t k = sh >= 64 ? 0ull : key[r] >> sh;
        ckey[cell] = k;
        cpbeg[cell] = (int)i;
        if (cell > lo.off[d]) cpend[cell - 1] = (int)i;
        cparent[cell] = up[r];
        if (d > 0) cchild[((int64_t)up[r] << dim) + (int)(k & ((1u << dim) - 1u))] = cell;
      }
      if (i == n - 1) cpend[lo.off[d + 1] - 1] = (int)n;
      if (d == D && i < n) leaf_of[i] = cell;
      up[r] = cell;
    }
  }
}

// The final particle order from the Dmax order: inside a leaf the input
// order, i.e. the particles sorted by their input index (vals), so each
// particle's place is its rank among its leaf's indices.  The result equals
// the stable sort of the depth-D keys from input order.
__global__ void k_leaf_order(const uint32_t *vals, const int *leaf_of, const int *cpbeg, const int *cpend, int64_t n,
                             uint32_t *pv) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int L = leaf_of[i], s = cpbeg[L], e = cpend[L];
  const uint32_t v = vals[i];
  int r = 0;
  for (int j = s; j < e; ++j) r += vals[j] < v ? 1 : 0;
  pv[s + r] = v;
}

// Adaptive targets, per cell g (flag[g - cell0]): bit 0, a target: the root,
// or a cell whose parent holds more than A particles (every ancestor then
// does too, since a cell's particles are a subset of its parent's); bit 1,
// an adaptive leaf: a target with at most A particles, or a leaf.  The
// adaptive leaves are appended to alist, their count kept in *acount.
__global__ void k_adaptive_flags(const int *pbeg, const int *pend, const int *parent, int cell0, int ncell,
                                 int first1, int leaf_first, int A, uint8_t *flag, int *alist, unsigned *acount) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
  const int g = cell0 + i;
  bool is_leaf = false;
  if (i < ncell) {
    const bool tgt = g < first1 || pend[parent[g]] - pbeg[parent[g]] > A;
    is_leaf = tgt && (pend[g] - pbeg[g] <= A || g >= leaf_first);
    flag[i] = (uint8_t)((tgt ? 1 : 0) | (is_leaf ? 2 : 0));
  }
  const unsigned m = __ballot_sync(0xffffffffu, is_leaf);
  unsigned base = 0;
  if (lane == 0 && m) base = atomicAdd(acount, (unsigned)__popc(m));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (is_leaf) alist[base + __popc(m & ((1u << lane) - 1u))] = g;
}

// Colleagues (|delta| <= 1 on every axis, same level, self included) of the
// cells of one level.  With c = 2P + b per axis (b the cell's child bit),
// the neighbour at offset delta is child ((b + delta) mod 2) of the parent's
// colleague at offset floor((b + delta) / 2), so each of the 3^dim slots is
// two dependent loads and no key decoding.
//
// With adaptive targets (aflag set) only target cells get a row: nothing
// reads the row of a cell that is no target (their parents' rows serve the
// targets, and a target's parent is a target).
template <int DIM>
__global__ void __launch_bounds__(256) k_colleagues(const uint64_t *ckey, const int *cparent, const int *cchild,
                                                    int *ccoll, int base, int count) {
  // one thread per (cell, slot): consecutive threads write consecutive slots.  (Blocks of 8 cells' slots, 72
  // threads in 2D, spent their time on the launch of blocks: 728 us for the 7.3 M cells of a 4M disk.)
  constexpr int NC = 1 << DIM, NS = DIM == 3 ? 27 : 9;
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int ci = (int)(idx / NS), s = (int)(idx % NS);
  if (ci >= count) return;
  const int c = base + ci;
  const int b = (int)(ckey[c] & (uint64_t)(NC - 1));
  int pslot = 0, child = 0, mul = 1;
#pragma unroll
  for (int a = 0; a < DIM; ++a) {
    const int delta = (s / mul) % 3 - 1;
    const int v = ((b >> a) & 1) + delta;  // in [-1, 2]
    const int f = (v + 2) / 2 - 1;        // floor(v / 2)
    pslot += (f + 1) * mul;
    child |= (v - 2 * f) << a;
    mul *= 3;
  }
  const int Q = ccoll[(int64_t)cparent[c] * NS + pslot];
  ccoll[(int64_t)c * NS + s] = Q >= 0 ? cchild[(int64_t)Q * NC + child] : -1;
}

// The same rows with adaptive targets, one thread per cell: most cells of the
// deep levels are no target and leave after one flag load, instead of 3^dim
// threads each; a target's thread writes its 3^dim slots.
template <int DIM>
__global__ void k_colleagues_targets(const uint64_t *ckey, const int *cparent, const int *cchild, int *ccoll,
                                     int base, int count, const uint8_t *aflag, int cell0) {
  constexpr int NC = 1 << DIM, NS = DIM == 3 ? 27 : 9;
  const int ci = blockIdx.x * blockDim.x + threadIdx.x;
  if (ci >= count) return;
  const int c = base + ci;
  if (!(aflag[c - cell0] & 1)) return;
  const int b = (int)(ckey[c] & (uint64_t)(NC - 1));
  const int *prow = ccoll + (int64_t)cparent[c] * NS;
  int *row = ccoll + (int64_t)c * NS;
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    int pslot = 0, child = 0, mul = 1;
#pragma unroll
    for (int a = 0; a < DIM; ++a) {
      const int delta = (s / mul) % 3 - 1;
      const int v = ((b >> a) & 1) + delta;  // in [-1, 2]
      const int f = (v + 2) / 2 - 1;        // floor(v / 2)
      pslot += (f + 1) * mul;
      child |= (v - 2 * f) << a;
      mul *= 3;
    }
    const int Q = prow[pslot];
    row[s] = Q >= 0 ? cchild[(int64_t)Q * NC + child] : -1;
  }
}

// Gathers particles into leaf order: the offset from the leaf's geometric
// centre split into FP32 hi + lo parts (x - c = hi + lo to ~48 bits), and the
// FP32 mass, used by P2M, L2P (hi only) and P2P (hi and lo).
__global__ void k_gather_particles(const double *pos, const double *mass, const uint32_t *perm, const int *leaf_of,
                                   const uint64_t *ckey, int64_t n, int dim, int depth, const double *geom,
                                   float4 *part, float4 *part_lo) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t j = perm[i];
  uint32_t q[3];
  morton_decode(dim, ckey[leaf_of[i]], q[0], q[1], q[2]);
  float r[3] = {0.f, 0.f, 0.f}, rl[3] = {0.f, 0.f, 0.f};
  const double inv = ldexp(1.0, -depth);
  for (int d = 0; d < dim; ++d) {
    double ext = geom[3 + d] - geom[d];
    double c = geom[d] + ((double)q[d] + 0.5) * (ext * inv);
    double v = pos[(int64_t)j * dim + d] - c;
    r[d] = (float)v;
    rl[d] = (float)(v - (double)r[d]);
  }
  part[i] = make_float4(r[0], r[1], r[2], (float)mass[j]);
  part_lo[i] = make_float4(rl[0], rl[1], rl[2], 0.f);
}

// ------------------------------------------------------------ host driver
static int bit_width_u64(uint64_t v) {
  int w = 0;
  while (v) {
    ++w;
    v >>= 1;
  }
  return w;
}

int launch_adaptive_flags(const Workspace &ws, const TreeState &t, int A, uint8_t *flag, int *list, cudaStream_t st) {
  if (t.depth < 1 || t.n_cells <= 0) return FMM_ERR_INVALID_ARGUMENT;
  CUDA_TRY(cudaMemsetAsync(list + t.n_cells, 0, sizeof(int), st));
  k_adaptive_flags<<<cdiv(t.n_cells, 256), 256, 0, st>>>(ws.cell_pbeg, ws.cell_pend, ws.cell_parent, t.cell0,
                                                          t.n_cells, t.level_off[1], t.level_off[t.depth], A, flag,
                                                          list, (unsigned *)(list + t.n_cells));
  CUDA_TRY(cudaGetLastError());
  return FMM_OK;
}

int build_tree(Workspace &ws, TreeState &t, const double *d_pos, const double *d_mass, int64_t n, int dim,
               int threshold, cudaStream_t st, int adaptive_leaf) {
  t.dim = dim;
  t.n = n;
  t.adaptive_leaf = 0;
  const int Dmax = ((64 / dim) >> dim) << dim;  // tree.cpp:38
  const int TPB = 256;
  const int nbN = cdiv(n, TPB);
  const int nblv = cdiv(n, LV_TILE);
  if (!ws.reserve_particles(n) || !ws.blev.reserve((size_t)nblv * (Dmax + 1))) return FMM_ERR_OUT_OF_MEMORY;
  uint32_t *lev = ws.lev;  // cells, then the largest cell, of every level
  const size_t cleared = ws.keep_err ? offsetof(TreeBack, err) : offsetof(TreeBack, ticket);  // with the error word
  CUDA_TRY(cudaMemsetAsync(lev, 0, cleared - offsetof(TreeBack, lev), st));
  k_aabb<<<std::min(nbN, WS_AABB_BLOCKS), TPB, 0, st>>>(d_pos, d_mass, n, dim, ws.box_u64, ws.ticket, ws.geom,
                                                       ws.dev_err);
  k_keys<<<nbN, TPB, 0, st>>>(d_pos, n, dim, Dmax, ws.geom, ws.keyA, ws.valA);
  ws.launches += 2;
  // sort all particles by their Dmax key
  uint64_t *kA = ws.keyA, *kB = ws.keyB;
  uint32_t *vA = ws.valA, *vB = ws.valB;
  int rc = radix_sort(ws, kA, vA, kB, vB, n, dim * Dmax, st);
  if (rc) return rc;
  k_levels<<<nblv, LV_BLOCK, 0, st>>>(kA, n, dim, Dmax, nblv, ws.blev.ptr, lev);
  ws.launches += 1;
  // the box, the finiteness check (keys of non-finite positions are clamped
  // into range, so what ran above is harmless) and the levels' sizes
  CUDA_TRY(cudaMemcpyAsync(&ws.host->tree, ws.bback.ptr, sizeof(TreeBack), cudaMemcpyDeviceToHost, st));
  CUDA_TRY(cudaStreamSynchronize(st));
  const uint32_t *hlev = ws.host->tree.lev;
  const unsigned int herr = ws.host->tree.err;
  if (ws.keep_err && (herr & FMM_DEV_ERR_NONFINITE_OUTPUT)) return FMM_ERR_NONFINITE_OUTPUT;  // of the pass before
  if (ws.keep_err && (herr & FMM_DEV_ERR_TIMEOUT)) return FMM_ERR_TIMEOUT;
  if (herr & FMM_DEV_ERR_NONFINITE_INPUT) return FMM_ERR_NONFINITE_INPUT;
  for (int d = 0; d < 3; ++d) {
    t.lo[d] = ws.host->tree.geom[d];
    t.hi[d] = ws.host->tree.geom[3 + d];
  }

  // depth loop, tree.cpp:43-69
  unsigned int max_n = (unsigned int)n;
  unsigned int depth = 0;
  do {
    uint64_t n_leafs = (uint64_t)(max_n - 1) / (unsigned)threshold + 1;
    depth += bit_width_u64(n_leafs) / dim + 1;
    if (depth > (unsigned)Dmax) depth = Dmax;
    max_n = hlev[LV_MAX + depth];
  } while (depth < (unsigned)Dmax && max_n > (unsigned)threshold);
  t.depth = (int)depth;
  const int D = t.depth;

  // the cells of all levels, contiguous from the root
  const int nc = 1 << dim, ns = dim == 3 ? 27 : 9;
  LevelOffsets lo;
  t.level_count.assign(D + 1, 0);
  t.level_off.assign(D + 2, 0);
  t.level_max.assign(D + 1, 0);
  int64_t cells = 0;
  for (int d = 0; d <= D; ++d) {
    lo.off[d] = t.level_off[d] = (int)cells;
    t.level_count[d] = (int)hlev[d];
    t.level_max[d] = (int)hlev[LV_MAX + d];
    cells += hlev[d];
    if (cells > (int64_t)INT32_MAX) return FMM_ERR_OUT_OF_MEMORY;
  }
  lo.off[D + 1] = t.level_off[D + 1] = (int)cells;
  t.cell0 = 0;
  t.n_cells = (int)cells;
  if (!ws.reserve_cells(cells, nc, ns)) return FMM_ERR_OUT_OF_MEMORY;
  CUDA_TRY(cudaMemsetAsync(ws.cell_child, 0xff, sizeof(int) * (size_t)cells * nc, st));
  k_level_scan<<<D + 1, SCAN_BLOCK, 0, st>>>(ws.blev.ptr, nblv);
  k_make_cells<<<nblv, LV_BLOCK, 0, st>>>(kA, n, dim, Dmax, D, nblv, ws.blev.ptr, lo, ws.cell_key, ws.cell_pbeg,
                                          ws.cell_pend, ws.cell_parent, ws.cell_child, ws.cell_coll, ws.leaf_of);
  ws.launches += 2;
  // final order: each leaf's particles in input order (tree.cpp:62-66).  The
  // Dmax order already groups the leaves; with leaves of at most
  // LEAF_ORDER_MAX particles only the order inside each leaf is redone, else
  // the leaf keys are sorted afresh from input order.
  uint32_t *pv = ws.valC;
  if (max_n <= (unsigned)LEAF_ORDER_MAX) {
    k_leaf_order<<<nbN, TPB, 0, st>>>(vA, ws.leaf_of, ws.cell_pbeg, ws.cell_pend, n, pv);
    ws.launches += 1;
  } else {
    uint64_t *lk = ws.keyC, *lkAlt = ws.keyA;
    uint32_t *pvAlt = ws.valA;
    k_leafkeys_input<<<nbN, TPB, 0, st>>>(d_pos, n, dim, Dmax, D, ws.geom, ws.keyC, ws.valC);
    ws.launches += 1;
    rc = radix_sort(ws, lk, pv, lkAlt, pvAlt, n, dim * D, st);
    if (rc) return rc;
  }
  t.d_perm = pv;
  // adaptive targets (3D trees of depth >= 3, as the force pass runs them):
  // the flags now, so that only target cells get colleague rows
  const uint8_t *aflag = nullptr;
  if (adaptive_leaf > 0 && dim == 3 && D >= 3) {
    if (!ws.reserve_adaptive(t.n_cells)) return FMM_ERR_OUT_OF_MEMORY;
    rc = launch_adaptive_flags(ws, t, adaptive_leaf, ws.aflag, ws.alist, st);
    if (rc) return rc;
    ws.launches += 1;
    t.adaptive_leaf = adaptive_leaf;
    aflag = ws.aflag;
  }
  // colleagues, top-down
  for (int d = 1; d <= D; ++d) {
    if (aflag)  // adaptive targets are 3D only
      k_colleagues_targets<3><<<cdiv(t.level_count[d], TPB), TPB, 0, st>>>(
          ws.cell_key, ws.cell_parent, ws.cell_child, ws.cell_coll, t.level_off[d], t.level_count[d], aflag, t.cell0);
    else
      (dim == 3 ? k_colleagues<3> : k_colleagues<2>)<<<cdiv((int64_t)t.level_count[d] * ns, 256), 256, 0, st>>>(
          ws.cell_key, ws.cell_parent, ws.cell_child, ws.cell_coll, t.level_off[d], t.level_count[d]);
    ws.launches += 1;
  }
  // particles in leaf order
  k_gather_particles<<<nbN, TPB, 0, st>>>(d_pos, d_mass, pv, ws.leaf_of, ws.cell_key, n, dim, D, ws.geom, ws.part,
                                             ws.part_lo);
  ws.launches += 1;
  CUDA_TRY(cudaGetLastError());
  return FMM_OK;
}

}  // namespace fmm
