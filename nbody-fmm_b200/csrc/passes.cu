// The FMM passes after the tree build: P2M, M2M, M2L, L2L, L2P and P2P
// (Tree::compute_accelerations, tree.cpp:93-111; Leaf::compute_acceleration,
// leaf.cpp:55-148).
//
// Translations are dense contractions.  Cells of one level with the same
// child index ("class": the parities of their coordinates) have the same
// set of interaction-list offsets (node_i.cpp:39-43: delta in
// [-2-c%2, 3-c%2] minus the neighbours), so a batch of 64 such target cells
// accumulates, slot by slot, Y[64 x K] += X_slot[64 x K] * T_slot[K x K] where
// X_slot gathers the source expansion of each target at that offset (zero if
// the cell does not exist).  M2M (8 child slots) and L2L (1 parent slot) use
// the same kernel.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

#include "expansions.cuh"
#include "m2l_tc.cuh"

namespace fmm {

// [dim == 3][class] -> list of (table offset index | colleague slot << 9 | child << 14)
__constant__ int c_m2l_slots[2][8][189];
__constant__ float c_rec1[FMM_MAX_P + 1][FMM_MAX_P + 1];  // (2l-1)/(l^2-m^2)
__constant__ float c_rec2[FMM_MAX_P + 1][FMM_MAX_P + 1];  // 1/(l^2-m^2)

void upload_class_tables() {
  // __constant__ memory is per device: upload once for every device used
  static std::mutex mu;
  static bool done[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return;
  std::lock_guard<std::mutex> lk(mu);
  if (done[dev]) return;
  done[dev] = true;
  static int h[2][8][189] = {};
  for (int dim = 2; dim <= 3; ++dim)
  for (int c = 0; c < (1 << dim); ++c) {
    int cb[3] = {c & 1, (c >> 1) & 1, (c >> 2) & 1};
    int k = 0;
    int lo[3], hi[3];
    for (int a = 0; a < 3; ++a) {
      lo[a] = a < dim ? -2 - cb[a] : 0;
      hi[a] = a < dim ? 3 - cb[a] : 0;
    }
    for (int dz = lo[2]; dz <= hi[2]; ++dz)
      for (int dy = lo[1]; dy <= hi[1]; ++dy)
        for (int dx = lo[0]; dx <= hi[0]; ++dx) {
          if (dx >= -1 && dx <= 1 && dy >= -1 && dy <= 1 && dz >= -1 && dz <= 1) continue;
          int dd[3] = {dx, dy, dz}, del[3], ch[3];
          for (int a = 0; a < 3; ++a) {
            int v = dd[a] + cb[a];         // in [-2, 3]
            del[a] = (v + 2) / 2 - 1;      // floor(v / 2)
            ch[a] = v - 2 * del[a];
          }
          int ti = dim == 3 ? (dx + 3) + 7 * (dy + 3) + 49 * (dz + 3) : (dx + 3) + 7 * (dy + 3);
          int cs = dim == 3 ? (del[0] + 1) + 3 * (del[1] + 1) + 9 * (del[2] + 1) : (del[0] + 1) + 3 * (del[1] + 1);
          int chi = ch[0] + 2 * ch[1] + (dim == 3 ? 4 * ch[2] : 0);
          h[dim - 2][c][k++] = ti | (cs << 9) | (chi << 14);
        }
  }
  cudaMemcpyToSymbol(c_m2l_slots, h, sizeof(h));
  float r1[FMM_MAX_P + 1][FMM_MAX_P + 1] = {}, r2[FMM_MAX_P + 1][FMM_MAX_P + 1] = {};
  for (int l = 0; l <= FMM_MAX_P; ++l)
    for (int m = 0; m < l; ++m) {
      r1[l][m] = (float)((2.0 * l - 1.0) / (double)(l * l - m * m));
      r2[l][m] = (float)(1.0 / (double)(l * l - m * m));
    }
  cudaMemcpyToSymbol(c_rec1, r1, sizeof(r1));
  cudaMemcpyToSymbol(c_rec2, r2, sizeof(r2));
}

// ------------------------------------------------------------ cp.async
__device__ inline void cp_async16(void *smem, const void *gmem, int src_bytes) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(src_bytes));
}
__device__ inline void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ inline void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

enum { MODE_M2L = 0, MODE_M2M = 1, MODE_L2L = 2 };
static constexpr int CT_TGT = 64;  // targets per batch
static constexpr int CT_THREADS = 256;

struct ContractArgs {
  const int4 *batches;  // {first (list offset or cell), count, level, class}
  const int *tlist;     // class-grouped target cells, or null (targets first + i)
  const float *X;
  float *Y;
  const float *tab;
  const int *cparent, *cchild, *ccoll, *cpbeg, *cpend;
  long long direct_max;  // M2L skips pairs with n_t * n_s <= direct_max (summed directly instead)
  const uint8_t *fdirect;  // M2L: per offset (dx+3) + 7(dy+3) + 49(dz+3): not well separated, summed directly
  const int *src_tab;    // M2L: [batch][slot][CT_TGT] source cells resolved ahead (or null)
  const int *slot_list;  // M2L: [batch][slot index] present slots, nslots_tab[batch] of them
  const int *nslots_tab;
  int cell0, K, KS, KP, dim, mode, slot_base, level_stride;
};

// M2L: the source cell of slot s of a target with nt particles and parent P;
// -1 if absent.
__device__ inline int m2l_source(const ContractArgs &a, int P, int nt, int s, int cls) {
  const int nc = 1 << a.dim, ns = a.dim == 3 ? 27 : 9;
  const int e = c_m2l_slots[a.dim - 2][cls][s];
  const int Q = a.ccoll[(int64_t)P * ns + ((e >> 9) & 31)];
  if (Q < 0) return -1;
  if (a.fdirect && a.fdirect[e & 511]) return -1;  // not well separated: direct far field
  const int src = a.cchild[(int64_t)Q * nc + ((e >> 14) & 7)];
  if (src >= 0 && a.direct_max > 0) {
    const long long nsrc = a.cpend[src] - a.cpbeg[src];
    if (nt * nsrc <= a.direct_max) return -1;  // evaluated by the direct far field
  }
  return src;
}

// A block's 64 targets x (32 J) outputs: warp w takes targets 8 w .. 8 w + 7,
// a lane the outputs lane + 32 j.  Per slot the operator and the gathered
// source rows come by cp.async into one of NS buffers; four threads copy a
// row, whose source index each loaded a slot earlier, so that the only wait of
// a slot is one barrier.  Bound by FP32 multiply-adds (64 x 81 x 96 at p = 8:
// 3.9 K cycles per slot and SM).  With the index looked up, shared and counted
// inside the slot, two barriers and a scalar shared load per target and input
// it took 10.7 K.
template <int J, int NS>
__global__ void __launch_bounds__(CT_THREADS) k_contract(ContractArgs a) {
  extern __shared__ __align__(16) float smem[];
  const int K = a.K, KS = a.KS, KP = a.KP;
  float *Ts = smem;                              // [NS][K][KP]
  float *Xs = Ts + (size_t)NS * K * KP;          // [NS][CT_TGT][KS]

  const int4 b = a.batches[blockIdx.x];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cnt = b.y, level = b.z, cls = b.w;
  const int nslots = a.mode == MODE_M2L ? a.nslots_tab[blockIdx.x] : (a.mode == MODE_M2M ? (1 << a.dim) : 1);
  // (a batch may have no source at all: the lists keep a cell whose only large pairs are with its neighbours)
  if (nslots == 0) return;
  const size_t tab_base = (size_t)blockIdx.x * 189;
  const int row = tid >> 2;  // the row this thread copies a quarter of
  const int row_tgt = row < cnt ? (a.tlist ? a.tlist[b.x + row] : b.x + row) : -1;

  float acc[8][J];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < J; ++j) acc[i][j] = 0.f;

  // operator slot and this row's source cell (-1: none) of slot s
  auto source = [&](int s, int &ts) -> int {
    if (a.mode == MODE_M2L) {
      const int slot = a.slot_list[tab_base + s];
      ts = (c_m2l_slots[a.dim - 2][cls][slot] & 511) + level * a.level_stride;
      return a.src_tab[(tab_base + slot) * CT_TGT + row];
    }
    ts = a.slot_base + (a.mode == MODE_M2M ? s : cls);
    if (row_tgt < 0) return -1;
    return a.mode == MODE_M2M ? a.cchild[((int64_t)row_tgt << a.dim) + s] : a.cparent[row_tgt];
  };
  auto prefetch = [&](int src, int ts, int buf) {
    const float *T = a.tab + (size_t)ts * K * KP;
    float *Td = Ts + (size_t)buf * K * KP;
    const int nT = K * KP / 4;
    for (int c = tid; c < nT; c += CT_THREADS) cp_async16(Td + 4 * c, T + 4 * c, 16);
    float *Xd = Xs + ((size_t)buf * CT_TGT + row) * KS;
    const float *g = a.X + (size_t)(src >= 0 ? src - a.cell0 : 0) * KS;
    for (int q = tid & 3; q < KS / 4; q += 4) cp_async16(Xd + 4 * q, g + 4 * q, src >= 0 ? 16 : 0);
    cp_async_commit();
  };

  int ts_nx, src_nx = source(0, ts_nx);
  if (NS == 2) {
    prefetch(src_nx, ts_nx, 0);
    if (nslots > 1) src_nx = source(1, ts_nx);
  }
  for (int s = 0; s < nslots; ++s) {
    const int buf = NS == 2 ? (s & 1) : 0;
    if (NS == 1) {
      if (s > 0) __syncthreads();  // everyone is done with the buffer
      prefetch(src_nx, ts_nx, 0);
      if (s + 1 < nslots) src_nx = source(s + 1, ts_nx);
    }
    cp_async_wait<0>();
    __syncthreads();  // slot s has landed for everyone; everyone is done with slot s - 1
    if (NS == 2 && s + 1 < nslots) {
      prefetch(src_nx, ts_nx, (s + 1) & 1);
      if (s + 2 < nslots) src_nx = source(s + 2, ts_nx);
    }
    const float *Tb = Ts + (size_t)buf * K * KP;
    const float *Xb = Xs + (size_t)buf * CT_TGT * KS + (size_t)(warp * 8) * KS;
    // four inputs at a time: one 16-byte broadcast load per target; a row's columns K .. KS - 1 are zero, the
    // operator has no such rows
    auto inputs = [&](int k, int m) {
      float av[8][4];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        *reinterpret_cast<float4 *>(av[i]) = *reinterpret_cast<const float4 *>(Xb + i * KS + k);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (q >= m) break;
        float bv[J];
#pragma unroll
        for (int j = 0; j < J; ++j) bv[j] = Tb[(k + q) * KP + lane + 32 * j];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < J; ++j) acc[i][j] = fmaf(av[i][q], bv[j], acc[i][j]);
      }
    };
    const int kf = K & ~3;
#pragma unroll 2
    for (int k = 0; k < kf; k += 4) inputs(k, 4);
    if (kf < K) inputs(kf, K - kf);
  }
  // write out
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = warp * 8 + i;
    if (r >= cnt) continue;
    const int tg = a.tlist ? a.tlist[b.x + r] : b.x + r;
    float *y = a.Y + (size_t)(tg - a.cell0) * KS;
#pragma unroll
    for (int j = 0; j < J; ++j) {
      int o = lane + 32 * j;
      if (o < K) {
        if (a.mode == MODE_M2M) y[o] = acc[i][j];
        else y[o] += acc[i][j];
      }
    }
  }
}

template <int J>
static void launch_contract_j(const ContractArgs &a, int nb, int stages, size_t sh, cudaStream_t st) {
  if (stages == 2) k_contract<J, 2><<<nb, CT_THREADS, sh, st>>>(a);
  else k_contract<J, 1><<<nb, CT_THREADS, sh, st>>>(a);
}

static size_t contract_smem(int K, int KS, int KP, int NS) {
  return sizeof(float) * ((size_t)NS * K * KP + (size_t)NS * CT_TGT * KS);
}

static int launch_contract(const ContractArgs &a, int nb, cudaStream_t st, int64_t &launches) {
  if (nb <= 0) return FMM_OK;
  int J = (a.K + 31) / 32;
  int stages = contract_smem(a.K, a.KS, a.KP, 2) <= 200 * 1024 ? 2 : 1;
  size_t sh = contract_smem(a.K, a.KS, a.KP, stages);
  if (sh > 227 * 1024) return FMM_ERR_UNSUPPORTED;
  // the shared-memory opt-in is per function and device
  static std::mutex mu;
  static size_t attr_set[64][8][3] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return FMM_ERR_CUDA;
  std::lock_guard<std::mutex> lk(mu);
  auto set_attr = [&](auto kern) { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh); };
  if (attr_set[dev][J][stages] < sh) {
    cudaError_t e = cudaSuccess;
    switch (J) {
      case 1: e = stages == 2 ? set_attr(k_contract<1, 2>) : set_attr(k_contract<1, 1>); break;
      case 2: e = stages == 2 ? set_attr(k_contract<2, 2>) : set_attr(k_contract<2, 1>); break;
      case 3: e = stages == 2 ? set_attr(k_contract<3, 2>) : set_attr(k_contract<3, 1>); break;
      case 4: e = stages == 2 ? set_attr(k_contract<4, 2>) : set_attr(k_contract<4, 1>); break;
      case 5: e = stages == 2 ? set_attr(k_contract<5, 2>) : set_attr(k_contract<5, 1>); break;
      case 6: e = stages == 2 ? set_attr(k_contract<6, 2>) : set_attr(k_contract<6, 1>); break;
      default: return FMM_ERR_UNSUPPORTED;
    }
    if (e != cudaSuccess) return FMM_ERR_CUDA;
    attr_set[dev][J][stages] = sh;
  }
  switch (J) {
    case 1: launch_contract_j<1>(a, nb, stages, sh, st); break;
    case 2: launch_contract_j<2>(a, nb, stages, sh, st); break;
    case 3: launch_contract_j<3>(a, nb, stages, sh, st); break;
    case 4: launch_contract_j<4>(a, nb, stages, sh, st); break;
    case 5: launch_contract_j<5>(a, nb, stages, sh, st); break;
    case 6: launch_contract_j<6>(a, nb, stages, sh, st); break;
    default: return FMM_ERR_UNSUPPORTED;
  }
  launches += 1;
  return FMM_OK;
}

// Resolves the source cell of every (slot, target) of each M2L batch ahead of
// the contraction (the lookups are chains of dependent loads, cheap when
// thousands are in flight) and lists, per batch, the slots with at least one
// source.  One block per batch of up to `tchunk` (64 or 128) targets; with
// pair_count set it also counts the (target, source) pairs, with lact / msrc
// set it flags the targets with a source and the sources.
__global__ void k_m2l_sources(ContractArgs a, int tchunk, int *src_tab, int *slot_list, int *nslots_tab,
                              int *tslot_list, unsigned long long *pair_count, const uint8_t *order_p16,
                              uint8_t *slot_p16, unsigned long long *nt_sum, uint8_t *lact, uint8_t *msrc,
                              int cell0) {
  __shared__ int s_flag[189];
  __shared__ int s_tgt[128], s_par[128], s_np[128];  // targets, their parents and sizes
  __shared__ int s_cnt;
  __shared__ unsigned long long s_nt;
  const int4 b = a.batches[blockIdx.x];
  const int tid = threadIdx.x;
  const int nsl = a.dim == 3 ? 189 : 27;
  if (tid < tchunk) {
    const int t = tid < b.y ? a.tlist[b.x + tid] : -1;
    s_tgt[tid] = t;
    s_par[tid] = t >= 0 ? a.cparent[t] : 0;
    s_np[tid] = t >= 0 ? a.cpend[t] - a.cpbeg[t] : 0;
  }
  for (int i = tid; i < 189; i += blockDim.x) s_flag[i] = 0;
  if (tid == 0) {
    s_cnt = 0;
    s_nt = 0;
  }
  __syncthreads();
  const size_t base = (size_t)blockIdx.x * 189;
  int cnt = 0;
  unsigned long long ntc = 0;
  for (int e = tid; e < nsl * tchunk; e += blockDim.x) {
    const int slot = e / tchunk, t = e % tchunk;
    int src = -1;
    if (s_tgt[t] >= 0) src = m2l_source(a, s_par[t], s_np[t], slot, b.w);
    src_tab[(base + slot) * tchunk + t] = src;
    if (src >= 0) {
      s_flag[slot] = 1;
      ++cnt;
      ntc += (unsigned long long)s_np[t];
      if (lact) lact[s_tgt[t] - cell0] = 1;
      if (msrc) msrc[src - cell0] = 1;
    }
  }
  if (pair_count && cnt) atomicAdd(&s_cnt, cnt);
  if (nt_sum && ntc) atomicAdd(&s_nt, ntc);
  __syncthreads();
  if (tid < 32) {
    int n = 0;
    for (int c0 = 0; c0 < nsl; c0 += 32) {
      const int sl = c0 + tid;
      const bool f = sl < nsl && s_flag[sl];
      const unsigned m = __ballot_sync(0xffffffffu, f);
      if (f) {
        const int at = n + __popc(m & ((1u << tid) - 1u));
        slot_list[base + at] = sl;
        const int ts = (c_m2l_slots[a.dim - 2][b.w][sl] & 511) + b.z * a.level_stride;
        if (tslot_list) tslot_list[base + at] = ts;
        if (slot_p16) slot_p16[base + at] = order_p16[ts];
      }
      n += __popc(m);
    }
    if (tid == 0) {
      nslots_tab[blockIdx.x] = n;
      if (pair_count && s_cnt) atomicAdd(pair_count, (unsigned long long)s_cnt);
      if (nt_sum && s_nt) atomicAdd(nt_sum, s_nt);
    }
  }
}

// ------------------------------------------------------------------ P2M
// One thread per particle (leaf order); each coefficient is summed over the
// particles of a leaf by a segmented warp reduction, then added by the
// segment's first lane.
__device__ inline float seg_sum(float v, const bool *same) {
#pragma unroll
  for (int o = 1, k = 0; o < 32; o <<= 1, ++k) {
    float t = __shfl_down_sync(0xffffffffu, v, o);
    if (same[k]) v += t;
  }
  return v;
}

__global__ void k_p2m3d(const float4 *part, const int *leaf_of, int64_t n, int cell0, float inv_s, int p, int KS,
                        float *M) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  bool valid = i < n;
  float4 q = valid ? part[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  int seg = valid ? leaf_of[i] : -1 - lane;
  bool same[5];
#pragma unroll
  for (int o = 1, k = 0; o < 32; o <<= 1, ++k) {
    int so = __shfl_down_sync(0xffffffffu, seg, o);
    same[k] = (lane + o < 32) && so == seg;
  }
  int sp = __shfl_up_sync(0xffffffffu, seg, 1);
  bool head = valid && (lane == 0 || sp != seg);
  float *Mrow = M + (size_t)(valid ? seg - cell0 : 0) * KS;
  const float x = q.x * inv_s, y = q.y * inv_s, z = q.z * inv_s, r2 = x * x + y * y + z * z, w = q.w;
  float dre = 1.f, dim_ = 0.f;
  for (int m = 0; m <= p; ++m) {
    if (m > 0) {
      float h = -0.5f / m;
      float nre = h * (x * dre - y * dim_), nim = h * (x * dim_ + y * dre);
      dre = nre;
      dim_ = nim;
    }
    float p1re = dre, p1im = dim_, p2re = 0.f, p2im = 0.f;
    for (int l = m; l <= p; ++l) {
      float cre, cim;
      if (l == m) {
        cre = dre;
        cim = dim_;
      } else {
        float a1 = c_rec1[l][m] * z, a2 = c_rec2[l][m] * r2;
        cre = a1 * p1re - a2 * p2re;
        cim = a1 * p1im - a2 * p2im;
        p2re = p1re;
        p2im = p1im;
        p1re = cre;
        p1im = cim;
      }
      float vr = seg_sum(w * cre, same);
      if (head) atomicAdd(Mrow + re_idx(l, m), vr);
      if (m > 0) {
        float vi = seg_sum(-w * cim, same);
        if (head) atomicAdd(Mrow + im_idx(l, m), vi);
      }
    }
  }
}

// ------------------------------------------------------------------ L2P
__device__ inline float2 lget(const float *Lr, int n, int m) {
  if (m > n) return make_float2(0.f, 0.f);
  if (m >= 0) return make_float2(Lr[re_idx(n, m)], m ? Lr[im_idx(n, m)] : 0.f);
  // m = -1: L_n^-1 = -conj(L_n^1)
  return make_float2(-Lr[re_idx(n, 1)], Lr[im_idx(n, 1)]);
}

// With `esrc` set, the expansion evaluated for the particles of a leaf is
// that of the leaf's deepest ancestor-or-self on a path to a cell with M2L
// contributions (esrc[leaf] = that cell, elev its level, -1: none, far field
// zero): below it the local expansion only moves by L2L, which is exact, so
// evaluating it there gives the same field without the L2L chain.  Offsets
// of the particles from level-d centres: `part` at the leaf level,
// lvl_off[(d - 2) n + i] above.
//
// P > 0: the order as a compile-time constant (P == p), so that the loops over
// (l, m) unroll completely and every coefficient index and recurrence factor
// is an immediate; P = 0 takes any p at run time.
template <int P, bool POT>
__global__ void k_l2p3d(const float4 *part, const int *leaf_of, int64_t n, int cell0, float inv_s, int p, int KS,
                        const float *L, float4 *far, const int *esrc, const uint8_t *elev, int leaf_first, int D,
                        const float4 *lvl_off, float inv_s0) {
  if (P) p = P;
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float4 q = part[i];
  int src = leaf_of[i];
  if (esrc) {
    const int lf = src - leaf_first;
    src = esrc[lf];
    if (src < 0) {
      far[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      return;
    }
    const int lev = elev[lf];
    if (lev < D) q = lvl_off[(size_t)(lev - 2) * n + i];
    inv_s = ldexpf(inv_s0, lev);
  }
  const float *Lr = L + (size_t)(src - cell0) * KS;
  const float x = q.x * inv_s, y = q.y * inv_s, z = q.z * inv_s, r2 = x * x + y * y + z * z;
  float gx = 0.f, gy = 0.f, gz = 0.f, ph = 0.f;
  float dre = 1.f, dim_ = 0.f;
#pragma unroll
  for (int m = 0; m <= p; ++m) {
    if (m > 0) {
      float h = -0.5f / m;
      float nre = h * (x * dre - y * dim_), nim = h * (x * dim_ + y * dre);
      dre = nre;
      dim_ = nim;
    }
    const float wm = m ? 2.f : 1.f;
    float p1re = dre, p1im = dim_, p2re = 0.f, p2im = 0.f;
#pragma unroll
    for (int l = m; l <= p; ++l) {
      float cre, cim;
      if (l == m) {
        cre = dre;
        cim = dim_;
      } else {
        float a1 = c_rec1[l][m] * z, a2 = c_rec2[l][m] * r2;
        cre = a1 * p1re - a2 * p2re;
        cim = a1 * p1im - a2 * p2im;
        p2re = p1re;
        p2im = p1im;
        p1re = cre;
        p1im = cim;
      }
      if (POT) {
        const float2 Lv = lget(Lr, l, m);
        ph += wm * (Lv.x * cre - Lv.y * cim);
      }
      if (l < p) {
        float2 A = lget(Lr, l + 1, m), Lm = lget(Lr, l + 1, m - 1), Lp = lget(Lr, l + 1, m + 1);
        gz += wm * (A.x * cre - A.y * cim);
        float axr = 0.5f * (Lm.x - Lp.x), axi = 0.5f * (Lm.y - Lp.y);
        gx += wm * (axr * cre - axi * cim);
        float sr = Lp.x + Lm.x, si = Lp.y + Lm.y;  // Re(-i S R / 2) = Im(S R) / 2
        gy += wm * 0.5f * (sr * cim + si * cre);
      }
    }
  }
  far[i] = make_float4(gx * inv_s * inv_s, gy * inv_s * inv_s, gz * inv_s * inv_s, ph * inv_s);
}

using L2P3dFn = void (*)(const float4 *, const int *, int64_t, int, float, int, int, const float *, float4 *, const int *,
                         const uint8_t *, int, int, const float4 *, float);

// The L2P instantiation for order p: unrolled for the orders 4 to 12 that the
// learned orders and the tensor cores cover, the generic one else (65,537
// particles at p = 10: P2M 109 us and L2P 30 us of a 1517 us pass with the
// generic kernels, 1431 us with these).
static L2P3dFn l2p3d_kernel(int p, bool pot) {
  switch (p) {
    case 4: return pot ? k_l2p3d<4, true> : k_l2p3d<4, false>;
    case 5: return pot ? k_l2p3d<5, true> : k_l2p3d<5, false>;
    case 6: return pot ? k_l2p3d<6, true> : k_l2p3d<6, false>;
    case 7: return pot ? k_l2p3d<7, true> : k_l2p3d<7, false>;
    case 8: return pot ? k_l2p3d<8, true> : k_l2p3d<8, false>;
    case 9: return pot ? k_l2p3d<9, true> : k_l2p3d<9, false>;
    case 10: return pot ? k_l2p3d<10, true> : k_l2p3d<10, false>;
    case 11: return pot ? k_l2p3d<11, true> : k_l2p3d<11, false>;
    case 12: return pot ? k_l2p3d<12, true> : k_l2p3d<12, false>;
    default: return pot ? k_l2p3d<0, true> : k_l2p3d<0, false>;
  }
}

// ------------------------------------------------------------------ 2D
// P2M / L2P of the complex-log expansions (power_set2D.cpp:9-21,
// local_set2D.cpp:60-69) with coefficients scaled by the cell size s:
// a~_k = sum_i m_i ((z_i - c)/s)^k, stored [a_0, Re a_1, Im a_1, ...].
__global__ void k_p2m2d(const float4 *part, const int *leaf_of, int64_t n, int cell0, float inv_s, int p, int KS,
                        float *M) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  bool valid = i < n;
  float4 q = valid ? part[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  int seg = valid ? leaf_of[i] : -1 - lane;
  bool same[5];
#pragma unroll
  for (int o = 1, k = 0; o < 32; o <<= 1, ++k) {
    int so = __shfl_down_sync(0xffffffffu, seg, o);
    same[k] = (lane + o < 32) && so == seg;
  }
  int sp = __shfl_up_sync(0xffffffffu, seg, 1);
  bool head = valid && (lane == 0 || sp != seg);
  float *Mrow = M + (size_t)(valid ? seg - cell0 : 0) * KS;
  const float x = q.x * inv_s, y = q.y * inv_s, w = q.w;
  float v = seg_sum(w, same);
  if (head) atomicAdd(Mrow, v);
  float pr = w, pi = 0.f;  // w (z/s)^k
  for (int k = 1; k <= p; ++k) {
    const float nr = pr * x - pi * y, ni = pr * y + pi * x;
    pr = nr;
    pi = ni;
    float vr = seg_sum(pr, same), vi = seg_sum(pi, same);
    if (head) {
      atomicAdd(Mrow + 2 * k - 1, vr);
      atomicAdd(Mrow + 2 * k, vi);
    }
  }
}

// L^ = [Re b_0, Re b_1, Im b_1, ...] with b^_n = b_n s^n represents
// sum_j m_j log(z - z_j); phi = -Re sum b^_n u^n and
// grad = (1/s) (-Re, +Im)(sum n b^_n u^(n-1)), u = (z - c)/s.
__global__ void k_l2p2d(const float4 *part, const int *leaf_of, int64_t n, int cell0, float inv_s, int p, int KS,
                        const float *L, float4 *far) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float4 q = part[i];
  const float *Lr = L + (size_t)(leaf_of[i] - cell0) * KS;
  const float x = q.x * inv_s, y = q.y * inv_s;
  float phr = Lr[0], dr = 0.f, di = 0.f, ur = 1.f, ui = 0.f;  // u^(n-1)
  for (int k = 1; k <= p; ++k) {
    const float br = Lr[2 * k - 1], bi = Lr[2 * k];
    dr += k * (br * ur - bi * ui);
    di += k * (br * ui + bi * ur);
    const float nr = ur * x - ui * y, ni = ur * y + ui * x;
    ur = nr;
    ui = ni;
    phr += br * ur - bi * ui;
  }
  far[i] = make_float4(-dr * inv_s, di * inv_s, 0.f, -phr);
}

// ------------------------------------------------------------------ P2P
// Error-free sum: s + e == a + b exactly (Knuth's TwoSum).
__device__ inline void two_sum(float a, float b, float &s, float &e) {
  s = a + b;
  float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}

// One pair: grad -= m d/|d|^3, phi += m/|d| (3D, leaf.cpp:118-142) or
// grad -= m d/|d|^2, phi -= m log|d| (2D, leaf.cpp:81-95), r^2 -> r^2 + eps2.
// 1/sqrt(x) by the SFU (PTX rsqrt.approx.ftz.f32, relative error below
// 2^-22.9), without the subnormal-input handling of rsqrtf: the r^2 of
// distinct particles here is far above the FP32 subnormal range.
__device__ __forceinline__ float rsqrt_sfu(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <int DIM, bool NEWTON = true, bool POT = true>
__device__ inline void pair_acc(float rx, float ry, float rz, float w, float eps2, float &ax, float &ay, float &az,
                                float &ph) {
  if (DIM == 3) {
    const float r2 = fmaf(rx, rx, fmaf(ry, ry, fmaf(rz, rz, eps2)));
    float inv = rsqrt_sfu(r2);
    if (NEWTON) inv = inv * fmaf(-0.5f * r2 * inv, inv, 1.5f);  // one Newton step
    const float mi = w * inv;
    const float mi3 = mi * inv * inv;
    ax = fmaf(-rx, mi3, ax);
    ay = fmaf(-ry, mi3, ay);
    az = fmaf(-rz, mi3, az);
    if (POT) ph += mi;
  } else {
    const float r2 = fmaf(rx, rx, fmaf(ry, ry, eps2));
    const float f = w / r2;
    ax = fmaf(-rx, f, ax);
    ay = fmaf(-ry, f, ay);
    if (POT) ph = fmaf(-0.5f * w, logf(r2), ph);
  }
}

// Fire-and-forget vector reduction into a float4 in global memory.
__device__ inline void red_add4(float4 *p, float x, float y, float z, float w) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}

struct P2PArgs {
  int leaf_first, nleaves, depth;
  int parts, chunk;  // k_p2p: warps per leaf, taking `chunk` of its targets at a time in turn
  const int *pbeg, *pend, *coll, *parent, *child, *leaf_of;
  const uint64_t *ckey;
  const float4 *part, *part_lo, *far;
  const uint32_t *perm;
  double hx, hy, hz;
  float eps2;
  long long direct_max;
  double G;
  double *acc, *pot;
  unsigned int *err;
  unsigned long long *pair_count;
};

// The cell holding position f = f0 + lane of a chunk of 32 concatenated
// positions, given the cell si0 holding f0; moves si0 to the cell holding
// f0 + 32.  s_pref[c] is the first position of cell c (every cell non-empty),
// s_pref[nsrc] the end; lanes past the end get the last cell (the caller masks
// them).  One shared load per lane, the cell starts inside the chunk as the
// bits of a warp-wide OR, and a population count (at most 32 cells overlap 32
// consecutive positions).
__device__ inline int chunk_cell(const int *s_pref, int nsrc, int f0, int &si0, int lane) {
  const int c = si0 + lane;
  const int rel = c < nsrc ? s_pref[c] - f0 : 32;  // lane 0: <= 0
  const unsigned bit = rel < 32 ? 1u << max(rel, 0) : 0u;
  const unsigned starts = __reduce_or_sync(0xffffffffu, bit);
  const int si = si0 + __popc(starts & (0xffffffffu >> (31 - lane))) - 1;
  const int last = __shfl_sync(0xffffffffu, si, 31);
  si0 = s_pref[last + 1] <= f0 + 32 ? last + 1 : last;
  return si;
}

// Lanes per target group for R targets per lane (largest power of two with
// ceil(nt / R) * Gl <= 32) and the work of the busiest lane per source:
// rounds x (R pairs of about 19 instructions with the hi + lo differences,
// and 4 for the two staged loads and the loop) / Gl.
__device__ inline void colleague_shape(int nt, int R, int &Gl, float &cost) {
  const int groups = (nt + R - 1) / R;
  Gl = 1;
  while (Gl * 2 * groups <= 32) Gl *= 2;
  const int rounds = (groups + 32 / Gl - 1) / (32 / Gl);
  cost = (float)rounds * (float)(19 * R + 4) / (float)Gl;
}

// The register blocking R in 1..4 with the least work on the busiest lane
// (larger R on ties), and its lanes per target group.
__device__ inline int best_shape(int nt, int &Gl) {
  if (nt <= 4) {  // one group of all lanes
    Gl = 32;
    return nt;
  }
  int bestR = 1;
  float best = 1e30f;
#pragma unroll
  for (int R = 1; R <= 4; ++R) {
    int G;
    float c;
    colleague_shape(nt, R, G, c);
    if (c <= best) {
      best = c;
      bestR = R;
      Gl = G;
    }
  }
  return bestR;
}

// A leaf's concatenated neighbours in shared memory: s_pref as in chunk_cell,
// s_cell[k] = (slot, index delta): the particle at position f is f + delta.
struct NearList {
  const int *pref;
  const int2 *cell;
  int n, total;
};

// One warp's targets [tb, tb + nt) of a leaf, R to a lane in groups of Gl
// lanes that share the sources (every Gl-th of each chunk of 32 staged through
// shared memory, shifted into the target leaf's frame), then the output.
template <int R, int DIM, bool POT>
__device__ bool near_targets(const P2PArgs &a, int tb, int nt, int Gl, const NearList &nl, const float2 *h,
                             float4 *s_hi, float4 *s_lo, int lane) {
  const int groups = (nt + R - 1) / R, gpr = 32 / Gl;
  bool bad = false;
  for (int g0 = 0; g0 < groups; g0 += gpr) {
    const int gi = g0 + lane / Gl, sub = lane % Gl;
    const bool live = gi < groups;
    float thx[R], tlx[R], thy[R], tly[R], thz[R], tlz[R], ax[R], ay[R], az[R], ph[R];
    int me[R];  // the target's particle index (the first target's for the lanes' padding)
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int ti = gi * R + r;
      me[r] = tb + (live && ti < nt ? ti : 0);
      const float4 t = a.part[me[r]], tl = a.part_lo[me[r]];
      thx[r] = t.x;
      thy[r] = t.y;
      thz[r] = t.z;
      tlx[r] = tl.x;
      tly[r] = tl.y;
      tlz[r] = tl.z;
      ax[r] = ay[r] = az[r] = ph[r] = 0.f;
    }
    int si0 = 0;
    for (int f0 = 0; f0 < nl.total; f0 += 32) {
      const int f = f0 + lane;
      const int si = chunk_cell(nl.pref, nl.n, f0, si0, lane);
      if (f < nl.total) {
        const int2 c = nl.cell[si];
        const int j = f + c.y;
        const float4 q = a.part[j], ql = a.part_lo[j];
        // + c_s - c_t, a hi + lo multiple of the leaf size per axis
        const float mx = (float)(c.x % 3 - 1), my = (float)((c.x / 3) % 3 - 1), mz = (float)(c.x / 9 - 1);
        float sx, sy, sz = 0.f, ex, ey, ez = 0.f;
        two_sum(q.x, mx * h[0].x, sx, ex);
        two_sum(q.y, my * h[1].x, sy, ey);
        if (DIM == 3) two_sum(q.z, mz * h[2].x, sz, ez);
        s_hi[lane] = make_float4(sx, sy, sz, q.w);
        s_lo[lane] = make_float4(ex + fmaf(mx, h[0].y, ql.x), ey + fmaf(my, h[1].y, ql.y),
                                 DIM == 3 ? ez + fmaf(mz, h[2].y, ql.z) : 0.f, __int_as_float(j));
      }
      __syncwarp();
      const int cnt = min(32, nl.total - f0);
      for (int k = sub; k < cnt; k += Gl) {
        const float4 q = s_hi[k], ql = s_lo[k];
        const int j = __float_as_int(ql.w);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if (j == me[r]) continue;
          const float rx = (thx[r] - q.x) + (tlx[r] - ql.x);
          const float ry = (thy[r] - q.y) + (tly[r] - ql.y);
          const float rz = DIM == 3 ? (thz[r] - q.z) + (tlz[r] - ql.z) : 0.f;
          pair_acc<DIM, true, POT>(rx, ry, rz, q.w, a.eps2, ax[r], ay[r], az[r], ph[r]);
        }
      }
      __syncwarp();
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      for (int o = 1; o < Gl; o <<= 1) {
        ax[r] += __shfl_xor_sync(0xffffffffu, ax[r], o);
        ay[r] += __shfl_xor_sync(0xffffffffu, ay[r], o);
        if (DIM == 3) az[r] += __shfl_xor_sync(0xffffffffu, az[r], o);
        if (POT) ph[r] += __shfl_xor_sync(0xffffffffu, ph[r], o);
      }
      const int ti = gi * R + r;
      if (sub == 0 && live && ti < nt) {
        const float4 fa = a.far[me[r]];
        const uint32_t o = a.perm[me[r]];
        const double vx = a.G * ((double)fa.x + ax[r]), vy = a.G * ((double)fa.y + ay[r]),
                     vz = DIM == 3 ? a.G * ((double)fa.z + az[r]) : 0.0;
        a.acc[DIM * (size_t)o] = vx;
        a.acc[DIM * (size_t)o + 1] = vy;
        if (DIM == 3) a.acc[3 * (size_t)o + 2] = vz;
        if (POT) a.pot[o] = a.G * ((double)fa.w + ph[r]);
        bad |= !(isfinite(vx) && isfinite(vy) && isfinite(vz));
      }
    }
  }
  return bad;
}

// One warp per target leaf.  Sources: the leaf itself (j != i) and its
// existing neighbours (leaf.cpp:118-142), concatenated, so that a warp's lanes
// stay busy whatever the neighbours' sizes: with 1 to 2 particles per leaf (a
// Plummer sphere's uniform-depth tree) a loop over the 27 neighbours left 30
// of 32 lanes idle.  The direct far field (interaction-list pairs summed
// particle by particle) has been added into `far` by k_direct_far before this
// kernel runs; this kernel adds the near field and writes the output.
//
// Near-field precision: x_i - x_j = t_i - (s_j + shift) with t_i, s_j the
// offsets from the two leaf centres and shift = c_s - c_t an exact multiple
// of the leaf size.  Offsets and shift are hi + lo FP32 pairs and s_hi +
// shift_hi is formed error-free (TwoSum), so each difference is rounded once,
// relative to itself, whatever the separation.
template <int DIM, bool POT>
__global__ void __launch_bounds__(256, 4) k_p2p(P2PArgs a) {
  constexpr int NS = DIM == 3 ? 27 : 9;
  __shared__ float4 s_hi_all[8][32], s_lo_all[8][32];
  __shared__ int2 s_cell_all[8][NS];
  __shared__ int s_pref_all[8][NS + 1];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int part = a.parts > 1 ? (int)(w % a.parts) : 0, wl = (int)(a.parts > 1 ? w / a.parts : w);
  if (wl >= a.nleaves) return;
  const int g = a.leaf_first + wl;
  const int lb = a.pbeg[g], le = a.pend[g];
  if (part > 0 && (int64_t)part * a.chunk >= le - lb) return;
  const int C = lane < NS ? a.coll[(int64_t)g * NS + lane] : -1;
  const int cb = C >= 0 ? a.pbeg[C] : 0, cn = C >= 0 ? a.pend[C] - cb : 0;
  int x = cn;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  const unsigned m = __ballot_sync(0xffffffffu, cn > 0);
  if (cn > 0) {
    const int at = __popc(m & ((1u << lane) - 1u));
    s_cell_all[wib][at] = make_int2(lane, cb - (x - cn));
    s_pref_all[wib][at + 1] = x;
  }
  if (lane == 0) s_pref_all[wib][0] = 0;
  __syncwarp();
  const int total = __shfl_sync(0xffffffffu, x, 31);
  const NearList nl{s_pref_all[wib], s_cell_all[wib], __popc(m), total};
  const float2 h[3] = {make_float2((float)a.hx, (float)(a.hx - (double)(float)a.hx)),
                       make_float2((float)a.hy, (float)(a.hy - (double)(float)a.hy)),
                       make_float2((float)a.hz, (float)(a.hz - (double)(float)a.hz))};
  bool bad = false;
  for (int64_t t0 = lb + (int64_t)part * a.chunk; t0 < le; t0 += (int64_t)a.parts * a.chunk) {
    const int tb = (int)t0, nt = min(a.chunk, le - tb);
    int Gl = 1;
    switch (best_shape(nt, Gl)) {
      case 1: bad |= near_targets<1, DIM, POT>(a, tb, nt, Gl, nl, h, s_hi_all[wib], s_lo_all[wib], lane); break;
      case 2: bad |= near_targets<2, DIM, POT>(a, tb, nt, Gl, nl, h, s_hi_all[wib], s_lo_all[wib], lane); break;
      case 3: bad |= near_targets<3, DIM, POT>(a, tb, nt, Gl, nl, h, s_hi_all[wib], s_lo_all[wib], lane); break;
      default: bad |= near_targets<4, DIM, POT>(a, tb, nt, Gl, nl, h, s_hi_all[wib], s_lo_all[wib], lane); break;
    }
  }
  if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(a.err, FMM_DEV_ERR_NONFINITE_OUTPUT);
  if (lane == 0 && a.pair_count && part == 0)
    atomicAdd(a.pair_count, (unsigned long long)((long long)(le - lb) * (total - 1)));
}

// Whether k_p2p's leaves are split over several warps of 16 targets: where the
// fullest leaf holds more than 32 particles, m, and m^2 is above twice the
// pairs of the mean leaf, (n / leaves)^2, times the leaves that one of the 4736
// warps at a time goes through.  Measured m^2 over that, without and with the
// split: 2.6 (300,000 uniform, 73 per leaf) 1.27 and 1.04 ms, 22 (20,000, 39
// per leaf) 0.19 and 0.09, 315 (a sphere of 300,000 with up to 300 per leaf)
// 4.05 and 1.00; 0.6 (2^20 uniform, 30 per leaf) 1.36 and 1.55, 1.4 (a 2D disk,
// 23 per leaf) 0.14 and 0.17.  A split leaf's other warps exist for every leaf
// and are mostly empty, so only up to 65,536 leaves (300,000 of up to 300 per
// leaf 2.16 and 2.35 ms, 570,000 of up to 128 1.20 and 2.11).
static bool near_split(int64_t n, int64_t nleaves, int64_t largest) {
  const double mean = (double)n / (double)nleaves;
  return nleaves <= 65536 && largest > 32 &&
         (double)largest * (double)largest > 2.0 * mean * mean * (double)nleaves / 4736.0;
}

// The 2D near field of small leaves: eight lanes per leaf, each with every
// eighth source for up to four targets in registers.  A leaf of one or two
// particles has about 15 sources, half of which a warp's lanes have nothing
// to do with, and k_p2p's staging and reductions over 32 lanes cost as much as
// the pairs.  A lane shifts its source into the target leaf's frame itself
// (the same hi + lo arithmetic as k_p2p).  (The same in 3D with 16 lanes per
// leaf lost: a sphere's few full leaves kept half warps busy long after the
// rest, 320 -> 500 us of a 65,537-particle pass.)
template <int R, bool POT>
__device__ __forceinline__ bool near2d_targets(const P2PArgs &a, int tb, int nt, int t0, const int2 *s_cell,
                                               const int *s_pref, int total, float2 hx, float2 hy, int sub) {
  float4 t[R], tl[R];
  float ax[R], ay[R], ph[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = nt > 0 ? tb + min(t0 + r, nt - 1) : 0;
    t[r] = a.part[i];
    tl[r] = a.part_lo[i];
    ax[r] = ay[r] = ph[r] = 0.f;
  }
  int si = 0;
  if (t0 < nt)
    for (int f = sub; f < total; f += 8) {
      while (s_pref[si + 1] <= f) ++si;
      const int2 c = s_cell[si];
      const int j = f + c.y;
      const float4 q = a.part[j], ql = a.part_lo[j];
      const float mx = (float)(c.x % 3 - 1), my = (float)(c.x / 3 - 1);
      float sx, sy, ex, ey;
      two_sum(q.x, mx * hx.x, sx, ex);
      two_sum(q.y, my * hy.x, sy, ey);
      ex += fmaf(mx, hx.y, ql.x);
      ey += fmaf(my, hy.y, ql.y);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (j == tb + t0 + r) continue;
        float az = 0.f;
        pair_acc<2, true, POT>((t[r].x - sx) + (tl[r].x - ex), (t[r].y - sy) + (tl[r].y - ey), 0.f, q.w, a.eps2, ax[r],
                               ay[r], az, ph[r]);
      }
    }
  __syncwarp();
  bool bad = false;
#pragma unroll
  for (int r = 0; r < R; ++r) {
#pragma unroll
    for (int o = 4; o; o >>= 1) {
      ax[r] += __shfl_xor_sync(0xffffffffu, ax[r], o);
      ay[r] += __shfl_xor_sync(0xffffffffu, ay[r], o);
      if (POT) ph[r] += __shfl_xor_sync(0xffffffffu, ph[r], o);
    }
    if (sub == r && t0 + r < nt) {
      const int i = tb + t0 + r;
      const float4 fa = a.far[i];
      const uint32_t o = a.perm[i];
      const double vx = a.G * ((double)fa.x + ax[r]), vy = a.G * ((double)fa.y + ay[r]);
      a.acc[2 * (size_t)o] = vx;
      a.acc[2 * (size_t)o + 1] = vy;
      if (POT) a.pot[o] = a.G * ((double)fa.w + ph[r]);
      bad |= !(isfinite(vx) && isfinite(vy));
    }
  }
  return bad;
}

// The mean leaf up to which 2D leaves may get octets: 300,000 particles of a
// disk at 5.8 per leaf 0.077 ms with octets and 0.112 with warps, at 15 per
// leaf (200,000) 0.112 and 0.105.
static constexpr int SMALL2D_MEAN = 8;

// Whether the leaves of a 2D near field get octets.  An octet is busy with its
// leaf of m particles for a time that grows as m^2, so that a full leaf may
// outlast all others: octets gained with leaves / m^2 = 33 (200,000 particles
// in clumps, m = 56, 0.097 against 0.122 ms with warps), 159 and 340 (2M, m =
// 57, 0.69 against 1.16) and lost at 21 (300,000, m = 84, 1.41 against 0.35),
// 19 (20,000, m = 25, 0.112 against 0.034) and 14.  At least 32 m^2 leaves also
// keep a warp's pair count within 32 bits.
static bool near2d_octets(int64_t n, int64_t nleaves, int64_t largest) {
  return n <= SMALL2D_MEAN * nleaves && 32 * largest * largest <= nleaves;
}

template <bool POT>
__global__ void __launch_bounds__(256) k_p2p2d_small(P2PArgs a) {
  __shared__ int2 s_cell_all[32][9];
  __shared__ int s_pref_all[32][10];
  const int lane = threadIdx.x & 31, sub = lane & 7, oct = threadIdx.x >> 3;
  const int64_t wl = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  int2 *s_cell = s_cell_all[oct];
  int *s_pref = s_pref_all[oct];
  // (octets past the end go along with no targets)
  const bool live = wl < a.nleaves;
  const int g = a.leaf_first + (live ? (int)wl : 0);
  const int tb = a.pbeg[g], nt = live ? a.pend[g] - tb : 0;
  int cb[2], cn[2], kept = 0, parts = 0;  // neighbours sub and, lane 7, the ninth
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int C = live && (k == 0 || sub == 7) ? a.coll[(int64_t)g * 9 + sub + k] : -1;
    cb[k] = C >= 0 ? a.pbeg[C] : 0;
    cn[k] = C >= 0 ? a.pend[C] - cb[k] : 0;
    kept += cn[k] > 0;
    parts += cn[k];
  }
  int at = kept, x = parts;  // inclusive scans over the octet
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, at, o, 8), z = __shfl_up_sync(0xffffffffu, x, o, 8);
    if (sub >= o) {
      at += y;
      x += z;
    }
  }
  const int total = __shfl_sync(0xffffffffu, x, 7, 8);
  at -= kept;
  x -= parts;
#pragma unroll
  for (int k = 0; k < 2; ++k)
    if (cn[k] > 0) {
      s_cell[at] = make_int2(sub + k, cb[k] - x);
      x += cn[k];
      s_pref[++at] = x;
    }
  if (sub == 0) s_pref[0] = 0;
  __syncwarp();
  const float2 hx = make_float2((float)a.hx, (float)(a.hx - (double)(float)a.hx)),
               hy = make_float2((float)a.hy, (float)(a.hy - (double)(float)a.hy));
  const int most = __reduce_max_sync(0xffffffffu, nt);
  bool bad = false;
  for (int t0 = 0; t0 < most; t0 += 4)
    switch (min(4, most - t0)) {  // warp-uniform
      case 1: bad |= near2d_targets<1, POT>(a, tb, nt, t0, s_cell, s_pref, total, hx, hy, sub); break;
      case 2: bad |= near2d_targets<2, POT>(a, tb, nt, t0, s_cell, s_pref, total, hx, hy, sub); break;
      case 3: bad |= near2d_targets<3, POT>(a, tb, nt, t0, s_cell, s_pref, total, hx, hy, sub); break;
      default: bad |= near2d_targets<4, POT>(a, tb, nt, t0, s_cell, s_pref, total, hx, hy, sub); break;
    }
  if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(a.err, FMM_DEV_ERR_NONFINITE_OUTPUT);
  const unsigned pairs = __reduce_add_sync(0xffffffffu, sub == 0 ? (unsigned)nt * (unsigned)max(total - 1, 0) : 0u);
  if (lane == 0 && a.pair_count) atomicAdd(a.pair_count, (unsigned long long)pairs);
}

// Adaptive targets: the colleague sums of the adaptive leaves.  An adaptive
// leaf B (any level, listed in alist[0 .. acount)) sums the particles of B
// itself (j != i) and of its colleagues at B's level: the pairs that the
// deeper levels' interaction lists and the leaf level's near field would sum
// in the uniform tree.  A colleague may hold millions of particles (a sparse
// cell next to a dense clump), so the work is cut into items of at most
// p2p_chunk sources of B's concatenated colleague list, each one warp's job;
// items of one B add into the far-field accumulator with vector reductions.
//
// Precision: colleagues touch B, so pairs can be far closer than the cell
// size.  Positions are taken relative to an origin inside B (its first
// particle) in FP64 and split into FP32 hi + lo parts; a difference
// (t_hi - s_hi) + (t_lo - s_lo) is then rounded once relative to itself, as
// in the uniform near field.  1/|r| is the SFU's rsqrt without a Newton step,
// as in the direct far field (relative error below 2^-22.9; with the step the
// 16M mixture's force error was the same, 7.7e-7, and the kernel 6 % slower).
// The chunk (sources per item) is a setting,
// fmm_config.p2p_chunk, 256 by default.
static constexpr int CL_CHUNK_DEFAULT = 256;

// Number of items of each listed adaptive leaf (0 past the list's end), over
// [0, ncell) so that the host needs no count.
__global__ void k_colleague_count(const int *alist, const unsigned *acount, int ncell, const int *coll,
                                  const int *pbeg, const int *pend, int ns, int chunk, uint32_t *cnt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ncell) return;
  uint32_t items = 0;
  if (i < (int)*acount) {
    const int B = alist[i];
    long long S = 0;
    for (int s = 0; s < ns; ++s) {
      const int C = coll[(int64_t)B * ns + s];
      if (C >= 0) S += pend[C] - pbeg[C];
    }
    items = pend[B] > pbeg[B] ? (uint32_t)((S + chunk - 1) / chunk) : 0u;
  }
  cnt[i] = items;
}

// items[off[i] + k] = (i, k) for the k-th chunk of listed leaf i.
__global__ void k_colleague_fill(const unsigned *acount, int ncell, const uint32_t *cnt, const uint32_t *off,
                                 int2 *items) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ncell || i >= (int)*acount) return;
  const uint32_t o = off[i], c = cnt[i];
  for (uint32_t k = 0; k < c; ++k) items[o + k] = make_int2(i, (int)k);
}

__device__ inline void split_hi_lo(double d, float &hi, float &lo) {
  hi = (float)d;
  lo = (float)(d - (double)hi);
}

// One item's concatenated source range [f0, f1), B's own particles at
// [bbeg, bend) in it, and the FP64 origin of the hi + lo offsets.
struct CollChunk {
  int f0, f1, bbeg, bend, ncoll;
  double ox, oy, oz;
};

// The targets of B, R to a lane, in target groups of Gl lanes that share the
// sources (every Gl-th of each chunk of 32 staged through shared memory).
// Only chunks that hold some of B's own particles test for j == i.
template <int R, int DIM, bool POT>
__device__ void colleague_targets(const P2PArgs &a, const double *xs, float4 *far, int tb, int nt, int Gl,
                                  const CollChunk &cc, const int *s_pref, const int *s_cell, float4 *s_hi,
                                  float4 *s_lo, int lane) {
  const int groups = (nt + R - 1) / R, gpr = 32 / Gl;
  for (int g0 = 0; g0 < groups; g0 += gpr) {
    const int gi = g0 + lane / Gl, sub = lane % Gl;
    const bool live = gi < groups;
    float2 tx[R], ty[R], tz[R];  // hi, lo
    float ax[R], ay[R], az[R], ph[R];
    int me[R];  // the target's particle index (target 0's for the lanes' padding)
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int ti = gi * R + r;
      me[r] = tb + (live && ti < nt ? ti : 0);
      split_hi_lo(xs[DIM * (size_t)me[r]] - cc.ox, tx[r].x, tx[r].y);
      split_hi_lo(xs[DIM * (size_t)me[r] + 1] - cc.oy, ty[r].x, ty[r].y);
      tz[r] = make_float2(0.f, 0.f);
      if (DIM == 3) split_hi_lo(xs[DIM * (size_t)me[r] + 2] - cc.oz, tz[r].x, tz[r].y);
      ax[r] = ay[r] = az[r] = ph[r] = 0.f;
    }
    for (int fb = cc.f0; fb < cc.f1; fb += 32) {
      const int f = fb + lane;
      if (f < cc.f1) {
        // colleague holding concatenated position f: the last k with s_pref[k] <= f
        int lo = 0, hi = cc.ncoll - 1;
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (s_pref[mid] <= f) lo = mid;
          else hi = mid - 1;
        }
        const int j = a.pbeg[s_cell[lo]] + (f - s_pref[lo]);
        float hx, lx, hy, ly, hz = 0.f, lz = 0.f;
        split_hi_lo(xs[DIM * (size_t)j] - cc.ox, hx, lx);
        split_hi_lo(xs[DIM * (size_t)j + 1] - cc.oy, hy, ly);
        if (DIM == 3) split_hi_lo(xs[DIM * (size_t)j + 2] - cc.oz, hz, lz);
        s_hi[lane] = make_float4(-hx, -lx, -hy, -ly);
        s_lo[lane] = make_float4(-hz, -lz, a.part[j].w, __int_as_float(j));
      }
      __syncwarp();
      const int cnt = min(32, cc.f1 - fb);
      if (fb < cc.bend && fb + cnt > cc.bbeg) {
        for (int k = sub; k < cnt; k += Gl) {
          const float4 q = s_hi[k], ql = s_lo[k];
          const int j = __float_as_int(ql.w);
#pragma unroll
          for (int r = 0; r < R; ++r) {
            if (j == me[r]) continue;
            const float2 dx = __fadd2_rn(tx[r], make_float2(q.x, q.y)), dy = __fadd2_rn(ty[r], make_float2(q.z, q.w)),
                         dz = __fadd2_rn(tz[r], make_float2(ql.x, ql.y));
            pair_acc<DIM, false, POT>(dx.x + dx.y, dy.x + dy.y, dz.x + dz.y, ql.z, a.eps2, ax[r], ay[r], az[r], ph[r]);
          }
        }
      } else {
        for (int k = sub; k < cnt; k += Gl) {
          const float4 q = s_hi[k], ql = s_lo[k];
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const float2 dx = __fadd2_rn(tx[r], make_float2(q.x, q.y)), dy = __fadd2_rn(ty[r], make_float2(q.z, q.w)),
                         dz = __fadd2_rn(tz[r], make_float2(ql.x, ql.y));
            pair_acc<DIM, false, POT>(dx.x + dx.y, dy.x + dy.y, dz.x + dz.y, ql.z, a.eps2, ax[r], ay[r], az[r], ph[r]);
          }
        }
      }
      __syncwarp();
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      for (int o = 1; o < Gl; o <<= 1) {
        ax[r] += __shfl_xor_sync(0xffffffffu, ax[r], o);
        ay[r] += __shfl_xor_sync(0xffffffffu, ay[r], o);
        az[r] += __shfl_xor_sync(0xffffffffu, az[r], o);
        if (POT) ph[r] += __shfl_xor_sync(0xffffffffu, ph[r], o);
      }
      const int ti = gi * R + r;
      if (sub == 0 && live && ti < nt) red_add4(far + tb + ti, ax[r], ay[r], az[r], ph[r]);
    }
  }
}

// One warp per item (grid-stride): B's targets R to a lane in groups of Gl
// lanes (colleague_targets), the item's sources staged 32 at a time through
// shared memory.
template <int DIM, bool POT>
__global__ void __launch_bounds__(256, 4) k_colleague_sum(P2PArgs a, const int *alist, const int2 *items,
                                                       const uint32_t *nitems, const double *xs, float4 *far,
                                                       int chunk) {
  constexpr int NS = DIM == 3 ? 27 : 9;
  __shared__ float4 s_hi_all[8][32], s_lo_all[8][32];
  __shared__ int s_pref_all[8][NS + 1], s_cell_all[8][NS];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  float4 *s_hi = s_hi_all[wib], *s_lo = s_lo_all[wib];
  int *s_pref = s_pref_all[wib], *s_cell = s_cell_all[wib];
  const int nwarps = (int)((gridDim.x * blockDim.x) >> 5);
  const int total = (int)*nitems;
  long long npairs = 0;
  for (int it = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); it < total; it += nwarps) {
    const int2 item = items[it];
    const int B = alist[item.x];
    const int tb = a.pbeg[B], nt = a.pend[B] - tb;
    // B's colleagues (B itself included), compacted, with the prefix of their sizes
    const int C = lane < NS ? a.coll[(int64_t)B * NS + lane] : -1;
    const int nc = C >= 0 ? a.pend[C] - a.pbeg[C] : 0;
    const unsigned m = __ballot_sync(0xffffffffu, C >= 0);
    int x = nc;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    const int ncoll = __popc(m);
    if (C >= 0) {
      const int at = __popc(m & ((1u << lane) - 1u));
      s_cell[at] = C;
      s_pref[at + 1] = x;  // inclusive prefix (zero-size colleagues repeat the previous value)
    }
    if (lane == 0) s_pref[0] = 0;
    __syncwarp();
    const int S = s_pref[ncoll];
    const int f0 = item.y * chunk, f1 = min(S, f0 + chunk);
    // B's own particles in the concatenation (the pairs j == i are skipped)
    const int bl = __ffs(__ballot_sync(0xffffffffu, C == B)) - 1;
    const int bend = __shfl_sync(0xffffffffu, x, bl), bbeg = bend - __shfl_sync(0xffffffffu, nc, bl);
    const double ox = xs[DIM * (size_t)tb], oy = xs[DIM * (size_t)tb + 1], oz = DIM == 3 ? xs[DIM * (size_t)tb + 2] : 0.0;
    int bestG = 1;
    const int bestR = best_shape(nt, bestG);
    const CollChunk cc{f0, f1, bbeg, bend, ncoll, ox, oy, oz};
    switch (bestR) {
      case 1: colleague_targets<1, DIM, POT>(a, xs, far, tb, nt, bestG, cc, s_pref, s_cell, s_hi, s_lo, lane); break;
      case 2: colleague_targets<2, DIM, POT>(a, xs, far, tb, nt, bestG, cc, s_pref, s_cell, s_hi, s_lo, lane); break;
      case 3: colleague_targets<3, DIM, POT>(a, xs, far, tb, nt, bestG, cc, s_pref, s_cell, s_hi, s_lo, lane); break;
      default: colleague_targets<4, DIM, POT>(a, xs, far, tb, nt, bestG, cc, s_pref, s_cell, s_hi, s_lo, lane); break;
    }
    if (lane == 0) npairs += (long long)nt * (f1 - f0) - max(0, min(f1, bend) - max(f0, bbeg));
  }
  if (lane == 0 && a.pair_count && npairs) atomicAdd(a.pair_count, (unsigned long long)npairs);
}

// The output: acc[perm[i]] = G * far[i] (and the potential), with the
// finiteness check, after every contribution was added into far.
template <int DIM>
__global__ void k_far_output(const float4 *far, const uint32_t *perm, int64_t n, double G, double *acc, double *pot,
                             unsigned int *err) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  bool bad = false;
  if (i < n) {
    const float4 f = far[i];
    const uint32_t o = perm[i];
    const double vx = G * (double)f.x, vy = G * (double)f.y, vz = G * (double)f.z;
    acc[DIM * (size_t)o] = vx;
    acc[DIM * (size_t)o + 1] = vy;
    if (DIM == 3) acc[3 * (size_t)o + 2] = vz;
    if (pot) pot[o] = G * (double)f.w;
    bad = !(isfinite(vx) && isfinite(vy) && isfinite(vz));
  }
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(err, FMM_DEV_ERR_NONFINITE_OUTPUT);
}

// --------------------------------------------------------- direct far field
// Offsets of every particle (leaf order) from the centre of its ancestor at
// each level d in [d0, d1], FP32, with the mass: the frames in which pairs of
// level-d cells are summed directly.  out[(d - d0) * n + i].
template <int DIM>
__global__ void k_level_offsets(const double *pos, const double *mass, const uint32_t *perm, const int *leaf_of,
                                const uint64_t *ckey, int64_t n, int depth, int d0, int d1, double lox, double loy,
                                double loz, double ex, double ey, double ez, float4 *out) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t qx, qy, qz;
  morton_decode(DIM, ckey[leaf_of[i]], qx, qy, qz);
  const uint32_t j = perm[i];
  const double px = pos[DIM * (size_t)j], py = pos[DIM * (size_t)j + 1], pz = DIM == 3 ? pos[3 * (size_t)j + 2] : 0.0;
  const float w = (float)mass[j];
  for (int d = d0; d <= d1; ++d) {
    const int sh = depth - d;
    const double inv = ldexp(1.0, -d);
    const double cx = lox + ((double)(qx >> sh) + 0.5) * (ex * inv);
    const double cy = loy + ((double)(qy >> sh) + 0.5) * (ey * inv);
    const double cz = DIM == 3 ? loz + ((double)(qz >> sh) + 0.5) * (ez * inv) : 0.0;
    out[(size_t)(d - d0) * n + i] =
        make_float4((float)(px - cx), (float)(py - cy), DIM == 3 ? (float)(pz - cz) : 0.f, w);
  }
}

static constexpr int DF_MAX_LEVELS = 33;

struct DirectArgs {
  // levels of the launch, coarse first: warps [w0[k], w0[k+1]) take the
  // cells first[k] + (warp - w0[k]), or with a target list (k_direct_far's
  // LIST) the cells tlist[first[k] + (warp - w0[k])]
  int nlev;
  int first[DF_MAX_LEVELS], w0[DF_MAX_LEVELS + 1];
  // k_direct_far's SPLIT: warp w takes item w of *nitems, (cell, part): the
  // part'th `chunk` targets of the cell
  int chunk;
  const int2 *items;
  const uint32_t *nitems;
  int cell[DF_MAX_LEVELS];           // first cell of each level
  const float4 *off[DF_MAX_LEVELS];  // particle offsets from their level-d ancestor's centre
  float h[DF_MAX_LEVELS][3];         // level-d cell size
  const int *pbeg, *pend, *coll, *parent, *child;
  const uint64_t *ckey;
  float eps2;
  long long direct_max;
  const uint8_t *fdirect;  // per offset: not well separated, always summed directly
  int any_fdirect;
  float4 *far;
  unsigned long long *pair_count;
  const int *tlist;        // adaptive targets: each level's targets, from first[k]
};

// One warp per level-d target cell T with n_T <= direct_max: the sources are
// the cells S of T's interaction list (node_i.cpp:39-43) with
// n_T * n_S <= direct_max, exactly the pairs the M2L contraction skips.
// Small T (NT <= 7 targets): every lane holds all targets and takes every
// 32nd particle of the concatenated sources; larger T: register-blocked
// target groups over sources staged through shared memory.
//
// With offsets that are not well separated (a box that is not near a cube)
// whole pairs of coarse cells are summed, and with one warp per cell the
// kernel waited for a few warps with thousands of targets: there (SPLIT) every
// `chunk` targets of a cell are an item of a list in the order of the cells, a
// warp each.  (As many warps for every cell of a level as for its largest left
// 94 to 99.8 % of them empty where a box holds a clump: a flattened halo of
// 60,000 particles with half of them in one cell on ten levels 36.9 ms, now 1.3;
// a flattened sphere of 2^20 35.5, now 24.1.)  The items come in runs of one
// cell, whose warps read the same sources; in the order in which atomics drew
// them that sphere took 42 ms.  Three blocks per SM: at four the loops over
// thousands of sources spill (32 ms).
//
// Per kept source cell si the warp keeps s_pref[si] (its first position in
// the concatenation; every cell non-empty) and s_cell[si] = (shift c_S - c_T,
// index delta): the particle at concatenated position f of cell si is
// off[f + delta].

// The source particle at concatenated position f of cell si, shifted into
// the target's frame.
__device__ inline float4 shifted_source(const float4 *off, const float4 *s_cell, int f, int si) {
  const float4 cd = s_cell[si];
  const float4 q = off[f + __float_as_int(cd.w)];
  return make_float4(q.x + cd.x, q.y + cd.y, q.z + cd.z, q.w);
}

template <int NT, int DIM, bool POT>
__device__ void direct_small(const DirectArgs &a, const float4 *off, int tb, int nt, const float4 *s_cell,
                             const int *s_pref, int nsrc, int lane) {
  float tx[NT], ty[NT], tz[NT], ax[NT], ay[NT], az[NT], ph[NT];
#pragma unroll
  for (int k = 0; k < NT; ++k) {
    float4 t = off[tb + (k < nt ? k : 0)];
    tx[k] = t.x;
    ty[k] = t.y;
    tz[k] = t.z;
    ax[k] = ay[k] = az[k] = ph[k] = 0.f;
  }
  const int total = s_pref[nsrc];
  int si0 = 0;
  for (int f0 = 0; f0 < total; f0 += 32) {
    const int f = f0 + lane;
    const int si = chunk_cell(s_pref, nsrc, f0, si0, lane);
    if (f < total) {
      const float4 q = shifted_source(off, s_cell, f, si);
#pragma unroll
      for (int k = 0; k < NT; ++k)
        pair_acc<DIM, false, POT>(tx[k] - q.x, ty[k] - q.y, tz[k] - q.z, q.w, a.eps2, ax[k], ay[k], az[k], ph[k]);
    }
  }
#pragma unroll
  for (int k = 0; k < NT; ++k) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      ax[k] += __shfl_xor_sync(0xffffffffu, ax[k], o);
      ay[k] += __shfl_xor_sync(0xffffffffu, ay[k], o);
      az[k] += __shfl_xor_sync(0xffffffffu, az[k], o);
      ph[k] += __shfl_xor_sync(0xffffffffu, ph[k], o);
    }
    if (lane == k && k < nt) red_add4(a.far + tb + k, ax[k], ay[k], az[k], ph[k]);
  }
}

// Larger T: each lane holds R targets and takes every Gl-th source of the
// chunks of 32 staged through shared memory; ceil(nt / R) target groups of
// Gl lanes, 32 / Gl groups per round.
template <int R, int DIM, bool POT>
__device__ void direct_blocked(const DirectArgs &a, const float4 *off, int tb, int nt, int Gl, const float4 *s_cell,
                               const int *s_pref, int nsrc, int lane, float4 *stage) {
  const int groups = (nt + R - 1) / R, gpr = 32 / Gl;
  const int total = s_pref[nsrc];
  for (int g0 = 0; g0 < groups; g0 += gpr) {
    const int gi = g0 + lane / Gl, sub = lane % Gl;
    float tx[R], ty[R], tz[R], ax[R], ay[R], az[R], ph[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int ti = gi * R + r;
      const float4 t = off[tb + (gi < groups && ti < nt ? ti : 0)];
      tx[r] = t.x;
      ty[r] = t.y;
      tz[r] = t.z;
      ax[r] = ay[r] = az[r] = ph[r] = 0.f;
    }
    int si0 = 0;
    for (int f0 = 0; f0 < total; f0 += 32) {
      const int f = f0 + lane;
      const int si = chunk_cell(s_pref, nsrc, f0, si0, lane);
      stage[lane] = f < total ? shifted_source(off, s_cell, f, si) : make_float4(0.f, 0.f, 0.f, 0.f);
      __syncwarp();
      const int cnt = min(32, total - f0);
      for (int k = sub; k < cnt; k += Gl) {
        const float4 sq = stage[k];
#pragma unroll
        for (int r = 0; r < R; ++r)
          pair_acc<DIM, false, POT>(tx[r] - sq.x, ty[r] - sq.y, tz[r] - sq.z, sq.w, a.eps2, ax[r], ay[r], az[r], ph[r]);
      }
      __syncwarp();
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      for (int o = 1; o < Gl; o <<= 1) {
        ax[r] += __shfl_xor_sync(0xffffffffu, ax[r], o);
        ay[r] += __shfl_xor_sync(0xffffffffu, ay[r], o);
        az[r] += __shfl_xor_sync(0xffffffffu, az[r], o);
        ph[r] += __shfl_xor_sync(0xffffffffu, ph[r], o);
      }
      const int ti = gi * R + r;
      if (sub == 0 && gi < groups && ti < nt) red_add4(a.far + tb + ti, ax[r], ay[r], az[r], ph[r]);
    }
  }
}

// Lanes per target group for R targets per lane (largest power of two with
// ceil(nt / R) * Gl <= 32), and the work of the busiest lane in units of
// the source count.
__device__ inline void blocked_shape(int nt, int R, int &Gl, float &cost) {
  const int groups = (nt + R - 1) / R;
  Gl = 1;
  while (Gl * 2 * groups <= 32) Gl *= 2;
  const int rounds = (groups + 32 / Gl - 1) / (32 / Gl);
  cost = (float)(rounds * R) / (float)Gl;
}

// The targets [tb, tb + nt) of one cell against its listed sources.
template <int DIM, bool POT>
__device__ __forceinline__ void direct_targets(const DirectArgs &a, const float4 *off, int tb, int nt,
                                               const float4 *s_cell, const int *s_pref, int nsrc, int lane,
                                               float4 *stage) {
  switch (nt) {
    case 1: direct_small<1, DIM, POT>(a, off, tb, nt, s_cell, s_pref, nsrc, lane); return;
    case 2: direct_small<2, DIM, POT>(a, off, tb, nt, s_cell, s_pref, nsrc, lane); return;
    case 3: direct_small<3, DIM, POT>(a, off, tb, nt, s_cell, s_pref, nsrc, lane); return;
    case 4: direct_small<4, DIM, POT>(a, off, tb, nt, s_cell, s_pref, nsrc, lane); return;
    case 5: direct_small<5, DIM, POT>(a, off, tb, nt, s_cell, s_pref, nsrc, lane); return;
    case 6: direct_small<6, DIM, POT>(a, off, tb, nt, s_cell, s_pref, nsrc, lane); return;
    case 7: direct_small<7, DIM, POT>(a, off, tb, nt, s_cell, s_pref, nsrc, lane); return;
    default: break;
  }
  // larger T: the register blocking R in 1..4 that minimises the busiest lane's work (largest R on ties)
  int bestR = 1, bestG = 1;
  float best = 1e30f;
#pragma unroll
  for (int R = 1; R <= 4; ++R) {
    int G;
    float c;
    blocked_shape(nt, R, G, c);
    if (c <= best) {  // ties: the larger R reuses each staged source for more targets
      best = c;
      bestR = R;
      bestG = G;
    }
  }
  switch (bestR) {
    case 1: direct_blocked<1, DIM, POT>(a, off, tb, nt, bestG, s_cell, s_pref, nsrc, lane, stage); break;
    case 2: direct_blocked<2, DIM, POT>(a, off, tb, nt, bestG, s_cell, s_pref, nsrc, lane, stage); break;
    case 3: direct_blocked<3, DIM, POT>(a, off, tb, nt, bestG, s_cell, s_pref, nsrc, lane, stage); break;
    default: direct_blocked<4, DIM, POT>(a, off, tb, nt, bestG, s_cell, s_pref, nsrc, lane, stage); break;
  }
}

template <int DIM, bool POT, bool LIST, bool SPLIT>
__global__ void __launch_bounds__(256, SPLIT ? 3 : DIM == 3 ? 4 : 6) k_direct_far(DirectArgs a) {
  constexpr int NS = DIM == 3 ? 27 : 9, NC = 1 << DIM, NCAND = NS * NC, NR = (NCAND + 31) / 32;
  constexpr int NSRC = DIM == 3 ? 189 : 27;  // interaction-list offsets
  __shared__ float4 s_cell_all[8][NSRC];
  __shared__ int s_pref_all[8][NSRC + 1];
  __shared__ float4 s_stage_all[8][32];
  __shared__ int s_dir_all[8][32];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int64_t wl = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int lv = a.nlev - 1;  // deep levels, which hold most of the warps, first
  int T, part = 0;
  if (SPLIT) {
    if (wl >= *a.nitems) return;
    const int2 it = a.items[wl];
    T = it.x;
    part = it.y;
    while (T < a.cell[lv]) --lv;
  } else {
    if (wl >= a.w0[a.nlev]) return;
    while (wl < a.w0[lv]) --lv;
    const int ci = a.first[lv] + (int)(wl - a.w0[lv]);
    T = LIST ? a.tlist[ci] : ci;
  }
  int tb = a.pbeg[T], nt = a.pend[T] - tb;
  if ((long long)nt > a.direct_max && !a.any_fdirect) return;
  const float4 *off = a.off[lv];
  float4 *s_cell = s_cell_all[wib];
  int *s_pref = s_pref_all[wib];
  const int P = a.parent[T];
  const int cls = (int)(a.ckey[T] & (uint64_t)(NC - 1));
  // kept sources have n_S <= ns_max (n_T n_S <= direct_max)
  const int ns_max = (int)min(a.direct_max, (long long)0x7fffffff) / max(nt, 1);
  int nsrc = 0, ptotal = 0;
  if (lane == 0) s_pref[0] = 0;
  // the existing colleagues, compacted, with their directions packed as
  // (dx+1) | (dy+1) << 2 | (dz+1) << 4 | slot << 8 in s_dir; then the
  // children of those only, all candidate loads in flight at once, child
  // then counts
  int *s_dir = s_dir_all[wib];
  const int Qlane = lane < NS ? a.coll[(size_t)P * NS + lane] : -1;
  const unsigned qmask = __ballot_sync(0xffffffffu, Qlane >= 0);
  if (Qlane >= 0)
    s_dir[__popc(qmask & ((1u << lane) - 1u))] = (lane % 3) | (((lane / 3) % 3) << 2) | ((lane / 9) << 4) | (lane << 8);
  __syncwarp();
  const int ncand = __popc(qmask) * NC;
  int qv[NR], nsv[NR], pbv[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    qv[r] = -1;
    if (r * 32 < ncand) {  // warp-uniform
      const int cand = r * 32 + lane;
      const int Q = __shfl_sync(0xffffffffu, Qlane, cand < ncand ? s_dir[cand / NC] >> 8 : 0);
      if (cand < ncand) qv[r] = a.child[(size_t)Q * NC + (cand % NC)];
    }
  }
  __syncwarp();
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    pbv[r] = qv[r] >= 0 ? a.pbeg[qv[r]] : 0;
    nsv[r] = qv[r] >= 0 ? a.pend[qv[r]] - pbv[r] : 0;
  }
  const float hx = a.h[lv][0], hy = a.h[lv][1], hz = a.h[lv][2];
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    if (r * 32 >= ncand) break;  // warp-uniform
    const int cand = r * 32 + lane;
    const int k = cand % NC, d = cand < ncand ? s_dir[cand / NC] : 0;
    int q = qv[r];
    const int ddx = 2 * ((d & 3) - 1) + (k & 1) - (cls & 1);
    const int ddy = 2 * (((d >> 2) & 3) - 1) + ((k >> 1) & 1) - ((cls >> 1) & 1);
    const int ddz = DIM == 3 ? 2 * (((d >> 4) & 3) - 1) + ((k >> 2) & 1) - ((cls >> 2) & 1) : 0;
    const bool adj = ddx >= -1 && ddx <= 1 && ddy >= -1 && ddy <= 1 && ddz >= -1 && ddz <= 1;
    const bool fd = a.any_fdirect && !adj && a.fdirect[(ddx + 3) + 7 * (ddy + 3) + (DIM == 3 ? 49 * (ddz + 3) : 0)];
    if (q >= 0 && (adj || (nsv[r] > ns_max && !fd))) q = -1;
    const unsigned mask = __ballot_sync(0xffffffffu, q >= 0);
    const int pos = nsrc + __popc(mask & ((1u << lane) - 1u));
    int x = q >= 0 ? nsv[r] : 0;  // inclusive scan of the kept counts
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (q >= 0) {
      // c_S - c_T, and the delta from concatenated position to particle index
      s_cell[pos] = make_float4(ddx * hx, ddy * hy, ddz * hz, __int_as_float(pbv[r] - (ptotal + x - nsv[r])));
      s_pref[pos + 1] = ptotal + x;
    }
    ptotal += __shfl_sync(0xffffffffu, x, 31);
    nsrc += __popc(mask);
  }
  __syncwarp();
  if (nsrc == 0) return;
  if (SPLIT) {
    tb += part * a.chunk;
    nt = min(a.chunk, nt - part * a.chunk);
  }
  if (lane == 0 && a.pair_count) atomicAdd(a.pair_count, (unsigned long long)((long long)nt * ptotal));
  direct_targets<DIM, POT>(a, off, tb, nt, s_cell, s_pref, nsrc, lane, s_stage_all[wib]);
}

// The 2D far field with small thresholds, eight lanes per target cell.  A 2D
// cell has 27 interaction-list offsets, and with 1 to 2 particles per leaf a
// target meets some 40 sources: one warp per cell spent 800 instruction slots
// on 45 pairs, most of them on its two rounds of candidates, on half-empty
// chunks and on the reduction over 32 lanes.  Lane s of an octet takes the
// four children of colleague s (one 16-byte load), lanes 0 .. 3 also one child
// of the ninth; the kept sources are concatenated as in k_direct_far, each
// lane takes every eighth of them for up to four targets in registers.
static constexpr long long FAR2D_MAX = 256;

// Whether a 2D far field takes octets: with leaves of few particles in the
// mean (in larger ones hardly a pair is kept: 23 per leaf 0.030 ms with octets
// and 0.017 with warps), and enough cells, since an octet is busy four times as
// long as a warp with the up to 27 direct_max pairs of a cell (direct_max 256:
// 69,000 cells 0.122 and 0.214 ms, 3,500 cells 0.042 and 0.019; direct_max 17:
// 14,000 cells 0.021 and 0.034, 2,600 cells 0.017 and 0.011).  Thresholds above
// FAR2D_MAX, which nothing sets by itself in 2D, stay with the warps: octets
// still gain a little at 512, lose at 1024 with full leaves and at 4096.
static bool far2d_octets(int64_t n, int64_t nleaves, int64_t ncells, int64_t direct_max) {
  return direct_max <= FAR2D_MAX && n <= SMALL2D_MEAN * nleaves && ncells >= 256 * direct_max;
}

template <int R, bool POT>
__device__ __forceinline__ void far2d_targets(const DirectArgs &a, const float4 *off, int tb, int nt, int t0,
                                              const float4 *s_cell, const int *s_pref, int total, int sub) {
  float tx[R], ty[R], ax[R], ay[R], ph[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const float4 t = nt > 0 ? off[tb + min(t0 + r, nt - 1)] : make_float4(0.f, 0.f, 0.f, 0.f);
    tx[r] = t.x;
    ty[r] = t.y;
    ax[r] = ay[r] = ph[r] = 0.f;
  }
  int si = 0;
  if (t0 < nt)
    for (int f = sub; f < total; f += 8) {
      while (s_pref[si + 1] <= f) ++si;
      const float4 q = shifted_source(off, s_cell, f, si);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float az = 0.f;
        pair_acc<2, false, POT>(tx[r] - q.x, ty[r] - q.y, 0.f, q.w, a.eps2, ax[r], ay[r], az, ph[r]);
      }
    }
  __syncwarp();
#pragma unroll
  for (int r = 0; r < R; ++r) {
#pragma unroll
    for (int o = 4; o; o >>= 1) {
      ax[r] += __shfl_xor_sync(0xffffffffu, ax[r], o);
      ay[r] += __shfl_xor_sync(0xffffffffu, ay[r], o);
      if (POT) ph[r] += __shfl_xor_sync(0xffffffffu, ph[r], o);
    }
    if (sub == r && t0 + r < nt) red_add4(a.far + tb + t0 + r, ax[r], ay[r], 0.f, ph[r]);
  }
}

template <bool POT>
__global__ void __launch_bounds__(256) k_direct_far2d(DirectArgs a) {
  __shared__ float4 s_cell_all[32][27];
  __shared__ int s_pref_all[32][28];
  const int lane = threadIdx.x & 31, sub = lane & 7, oct = threadIdx.x >> 3;
  const int idx = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3);
  float4 *s_cell = s_cell_all[oct];
  int *s_pref = s_pref_all[oct];
  // (octets past the end or with too large a cell go along with no targets)
  bool live = idx < a.w0[a.nlev];
  int lv = a.nlev - 1, tb = 0, nt = 0, P = 0, cls = 0;
  if (live) {
    while (idx < a.w0[lv]) --lv;
    const int T = a.first[lv] + (idx - a.w0[lv]);
    tb = a.pbeg[T];
    nt = a.pend[T] - tb;
    live = nt <= a.direct_max;
    P = a.parent[T];
    cls = (int)(a.ckey[T] & 3);
  }
  const float4 *off = a.off[lv];
  int q[5];
  const int Qa = live ? a.coll[(size_t)P * 9 + sub] : -1, Qb = live && sub < 4 ? a.coll[(size_t)P * 9 + 8] : -1;
  const int4 ch = Qa >= 0 ? reinterpret_cast<const int4 *>(a.child)[Qa] : make_int4(-1, -1, -1, -1);
  q[0] = ch.x;
  q[1] = ch.y;
  q[2] = ch.z;
  q[3] = ch.w;
  q[4] = Qb >= 0 ? a.child[(size_t)Qb * 4 + sub] : -1;
  int pb[5], ns[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    pb[k] = q[k] >= 0 ? a.pbeg[q[k]] : 0;
    ns[k] = q[k] >= 0 ? a.pend[q[k]] - pb[k] : 0;
  }
  const int ns_max = live ? (int)a.direct_max / max(nt, 1) : 0;
  int kept = 0, parts = 0;  // this lane's kept sources and their particles
  int ddx[5], ddy[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const int slot = k < 4 ? sub : 8, c = k < 4 ? k : sub;
    ddx[k] = 2 * (slot % 3 - 1) + (c & 1) - (cls & 1);
    ddy[k] = 2 * (slot / 3 - 1) + ((c >> 1) & 1) - (cls >> 1);
    const bool adj = ddx[k] >= -1 && ddx[k] <= 1 && ddy[k] >= -1 && ddy[k] <= 1;
    if (adj || ns[k] > ns_max) ns[k] = 0;
    kept += ns[k] > 0;
    parts += ns[k];
  }
  int at = kept, x = parts;  // inclusive scans over the octet
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, at, o, 8), z = __shfl_up_sync(0xffffffffu, x, o, 8);
    if (sub >= o) {
      at += y;
      x += z;
    }
  }
  const int total = __shfl_sync(0xffffffffu, x, 7, 8);
  at -= kept;
  x -= parts;
  const float hx = a.h[lv][0], hy = a.h[lv][1];
#pragma unroll
  for (int k = 0; k < 5; ++k)
    if (ns[k] > 0) {
      // c_S - c_T, and the delta from concatenated position to particle index
      s_cell[at] = make_float4(ddx[k] * hx, ddy[k] * hy, 0.f, __int_as_float(pb[k] - x));
      x += ns[k];
      s_pref[++at] = x;
    }
  if (sub == 0) s_pref[0] = 0;
  if (total == 0) nt = 0;
  __syncwarp();
  const int pairs = __reduce_add_sync(0xffffffffu, sub == 0 ? nt * total : 0);
  if (pairs == 0) return;  // warp-uniform
  if (lane == 0 && a.pair_count) atomicAdd(a.pair_count, (unsigned long long)pairs);
  const int most = __reduce_max_sync(0xffffffffu, live ? nt : 0);
  if (!live) nt = 0;
  for (int t0 = 0; t0 < most; t0 += 4)
    switch (min(4, most - t0)) {  // warp-uniform
      case 1: far2d_targets<1, POT>(a, off, tb, nt, t0, s_cell, s_pref, total, sub); break;
      case 2: far2d_targets<2, POT>(a, off, tb, nt, t0, s_cell, s_pref, total, sub); break;
      case 3: far2d_targets<3, POT>(a, off, tb, nt, t0, s_cell, s_pref, total, sub); break;
      default: far2d_targets<4, POT>(a, off, tb, nt, t0, s_cell, s_pref, total, sub); break;
    }
}

// ------------------------------------------------------------------ lists
// The level of cell g in [off[lo], off[D + 1]).
__device__ inline int cell_level(const LevelOffsets &lv, int lo, int D, int g) {
  while (lo < D && g >= lv.off[lo + 1]) ++lo;
  return lo;
}

// List keys (level << dim | class) of the cells of levels 2 .. D: key_all for
// L2L (every cell; null: not wanted), key_m2l for M2L with 255 for cells that
// cannot have an M2L pair under the direct-pair rule (every child S of the
// parent's colleagues has n_T * n_S <= direct_max; adjacency is ignored, so
// the test only errs towards keeping a cell), and with adaptive targets
// (aflag set) for cells that are no target.
//
// A warp takes CW cells: one lane each for the flags and keys, then eight
// lanes per cell that has to be looked at, four cells at a time, over the
// parent's colleagues (one thread each waited for up to 216 loads one after
// another: 130 us of a 4096-particle pass, where there is little else to
// run).  CW = 32 for many cells, of which most need no look (44 M cells of a
// 16M mixture: 2.4 ms with four cells per warp), 4 to spread few cells over
// more warps.
template <int DIM, int CW>
__global__ void k_class_keys(const uint64_t *ckey, const int *cpbeg, const int *cpend, const int *cparent,
                             const int *ccoll, const int *cchild, long long direct_max, LevelOffsets lv, int D,
                             uint8_t *keys_all, uint8_t *keys_m2l, const uint8_t *aflag, int cell0) {
  constexpr int NC = 1 << DIM, NS = DIM == 3 ? 27 : 9;
  const int lane = threadIdx.x & 31, sub = lane & 7, oct = lane >> 3;
  const int first = lv.off[2];
  const int i = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * CW + lane;
  const int g = first + i;
  const bool in = lane < CW && g < lv.off[D + 1];
  const bool target = in && (!aflag || (aflag[g - cell0] & 1));
  unsigned look = direct_max > 0 ? __ballot_sync(0xffffffffu, target) : 0u;
  unsigned m2l = direct_max > 0 ? 0u : __ballot_sync(0xffffffffu, target);
  int nt_me = 0, par_me = 0;
  if (target && direct_max > 0) {
    nt_me = cpend[g] - cpbeg[g];
    par_me = cparent[g];
  }
  while (look) {  // the next four cells, one per octet
    unsigned rest = look;
    for (int q = 0; q < oct; ++q) rest &= rest - 1;
    const int b = __ffs(rest) - 1;  // -1: none left for this octet
    const long long nt = __shfl_sync(0xffffffffu, nt_me, b & 31);
    const int par = __shfl_sync(0xffffffffu, par_me, b & 31);
    const int *pc = ccoll + (int64_t)par * NS;
    bool open = b >= 0, hit = false;
    for (int s0 = 0; s0 < NS; s0 += 8) {
      if (!__any_sync(0xffffffffu, open)) break;
      const int s = s0 + sub;
      bool found = false;
      const int Q = open && s < NS ? pc[s] : -1;
      if (Q >= 0 && nt * (cpend[Q] - cpbeg[Q]) > direct_max) {
        int q[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) q[c] = cchild[(int64_t)Q * NC + c];
#pragma unroll
        for (int c = 0; c < NC; ++c) found |= q[c] >= 0 && nt * (cpend[q[c]] - cpbeg[q[c]]) > direct_max;
      }
      if (__ballot_sync(0xffffffffu, found) & (0xffu << (8 * oct))) {
        hit = true;
        open = false;
      }
    }
    m2l |= __reduce_or_sync(0xffffffffu, hit ? 1u << b : 0u);
#pragma unroll
    for (int q = 0; q < 4; ++q) look &= look - 1;  // (zero stays zero)
  }
  if (in) {
    const uint8_t k = (uint8_t)((cell_level(lv, 2, D, g) << DIM) | (int)(ckey[g] & (NC - 1)));
    if (keys_all) keys_all[i] = k;
    keys_m2l[i] = (m2l >> lane) & 1 ? k : (uint8_t)255;
  }
}

// ------------------------------------------------------------ M shortcut
// Multipoles are formed only for the cells M2L reads (its sources) and for
// its targets (their spectrum is a feature of the learned orders), plus what
// M2M needs to form those.  A needed cell with at most P2M_DIRECT_MAX
// particles, or a leaf, takes its multipole straight from its particles
// (mode 1); a larger one sums its children by M2M (mode 2), which makes all
// of them needed.  mode 0: not formed.
static constexpr int P2M_DIRECT_MAX = 64;

//
// It also marks (needs) every ancestor-or-self at levels >= 2 of the cells
// with M2L contributions (lact): the cells whose local expansion is needed
// below them.
__global__ void k_m_mode(const uint8_t *lact, const uint8_t *msrc, int first2, int leaf_first, int count,
                         const int *parent, const int *pbeg, const int *pend, int cell0, int tmax, uint8_t *mode,
                         int *list1, unsigned *count1, uint8_t *needs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
  const int c = first2 + i;
  if (i < count && lact[c - cell0])
    for (int a = c; a >= first2 && !needs[a - cell0]; a = parent[a])  // stops where another walk already passed
      needs[a - cell0] = 1;
  int md = 0;
  if (i < count) {
    int a = c;
    bool req = lact[a - cell0] || msrc[a - cell0];
    while (!req) {  // needed through a chain of M2M ancestors
      const int P = parent[a];
      if (P < first2 || pend[P] - pbeg[P] <= tmax) break;
      a = P;
      req = lact[a - cell0] || msrc[a - cell0];
    }
    md = !req ? 0 : (c >= leaf_first || pend[c] - pbeg[c] <= tmax) ? 1 : 2;
    mode[c - cell0] = (uint8_t)md;
  }
  // the mode-1 cells, appended a warp at a time (ascending within a warp)
  const unsigned m1 = __ballot_sync(0xffffffffu, md == 1);
  if (m1) {
    unsigned at = 0;
    if (lane == 0) at = atomicAdd(count1, (unsigned)__popc(m1));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (md == 1) list1[at + __popc(m1 & ((1u << lane) - 1u))] = c;
  }
}

// Zeroes the rows (KS floats, KS a multiple of 4) of X of the cells
// [first, first + count) with fx[c] == wx, and those of Y with fy[c] == wy:
// a warp reads the flags of 32 cells at once and stores each flagged row
// with all its lanes.
__global__ void k_zero_rows(const uint8_t *fx, uint8_t wx, float *X, const uint8_t *fy, uint8_t wy, float *Y,
                            int first, int count, int cell0, int KS) {
  const int lane = threadIdx.x & 31;
  const int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t i0 = w0 * 32; i0 < count; i0 += nw * 32) {
    const int64_t i = i0 + lane;
    const int c = first + (int)i;
    const bool in = i < count;
    unsigned mx = __ballot_sync(0xffffffffu, in && fx[c - cell0] == wx);
    unsigned my = __ballot_sync(0xffffffffu, in && fy[c - cell0] == wy);
    while (mx | my) {
      const bool isx = mx != 0;
      unsigned &m = isx ? mx : my;
      const int b = __ffs(m) - 1;
      m &= m - 1;
      float4 *row = reinterpret_cast<float4 *>((isx ? X : Y) + (size_t)(first + (int)i0 + b - cell0) * KS);
      for (int q = lane; q < (KS >> 2); q += 32) row[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
}

// List keys of the cells of levels 2 .. D, two lists of n: the cells that
// need L2L (levels >= 3) by (level, class); the M2M rows, with child_rows
// (tensor-core M2M, rows are children) the children of mode-2 cells by
// (level, class), else (CUDA-core M2M, rows are parents) the mode-2 cells by
// (level, 0).  255: in no list.
__global__ void k_row_keys(const uint64_t *ckey, const uint8_t *needs, const uint8_t *mode, const int *parent,
                           LevelOffsets lv, int D, int dim, int cell0, int child_rows, int n, uint8_t *keys) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int g = lv.off[2] + i, d = cell_level(lv, 2, D, g);
  const int cls = (int)(ckey[g] & ((1u << dim) - 1));
  keys[i] = d >= 3 && needs[g - cell0] ? (uint8_t)((d << dim) | cls) : (uint8_t)255;
  const bool row = child_rows ? d >= 3 && mode[parent[g] - cell0] == 2 : mode[g - cell0] == 2;
  keys[(int64_t)n + i] = row ? (uint8_t)((d << dim) | (child_rows ? cls : 0)) : (uint8_t)255;
}

struct P2MListArgs {
  int nlev;                          // levels 2 .. nlev + 1
  int first[DF_MAX_LEVELS + 1];      // first cell of each level; first[nlev]: end
  const float4 *off[DF_MAX_LEVELS];  // particle offsets from the level's cell centres, mass in w
  float inv_s[DF_MAX_LEVELS];        // 2^level / emax
  const int *pbeg, *pend;
  const int *list;                   // the mode-1 cells
  const unsigned *count;             // their number
  int cell0, p, K, KS;
  int rs;                            // shared-memory row stride: K rounded up to odd
  float *M;
};
static constexpr int P2M_WARPS = 5, P2M_KC = (FMM_MAX_P * FMM_MAX_P + 2 * FMM_MAX_P + 4 + 31) / 32;

// One particle's contributions w R~_l^m (real parts, then -imaginary parts
// as the layout stores them) into a shared-memory row.
template <int P>
__device__ inline void p2m_row(float x, float y, float z, float w, int p, float *row) {
  if (P) p = P;
  const float r2 = x * x + y * y + z * z;
  float dre = 1.f, dim_ = 0.f;
#pragma unroll
  for (int m = 0; m <= p; ++m) {
    if (m > 0) {
      const float h = -0.5f / m;
      const float nre = h * (x * dre - y * dim_), nim = h * (x * dim_ + y * dre);
      dre = nre;
      dim_ = nim;
    }
    float p1re = dre, p1im = dim_, p2re = 0.f, p2im = 0.f;
#pragma unroll
    for (int l = m; l <= p; ++l) {
      float cre, cim;
      if (l == m) {
        cre = dre;
        cim = dim_;
      } else {
        const float a1 = c_rec1[l][m] * z, a2 = c_rec2[l][m] * r2;
        cre = a1 * p1re - a2 * p2re;
        cim = a1 * p1im - a2 * p2im;
        p2re = p1re;
        p2im = p1im;
        p1re = cre;
        p1im = cim;
      }
      row[re_idx(l, m)] = w * cre;
      if (m > 0) row[im_idx(l, m)] = -w * cim;
    }
  }
}

// P2M of the mode-1 cells (their own particles at their own level, no M2M).
// Persistent warps take the list 32 (8 or 16 for short lists) cells at a
// time.  Consecutive cells of at most 32 particles share 32-particle chunks;
// a larger cell takes chunks of its own with a running sum.  In a chunk each
// lane writes the contributions of one particle as a row of a shared-memory
// tile (odd stride: conflict-free), then the lanes sum each cell's rows
// column by column, in particle order, and store the cell's row once,
// padding columns zero (no atomics, no reductions across lanes).  PO > 0:
// the order as a compile-time constant (PO == a.p, the row loops unrolled);
// PO = 0: any order.
template <int PO>
__global__ void __launch_bounds__(32 * P2M_WARPS) k_p2m_list(P2MListArgs a) {
  extern __shared__ float s_tile[];
  // locals, not writes into a (which would copy the parameter block to local memory)
  const int ord = PO ? PO : a.p, K = PO ? (PO + 1) * (PO + 1) : a.K;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  float *S = s_tile + (size_t)wib * 32 * a.rs;
  const unsigned total = *a.count;
  // cells per group: 32, or fewer when the list is short, so that the warps
  // share the work evenly
  const unsigned nw = (unsigned)gridDim.x * P2M_WARPS;
  const unsigned G = total >= nw * 128u ? 32u : total >= nw * 32u ? 16u : 8u;
  for (unsigned g0 = ((unsigned)blockIdx.x * P2M_WARPS + wib) * G; g0 < total; g0 += nw * G) {
    const int gcount = (int)min(G, total - g0);
    const bool has = lane < gcount;
    const int c = has ? a.list[g0 + lane] : 0;
    int pb = 0, n = 0, lv = 0;
    if (has) {
      pb = a.pbeg[c];
      n = a.pend[c] - pb;
      while (lv + 1 < a.nlev && c >= a.first[lv + 1]) ++lv;
    }
    // inclusive prefix of the sizes of the cells of at most 32 particles
    int P = has && n <= 32 ? n : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, P, o);
      if (lane >= o) P += y;
    }
    const unsigned bigmask = __ballot_sync(0xffffffffu, has && n > 32);
    int j = 0;
    while (j < gcount) {  // warp-uniform
      const int nj = __shfl_sync(0xffffffffu, n, j);
      if (nj > 32) {  // a large cell: chunks of 32 with a running sum
        const int cb = __shfl_sync(0xffffffffu, c, j), pbj = __shfl_sync(0xffffffffu, pb, j);
        const int lvj = __shfl_sync(0xffffffffu, lv, j);
        const float4 *off = a.off[lvj];
        const float inv_s = a.inv_s[lvj];
        float acc[P2M_KC];
#pragma unroll
        for (int t = 0; t < P2M_KC; ++t) acc[t] = 0.f;
        for (int e0 = 0; e0 < nj; e0 += 32) {
          const int cnt = min(32, nj - e0);
          const float4 q = lane < cnt ? off[pbj + e0 + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
          p2m_row<PO>(q.x * inv_s, q.y * inv_s, q.z * inv_s, q.w, ord, S + lane * a.rs);
          __syncwarp();
#pragma unroll
          for (int t = 0; t < P2M_KC; ++t) {
            const int col = lane + 32 * t;
            if (col < K)
              for (int r = 0; r < cnt; ++r) acc[t] += S[r * a.rs + col];
          }
          __syncwarp();
        }
        float *mrow = a.M + (size_t)(cb - a.cell0) * a.KS;
#pragma unroll
        for (int t = 0; t < P2M_KC; ++t) {
          const int col = lane + 32 * t;
          if (col < a.KS) mrow[col] = col < K ? acc[t] : 0.f;
        }
        ++j;
        continue;
      }
      // a chunk of consecutive small cells j .. j1 (up to the next large cell)
      const int start = j > 0 ? __shfl_sync(0xffffffffu, P, j - 1) : 0;
      const unsigned after = bigmask & ~(0xffffffffu >> (31 - j));  // large cells after j
      const int jb = after ? __ffs(after) - 1 : gcount;
      const unsigned fit = __ballot_sync(0xffffffffu, lane >= j && lane < jb && P - start <= 32);
      const int j1 = 31 - __clz(fit);
      const int used = __shfl_sync(0xffffffffu, P, j1) - start;
      const int rel = lane >= j && lane <= j1 ? P - n - start : 32;  // each cell's first row
      const unsigned starts = __reduce_or_sync(0xffffffffu, rel < 32 ? 1u << rel : 0u);
      const int myk = j + __popc(starts & (0xffffffffu >> (31 - lane))) - 1;
      const int s0 = __shfl_sync(0xffffffffu, P - n, myk) - start;
      const int mpb = __shfl_sync(0xffffffffu, pb, myk), mlv = __shfl_sync(0xffffffffu, lv, myk);
      const float4 q = lane < used ? a.off[mlv][mpb + lane - s0] : make_float4(0.f, 0.f, 0.f, 0.f);
      const float inv_s = a.inv_s[mlv];
      p2m_row<PO>(q.x * inv_s, q.y * inv_s, q.z * inv_s, q.w, ord, S + lane * a.rs);
      __syncwarp();
      for (int k = j; k <= j1; ++k) {
        const int r0 = __shfl_sync(0xffffffffu, P - n, k) - start, nk = __shfl_sync(0xffffffffu, n, k);
        const int ck = __shfl_sync(0xffffffffu, c, k);
        float *mrow = a.M + (size_t)(ck - a.cell0) * a.KS;
        for (int col = lane; col < a.KS; col += 32) {
          float v = 0.f;
          if (col < K)
            for (int r = r0; r < r0 + nk; ++r) v += S[r * a.rs + col];
          mrow[col] = v;
        }
      }
      __syncwarp();
      j = j1 + 1;
    }
  }
}

// Launches k_p2m_list<P> with its dynamic shared memory (32 rows of rs
// floats per warp), raising the instantiation's limit once per device.
template <int P>
static int launch_p2m_list(const P2MListArgs &pm, cudaStream_t st) {
  const size_t psh = sizeof(float) * (size_t)P2M_WARPS * 32 * pm.rs;
  {
    static std::mutex mu;
    static size_t attr[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return FMM_ERR_CUDA;
    std::lock_guard<std::mutex> lk(mu);
    if (attr[dev] < psh) {
      CUDA_TRY(cudaFuncSetAttribute(k_p2m_list<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)psh));
      CUDA_TRY(cudaFuncSetAttribute(k_p2m_list<P>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                    cudaSharedmemCarveoutMaxShared));
      attr[dev] = psh;
    }
  }
  k_p2m_list<P><<<148 * 2, 32 * P2M_WARPS, psh, st>>>(pm);
  return FMM_OK;
}

// ------------------------------------------------------------ L2L shortcut
// Per leaf: its deepest ancestor-or-self with a needed local expansion.
__global__ void k_leaf_esrc(int leaf_first, int nleaves, int D, int first2, const int *parent, const uint8_t *needs,
                            int cell0, int *esrc, uint8_t *elev) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nleaves) return;
  int c = leaf_first + i, lev = D;
  while (c >= first2 && !needs[c - cell0]) {
    c = parent[c];
    --lev;
  }
  esrc[i] = c >= first2 ? c : -1;
  elev[i] = (uint8_t)(c >= first2 ? lev : 0);
}

// ------------------------------------------------------------ separation
// Offset o = (dx+3) + 7(dy+3) + 49(dz+3) (cells of the box with extents ex):
// the two cells' radii summed over the distance of their centres exceeds
// FMM_RHO_MAX, so their multipole expansion may not converge.
__host__ __device__ inline bool offset_not_well_separated(int o, int dim, double ex, double ey, double ez) {
  if (dim == 2 && o >= 49) return false;  // 2D offsets: (dx+3) + 7(dy+3)
  const int dx = o % 7 - 3, dy = (o / 7) % 7 - 3, dz = dim == 3 ? o / 49 - 3 : 0;
  const double diag2 = ex * ex + ey * ey + (dim == 3 ? ez * ez : 0.0);
  const double dist2 = dx * ex * dx * ex + dy * ey * dy * ey + (dim == 3 ? dz * ez * dz * ez : 0.0);
  return dist2 > 0.0 && sqrt(diag2) > FMM_RHO_MAX * sqrt(dist2);
}

__global__ void k_fdirect_table(int dim, double ex, double ey, double ez, uint8_t *out) {
  const int o = threadIdx.x;
  if (o < 343) out[o] = offset_not_well_separated(o, dim, ex, ey, ez) ? 1 : 0;
}

// ------------------------------------------------------------ pair orders
// FMM_ORDER_GEOMETRIC: for every M2L operator slot (offset D of source from
// target, in cell sizes), the order whose truncation bound rho^(q+1),
// rho = (sum of the two cells' radii) / |D|, matches the closest offset's at
// order p, plus `margin`, clamped to [min(4, p), p]; stored as the padded
// width of that order's expansion length.
__global__ void k_order_table(int dim, int p, int margin, int n_slots, int per_level, float ax, float ay, float az,
                              uint8_t *out) {
  __shared__ float s_ref;
  const float diag = sqrtf(ax * ax + ay * ay + (dim == 3 ? az * az : 0.f));  // radius sum of two cells
  if (threadIdx.x == 0) {
    float ref = 0.f;
    for (int t = 0; t < per_level; ++t) {
      const int dx = t % 7 - 3, dy = (t / 7) % 7 - 3, dz = dim == 3 ? t / 49 - 3 : 0;
      if (max(abs(dx), max(abs(dy), abs(dz))) < 2) continue;  // neighbours never interact by M2L
      const float R = sqrtf(dx * dx * ax * ax + dy * dy * ay * ay + dz * dz * az * az);
      ref = fmaxf(ref, diag / R);
    }
    s_ref = ref;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < n_slots; t += blockDim.x) {
    const int o = t % per_level;
    const int dx = o % 7 - 3, dy = (o / 7) % 7 - 3, dz = dim == 3 ? o / 49 - 3 : 0;
    const float R = sqrtf(dx * dx * ax * ax + dy * dy * ay * ay + dz * dz * az * az);
    const float rho = R > 0.f ? diag / R : 1.f;
    int q = p;
    if (rho < 1.f && s_ref < 1.f && max(abs(dx), max(abs(dy), abs(dz))) >= 2) {
      q = (int)ceilf((p + 1) * logf(s_ref) / logf(rho)) - 1 + margin;
      q = max(min(q, p), min(4, p));
    }
    const int K = dim == 3 ? (q + 1) * (q + 1) : 2 * q + 1;
    out[t] = (uint8_t)((K + 15) & ~15);
  }
}

// Adaptive targets of one level for the direct far field: the cells with
// flag bit 0 that can have direct pairs, appended to seg (warp-aggregated;
// their order within the level is free), their count in *cnt.
__global__ void k_level_targets(const uint8_t *aflag, int cell0, int first, int count, const int *pbeg,
                                const int *pend, long long direct_max, int any_fdirect, int *seg, unsigned *cnt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
  const int g = first + i;
  const bool tgt = i < count && (aflag[g - cell0] & 1) &&
                   ((long long)(pend[g] - pbeg[g]) <= direct_max || any_fdirect);
  const unsigned m = __ballot_sync(0xffffffffu, tgt);
  unsigned base = 0;
  if (lane == 0 && m) base = atomicAdd(cnt, (unsigned)__popc(m));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (tgt) seg[base + __popc(m & ((1u << lane) - 1u))] = g;
}

// FP64 positions in leaf order: xs[i] = pos[perm[i]].
__global__ void k_gather_pos(const double *pos, const uint32_t *perm, int64_t n, int dim, double *xs) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const size_t o = (size_t)perm[i] * dim;
  for (int k = 0; k < dim; ++k) xs[(size_t)i * dim + k] = pos[o + k];
}

// ------------------------------------------------------------ driver

int run_fmm_passes(Workspace &ws, TreeState &t, OpTables &ops, ExpBuffers &eb, const double *d_pos_g,
                   const double *d_mass_g, int p, double eps2, double G,
                   const PassGeom &g, double *d_acc, double *d_pot, int m2l_mode, int64_t direct_max,
                   const OrderOpts &order, cudaStream_t st, fmm_stats &stats, cudaEvent_t *ev,
                   int adaptive_leaf, int p2p_chunk, int m2l_run) {
  const int dim = t.dim, D = t.depth, KS = ops.KS;
  const int64_t n = t.n;
  const bool want_pot = d_pot != nullptr;  // the potential is summed only when it is asked for
  const int ncell = t.n_cells, cell0 = t.cell0;
  const int TPB = 256;
  if (!eb.M.reserve((size_t)ncell * KS) || !eb.L.reserve((size_t)ncell * KS)) return FMM_ERR_OUT_OF_MEMORY;
  // 3D shortcuts: local expansions only on paths to cells with M2L
  // contributions (L2P from each leaf's deepest such ancestor), multipoles
  // only for what M2L reads (P2M straight into small cells, M2M above them);
  // only the rows that are summed into start at zero
  if (!(t.dim == 3 && D >= 3)) {
    CUDA_TRY(cudaMemsetAsync(eb.M.ptr, 0, sizeof(float) * (size_t)ncell * KS, st));
    CUDA_TRY(cudaMemsetAsync(eb.L.ptr, 0, sizeof(float) * (size_t)ncell * KS, st));
  }
  // tensor-core translations: 128-target batches, BF16 split operator images
  const int P16 = (ops.K + 15) & ~15;
  const bool tc = m2l_mode == FMM_M2L_TC && P16 <= TC_MAX_P16;
  const int tchunk = tc ? 128 : CT_TGT;
  const bool split96 = ops.img96 != nullptr;  // M2L tiles up to 96 wide run in a kernel of their own
  // counters that start at zero, in one buffer: bucket sizes of the two list
  // steps, work counters of the tensor-core launches, listed P2M cells, items
  // of the far field
  if (!eb.zeros.reserve(1024 + TC_MAX_LAUNCHES + 2)) return FMM_ERR_OUT_OF_MEMORY;
  CUDA_TRY(cudaMemsetAsync(eb.zeros.ptr, 0, (1024 + TC_MAX_LAUNCHES + 2) * sizeof(uint32_t), st));
  uint32_t *const cls_count = eb.zeros.ptr;
  unsigned int *const tc_work = eb.zeros.ptr + 1024, *const p2m_count = tc_work + TC_MAX_LAUNCHES,
               *const far_items = p2m_count + 1;
  int tc_k = 0;  // tensor-core launches so far (work counter index)
  if (tc && D >= 2) {
    if (2 * D + 2 > TC_MAX_LAUNCHES) return FMM_ERR_UNSUPPORTED;
  }
  const double emax = g.emax > 0 ? g.emax : 1.0;
  const double sD = std::ldexp(emax, -D);
  // offsets whose cells are not well separated for this box (summed
  // directly): flags on the device, and on the host whether there are any
  // (the same FP64 arithmetic, IEEE square roots, so both agree)
  int any_fdirect = 0;
  for (int o = 0; o < 343; ++o)
    if (offset_not_well_separated(o, dim, g.ext[0], g.ext[1], g.ext[2])) {
      const int dd[3] = {o % 7 - 3, (o / 7) % 7 - 3, dim == 3 ? o / 49 - 3 : 0};
      if (std::abs(dd[0]) > 1 || std::abs(dd[1]) > 1 || std::abs(dd[2]) > 1) any_fdirect = 1;
    }
  if (!eb.fdirect.reserve(343)) return FMM_ERR_OUT_OF_MEMORY;
  k_fdirect_table<<<1, 352, 0, st>>>(dim, g.ext[0], g.ext[1], g.ext[2], eb.fdirect.ptr);
  ws.launches += 1;
  const float inv_sD = (float)(1.0 / sD);

  // class-grouped target lists of levels >= 2: the cells with possible M2L
  // pairs (for M2L) and, without the shortcuts (which build their own lists
  // below), every cell (for M2M and L2L) and consecutive M2M parents
  const bool shortcut = dim == 3 && D >= 3;
  // adaptive targets (3D shortcut pass only): flags and the adaptive leaves
  const bool adaptive = shortcut && adaptive_leaf > 0;
  if (adaptive && t.adaptive_leaf != adaptive_leaf) {  // not computed with the tree
    if (!ws.reserve_adaptive(ncell)) return FMM_ERR_OUT_OF_MEMORY;
    int rc = launch_adaptive_flags(ws, t, adaptive_leaf, ws.aflag, ws.alist, st);
    if (rc) return rc;
    ws.launches += 1;
  }
  std::vector<int> lvl_b0(D + 2, 0), lvl_b1(D + 2, 0), m2l_b0(D + 2, 0), m2l_b1(D + 2, 0);
  std::vector<int> m2m_b0(D + 1, 0), m2m_b1(D + 1, 0);
  int ntl = 0;
  const int *tl = nullptr, *tl_m2l = nullptr;
  size_t nhb = 0;
  LevelOffsets lvo{};
  for (int d = 0; d <= D + 1; ++d) lvo.off[d] = t.level_off[d];
  if (D >= 2) {
    ntl = t.level_off[D] + t.level_count[D] - t.level_off[2];
    // lists: every cell (without the shortcuts), then the M2L targets
    const int nlist = shortcut ? 1 : 2;
    if (!eb.tlist.reserve((size_t)nlist * ntl) || !eb.lkey.reserve((size_t)2 * ntl))
      return FMM_ERR_OUT_OF_MEMORY;
    uint8_t *k_all = shortcut ? nullptr : eb.lkey.ptr, *k_m2l = eb.lkey.ptr + (shortcut ? 0 : ntl);
    const int cw = ntl < (1 << 20) ? 4 : 32;
    auto ck_kern = dim == 3 ? (cw == 4 ? k_class_keys<3, 4> : k_class_keys<3, 32>)
                            : (cw == 4 ? k_class_keys<2, 4> : k_class_keys<2, 32>);
    ck_kern<<<cdiv(cdiv(ntl, cw) * (int64_t)32, TPB), TPB, 0, st>>>(ws.cell_key, ws.cell_pbeg, ws.cell_pend, ws.cell_parent,
                                                         ws.cell_coll, ws.cell_child, direct_max, lvo, D, k_all, k_m2l,
                                                         adaptive ? ws.aflag : nullptr, cell0);
    ws.launches += 1;
    // (the counts of the M2L list are read from 256 on)
    bucket_lists(ws, eb.lkey.ptr, nlist, ntl, lvo.off[2], eb.tlist.ptr, cls_count + (shortcut ? 256 : 0), st);
    if (!ws.ok) return FMM_ERR_OUT_OF_MEMORY;
    tl = eb.tlist.ptr;
    tl_m2l = eb.tlist.ptr + (shortcut ? 0 : ntl);
    const uint32_t *hc = ws.host->hist;
    CUDA_TRY(cudaMemcpyAsync(ws.host->hist, cls_count, sizeof(ws.host->hist), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaStreamSynchronize(st));
    const int ncls = 1 << dim;
    // batch count, then the table written straight into pinned staging
    size_t cnt_b = 0;
    for (int pass = shortcut ? 1 : 0; pass < 2; ++pass)
      for (int d = 2; d <= D; ++d)
        for (int c = 0; c < ncls; ++c) cnt_b += ((size_t)hc[256 * pass + ((d << dim) | c)] + tchunk - 1) / tchunk;
    if (!shortcut)
      for (int d = D - 1; d >= 2; --d) cnt_b += ((size_t)t.level_count[d] + tchunk - 1) / tchunk;
    if (!eb.hbatches.reserve(cnt_b + 1, st)) return FMM_ERR_OUT_OF_MEMORY;
    int4 *hb = eb.hbatches.ptr;
    for (int pass = shortcut ? 1 : 0; pass < 2; ++pass) {
      const uint32_t *h = hc + 256 * pass;
      int off = 0;
      for (int d = 2; d <= D; ++d) {
        (pass ? m2l_b0 : lvl_b0)[d] = (int)nhb;
        for (int c = 0; c < ncls; ++c) {
          const int cnt = (int)h[(d << dim) | c];
          for (int s0 = 0; s0 < cnt; s0 += tchunk) hb[nhb++] = make_int4(off + s0, std::min(tchunk, cnt - s0), d, c);
          off += cnt;
        }
        (pass ? m2l_b1 : lvl_b1)[d] = (int)nhb;
      }
    }
    // M2M batches (levels D-1 .. 2, consecutive cells)
    for (int d = D - 1; d >= 2 && !shortcut; --d) {
      m2m_b0[d] = (int)nhb;
      for (int s = 0; s < t.level_count[d]; s += tchunk)
        hb[nhb++] = make_int4(t.level_off[d] + s, std::min(tchunk, t.level_count[d] - s), d, -1);
      m2m_b1[d] = (int)nhb;
    }
  }
  if (!eb.batches.reserve(nhb + 1)) return FMM_ERR_OUT_OF_MEMORY;
  if (nhb)
    CUDA_TRY(cudaMemcpyAsync(eb.batches.ptr, eb.hbatches.ptr, nhb * sizeof(int4), cudaMemcpyHostToDevice, st));

  ContractArgs ca;
  ca.batches = eb.batches.ptr;
  ca.tlist = nullptr;
  ca.tab = ops.tab.ptr;
  ca.cparent = ws.cell_parent;
  ca.cchild = ws.cell_child;
  ca.ccoll = ws.cell_coll;
  ca.cpbeg = ws.cell_pbeg;
  ca.cpend = ws.cell_pend;
  ca.direct_max = direct_max;
  ca.fdirect = any_fdirect ? eb.fdirect.ptr : nullptr;
  ca.src_tab = nullptr;
  ca.slot_list = nullptr;
  ca.nslots_tab = nullptr;
  ca.cell0 = cell0;
  ca.K = ops.K;
  ca.KS = KS;
  ca.KP = ops.KP;
  ca.dim = dim;
  ca.level_stride = dim == 2 ? 49 : 0;
  CUDA_TRY(cudaMemsetAsync(ws.counters, 0, 8 * sizeof(unsigned long long), st));
  TcArgs ta{};
  ta.cchild = ws.cell_child;
  ta.cparent = ws.cell_parent;
  ta.nchild = 1 << dim;
  ta.bimg = ops.img;
  ta.cell0 = cell0;
  ta.K = ops.K;
  ta.KS = KS;
  ta.P16 = P16;
  ta.err = ws.dev_err;
  ta.run_slots = m2l_run;

  uint8_t *lact = nullptr, *needs = nullptr, *msrc = nullptr, *mmode = nullptr;
  if (shortcut) {
    if (!eb.lact.reserve(4 * (size_t)ncell)) return FMM_ERR_OUT_OF_MEMORY;
    CUDA_TRY(cudaMemsetAsync(eb.lact.ptr, 0, 4 * (size_t)ncell, st));
    lact = eb.lact.ptr;
    needs = lact + ncell;
    msrc = lact + 2 * (size_t)ncell;
    mmode = lact + 3 * (size_t)ncell;
  }
  // M2L plan, all levels: the source of every (slot, target) of each batch
  // and, with variable orders, the geometric widths
  ContractArgs cm = ca;
  cm.mode = MODE_M2L;
  cm.slot_base = 0;
  cm.tlist = tl_m2l;
  cm.X = eb.M.ptr;
  cm.Y = eb.L.ptr;
  cm.batches = eb.batches.ptr + m2l_b0[2];
  const int nbm = D >= 2 ? m2l_b1[D] - m2l_b0[2] : 0;
  const bool geometric = tc && order.mode == FMM_ORDER_GEOMETRIC;
  const bool learned = tc && dim == 3 && order.mode == FMM_ORDER_LEARNED && order.params;
  const bool collect = tc && dim == 3 && order.ntiles > 0 && ops.tab64.ptr;
  const bool var_order = geometric || learned;
  const float ax = (float)(g.ext[0] / emax), ay = (float)(g.ext[1] / emax),
              az = (float)(dim == 3 ? g.ext[2] / emax : 0.0);
  if (D >= 2) {
    if (!eb.m2l_src.reserve((size_t)nbm * 189 * tchunk) || !eb.m2l_list.reserve((size_t)nbm * 189) ||
        !eb.m2l_nslots.reserve(nbm) || !eb.m2l_tslot.reserve((size_t)nbm * 189))
      return FMM_ERR_OUT_OF_MEMORY;
    if (var_order && !eb.m2l_w.reserve((size_t)nbm * 189)) return FMM_ERR_OUT_OF_MEMORY;
    if (geometric) {
      if (!eb.order_p16.reserve(ops.n_m2l)) return FMM_ERR_OUT_OF_MEMORY;
      k_order_table<<<1, 256, 0, st>>>(dim, p, order.margin, ops.n_m2l, dim == 3 ? 343 : 49, ax, ay, az,
                                       eb.order_p16.ptr);
      ws.launches += 1;
    }
    if (nbm > 0) {
      // few batches: more threads for each, so that the chains of loads overlap
      k_m2l_sources<<<nbm, nbm < 2 * 148 ? 1024 : 256, 0, st>>>(cm, tchunk, eb.m2l_src.ptr, eb.m2l_list.ptr, eb.m2l_nslots.ptr,
                                         tc ? eb.m2l_tslot.ptr : nullptr, ws.counters,
                                         geometric ? eb.order_p16.ptr : nullptr, geometric ? eb.m2l_w.ptr : nullptr,
                                         ws.counters + 4, lact, msrc, cell0);
      ws.launches += 1;
    }
  }
  // particle offsets from their ancestors' centres, levels 2..D-1 (P2M and
  // L2P shortcuts, direct far field)
  const bool need_lvl_off = D > 2 && (shortcut || direct_max > 0 || any_fdirect);
  if (need_lvl_off) {
    if (!eb.lvl_off.reserve((size_t)n * (D - 2))) return FMM_ERR_OUT_OF_MEMORY;
    auto lo_kern = dim == 3 ? k_level_offsets<3> : k_level_offsets<2>;
    lo_kern<<<cdiv(n, TPB), TPB, 0, st>>>(d_pos_g, d_mass_g, t.d_perm, ws.leaf_of, ws.cell_key, n, D, 2, D - 1,
                                          g.lo[0], g.lo[1], g.lo[2], g.ext[0], g.ext[1], g.ext[2], eb.lvl_off.ptr);
    ws.launches += 1;
  }
  // shortcut lists: the cells that need L2L and the M2M rows, each grouped
  // by (level, class), from one histogram read-back
  const int *tl2 = tl, *tlm = nullptr;
  const int4 *b2 = eb.batches.ptr;
  std::vector<int> l2_b0(lvl_b0), l2_b1(lvl_b1), um_b0(D + 2, 0), um_b1(D + 2, 0);
  if (shortcut) {
    const int first2 = t.level_off[2], leaf_first = t.level_off[D];
    if (!eb.p2m_list.reserve((size_t)ntl)) return FMM_ERR_OUT_OF_MEMORY;
    k_m_mode<<<cdiv(ntl, TPB), TPB, 0, st>>>(lact, msrc, first2, leaf_first, ntl, ws.cell_parent, ws.cell_pbeg,
                                             ws.cell_pend, cell0, P2M_DIRECT_MAX, mmode, eb.p2m_list.ptr,
                                             p2m_count, needs);
    ws.launches += 1;
    // L2L rows: levels 3..D; M2M rows: children at levels 3..D (tensor
    // cores) or the mode-2 parents at levels 2..D-1
    const int m_lo = tc ? 3 : 2, m_hi = tc ? D : D - 1;
    if (!eb.rows.reserve(2 * (size_t)ntl)) return FMM_ERR_OUT_OF_MEMORY;
    k_row_keys<<<cdiv(ntl, TPB), TPB, 0, st>>>(ws.cell_key, needs, mmode, ws.cell_parent, lvo, D, dim, cell0,
                                               tc ? 1 : 0, ntl, eb.lkey.ptr);
    ws.launches += 1;
    bucket_lists(ws, eb.lkey.ptr, 2, ntl, first2, eb.rows.ptr, cls_count + 512, st);
    if (!ws.ok) return FMM_ERR_OUT_OF_MEMORY;
    const uint32_t *hc = ws.host->hist;
    CUDA_TRY(cudaMemcpyAsync(ws.host->hist, cls_count + 512, sizeof(ws.host->hist), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaStreamSynchronize(st));
    const int ncls = 1 << dim;
    size_t cnt_b = 0, nb2 = 0;
    for (int d = 3; d <= D; ++d)
      for (int c = 0; c < ncls; ++c) cnt_b += ((size_t)hc[(d << dim) | c] + tchunk - 1) / tchunk;
    for (int d = m_lo; d <= m_hi; ++d)
      for (int c = 0; c < (tc ? ncls : 1); ++c) cnt_b += ((size_t)hc[256 + ((d << dim) | c)] + tchunk - 1) / tchunk;
    if (!eb.hbatches2.reserve(cnt_b + 1, st)) return FMM_ERR_OUT_OF_MEMORY;
    int4 *hb2 = eb.hbatches2.ptr;
    int off = 0;
    for (int d = 3; d <= D; ++d) {
      l2_b0[d] = (int)nb2;
      for (int c = 0; c < ncls; ++c) {
        const int cnt = (int)hc[(d << dim) | c];
        for (int s0 = 0; s0 < cnt; s0 += tchunk) hb2[nb2++] = make_int4(off + s0, std::min(tchunk, cnt - s0), d, c);
        off += cnt;
      }
      l2_b1[d] = (int)nb2;
    }
    off = 0;
    for (int d = m_lo; d <= m_hi; ++d) {
      um_b0[d] = (int)nb2;
      for (int c = 0; c < (tc ? ncls : 1); ++c) {
        const int cnt = (int)hc[256 + ((d << dim) | c)];
        for (int s0 = 0; s0 < cnt; s0 += tchunk)
          hb2[nb2++] = make_int4(off + s0, std::min(tchunk, cnt - s0), d, tc ? c : -1);
        off += cnt;
      }
      um_b1[d] = (int)nb2;
    }
    if (!eb.batches2.reserve(nb2 + 1)) return FMM_ERR_OUT_OF_MEMORY;
    if (nb2)
      CUDA_TRY(cudaMemcpyAsync(eb.batches2.ptr, hb2, nb2 * sizeof(int4), cudaMemcpyHostToDevice, st));
    tl2 = eb.rows.ptr;
    tlm = eb.rows.ptr + ntl;
    b2 = eb.batches2.ptr;
    if (!eb.esrc.reserve((size_t)t.level_count[D]) || !eb.elev.reserve((size_t)t.level_count[D]))
      return FMM_ERR_OUT_OF_MEMORY;
    k_leaf_esrc<<<cdiv(t.level_count[D], TPB), TPB, 0, st>>>(leaf_first, t.level_count[D], D, first2, ws.cell_parent,
                                                              needs, cell0, eb.esrc.ptr, eb.elev.ptr);
    // rows summed into: M of the M2M cells, L of the cells that need L
    k_zero_rows<<<std::max(1, std::min(cdiv((int64_t)ntl, TPB), 148 * 32)), TPB, 0, st>>>(
        mmode, 2, eb.M.ptr, needs, 1, eb.L.ptr, first2, ntl, cell0, KS);
    ws.launches += 2;
  }

  if (ev) cudaEventRecord(ev[1], st);
  // P2M
  if (shortcut) {
    if (D - 1 > DF_MAX_LEVELS) return FMM_ERR_UNSUPPORTED;
    P2MListArgs pm;
    pm.nlev = D - 1;
    for (int d = 2; d <= D; ++d) {
      pm.first[d - 2] = t.level_off[d];
      pm.off[d - 2] = d == D ? ws.part : eb.lvl_off.ptr + (size_t)(d - 2) * n;
      pm.inv_s[d - 2] = (float)(std::ldexp(1.0, d) / emax);
    }
    pm.first[D - 1] = t.level_off[D] + t.level_count[D];
    pm.pbeg = ws.cell_pbeg;
    pm.pend = ws.cell_pend;
    pm.list = eb.p2m_list.ptr;
    pm.count = p2m_count;
    pm.cell0 = cell0;
    pm.p = p;
    pm.K = ops.K;
    pm.KS = KS;
    pm.rs = ops.K | 1;
    pm.M = eb.M.ptr;
    int ps;
    switch (p) {  // as the L2P
      case 4: ps = launch_p2m_list<4>(pm, st); break;
      case 5: ps = launch_p2m_list<5>(pm, st); break;
      case 6: ps = launch_p2m_list<6>(pm, st); break;
      case 7: ps = launch_p2m_list<7>(pm, st); break;
      case 8: ps = launch_p2m_list<8>(pm, st); break;
      case 9: ps = launch_p2m_list<9>(pm, st); break;
      case 10: ps = launch_p2m_list<10>(pm, st); break;
      case 11: ps = launch_p2m_list<11>(pm, st); break;
      case 12: ps = launch_p2m_list<12>(pm, st); break;
      default: ps = launch_p2m_list<0>(pm, st); break;
    }
    if (ps != FMM_OK) return ps;
  } else if (dim == 3) {
    k_p2m3d<<<cdiv(n, TPB), TPB, 0, st>>>(ws.part, ws.leaf_of, n, cell0, inv_sD, p, KS, eb.M.ptr);
  } else {
    k_p2m2d<<<cdiv(n, TPB), TPB, 0, st>>>(ws.part, ws.leaf_of, n, cell0, inv_sD, p, KS, eb.M.ptr);
  }
  ws.launches += 1;
  // M2M, bottom-up
  for (int d = D - 1; d >= 2 && tc; --d) {  // children of level d + 1 by class
    TcArgs t2 = ta;
    t2.mode = TC_M2M;
    t2.batches = shortcut ? b2 + um_b0[d + 1] : eb.batches.ptr + lvl_b0[d + 1];
    t2.tlist = shortcut ? tlm : tl;
    t2.op_base = ops.off_m2m;
    t2.X = eb.M.ptr;
    t2.Y = eb.M.ptr;
    const int nb = shortcut ? um_b1[d + 1] - um_b0[d + 1] : lvl_b1[d + 1] - lvl_b0[d + 1];
    int rc = tc_launch(t2, nb, tc_work + tc_k++, st, ws.launches);
    if (rc) return rc;
  }
  for (int d = D - 1; d >= 2 && !tc; --d) {  // cells of level d gather their children
    ContractArgs c2 = ca;
    c2.mode = MODE_M2M;
    c2.slot_base = ops.off_m2m;
    c2.tlist = shortcut ? tlm : nullptr;
    c2.X = eb.M.ptr;
    c2.Y = eb.M.ptr;
    c2.batches = shortcut ? b2 + um_b0[d] : eb.batches.ptr + m2m_b0[d];
    const int nb = shortcut ? um_b1[d] - um_b0[d] : m2m_b1[d] - m2m_b0[d];
    int rc = launch_contract(c2, nb, st, ws.launches);
    if (rc) return rc;
  }
  if (ev) cudaEventRecord(ev[2], st);
  // M2L, all levels in one launch
  if (D >= 2) {
    TileArgs tla;
    if (learned || collect) {
      if (!eb.cf.reserve((size_t)ncell * ORD_CF) || !eb.frms.reserve(3)) return FMM_ERR_OUT_OF_MEMORY;
      int rc = order_cell_features(eb.M.ptr, ws.cell_pbeg, ws.cell_pend, t.level_off[2], ntl, cell0, p, KS, mmode,
                                   eb.cf.ptr, ws.part, n, eb.frms.ptr + 2, st, ws.launches);
      if (rc) return rc;
      tla.batches = cm.batches;
      tla.tlist = tl_m2l;
      tla.src_tab = eb.m2l_src.ptr;
      tla.slot_list = eb.m2l_list.ptr;
      tla.tslot_list = eb.m2l_tslot.ptr;
      tla.nslots = eb.m2l_nslots.ptr;
      tla.pbeg = ws.cell_pbeg;
      tla.pend = ws.cell_pend;
      tla.cf = eb.cf.ptr;
      tla.mtot = eb.frms.ptr + 2;
      tla.cell0 = cell0;
      tla.ax = ax;
      tla.ay = ay;
      tla.az = az;
    }
    if (learned && nbm > 0) {
      InferArgs ia;
      ia.t = tla;
      ia.params = order.params;
      ia.frms = eb.frms.ptr;
      ia.nt_sum = ws.counters + 4;
      ia.n = n;
      ia.p = p;
      ia.tol = order.tol;
      ia.emax = emax;
      ia.slot_p16 = eb.m2l_w.ptr;
      int rc = order_infer(ia, nbm, st, ws.launches);
      if (rc) return rc;
    }
    if (collect && nbm > 0) {
      int rc = order_sample_tiles(tla, nbm, order.ntiles, order.seed, order.tiles, order.feat, order.pairs, st,
                                  ws.launches);
      if (!rc) {
        ProbeArgs pa;
        pa.pairs = order.pairs;
        pa.n = order.ntiles * 128;
        pa.pos = d_pos_g;
        pa.mass = d_mass_g;
        pa.perm = t.d_perm;
        pa.pbeg = ws.cell_pbeg;
        pa.pend = ws.cell_pend;
        pa.ckey = ws.cell_key;
        pa.tab64 = ops.tab64.ptr;
        pa.p = p;
        pa.K = ops.K;
        pa.KP = ops.KP;
        for (int k = 0; k < 3; ++k) {
          pa.g.lo[k] = g.lo[k];
          pa.g.ext[k] = g.ext[k];
        }
        pa.g.emax = emax;
        pa.labels = order.pair_labels;
        rc = order_probe_errors(pa, st, ws.launches);
      }
      if (!rc) rc = order_tile_labels(order.pair_labels, order.ntiles, eb.frms.ptr + 2, order.labels, order.feat, st,
                                      ws.launches);
      if (rc) return rc;
    }
    int rc;
    if (tc) {
      TcArgs t2 = ta;
      t2.mode = TC_M2L;
      t2.batches = cm.batches;
      t2.tlist = tl_m2l;
      t2.src_tab = eb.m2l_src.ptr;
      t2.slot_list = eb.m2l_list.ptr;
      t2.tslot_list = eb.m2l_tslot.ptr;
      t2.nslots = eb.m2l_nslots.ptr;
      t2.X = eb.M.ptr;
      t2.Y = eb.L.ptr;
      t2.tiles = ws.counters + 2;
      t2.widths = ws.counters + 5;
      t2.slot_p16 = var_order ? eb.m2l_w.ptr : nullptr;
      if (split96 && nbm > 0) {
        // narrow tiles (w <= 96) in a 96-wide kernel (two CTAs per SM), the others in the 176-wide
        // kernel; both add into L
        const size_t ns = (size_t)nbm * 189;
        if (!eb.m2l_split.reserve(4 * ns + 2 * (size_t)nbm) || !eb.m2l_split_w.reserve(2 * ns))
          return FMM_ERR_OUT_OF_MEMORY;
        int *lo_s = eb.m2l_split.ptr, *lo_t = lo_s + ns, *hi_s = lo_t + ns, *hi_t = hi_s + ns;
        int *lo_n = hi_t + ns, *hi_n = lo_n + nbm;
        uint8_t *lo_w = eb.m2l_split_w.ptr, *hi_w = lo_w + ns;
        rc = tc_split_slots(eb.m2l_list.ptr, eb.m2l_tslot.ptr, eb.m2l_w.ptr, eb.m2l_nslots.ptr, nbm, 96, lo_s, lo_t,
                            lo_w, lo_n, hi_s, hi_t, hi_w, hi_n, st, ws.launches);
        if (!rc) {
          TcArgs lo = t2;
          lo.P16 = 96;
          lo.bimg = ops.img96;
          lo.slot_list = lo_s;
          lo.tslot_list = lo_t;
          lo.slot_p16 = lo_w;
          lo.nslots = lo_n;
          rc = tc_launch(lo, nbm, tc_work + tc_k++, st, ws.launches);
        }
        if (!rc) {
          TcArgs hi = t2;
          hi.slot_list = hi_s;
          hi.tslot_list = hi_t;
          hi.slot_p16 = hi_w;
          hi.nslots = hi_n;
          rc = tc_launch(hi, nbm, tc_work + tc_k++, st, ws.launches);
        }
      } else {
        rc = tc_launch(t2, nbm, tc_work + tc_k++, st, ws.launches);
      }
    } else {
      cm.src_tab = eb.m2l_src.ptr;
      cm.slot_list = eb.m2l_list.ptr;
      cm.nslots_tab = eb.m2l_nslots.ptr;
      rc = launch_contract(cm, nbm, st, ws.launches);
    }
    if (rc) return rc;
  }
  if (ev) cudaEventRecord(ev[3], st);
  // L2L, top-down: every cell of levels >= 3, or with the shortcut only the
  // cells that need a local expansion (their own class-grouped list)
  for (int d = 3; d <= D && tc; ++d) {
    TcArgs t2 = ta;
    t2.mode = TC_L2L;
    t2.batches = b2 + l2_b0[d];
    t2.tlist = tl2;
    t2.op_base = ops.off_l2l;
    t2.X = eb.L.ptr;
    t2.Y = eb.L.ptr;
    int rc = tc_launch(t2, l2_b1[d] - l2_b0[d], tc_work + tc_k++, st, ws.launches);
    if (rc) return rc;
  }
  for (int d = 3; d <= D && !tc; ++d) {
    ContractArgs c2 = ca;
    c2.mode = MODE_L2L;
    c2.slot_base = ops.off_l2l;
    c2.tlist = tl2;
    c2.X = eb.L.ptr;
    c2.Y = eb.L.ptr;
    c2.batches = b2 + l2_b0[d];
    int rc = launch_contract(c2, l2_b1[d] - l2_b0[d], st, ws.launches);
    if (rc) return rc;
  }
  // adaptive targets: the direct far field's targets per level and the
  // colleague-sum items, counted on the device and read back together
  // (timed with the downward pass)
  const unsigned *const ntgt = ws.host->ntgt;
  uint32_t n_items = 0;
  const int cl_chunk = p2p_chunk > 0 ? p2p_chunk : CL_CHUNK_DEFAULT;
  if (adaptive) {
    const int ncl = t.level_off[D] + t.level_count[D] - t.level_off[2];
    if (!eb.ftl.reserve((size_t)ncl + D + 2) || !eb.ccnt.reserve(2 * (size_t)ncell)) return FMM_ERR_OUT_OF_MEMORY;
    unsigned *cnt = (unsigned *)(eb.ftl.ptr + ncl);
    CUDA_TRY(cudaMemsetAsync(cnt, 0, sizeof(unsigned) * (D + 2), st));
    for (int d = 2; d <= D; ++d)
      k_level_targets<<<cdiv(t.level_count[d], TPB), TPB, 0, st>>>(
          ws.aflag, cell0, t.level_off[d], t.level_count[d], ws.cell_pbeg, ws.cell_pend, direct_max,
          any_fdirect, eb.ftl.ptr + (t.level_off[d] - t.level_off[2]), cnt + d);
    const unsigned *acount = (const unsigned *)(ws.alist + ncell);
    uint32_t *ccnt = eb.ccnt.ptr, *coff = eb.ccnt.ptr + ncell;
    k_colleague_count<<<cdiv(ncell, TPB), TPB, 0, st>>>(ws.alist, acount, ncell, ws.cell_coll, ws.cell_pbeg,
                                                         ws.cell_pend, dim == 3 ? 27 : 9, cl_chunk, ccnt);
    exclusive_scan(ws, ccnt, coff, ncell, cnt + D + 1, st);
    if (!ws.ok) return FMM_ERR_OUT_OF_MEMORY;
    ws.launches += D;
    CUDA_TRY(cudaMemcpyAsync(ws.host->ntgt, cnt, sizeof(unsigned) * (D + 2), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaStreamSynchronize(st));
    n_items = ntgt[D + 1];
    if (!eb.citems.reserve((size_t)n_items + 1)) return FMM_ERR_OUT_OF_MEMORY;
    k_colleague_fill<<<cdiv(ncell, TPB), TPB, 0, st>>>(acount, ncell, ccnt, coff, eb.citems.ptr);
    ws.launches += 1;
  }
  // L2P
  if (dim == 3)
    l2p3d_kernel(p, want_pot)<<<cdiv(n, TPB), TPB, 0, st>>>(ws.part, ws.leaf_of, n, cell0, inv_sD, p, KS, eb.L.ptr,
                                                           ws.far, shortcut ? eb.esrc.ptr : nullptr,
                                                           shortcut ? eb.elev.ptr : nullptr, t.level_off[D], D,
                                                           eb.lvl_off.ptr, (float)(1.0 / emax));
  else
    k_l2p2d<<<cdiv(n, TPB), TPB, 0, st>>>(ws.part, ws.leaf_of, n, cell0, inv_sD, p, KS, eb.L.ptr, ws.far);
  ws.launches += 1;
  if (ev) cudaEventRecord(ev[4], st);
  // direct far field, all levels >= 2 (they have interaction lists) in one
  // launch, coarse levels first so that their long warps start early
  if ((direct_max > 0 || any_fdirect) && D >= 2) {
    if (D + 1 > DF_MAX_LEVELS) return FMM_ERR_UNSUPPORTED;
    DirectArgs da;
    da.pbeg = ws.cell_pbeg;
    da.pend = ws.cell_pend;
    da.coll = ws.cell_coll;
    da.parent = ws.cell_parent;
    da.child = ws.cell_child;
    da.ckey = ws.cell_key;
    da.eps2 = (float)eps2;
    da.direct_max = direct_max;
    da.fdirect = eb.fdirect.ptr;
    da.any_fdirect = any_fdirect;
    da.far = ws.far;
    da.pair_count = ws.counters + 3;
    // adaptive targets: each level's targets listed in its own segment of
    // the list (the level's cells in order, gaps after the targets)
    da.tlist = adaptive ? eb.ftl.ptr : nullptr;
    da.nlev = 0;
    // targets per warp where cells are split: few enough that n of them give
    // a few thousand warps, up to the 128 of four targets per lane
    da.chunk = n < (1 << 17) ? 32 : n < (1 << 19) ? 64 : 128;
    int64_t nw = 0;
    int64_t nitems = 0;  // a bound on the items: a level's last parts, then n / chunk full ones
    for (int d = 2; d <= D; ++d) {
      const int k = da.nlev++;
      da.cell[k] = t.level_off[d];
      const double invd = std::ldexp(1.0, -d);
      da.first[k] = adaptive ? t.level_off[d] - t.level_off[2] : t.level_off[d];
      da.w0[k] = (int)nw;
      da.off[k] = d == D ? ws.part : eb.lvl_off.ptr + (size_t)(d - 2) * n;
      da.h[k][0] = (float)(g.ext[0] * invd);
      da.h[k][1] = (float)(g.ext[1] * invd);
      da.h[k][2] = (float)(g.ext[2] * invd);
      const int64_t nc = adaptive ? (int64_t)ntgt[d] : (int64_t)t.level_count[d];
      nw += nc;
      nitems += nc + std::min(n / da.chunk, nc * ((t.level_max[d] - 1) / da.chunk));
    }
    da.w0[da.nlev] = (int)nw;
    if (any_fdirect) {
      if (!eb.fitems.reserve((size_t)nitems)) return FMM_ERR_OUT_OF_MEMORY;
      split_items(ws, adaptive ? ws.aflag : nullptr, cell0, t.level_off[2], t.level_off[D + 1] - t.level_off[2],
                  da.chunk, eb.fitems.ptr, far_items, st);
      if (!ws.ok) return FMM_ERR_OUT_OF_MEMORY;
    }
    da.items = eb.fitems.ptr;
    da.nitems = far_items;
    const int64_t grid = cdiv((any_fdirect ? nitems : nw) * 32, TPB);
    auto pick = [&](auto plain, auto split) { return any_fdirect ? split : plain; };
    void (*kern)(DirectArgs);
    if (adaptive)
      kern = want_pot ? pick(k_direct_far<3, true, true, false>, k_direct_far<3, true, true, true>)
                      : pick(k_direct_far<3, false, true, false>, k_direct_far<3, false, true, true>);
    else if (dim == 3)
      kern = want_pot ? pick(k_direct_far<3, true, false, false>, k_direct_far<3, true, false, true>)
                      : pick(k_direct_far<3, false, false, false>, k_direct_far<3, false, false, true>);
    else
      kern = want_pot ? pick(k_direct_far<2, true, false, false>, k_direct_far<2, true, false, true>)
                      : pick(k_direct_far<2, false, false, false>, k_direct_far<2, false, false, true>);
    // (4M clumped disk, threshold 43: 6.9 -> 2.8 ms)
    const bool octets = dim == 2 && !any_fdirect && far2d_octets(n, t.level_count[D], nw, direct_max);
    if (octets) (want_pot ? k_direct_far2d<true> : k_direct_far2d<false>)<<<cdiv(nw * 8, TPB), TPB, 0, st>>>(da);
    else if (grid > 0) kern<<<(unsigned)grid, TPB, 0, st>>>(da);
    ws.launches += 1;
  }
  if (ev) cudaEventRecord(ev[6], st);
  // P2P + output
  const double inv2D = std::ldexp(1.0, -D);
  P2PArgs pa;
  pa.leaf_first = t.level_off[D];
  pa.nleaves = t.level_count[D];
  pa.depth = D;
  pa.pbeg = ws.cell_pbeg;
  pa.pend = ws.cell_pend;
  pa.coll = ws.cell_coll;
  pa.parent = ws.cell_parent;
  pa.child = ws.cell_child;
  pa.leaf_of = ws.leaf_of;
  pa.ckey = ws.cell_key;
  pa.part = ws.part;
  pa.part_lo = ws.part_lo;
  pa.far = ws.far;
  pa.perm = t.d_perm;
  pa.hx = g.ext[0] * inv2D;
  pa.hy = g.ext[1] * inv2D;
  pa.hz = g.ext[2] * inv2D;
  pa.eps2 = (float)eps2;
  pa.direct_max = direct_max;
  pa.G = G;
  pa.acc = d_acc;
  pa.pot = d_pot;
  pa.err = ws.dev_err;
  pa.pair_count = ws.counters + 1;
  // one warp per leaf, or where the fullest leaf's warp outlasts the kernel one
  // per 16 targets
  pa.parts = 1;
  pa.chunk = t.level_max[D];
  if (near_split(n, pa.nleaves, t.level_max[D])) {
    pa.chunk = 16;
    pa.parts = std::min(cdiv(t.level_max[D], pa.chunk), 16);
  }
  const int pgrid = cdiv((int64_t)pa.nleaves * pa.parts * 32, TPB);
  if (adaptive) {
    // every particle lies in exactly one adaptive leaf: its colleague sums
    // add into far, then every particle's output is written
    if (!eb.xs.reserve((size_t)n * 3)) return FMM_ERR_OUT_OF_MEMORY;
    k_gather_pos<<<cdiv(n, TPB), TPB, 0, st>>>(d_pos_g, t.d_perm, n, dim, eb.xs.ptr);
    const uint32_t *nit = (const uint32_t *)(eb.ftl.ptr + (t.level_off[D] + t.level_count[D] - t.level_off[2])) + D + 1;
    if (n_items > 0) {
      const int cgrid = (int)std::min<int64_t>(cdiv((int64_t)n_items * 32, TPB), 148 * 16);
      if (want_pot) k_colleague_sum<3, true><<<cgrid, TPB, 0, st>>>(pa, ws.alist, eb.citems.ptr, nit, eb.xs.ptr, ws.far,
                                                                  cl_chunk);
      else k_colleague_sum<3, false><<<cgrid, TPB, 0, st>>>(pa, ws.alist, eb.citems.ptr, nit, eb.xs.ptr, ws.far,
                                                                   cl_chunk);
    }
    k_far_output<3><<<cdiv(n, TPB), TPB, 0, st>>>(ws.far, t.d_perm, n, G, d_acc, d_pot, ws.dev_err);
    ws.launches += 3;
  } else if (dim == 2 && near2d_octets(n, pa.nleaves, t.level_max[D])) {
    // (4M clumped disk, 1.6 particles per leaf: 2.05 -> 0.81 ms)
    (want_pot ? k_p2p2d_small<true> : k_p2p2d_small<false>)<<<cdiv((int64_t)pa.nleaves * 8, TPB), TPB, 0, st>>>(pa);
  } else if (dim == 3) {
    if (want_pot) k_p2p<3, true><<<pgrid, TPB, 0, st>>>(pa);
    else k_p2p<3, false><<<pgrid, TPB, 0, st>>>(pa);
  } else {
    if (want_pot) k_p2p<2, true><<<pgrid, TPB, 0, st>>>(pa);
    else k_p2p<2, false><<<pgrid, TPB, 0, st>>>(pa);
  }
  ws.launches += 1;
  if (ev) cudaEventRecord(ev[5], st);
  stats.n_cells = ncell;
  CUDA_TRY(cudaGetLastError());
  return FMM_OK;
}

}  // namespace fmm
