// Translations (M2L, M2M, L2L) on the 5th-generation tensor cores (tcgen05).
#pragma once
#include <cuda_bf16.h>

#include "tree.cuh"

namespace fmm {

enum { TC_M2L = 0, TC_M2M = 1, TC_L2L = 2 };

// Largest padded expansion length the tensor-core kernel takes (K <= 176:
// 3D p <= 12, 2D p <= 87).
static constexpr int TC_MAX_P16 = 176;

struct TcArgs {
  int mode;                 // TC_M2L, TC_M2M or TC_L2L
  const int4 *batches;      // {tlist offset, count, level, class}, up to 128 cells each
  const int *tlist;         // class-grouped cells: targets (M2L, L2L) or children (M2M)
  const int *src_tab;       // M2L: [batch][slot][128] source cell per target, -1 if none
  const int *slot_list;     // M2L: [batch][i] present slots
  const int *tslot_list;    // M2L: [batch][i] operator-table slot of each present slot
  const int *nslots;        // M2L: [batch]
  const uint8_t *slot_p16;  // M2L: [batch][i] padded width (16 * ceil(K_i / 16)) of each present slot's
                            // order, null = every slot at full order
  const int *cchild;        // children of each cell (nchild per cell, -1 if absent)
  const int *cparent;       // parent of each cell (M2M destination, L2L source)
  int nchild;               // 8 in 3D, 4 in 2D
  int op_base;              // M2M / L2L: operator-table slot of child class 0
  const float *X;           // source expansions, KS floats per cell
  float *Y;                 // target expansions (accumulated into)
  const uint16_t *bimg;     // BF16 split operator images of width P16: 3 * P16^2 per table slot
  int cell0, K, KS, P16;    // P16: width of the kernel, K rounded up to 16 (narrow M2L tiles: less)
  unsigned int *err;
  unsigned long long *tiles;  // M2L: number of (batch, slot) tiles contracted (nullable)
  unsigned long long *widths; // M2L: sum of the tiles' padded widths (nullable)
  int run_slots;            // M2L: slots per work item requested (fmm_config.m2l_run; 0: the launcher's rule)
  int chunk_slots;          // M2L: slots per work item (set by the launcher; a batch of more slots is
                            // split into items whose sums all add into the targets)
};

// K rows of one operator copy: a whole split up to 48, half of it up to 128,
// else a third (four copies and the three A splits fill the shared memory of
// one CTA at 176, and of two at 96).
__host__ __device__ constexpr int tc_kpart(int P16) {
  return P16 <= 48 ? P16 : P16 <= 128 ? ((P16 / 16 + 1) / 2) * 16 : ((P16 / 16 + 2) / 3) * 16;
}

// The three-part BF16 split of two values at once (round to nearest); each
// 32-bit word holds (a, b) with a in the low half.
__device__ inline uint32_t bf2_pack(float a, float b) {
  const __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&t);
}
__device__ inline void split3x2(float a, float b, uint32_t &h, uint32_t &m, uint32_t &l) {
  h = bf2_pack(a, b);
  const float ra = a - __uint_as_float(h << 16), rb = b - __uint_as_float(h & 0xffff0000u);
  m = bf2_pack(ra, rb);
  const float sa = ra - __uint_as_float(m << 16), sb = rb - __uint_as_float(m & 0xffff0000u);
  l = bf2_pack(sa, sb);
}

// Operator image of width W: for each split s, B = T^T (n: output, k: input)
// of the first W rows and columns, W^2 values; element (n, k) at
// ((k/8) * (W/8) + n/8) * 64 + (n%8) * 8 + k%8, so that the first w rows (k)
// are a contiguous prefix.  Stores the inputs k0 .. k0 + 7 of output n.
__device__ inline void tc_store_image(uint16_t *img, int W, int n, int k0, const float *v) {
  uint32_t h[4], m[4], l[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) split3x2(v[2 * q], v[2 * q + 1], h[q], m[q], l[q]);
  const size_t bsplit = (size_t)W * W, at = ((size_t)(k0 / 8) * (W / 8) + n / 8) * 64 + (n % 8) * 8;
  *(uint4 *)(img + at) = make_uint4(h[0], h[1], h[2], h[3]);
  *(uint4 *)(img + bsplit + at) = make_uint4(m[0], m[1], m[2], m[3]);
  *(uint4 *)(img + 2 * bsplit + at) = make_uint4(l[0], l[1], l[2], l[3]);
}

// The images of width W of FP32 matrices tab (K x KP each).
int tc_build_images(const float *tab, int n_slots, int K, int KP, int W, uint16_t *img, cudaStream_t st,
                    int64_t &launches);
// Launches one translation pass over nb batches; `work` is a zeroed device
// counter the persistent CTAs take batches from.
int tc_launch(const TcArgs &a, int nb, unsigned int *work, cudaStream_t st, int64_t &launches);

// Splits the present slots of every M2L batch by padded width: slots with
// w <= wsplit into (lo_*), the others into (hi_*), each [batch][189] with counts.
int tc_split_slots(const int *slot_list, const int *tslot_list, const uint8_t *slot_p16, const int *nslots, int nbm,
                   int wsplit, int *lo_slot, int *lo_tslot, uint8_t *lo_w, int *lo_n, int *hi_slot, int *hi_tslot,
                   uint8_t *hi_w, int *hi_n, cudaStream_t st, int64_t &launches);

// Work counters per pass (one per launch).
static constexpr int TC_MAX_LAUNCHES = 80;

}  // namespace fmm
