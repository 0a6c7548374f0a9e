// Translations on the 5th-generation tensor cores (tcgen05, sm_100a): M2L,
// M2M and L2L as batched dense contractions.
//
// A CTA takes up to 128 target cells that share their translation slots:
//   M2L  cells of one level and one child class (same interaction offsets),
//        one slot per offset present in the batch;
//   M2M  cells of one level and one child class, one slot: the rows are the
//        children and the results are added into their parents;
//   L2L  cells of one level and one child class, one slot (the parent).
// For each slot it computes D[128 x N] = A_slot[128 x K] * B_slot[K x N],
// where row r of A_slot is the source expansion of target r at that slot
// (zero if absent) and B_slot the slot's operator (transposed), and adds D
// to the running sum R.  D and R live in tensor memory (TMEM), lane r =
// target r; R is written to the targets' expansions at the end.
//
// Precision: every FP32 operand x is split into three BF16 parts
// x = x1 + x2 + x3 (8 significant bits each, 24 in all), and the product is
// the sum of the six split products with total order <= 2
// (x1y1 + x1y2 + x2y1 + x1y3 + x2y2 + x3y1); the dropped terms are below
// 2^-24 relative.  The tensor core's own FP32 accumulation truncates at the
// accumulator's magnitude, so D starts afresh for every slot and takes its
// split products smallest first; R += D is done by the threads in FP32
// (round to nearest), which keeps the contraction at FP32 accuracy.
//
// Pipeline.  Eight worker warps form the A operand and add D to R, one warp
// issues the MMAs, and one streams the operator's BF16 images through four
// shared-memory buffers by bulk asynchronous copies completing on mbarriers
// (part of one split's K rows per copy), so that copies run up to three ahead
// of the MMAs.  The workers prefetch the next slot's source rows into
// registers while the MMAs run, then split them into the A operand once the
// MMAs have released it.
//
// What bounds it: at width 176 the tensor pipe (66 MMAs of N = 176, about
// 5.8 K cycles) and, in series with it, forming A and adding D (3.5 K), about
// 10 K cycles per slot; below that the smaller MMAs are held by their shared-
// memory reads.  Why this split: with one thread of four worker warps issuing
// the MMAs between its own loads a 176-wide slot took 28 K cycles, 18 K of
// them in the issue (134 cycles per MMA, the descriptor arithmetic of a loop
// that was not unrolled) and 4.8 K in forming A and adding D.  Hence an
// issuing thread of its own with descriptors advanced by constants, one MMA
// over all columns (N = w) instead of two halves (A is read once), a copying
// warp and eight warps for the conversions: the M2L phase of the 16M mixture
// at p = 12 with learned orders went from 35.0 to 15.8 ms.  Tried and not
// kept: writing the second and third splits of A while the last product runs
// (17.0 ms: the stores and the MMAs share the shared-memory bandwidth).
//
// Shared-memory operands use the K-major layout without swizzle: 8-row x
// 16-byte core matrices, rows of a core matrix contiguous, 8-row groups
// SBO = 128 B apart and 16-byte K chunks LBO apart.  Every wait on an
// mbarrier gives up after about a second; the kernel then issues nothing more,
// flags the device error word, waits for its MMAs and copies in flight (again
// with a limit), releases its TMEM and returns.
#include <algorithm>
#include <mutex>

#include "m2l_tc.cuh"

namespace fmm {

static constexpr int TC_M = 128;
static constexpr int TC_MAX_SLOTS = 189;

__device__ inline uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// SM100 shared-memory matrix descriptor: start >> 4 [0,14), LBO >> 4
// [16,30), SBO >> 4 [32,46), version 1 [46,48), no swizzle [61,64) = 0.
__device__ inline uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// A thread takes 8 consecutive k of one n: reads coalesced over n, 16-byte
// stores.
__global__ void k_tc_images(const float *tab, int K, int KP, int W, uint16_t *img) {
  const float *T = tab + (size_t)blockIdx.x * K * KP;
  uint16_t *out = img + (size_t)blockIdx.x * 3 * W * W;
  for (int e = threadIdx.x; e < W * (W / 8); e += blockDim.x) {
    const int n = e % W, k0 = (e / W) * 8;
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = (n < K && k0 + q < K) ? T[(size_t)(k0 + q) * KP + n] : 0.f;
    tc_store_image(out, W, n, k0, v);
  }
}

// ------------------------------------------------------------ primitives
__device__ inline void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

// Whether the phase with the given parity has completed (waits a little).
__device__ inline bool mbar_try(uint32_t addr, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred P1;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, P1;\n\t}"
      : "=r"(done)
      : "r"(addr), "r"(parity)
      : "memory");
  return done != 0;
}

// Waits for the completion of the phase with the given parity; false after
// about 2^31 clocks (about a second).
__device__ inline bool mbar_wait(uint64_t *bar, uint32_t parity) {
  const uint32_t addr = smem_u32(bar);
  if (mbar_try(addr, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_try(addr, parity))
    if (clock64() - t0 > (1ll << 31)) return false;
  return true;
}

// Bulk copy global -> shared completing on an mbarrier (no multicast).
__device__ inline void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

__device__ inline void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ inline void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum));
}

// One lane of a converged warp, the same one each time.
__device__ inline bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "elect.sync _|P, 0xffffffff;\n\t"
      "selp.b32 %0, 1, 0, P;\n\t}"
      : "=r"(p));
  return p != 0;
}

__device__ inline void mma_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

__device__ inline void tmem_ld16(uint32_t addr, uint32_t *r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(addr));
}

__device__ inline void tmem_st16(uint32_t addr, const uint32_t *r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15, %16};" ::"r"(addr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

__device__ inline void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ inline void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ------------------------------------------------------------------ kernel
// Persistent: each CTA takes batches from the launch's work counter and runs
// their slots as one stream, so the operator copies and the source-row
// prefetch of the next batch overlap the MMAs of the current one.  Batch
// metadata is double-buffered in shared memory (current, next).
//
// Barriers: s_a (the workers have written A and read D), s_full / s_mma (an
// operator copy has landed in a buffer / its MMAs are done), s_done (the
// slot's MMAs are done), s_drain (after a wait that gave up: all MMAs issued are
// done).  A wait that gives up makes its thread skip the rest of the batch; all
// threads meet at the batch's end and leave together.
static constexpr int TC_WORKERS = 256, TC_THREADS = TC_WORKERS + 64, TC_NBUF = 4;

// CTAs per SM: two where shared memory and TMEM (512 columns) hold them, at
// 96 registers a thread.  (Three of the narrow kernels' at 64 registers
// spilled: 1.26 against 1.10 ms for the 48-wide M2L of a 4M 2D pass.)
__host__ __device__ constexpr int tc_per_sm(int P16) { return P16 <= 96 ? 2 : 1; }

template <int P16>
__global__ void __launch_bounds__(TC_THREADS, tc_per_sm(P16)) k_tc_translate(TcArgs a, int nb, unsigned int *work) {
  constexpr int KH = tc_kpart(P16);  // K rows per operator copy
  constexpr int KC = P16 / 8;       // 16-byte K chunks
  constexpr int ASPLIT = TC_M * P16;
  constexpr int BTILE = KH * P16;
  constexpr uint32_t NCOLS = P16 <= 64 ? 128u : P16 <= 128 ? 256u : 512u;
  constexpr uint32_t RCOL = NCOLS / 2;  // running sum R; D at column 0
  constexpr uint32_t LBO_A = (TC_M / 8) * 128, LBO_B = (P16 / 8) * 128;

  extern __shared__ __align__(1024) uint8_t smem[];
  uint16_t *As = (uint16_t *)smem;  // 3 splits
  uint16_t *Bs = As + 3 * ASPLIT;   // TC_NBUF buffers
  __shared__ __align__(8) uint64_t s_full[TC_NBUF], s_mma[TC_NBUF], s_a, s_done, s_drain;
  __shared__ uint32_t s_tmem;
  __shared__ short s_slot[2][TC_MAX_SLOTS], s_op[2][TC_MAX_SLOTS];  // 16-bit: two 96-wide CTAs fit an SM
  __shared__ uint8_t s_w[2][TC_MAX_SLOTS];  // padded width of each slot's order
  __shared__ int s_n[2], s_b[2];
  __shared__ int s_grab;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // a worker reads D and R at TMEM lane `trow` (a warp reaches the 32 lanes of
  // its index mod 4; warps 0-3 take the even 16-column groups, 4-7 the odd
  // ones) and gathers for A the 16 rows from 16 warp, as rows `grow`
  const int trow = (warp & 3) * 32 + lane, grow = (warp & 7) * 16 + (lane & 15);

  // Takes the next work item with at least one slot into metadata buffer
  // `buf` (s_n[buf] = 0 when the work is exhausted) and sets this thread's
  // targets (rows trow and grow).  An item is a batch, or for M2L a run of up
  // to chunk_slots of its present slots (item = batch * chunks + run).
  const int chunks = a.mode == TC_M2L ? (TC_MAX_SLOTS + a.chunk_slots - 1) / a.chunk_slots : 1;
  // Thread 0 draws the item after the one it hands out, so that nobody waits
  // for the counter; the first item of a CTA is its own index.
  int drawn = (int)blockIdx.x;
  auto load_meta = [&](int buf, int &tg, int &tgg) {
    tg = tgg = -1;
    while (true) {
      if (tid == 0) {
        s_grab = drawn;
        if (drawn < nb * chunks)
          drawn = (int)gridDim.x < nb * chunks ? (int)(gridDim.x + atomicAdd(work, 1u)) : nb * chunks;
      }
      __syncthreads();
      const int item = s_grab;
      if (item >= nb * chunks) {
        if (tid == 0) {
          s_n[buf] = 0;
          s_b[buf] = -1;
        }
        __syncthreads();
        return;
      }
      const int b = item / chunks, s0 = (item % chunks) * a.chunk_slots;
      const int4 bt = a.batches[b];
      int n = 0;
      if (a.mode == TC_M2L) {
        n = max(0, min(a.chunk_slots, a.nslots[b] - s0));
        const size_t tb = (size_t)b * TC_MAX_SLOTS + s0;
        for (int i = tid; i < n; i += TC_THREADS) {
          s_slot[buf][i] = (short)a.slot_list[tb + i];
          s_op[buf][i] = (short)a.tslot_list[tb + i];
          s_w[buf][i] = a.slot_p16 ? a.slot_p16[tb + i] : (uint8_t)P16;
        }
      } else {
        if (tid == 0) {
          s_slot[buf][0] = 0;
          s_op[buf][0] = (short)(a.op_base + bt.w);
          s_w[buf][0] = (uint8_t)P16;
        }
        n = bt.y > 0 ? 1 : 0;
      }
      if (n) {
        if (trow < bt.y) tg = a.tlist ? a.tlist[bt.x + trow] : bt.x + trow;
        if (grow < bt.y) tgg = a.tlist ? a.tlist[bt.x + grow] : bt.x + grow;
      }
      if (tid == 0) {
        s_n[buf] = n;
        s_b[buf] = b;
      }
      __syncthreads();  // also keeps s_grab until everyone has read it
      if (warp == 8 && n && a.mode == TC_M2L && (a.tiles || a.widths)) {
        unsigned ws = 0;
        for (int i = lane; i < n; i += 32) ws += s_w[buf][i];
        ws = __reduce_add_sync(0xffffffffu, ws);
        if (lane == 0 && a.tiles) atomicAdd(a.tiles, (unsigned long long)n);
        if (lane == 0 && a.widths) atomicAdd(a.widths, (unsigned long long)ws);
      }
      if (n) return;
    }
  };

  // Launched while the kernel before it drains (tc_launch_p).  The M2L lists
  // are its predecessor's work; the rows and batches of M2M and L2L and the
  // operators are older (the predecessor itself waited for them), so only the
  // expansions are waited for, below.
  if (a.mode == TC_M2L) asm volatile("griddepcontrol.wait;" ::: "memory");
  int tg_cur, tgg_cur, tg_nxt, tgg_nxt;
  load_meta(0, tg_cur, tgg_cur);
  if (s_n[0] == 0) {
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the launches form a chain: none ends before its predecessor
    return;
  }
  load_meta(1, tg_nxt, tgg_nxt);

  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                 "r"(NCOLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int i = 0; i < TC_NBUF; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&s_mma[i], 1);
    }
    mbar_init(&s_a, TC_WORKERS / 32);
    mbar_init(&s_done, 1);
    mbar_init(&s_drain, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;

  int c = 0;           // metadata buffer of the current batch
  bool ok = true;
  uint32_t sidx = 0;   // slots of the batches before the current one (parity of s_a and s_done)

  if (warp == 9) {
    // ------------------------------------------------------ operator copies
    // Copy g (over all slots of all batches: splits in the order 2, 1, 0, of
    // each the parts of KH of the slot's first w K rows) goes to buffer
    // g % TC_NBUF once the MMAs of copy g - TC_NBUF are done.  Up to TC_NBUF
    // copies of the next batch are issued before the batch ends.
    uint32_t g = 0;
    int ahead = 0;  // copies of the current batch issued during the one before
    auto stream = [&](int buf, int skip, int most) -> int {  // the batch's copies [skip, most)
      int k = 0;
      for (int i = 0; i < s_n[buf]; ++i) {
        const int w = s_w[buf][i], np = (w + KH - 1) / KH;
        if (k + 3 * np <= skip) {
          k += 3 * np;
          continue;
        }
        const uint16_t *img = a.bimg + (size_t)s_op[buf][i] * 3 * P16 * P16;
        for (int s = 2; s >= 0; --s)
          for (int h = 0; h < np; ++h, ++k) {
            if (k < skip) continue;
            if (k >= most) return k;
            const uint32_t b = g % TC_NBUF;
            if (g >= TC_NBUF &&
                !__all_sync(0xffffffffu, mbar_wait(&s_mma[b], ((g / TC_NBUF) - 1) & 1))) {
              ok = false;
              return k;
            }
            if (lane == 0)
              bulk_load(Bs + b * BTILE, img + (size_t)s * P16 * P16 + (size_t)h * KH * P16,
                        (uint32_t)min(w - h * KH, KH) * P16 * 2, &s_full[b]);
            __syncwarp();
            ++g;
          }
      }
      return k;
    };
    while (true) {
      stream(c, ahead, 1 << 30);
      ahead = ok ? stream(c ^ 1, 0, TC_NBUF) : 0;
      const bool mine = ok;
      ok = __syncthreads_and(ok);
      if (!ok) {
        if (!mine && lane == 0) atomicOr(a.err, FMM_DEV_ERR_TIMEOUT);
        break;
      }
      if (s_n[c ^ 1] == 0) break;
      c ^= 1;
      load_meta(c ^ 1, tg_nxt, tgg_nxt);
    }
    if (!ok)  // the last copy into each buffer may still be in flight
      for (uint32_t q = g > TC_NBUF ? g - TC_NBUF : 0; q < g; ++q)
        if (!mbar_wait(&s_full[q % TC_NBUF], (q / TC_NBUF) & 1)) break;
  } else if (warp == 8) {
    // ---------------------------------------------------------------- MMAs
    uint32_t g = 0;  // operator copies consumed
    // A and B descriptors: the high words are constant, the low words hold
    // the address and advance by constants from one K step to the next
    const uint64_t adesc0 = smem_desc(smem_u32(As), LBO_A, 128), bdesc0 = smem_desc(smem_u32(Bs), LBO_B, 128);
    // K steps [0, nk) of A split sa, from K row h KH, against copy q;
    // first: D starts afresh
    auto mma_steps = [&](int sa, int h, uint32_t q, int nk, uint32_t idesc, bool first) {
      const uint64_t ad = adesc0 + (uint32_t)((sa * ASPLIT * 2 + h * (KH / 8) * (int)LBO_A) >> 4);
      const uint64_t bd = bdesc0 + (((q % TC_NBUF) * (uint32_t)(BTILE * 2)) >> 4);
#pragma unroll
      for (int ks = 0; ks < KH / 16; ++ks)
        if (ks < nk)
          mma_bf16(tmem, ad + (uint32_t)(ks * 2 * (int)LBO_A >> 4), bd + (uint32_t)(ks * 2 * (int)LBO_B >> 4), idesc,
                   first && ks == 0 ? 0u : 1u);
    };
    // The products of one slot of width w; false, with nothing more issued, as
    // soon as a wait for a copy gives up.
    auto issue = [&](int w) -> bool {
      const int np = (w + KH - 1) / KH;
      const uint32_t idesc =
          (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(w >> 3) << 17) | ((uint32_t)(TC_M >> 4) << 24);
#pragma unroll
      for (int s = 2; s >= 0; --s)
        for (int h = 0; h < np; ++h, ++g) {
          if (!mbar_wait(&s_full[g % TC_NBUF], (g / TC_NBUF) & 1)) return false;
          const int nk = min(w - h * KH, KH) / 16;
          if (s == 2) {
            mma_steps(0, h, g, nk, idesc, h == 0);
            mma_commit(&s_mma[g % TC_NBUF]);
          } else if (s == 1) {
            mma_steps(1, h, g, nk, idesc, false);
            mma_steps(0, h, g, nk, idesc, false);
            mma_commit(&s_mma[g % TC_NBUF]);
          } else {
            mma_steps(2, h, g, nk, idesc, false);
            mma_steps(1, h, g, nk, idesc, false);
            if (h == np - 1) {  // the largest product (x1 y1) last, over all parts (np <= TC_NBUF: all resident)
              for (int q = 0; q < np; ++q) {
                const uint32_t gq = g - (uint32_t)(np - 1 - q);
                mma_steps(0, q, gq, min(w - q * KH, KH) / 16, idesc, false);
                mma_commit(&s_mma[gq % TC_NBUF]);
              }
              mma_commit(&s_done);
            }
          }
        }
      return true;
    };
    const bool lead = elect_one();
    while (true) {
      const int n = s_n[c];
      // one thread waits and issues, without a warp-wide step in between
      for (int j = 0; lead && j < n && ok; ++j) {
        ok = mbar_wait(&s_a, (sidx + (uint32_t)j) & 1);
        if (!ok) break;
        tc_fence_after();
        ok = issue(s_w[c][j]);
      }
      __syncwarp();
      sidx += (uint32_t)n;
      const bool mine = ok;
      ok = __syncthreads_and(ok);
      if (!ok) {
        if (!mine) atomicOr(a.err, FMM_DEV_ERR_TIMEOUT);
        break;
      }
      if (s_n[c ^ 1] == 0) break;
      c ^= 1;
      load_meta(c ^ 1, tg_nxt, tgg_nxt);
    }
  } else {
    // ------------------------------------------------------------- workers
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    const int half = warp >> 2, r8 = lane & 7;
    // source cell of row `grow` (target tgg) for slot i of metadata buffer
    // `buf`.  The source index of a slot is loaded one slot ahead of its
    // rows, so that only the row loads are left in the window of the MMAs.
    auto src_of = [&](int buf, int i, int tgg) -> int {
      if (tgg < 0) return -1;
      if (a.mode == TC_M2L) return a.src_tab[((size_t)s_b[buf] * TC_MAX_SLOTS + s_slot[buf][i]) * TC_M + grow];
      if (a.mode == TC_M2M) return tgg;
      return a.cparent[tgg];
    };
    // A warp gathers its 16 rows together, in units of 8 columns of one row
    // (32 bytes, one load): the 8 lanes of an octet take 8 rows of one column
    // chunk and the 4 octets consecutive chunks, so that a load instruction
    // reads 8 rows x 128 contiguous bytes, each sector once, and the 16-byte
    // stores of an octet into a core matrix of A fill 128 contiguous bytes.
    // (One row per thread touched 32 lines per instruction, half a sector
    // each.)  Unit 4 u + octet of the slot's 2 (w / 8): row group (unit) /
    // (w / 8), column chunk (unit) % (w / 8).
    float rv[KC / 2][8];
    auto fetch = [&](int w, int src) {
      const int nkc = w >> 3;      // the slot's order needs its first w inputs
      const int kmax = a.KS >> 3;  // chunks that exist in memory (KS is a multiple of 8)
      int kc = lane >> 3, rg = 0;
      while (kc >= nkc) kc -= nkc, ++rg;
#pragma unroll
      for (int u = 0; u < KC / 2; ++u) {
        if (2 * u >= nkc) break;
        const int sr = __shfl_sync(0xffffffffu, src, 8 * rg + r8);
        if (sr >= 0 && kc < kmax) {
          const float *x = a.X + (size_t)(sr - a.cell0) * a.KS + 8 * kc;
          asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                       : "=f"(rv[u][0]), "=f"(rv[u][1]), "=f"(rv[u][2]), "=f"(rv[u][3]), "=f"(rv[u][4]),
                         "=f"(rv[u][5]), "=f"(rv[u][6]), "=f"(rv[u][7])
                       : "l"(x));
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) rv[u][e] = 0.f;
        }
        kc += 4;
        while (kc >= nkc) kc -= nkc, ++rg;
      }
    };
    // A operand of the next slot from the prefetched rows: two values per
    // conversion (cvt.rn.bf16x2.f32).  Columns K..KS-1 of a row are zero in
    // memory and beyond KS the prefetch is zero, so no masking is needed.
    auto write_a = [&](int w) {
      const int nkc = w >> 3;  // the MMAs of a slot of width w read only its first w columns
      int kc = lane >> 3, rg = 0;
      while (kc >= nkc) kc -= nkc, ++rg;
#pragma unroll
      for (int u = 0; u < KC / 2; ++u) {
        if (2 * u >= nkc) break;
        uint32_t h[4], m[4], l[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) split3x2(rv[u][2 * e], rv[u][2 * e + 1], h[e], m[e], l[e]);
        const int off = (kc * (TC_M / 8) + warp * 2 + rg) * 64 + r8 * 8;
        *(uint4 *)(As + off) = make_uint4(h[0], h[1], h[2], h[3]);
        *(uint4 *)(As + ASPLIT + off) = make_uint4(m[0], m[1], m[2], m[3]);
        *(uint4 *)(As + 2 * ASPLIT + off) = make_uint4(l[0], l[1], l[2], l[3]);
        kc += 4;
        while (kc >= nkc) kc -= nkc, ++rg;
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      tc_fence_before();  // D and R of the slot before have been read
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_a);
    };
    const int src0 = src_of(0, 0, tgg_cur);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    fetch(s_w[0][0], src0);
    while (true) {
      const int n = s_n[c];
      // the source index of the next slot to fetch
      int src_nx = n > 1 ? src_of(c, 1, tgg_cur) : s_n[c ^ 1] ? src_of(c ^ 1, 0, tgg_nxt) : -1;
      int wr = 0;  // columns of R written so far
      for (int j = 0; j < n && ok; ++j) {
        const uint32_t si = sidx + (uint32_t)j;
        const int w = s_w[c][j];
        write_a(w);
        // rows of the next slot, in flight during the MMAs
        if (j + 1 < n) {
          fetch(s_w[c][j + 1], src_nx);
          src_nx = j + 2 < n ? src_of(c, j + 2, tgg_cur) : s_n[c ^ 1] ? src_of(c ^ 1, 0, tgg_nxt) : -1;
        } else if (s_n[c ^ 1]) {
          fetch(s_w[c ^ 1][0], src_nx);
        }
        // tcgen05.ld/st are warp-collective: the whole warp goes on only if it saw the commit
        if (!__all_sync(0xffffffffu, mbar_wait(&s_done, si & 1))) {
          ok = false;
          break;
        }
        tc_fence_after();
        // R += D (the slot's first w columns)
#pragma unroll
        for (int c0 = 0; c0 < P16; c0 += 32) {
          const int cc = c0 + 16 * half;
          if (cc < w) {
            uint32_t d[16];
            tmem_ld16(tmem + lane_off + (uint32_t)cc, d);
            if (cc < wr) {
              uint32_t r[16];
              tmem_ld16(tmem + lane_off + RCOL + (uint32_t)cc, r);
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
              for (int e = 0; e < 16; ++e) d[e] = __float_as_uint(__uint_as_float(d[e]) + __uint_as_float(r[e]));
            } else {
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            }
            tmem_st16(tmem + lane_off + RCOL + (uint32_t)cc, d);
          }
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        wr = max(wr, w);
      }
      sidx += (uint32_t)n;
      // epilogue: R into the targets' expansions (fire-and-forget vector
      // reductions; M2M rows of several batches meet in one parent)
      if (ok) {
        const int dst = a.mode == TC_M2M ? (tg_cur >= 0 ? a.cparent[tg_cur] : -1) : tg_cur;
        float *y = a.Y + (size_t)(dst >= 0 ? dst - a.cell0 : 0) * a.KS;
#pragma unroll
        for (int c0 = 0; c0 < P16; c0 += 32) {
          const int cc = c0 + 16 * half;
          if (cc < wr) {
            uint32_t r[16];
            tmem_ld16(tmem + lane_off + RCOL + (uint32_t)cc, r);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (dst >= 0) {
#pragma unroll
              for (int q = 0; q < 4; ++q)
                if (cc + 4 * q < a.KS)
                  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(y + cc + 4 * q), "r"(r[4 * q]),
                               "r"(r[4 * q + 1]), "r"(r[4 * q + 2]), "r"(r[4 * q + 3])
                               : "memory");
            }
          }
        }
      }
      // advance: the next batch becomes current; take the one after it
      const bool mine = ok;
      ok = __syncthreads_and(ok);
      if (!mine && lane == 0) atomicOr(a.err, FMM_DEV_ERR_TIMEOUT);
      if (!ok || s_n[c ^ 1] == 0) break;
      c ^= 1;
      tg_cur = tg_nxt;
      tgg_cur = tgg_nxt;
      load_meta(c ^ 1, tg_nxt, tgg_nxt);
    }
  }

  tc_fence_before();
  __syncthreads();
  // After a wait that gave up, what was issued may still be writing D: it is
  // waited for before the columns are freed (by the same elected thread; here
  // and not where the issuing warp leaves its loop, which cost the M2L 2 %).
  if (warp == 8 && !ok) {
    if (elect_one()) {
      mma_commit(&s_drain);
      mbar_wait(&s_drain, 0);
    }
    __syncwarp();
  }
  if (warp == 8) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(NCOLS));
}

// ------------------------------------------------------------------ host
static size_t tc_dyn_smem(int P16) {
  return (size_t)3 * TC_M * P16 * 2 + (size_t)TC_NBUF * P16 * tc_kpart(P16) * 2;
}

int tc_build_images(const float *tab, int n_slots, int K, int KP, int W, uint16_t *img, cudaStream_t st,
                    int64_t &launches) {
  k_tc_images<<<n_slots, 256, 0, st>>>(tab, K, KP, W, img);
  launches += 1;
  return cudaGetLastError() == cudaSuccess ? FMM_OK : FMM_ERR_CUDA;
}

template <int P16>
static int tc_launch_p(const TcArgs &a, int nb, unsigned int *work, cudaStream_t st) {
  // at most as many CTAs per SM as TMEM has room for
  size_t sh = tc_dyn_smem(P16);
  sh = std::max(sh, P16 <= 64 ? (size_t)60 * 1024 : P16 <= 128 ? (size_t)80 * 1024 : (size_t)120 * 1024);
  // the shared-memory opt-in is per function and device
  static std::mutex mu;
  static size_t attr[64] = {};
  static int per_sm_dev[64] = {};
  int dev = 0, nsm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 ||
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return FMM_ERR_CUDA;
  int per_sm = 0;
  {
    std::lock_guard<std::mutex> lk(mu);
    if (attr[dev] < sh) {
      // the largest shared-memory carveout, so that two CTAs of the narrow
      // kernels fit one SM
      if (cudaFuncSetAttribute(k_tc_translate<P16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh) !=
              cudaSuccess ||
          cudaFuncSetAttribute(k_tc_translate<P16>, cudaFuncAttributePreferredSharedMemoryCarveout,
                               cudaSharedmemCarveoutMaxShared) != cudaSuccess)
        return FMM_ERR_CUDA;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_dev[dev], k_tc_translate<P16>, TC_THREADS, sh) !=
              cudaSuccess ||
          per_sm_dev[dev] < 1)
        return FMM_ERR_CUDA;
      attr[dev] = sh;
    }
    per_sm = per_sm_dev[dev];
  }
  // the narrow kernels' CTAs share an SM whatever the occupancy query says
  // (they take work from a counter, so a CTA that cannot start at once only
  // finds less work)
  per_sm = std::max(per_sm, tc_per_sm(P16));
  // M2L with fewer than four batches per CTA: runs of at most 24 slots as
  // work items, so that the CTAs finish together; fewer slots (down to 4)
  // while there are not four items per CTA
  TcArgs b = a;
  b.chunk_slots = TC_MAX_SLOTS;
  if (a.mode == TC_M2L && nb < 4 * per_sm * nsm)
    b.chunk_slots = std::max(4, std::min(24, (int)((int64_t)nb * TC_MAX_SLOTS / (4 * per_sm * nsm))));
  if (a.mode == TC_M2L && a.run_slots > 0) b.chunk_slots = std::min(a.run_slots, TC_MAX_SLOTS);
  const int chunks = a.mode == TC_M2L ? (TC_MAX_SLOTS + b.chunk_slots - 1) / b.chunk_slots : 1;
  const int grid = std::min(nb * chunks, per_sm * nsm);
  // programmatic launch: the set-up, the metadata and the first operator
  // copies run while the kernel before it drains (a small system's M2M and
  // L2L are a chain of launches of one work item per CTA)
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(TC_THREADS);
  cfg.dynamicSmemBytes = sh;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_tc_translate<P16>, b, nb, work) == cudaSuccess ? FMM_OK : FMM_ERR_CUDA;
}

__global__ void k_tc_split(const int *slot_list, const int *tslot_list, const uint8_t *slot_p16, const int *nslots,
                           int wsplit, int *lo_slot, int *lo_tslot, uint8_t *lo_w, int *lo_n, int *hi_slot,
                           int *hi_tslot, uint8_t *hi_w, int *hi_n) {
  const size_t base = (size_t)blockIdx.x * TC_MAX_SLOTS;
  const int n = nslots[blockIdx.x];
  __shared__ int s_lo, s_hi;
  if (threadIdx.x == 0) s_lo = s_hi = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  // warps take 32 slots at a time, in order, so the compacted lists keep the order
  for (int i0 = 0; i0 < n; i0 += 32) {
    if (threadIdx.x < 32) {
      const int i = i0 + lane;
      const bool ok = i < n;
      const int w = ok ? slot_p16[base + i] : 0;
      const bool lo = ok && w <= wsplit, hi = ok && w > wsplit;
      const unsigned ml = __ballot_sync(0xffffffffu, lo), mh = __ballot_sync(0xffffffffu, hi);
      const unsigned below = (1u << lane) - 1u;
      if (lo) {
        const int at = s_lo + __popc(ml & below);
        lo_slot[base + at] = slot_list[base + i];
        lo_tslot[base + at] = tslot_list[base + i];
        lo_w[base + at] = (uint8_t)w;
      }
      if (hi) {
        const int at = s_hi + __popc(mh & below);
        hi_slot[base + at] = slot_list[base + i];
        hi_tslot[base + at] = tslot_list[base + i];
        hi_w[base + at] = (uint8_t)w;
      }
      __syncwarp();
      if (lane == 0) {
        s_lo += __popc(ml);
        s_hi += __popc(mh);
      }
      __syncwarp();
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    lo_n[blockIdx.x] = s_lo;
    hi_n[blockIdx.x] = s_hi;
  }
}

int tc_split_slots(const int *slot_list, const int *tslot_list, const uint8_t *slot_p16, const int *nslots, int nbm,
                   int wsplit, int *lo_slot, int *lo_tslot, uint8_t *lo_w, int *lo_n, int *hi_slot, int *hi_tslot,
                   uint8_t *hi_w, int *hi_n, cudaStream_t st, int64_t &launches) {
  if (nbm <= 0) return FMM_OK;
  k_tc_split<<<nbm, 32, 0, st>>>(slot_list, tslot_list, slot_p16, nslots, wsplit, lo_slot, lo_tslot, lo_w, lo_n,
                                 hi_slot, hi_tslot, hi_w, hi_n);
  launches += 1;
  return cudaGetLastError() == cudaSuccess ? FMM_OK : FMM_ERR_CUDA;
}

int tc_launch(const TcArgs &a, int nb, unsigned int *work, cudaStream_t st, int64_t &launches) {
  if (nb <= 0) return FMM_OK;
  launches += 1;
  switch (a.P16) {
    case 16: return tc_launch_p<16>(a, nb, work, st);
    case 32: return tc_launch_p<32>(a, nb, work, st);
    case 48: return tc_launch_p<48>(a, nb, work, st);
    case 64: return tc_launch_p<64>(a, nb, work, st);
    case 80: return tc_launch_p<80>(a, nb, work, st);
    case 96: return tc_launch_p<96>(a, nb, work, st);
    case 112: return tc_launch_p<112>(a, nb, work, st);
    case 128: return tc_launch_p<128>(a, nb, work, st);
    case 144: return tc_launch_p<144>(a, nb, work, st);
    case 160: return tc_launch_p<160>(a, nb, work, st);
    case 176: return tc_launch_p<176>(a, nb, work, st);
    default: return FMM_ERR_UNSUPPORTED;
  }
}

}  // namespace fmm
