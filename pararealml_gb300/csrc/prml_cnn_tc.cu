/*
 * 32 -> 32 channel 3x3 convolutions of the residual CNN on the 5th-generation
 * tensor cores (tcgen05, accumulators in tensor memory).
 *
 * Implicit GEMM: M = 128 pixels (one row segment of one image), K = 32 input
 * channels of one column tap.  One staged input row feeds the (up to) three
 * output rows around it at once: N = 3 x 32 output channels, the weights of
 * the three row taps side by side, accumulated into three neighbouring
 * 32-column accumulators in tensor memory.  So an input row costs 6
 * tcgen05.mma.kind::f16 (bf16 x bf16 -> f32, M128 N96 K16; 3 column taps x 2
 * halves of K).  What bounds a narrow MMA is reading A (128 pixels) from
 * shared memory, not N: 18 MMAs of N = 32 per output row took 1200 cycles a
 * tile and were the bound.  Each output still sums its 9 taps x 2 halves in
 * the same order, from an accumulator that the epilogue left zeroed.  Only
 * MMAs of one shape and accumulator are pipelined in order, so the next input
 * row, whose accumulators lie one row further, waits for this one's MMAs (the
 * commit that frees the row); the other CTA of the SM fills the gap.
 * Measured, a layer of 16 images of 257^2: forward 56 -> 35 us, data gradient
 * 58 -> 39 (135 MB read and written: 20 us), the CTA's chain of row loads,
 * MMAs and epilogue being what is left (35 with the MMAs taken out before); of
 * one image 21 -> 10.
 *
 * Work item: a band of output rows of one 128-pixel column segment (band_rows
 * chooses the band).  A CTA walks down the band; the input rows stream through
 * a ring of 8 staged rows: ONE TMA box load of 130 whole pixels (64 bytes
 * each, zero filled outside the image) with the 64-byte swizzle.  That is the
 * SWIZZLE_64B K-major canonical layout (rows of 64 bytes = all 32 input
 * channels, 8-row groups 512 bytes apart), so the A matrix of column tap dx
 * and K half kk starts at pixel dx, byte 32 kk.  B operand: the packed weights
 * [dx][chunk][row tap, n][8], staged once per CTA (no swizzle).
 *
 * Up to TAIL_W columns left over by the 128-pixel segments (rows of 2^k + 1
 * vertices leave one) are not a segment of their own, which would spend a
 * whole tile per row on them: a tail item is 16 rows x 8 pixels as one M =
 * 128 tile.  Its box of 18 rows x 16 pixels is staged at 1024 bytes a row, so
 * the 8-row groups of the A matrix are 1024 bytes apart and row tap dy is a
 * start one staged row further.  257-wide rows: 3 tiles a row before, 2 1/16
 * now.
 *
 * Roles per CTA (320 threads): warp 8 issues the row loads, warp 9 issues
 * the MMAs into one of eight 32-column TMEM accumulators and releases each
 * row (tcgen05.commit) once its MMAs have been issued, and
 * two epilogue warpgroups (warps 0-3 and 4-7, alternating tiles; warp w reads
 * TMEM lanes 32 (w mod 4) ..) read an accumulator back with tcgen05.ld, apply
 * bias + ReLU (forward) or the ReLU mask of the layer input (data gradient)
 * and store bf16 NHWC.  Every mbarrier wait is bounded: on a timeout the CTA
 * raises a device status flag, drains its in-flight copies and MMAs (again
 * bounded), frees its tensor memory and returns.
 */
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "prml_internal.h"

namespace {

typedef __nv_bfloat16 bf16;

constexpr int HC = 32;                     /* channels in and out */
constexpr int TM = 128;                    /* pixels per tile */
constexpr int SEG = TM + 2;                /* staged pixels per row */
constexpr int PIX_BYTES = HC * 2;          /* one staged pixel: 64 bytes */
constexpr unsigned TX_BYTES = SEG * PIX_BYTES; /* one staged row: 8320 bytes */
/* rows start on 1024-byte boundaries (the swizzle pattern repeats every 512) */
constexpr int ROW_BYTES = (int)((TX_BYTES + 1023) / 1024 * 1024);
constexpr int NROW = 8;                    /* staged-row ring (a power of two) */
constexpr int BAND = 16;                   /* most output rows per work item; rows of a tail item */
constexpr int TAIL_W = 8;                  /* most columns of a tail item */
constexpr int TAIL_SEG = 16;               /* staged pixels per row of a tail item (TAIL_W + 2 used) */
constexpr int TAIL_PITCH = TAIL_SEG * PIX_BYTES;
constexpr unsigned TAIL_TX = (BAND + 2) * TAIL_PITCH;
constexpr int W_BYTES = 9 * 4 * HC * 16;   /* [dx][chunk][dy' n][8], dy' = 2 - dy */
constexpr int W_CHUNK = 3 * HC * 16;       /* bytes of one chunk (8 input channels) of one column tap */
constexpr int NACC = 8;
constexpr int TMEM_COLS = 256;             /* NACC x 32 columns: two CTAs hold an SM's tensor memory */
constexpr int EPI_GROUPS = 2;              /* epilogue warpgroups, alternating tiles */
constexpr int TMA_WARP = 4 * EPI_GROUPS, MMA_WARP = TMA_WARP + 1;
constexpr int THREADS = (MMA_WARP + 1) * 32;
static_assert(NACC % EPI_GROUPS == 0, "each group owns whole accumulators");
constexpr int BAR_BYTES = 384;
constexpr int SMEM_BYTES = NROW * ROW_BYTES + W_BYTES + BAR_BYTES + HC * 4 + 16 + 1024; /* + alignment slack */
constexpr unsigned long long kWaitNs = 2000000000ull; /* 2 s */
static_assert(ROW_BYTES % 1024 == 0, "swizzled TMA destinations start on 1024-byte boundaries");
static_assert((NROW * ROW_BYTES + W_BYTES) % 128 == 0, "weights and barriers aligned");
static_assert((2 * NROW + 2 * NACC + 1) * 8 <= BAR_BYTES, "barrier area");
static_assert(TAIL_TX <= 2 * ROW_BYTES && TAIL_PITCH == 1024, "a tail box fills two ring slots, rows on 1024 bytes");
static_assert(NROW >= 4 && (NROW & (NROW - 1)) == 0, "ring of a power of two >= 4 rows");
static_assert((HC * 16 >> 4) < (1 << 14) && (512 >> 4) < (1 << 14), "descriptor offsets fit 14 bits");
static_assert(NROW * ROW_BYTES + W_BYTES < (1 << 18), "descriptor start fields (addr >> 4, 14 bits) never carry");

/* instruction descriptor, kind::f16: D f32, A bf16, B bf16, both K-major,
 * M = 128, N = 32 blocks */
__device__ __forceinline__ constexpr unsigned idesc(int blocks) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(blocks * (HC >> 3)) << 17) | ((unsigned)(TM >> 4) << 24);
}

__device__ int g_cnn_tc_status;

/* The next launch may start once every CTA of this one has got its tensor
 * memory; nothing global is touched before the previous launch is complete. */
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ unsigned saddr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void bar_init(unsigned long long* b, unsigned n) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(b)), "r"(n) : "memory");
}

__device__ __forceinline__ bool bar_try(unsigned long long* b, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(saddr(b)), "r"(parity)
      : "memory");
  return ok != 0;
}

/* bounded wait; false after kWaitNs */
__device__ __forceinline__ bool bar_wait(unsigned long long* b, unsigned parity) {
  if (bar_try(b, parity)) return true;
  const unsigned long long t0 = now_ns();
  while (!bar_try(b, parity))
    if (now_ns() - t0 > kWaitNs) return false;
  return true;
}

__device__ __forceinline__ void bar_arrive(unsigned long long* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(saddr(b)) : "memory");
}

__device__ __forceinline__ void bar_expect_tx(unsigned long long* b, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(b)), "r"(bytes) : "memory");
}

/* one staged row: box {32, 130, 1, 1} at (0, x, y, b), 64-byte swizzle */
__device__ __forceinline__ void tma_row(void* dst, const CUtensorMap* map, int x, int y, int b,
                                        unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cta.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(saddr(dst)),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(0), "r"(x), "r"(y), "r"(b), "r"(saddr(bar))
      : "memory");
}

/* no-swizzle K-major shared memory descriptor */
__device__ __forceinline__ unsigned long long smem_desc(unsigned addr, unsigned lbo, unsigned sbo) {
  return (unsigned long long)((addr >> 4) & 0x3FFFu) | ((unsigned long long)((lbo >> 4) & 0x3FFFu) << 16) |
         ((unsigned long long)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

/* SWIZZLE_64B K-major descriptor (8-row groups 512 bytes apart).  The
 * swizzle follows the absolute shared-memory address bits, as the TMA
 * writes it, so a start shifted by whole pixels or by 32 bytes inside a row
 * needs no base offset (measured: base offset 0 matches the reference
 * convolution, the address-derived one does not). */
__device__ __forceinline__ unsigned long long smem_desc_sw64(unsigned addr, unsigned sbo = 512u) {
  return (unsigned long long)((addr >> 4) & 0x3FFFu) | (1ull << 16) | ((unsigned long long)(sbo >> 4) << 32) |
         (1ull << 46) | (4ull << 61);
}

__device__ __forceinline__ void mma_f16(unsigned d_tmem, unsigned long long a, unsigned long long b, unsigned id,
                                        unsigned accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(id), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void mma_commit(unsigned long long* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(saddr(bar))
               : "memory");
}

__device__ __forceinline__ void tmem_ld32(unsigned taddr, float (&v)[32]) {
  unsigned r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
      "%13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, "
      "[%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

/* zeroes 32 columns of the warp's 32 lanes */
__device__ __forceinline__ void tmem_zero32(unsigned taddr) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, "
      "%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1};" ::"r"(taddr),
      "r"(0)
      : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

/* Work items of a layer: bands of `band` rows of the 128-pixel segments, then
 * the tail items. */
struct Items {
  int segs, nbands, band, main, groups, total, H, W;
};

struct Item {
  int b, r0, rows, x0; /* image, output rows [r0, r0 + rows), first column */
  bool tail;           /* a tail item: rows x (at most TAIL_W) columns, one tile */
  __device__ __forceinline__ int tiles() const { return tail ? 1 : rows; }
};

__host__ __device__ __forceinline__ Items make_items(int B, int H, int W, int band) {
  Items n;
  const int left = W % TM;
  const bool tail = left >= 1 && left <= TAIL_W;
  n.segs = W / TM + (left && !tail ? 1 : 0);
  n.band = band;
  n.nbands = (H + band - 1) / band;
  n.groups = tail ? (H + BAND - 1) / BAND : 0;
  n.main = B * n.segs * n.nbands;
  n.total = n.main + B * n.groups;
  n.H = H;
  n.W = W;
  return n;
}

/* Rows of a band: the rows a slot takes when all rows of all segments are
 * dealt evenly in as few rounds of at most BAND rows as it takes.  Fixed 16-row
 * bands left a batch of one 257^2 image 51 of the 304 slots busy for 16 rows
 * each (21 us a layer) and 16 images 1.8 rounds. */
int band_rows(int B, int H, int W, int slots) {
  const Items one = make_items(B, H, W, BAND);
  const long long total = (long long)B * H * (one.segs > 0 ? one.segs : 1);
  const long long rounds = (total + (long long)slots * BAND - 1) / ((long long)slots * BAND);
  const long long band = (total + slots * rounds - 1) / (slots * rounds);
  return (int)(band < 1 ? 1 : (band > BAND ? BAND : band));
}

__device__ __forceinline__ Item item_at(int t, const Items& n) {
  Item it;
  it.tail = t >= n.main;
  if (it.tail) {
    t -= n.main;
    it.b = t / n.groups;
    it.r0 = (t - it.b * n.groups) * BAND;
    it.x0 = n.segs * TM;
    it.rows = n.H - it.r0 < BAND ? n.H - it.r0 : BAND;
    return it;
  }
  const int per_img = n.segs * n.nbands;
  it.b = t / per_img;
  const int r = t - it.b * per_img;
  const int band = r / n.segs;
  it.x0 = (r - band * n.segs) * TM;
  it.r0 = band * n.band;
  it.rows = n.H - it.r0 < n.band ? n.H - it.r0 : n.band;
  return it;
}

/* MODE 0: y = relu(conv(x, w) + bias).  MODE 1: y = conv(x, w) * (mask > 0).
 * w: [tap][n][k] bf16 (n = output channel). */
template <int MODE>
__global__ void __launch_bounds__(THREADS, 2) mid_conv_tc(const __grid_constant__ CUtensorMap xmap,
                                                          const __grid_constant__ CUtensorMap tmap,
                                                          const bf16* __restrict__ w,
                                                          const float* __restrict__ bias,
                                                          const bf16* __restrict__ mask, bf16* __restrict__ y,
                                                          const Items n) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* base = smem_raw + ((1024u - (saddr(smem_raw) & 1023u)) & 1023u);
  unsigned char* rows = base;
  unsigned char* wsm = base + NROW * ROW_BYTES;
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(wsm + W_BYTES);
  unsigned long long* full = bars;                 /* [NROW] */
  unsigned long long* empty = bars + NROW;         /* [NROW] */
  unsigned long long* accfull = bars + 2 * NROW;   /* [NACC] */
  unsigned long long* accempty = accfull + NACC;   /* [NACC] */
  unsigned long long* done = accempty + NACC;      /* all MMAs complete */
  float* bias_s = reinterpret_cast<float*>(wsm + W_BYTES + BAR_BYTES);
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(bias_s + HC);
  __shared__ int abort_flag;
  __shared__ int loads_issued;  /* row loads issued by the producer */
  __shared__ int loads_waited;  /* row loads the MMA warp has seen land */

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int s = 0; s < NROW; ++s) {
      bar_init(&full[s], 1);
      bar_init(&empty[s], 1);
    }
    for (int a = 0; a < NACC; ++a) {
      bar_init(&accfull[a], 1);
      bar_init(&accempty[a], 4 * 32);
    }
    bar_init(done, 1);
    abort_flag = 0;
    loads_issued = 0;
    loads_waited = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(tmem_slot)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = *tmem_slot;
  if (warp < 4)
    for (int a = 0; a < NACC; ++a) tmem_zero32(tmem + ((unsigned)(warp * 32) << 16) + (unsigned)(a * HC));
  let_next_start();
  wait_previous();

  /* weights [dy][dx][n][k] -> [dx][chunk][2 - dy][n][8], bias */
  for (int i = tid; i < 9 * HC * 4; i += THREADS) {
    const int tap = i / (HC * 4), rem = i - tap * HC * 4, co = rem >> 2, c = rem & 3;
    const uint4 v = *reinterpret_cast<const uint4*>(w + (tap * HC + co) * HC + c * 8);
    *reinterpret_cast<uint4*>(wsm + (((tap % 3) * 4 + c) * 3 * HC + (2 - tap / 3) * HC + co) * 16) = v;
  }
  if (MODE == 0 && tid < HC) bias_s[tid] = bias[tid];
  /* generic-proxy weight stores must be visible to the tensor cores */
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  if (warp == TMA_WARP) {
    /* ---- row loads; a tail box takes two ring slots, the first one even
     * (the slot skipped for that completes without a copy) */
    if (lane == 0) {
      int L = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < n.total && ok; t += gridDim.x) {
        const Item it = item_at(t, n);
        const int loads = it.tail ? 2 + (L & 1) : it.rows + 2;
        for (int j = 0; j < loads; ++j, ++L) {
          const int q = L % NROW;
          unsigned char* dst = rows + q * ROW_BYTES;
          ok = bar_wait(&empty[q], ((L / NROW) & 1) ^ 1) && !*(volatile int*)&abort_flag &&
               (saddr(dst) & 1023u) == 0; /* the last test: never issue a misaligned copy */
          if (ok && it.tail && loads - j == 2) /* the box also writes the next slot */
            ok = bar_wait(&empty[q + 1], (((L + 1) / NROW) & 1) ^ 1);
          if (!ok) break;
          if (!it.tail) {
            bar_expect_tx(&full[q], TX_BYTES);
            tma_row(dst, &xmap, it.x0 - 1, it.r0 - 1 + j, it.b, &full[q]);
          } else if (loads - j == 2) {
            bar_expect_tx(&full[q], TAIL_TX);
            tma_row(dst, &tmap, it.x0 - 1, it.r0 - 1, it.b, &full[q]);
          } else {
            bar_arrive(&full[q]);
          }
          loads_issued = L + 1;
        }
      }
      if (!ok) atomicExch(&abort_flag, 1);
    }
  } else if (warp == MMA_WARP) {
    /* ---- MMA issuer */
    if (lane == 0) {
      const unsigned wbase = saddr(wsm);
      int L = 0, T = 0; /* ring slots and accumulators used so far */
      bool ok = (wbase & 15u) == 0;
      /* descriptors are linear in the start address (field = addr >> 4, no
       * carry for shared addresses): ring slots are ROW_BYTES apart */
      const unsigned long long adesc0 = smem_desc_sw64(saddr(rows));
      const unsigned long long tdesc0 = smem_desc_sw64(saddr(rows), TAIL_PITCH);
      const unsigned long long bdesc = smem_desc(wbase, W_CHUNK, 128);
      auto landed = [&](int l) {
        if (!bar_wait(&full[l % NROW], (l / NROW) & 1)) return false;
        loads_waited = l + 1;
        return true;
      };
      auto acc_free = [&](int a) {
        return bar_wait(&accempty[a % NACC], ((a / NACC) & 1) ^ 1) && !*(volatile int*)&abort_flag;
      };
      /* column tap dx, K half kk of one A row for row-tap blocks [blk, blk + cnt) into the accumulator of tile a */
      auto mma = [&](unsigned long long ar, int dx, int kk, int a, int blk, int cnt) {
        mma_f16(tmem + (unsigned)((a % NACC) * HC), ar + (unsigned long long)((dx * PIX_BYTES + kk * 32) >> 4),
                bdesc + (unsigned long long)(((dx * 4 + 2 * kk) * W_CHUNK + blk * HC * 16) >> 4), idesc(cnt), 1u);
      };
      for (int t = blockIdx.x; t < n.total && ok; t += gridDim.x) {
        const Item it = item_at(t, n);
        if (it.tail) {
          if (L & 1) {
            if (!(ok = landed(L))) break;
            bar_arrive(&empty[L % NROW]);
            ++L;
          }
          ok = landed(L) && landed(L + 1) && acc_free(T);
          if (!ok) break;
          tc_fence_after();
          const unsigned long long ar = tdesc0 + (unsigned long long)((L % NROW) * (ROW_BYTES >> 4));
#pragma unroll
          for (int tap = 0; tap < 9; ++tap)
#pragma unroll
            for (int kk = 0; kk < 2; ++kk)
              mma(ar + (unsigned long long)((tap / 3) * (TAIL_PITCH >> 4)), tap % 3, kk, T, 2 - tap / 3, 1);
          mma_commit(&accfull[T % NACC]);
          mma_commit(&empty[L % NROW]);
          mma_commit(&empty[(L + 1) % NROW]);
          L += 2;
          ++T;
          continue;
        }
        for (int j = 0; j < it.rows + 2 && ok; ++j, ++L) {
          /* input row j feeds output rows lo .. hi of the band: row i through
           * row tap j - i, weight block 2 - (j - i) */
          const int lo = j > 2 ? j - 2 : 0, hi = j < it.rows ? j : it.rows - 1;
          ok = landed(L) && (j >= it.rows || acc_free(T + j)) &&
               (j == 0 || bar_wait(&empty[(L - 1) % NROW], ((L - 1) / NROW) & 1));
          if (!ok) break;
          tc_fence_after();
          const unsigned long long ar = adesc0 + (unsigned long long)((L % NROW) * (ROW_BYTES >> 4));
          /* their accumulators may wrap around the ring */
          const int blk = 2 - (j - lo), cnt = hi - lo + 1, room = NACC - (T + lo) % NACC;
          const int c0 = cnt < room ? cnt : room;
#pragma unroll
          for (int k = 0; k < 6; ++k) {
            mma(ar, k >> 1, k & 1, T + lo, blk, c0);
            if (c0 < cnt) mma(ar, k >> 1, k & 1, T + lo + c0, blk + c0, cnt - c0);
          }
          if (j >= 2) mma_commit(&accfull[(T + j - 2) % NACC]); /* that output row is complete */
          mma_commit(&empty[L % NROW]);
        }
        T += it.rows;
      }
      if (!ok) atomicExch(&abort_flag, 1);
      mma_commit(done); /* arrives once every MMA issued above has completed */
      bar_wait(done, 0);
    }
  } else {
    /* ---- epilogue: group g takes the tiles T with T mod EPI_GROUPS == g;
     * warp w owns TMEM lanes 32 (w mod 4) .. = tile pixels */
    const int group = warp >> 2, wq = warp & 3;
    int T = 0;
    bool go = true;
    for (int t = blockIdx.x; t < n.total && go; t += gridDim.x) {
      const Item it = item_at(t, n);
      const int tiles = it.tiles();
      for (int i = 0; i < tiles; ++i, ++T) {
        if (T % EPI_GROUPS != group) continue;
        const int a = T % NACC;
        const bool ok = bar_wait(&accfull[a], (T / NACC) & 1);
        if (__any_sync(0xffffffffu, !ok) || *(volatile int*)&abort_flag) {
          atomicExch(&abort_flag, 1);
          go = false;
          break;
        }
        tc_fence_after();
        float v[32];
        const unsigned acc = tmem + ((unsigned)(wq * 32) << 16) + (unsigned)(a * HC);
        tmem_ld32(acc, v);
        tmem_zero32(acc); /* the next tile's first products add to zero */
        tc_fence_before();
        bar_arrive(&accempty[a]);
        const int m = wq * 32 + lane;
        const int gx = it.x0 + (it.tail ? m % TAIL_W : m), gy = it.tail ? m / TAIL_W : i;
        if (gx < n.W && gy < it.rows) {
          const long long p = ((long long)it.b * n.H + it.r0 + gy) * n.W + gx;
          if (MODE == 0) {
#pragma unroll
            for (int k = 0; k < 32; ++k) v[k] = fmaxf(v[k] + bias_s[k], 0.f);
          } else {
            const uint4* mp = reinterpret_cast<const uint4*>(mask + p * HC);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const uint4 m = mp[q];
              const __nv_bfloat162* mh = reinterpret_cast<const __nv_bfloat162*>(&m);
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float2 f = __bfloat1622float2(mh[j]);
                if (!(f.x > 0.f)) v[q * 8 + 2 * j] = 0.f;
                if (!(f.y > 0.f)) v[q * 8 + 2 * j + 1] = 0.f;
              }
            }
          }
          uint4* yp = reinterpret_cast<uint4*>(y + p * HC);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint4 o;
            __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
            for (int j = 0; j < 4; ++j) oh[j] = __floats2bfloat162_rn(v[q * 8 + 2 * j], v[q * 8 + 2 * j + 1]);
            yp[q] = o;
          }
        }
      }
    }
  }

  /* ---- drain (bounded) and free tensor memory */
  __syncthreads();
  if (abort_flag) {
    if (tid == 0) atomicExch(&g_cnn_tc_status, 1);
    if (warp == TMA_WARP && lane == 0) {
      /* row loads issued but never seen by the MMA warp */
      for (int j = loads_waited; j < loads_issued; ++j) bar_wait(&full[j % NROW], (j / NROW) & 1);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
}

/* ---- weight and bias gradient of the 32 -> 32 convolutions ------------------
 * dW[dy][dx][co][ci] = sum over pixels p of g[p][co] x[p + (dy - 1, dx - 1)][ci]
 * (x zero outside the image) as tcgen05 MMAs whose K is pixels.  D (M = 128,
 * f32 in TMEM) row 32 j + ci holds the column shift j - 1 of input channel ci;
 * j = 3 (a shift of +2) is computed and discarded, so one MMA covers a kernel
 * row's three taps.  One staged input row meets the (up to) three gradient
 * rows around it at once: N = 3 x 32 output channels, one 32-column
 * accumulator per kernel row (dy in columns 32 (2 - dy) ..), so an input row
 * costs 8 MMAs of N = 96 where an output row took 24 of N = 32.  Both operands
 * are the staged NHWC rows read MN-major with the 64-byte swizzle (a pixel's
 * 32 channels are one 64-byte row of a swizzle atom, 8 pixels one 512-byte
 * atom): A = the input row from one pixel left of the K block, its four 32-row
 * MN blocks one pixel (64 bytes, the leading byte offset) apart, 8-pixel K
 * groups 512 bytes (the stride byte offset) apart; B = gradient rows, MN
 * blocks one ring slot apart.  A tail item (16 rows x 8 pixels) is one K of
 * 128 pixels: its 8-pixel groups are rows, 1024 bytes apart in A.
 * A CTA walks items as the convolution does, accumulates over all of them, and
 * writes its partial dW [tap][co][ci] and bias sums once at the end.  Roles:
 * warp 4 loads rows (input rows through a ring of WG_NX, gradient rows through
 * a ring of WG_NG), warp 5 issues the MMAs, warps 0-3 sum the staged gradient
 * rows per channel (a pass of its own over the gradient took 20 us of a
 * layer's 90 at 16 x 257^2) and read the accumulators back.  Waits are bounded
 * as in the convolution.
 * Measured, 16 images of 257^2: 56 -> 35 us, and 36 us of four more launches
 * (bias pass, two reductions, transposition) became 7 (reduce_wgrad). */
constexpr int WG_G_BYTES = TM * PIX_BYTES; /* one gradient row, 8192 bytes */
constexpr int WG_NX = 4, WG_NG = 8;
constexpr int WG_PART = 9 * HC * HC + HC;  /* floats of a CTA's partial: dW, then the bias sums */
constexpr int WG_TMEM_COLS = 128;          /* 3 x 32 used */
constexpr int WG_TMA_WARP = 4, WG_MMA_WARP = 5;
constexpr int WG_THREADS = 6 * 32;
/* + alignment slack + room for reads of the discarded shift past a row */
constexpr int WG_SMEM = WG_NX * ROW_BYTES + WG_NG * WG_G_BYTES + BAR_BYTES + 1024 + 2048;
constexpr unsigned kMnMajor = (1u << 15) | (1u << 16); /* A and B MN-major */
static_assert(WG_G_BYTES % 1024 == 0, "gradient rows start on 1024-byte boundaries");
static_assert((2 * WG_NX + 2 * WG_NG + 1) * 8 <= BAR_BYTES, "barrier area");
static_assert(BAND * TAIL_W * PIX_BYTES == WG_G_BYTES, "a tail item's gradient fills one slot");
static_assert(WG_NX * ROW_BYTES + WG_NG * WG_G_BYTES + BAR_BYTES < (1 << 18), "descriptor start fields never carry");

/* SWIZZLE_64B MN-major descriptor: MN blocks of 32 elements `lbo` bytes
 * apart, 8-row K groups `sbo` bytes apart */
__device__ __forceinline__ unsigned long long smem_desc_mn_sw64(unsigned addr, unsigned lbo, unsigned sbo = 512u) {
  return (unsigned long long)((addr >> 4) & 0x3FFFu) | ((unsigned long long)((lbo >> 4) & 0x3FFFu) << 16) |
         ((unsigned long long)(sbo >> 4) << 32) | (1ull << 46) | (4ull << 61);
}

__global__ void __launch_bounds__(WG_THREADS, 2) mid_wgrad_tc(const __grid_constant__ CUtensorMap xmap,
                                                              const __grid_constant__ CUtensorMap gmap,
                                                              const __grid_constant__ CUtensorMap xtail,
                                                              const __grid_constant__ CUtensorMap gtail,
                                                              float* __restrict__ partial, const Items n) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* base = smem_raw + ((1024u - (saddr(smem_raw) & 1023u)) & 1023u);
  unsigned char* xrows = base;
  unsigned char* grows = base + WG_NX * ROW_BYTES;
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(grows + WG_NG * WG_G_BYTES);
  unsigned long long* xfull = bars;                  /* [WG_NX] */
  unsigned long long* xempty = bars + WG_NX;         /* [WG_NX] */
  unsigned long long* gfull = bars + 2 * WG_NX;      /* [WG_NG] */
  unsigned long long* gempty = gfull + WG_NG;        /* [WG_NG] */
  unsigned long long* done = gempty + WG_NG;         /* all MMAs complete */
  __shared__ unsigned tmem_slot;
  __shared__ int abort_flag;
  __shared__ int xl_issued, xl_waited, gl_issued, gl_waited;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  __shared__ float bias_sum[4][HC];

  if (tid == 0) {
    for (int q = 0; q < WG_NX; ++q) {
      bar_init(&xfull[q], 1);
      bar_init(&xempty[q], 1);
    }
    for (int q = 0; q < WG_NG; ++q) {
      bar_init(&gfull[q], 1);
      bar_init(&gempty[q], 1 + 4); /* the MMAs and the four summing warps */
    }
    bar_init(done, 1);
    abort_flag = 0;
    xl_issued = xl_waited = gl_issued = gl_waited = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(&tmem_slot)),
                 "r"(WG_TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = tmem_slot;
  if (warp < 4)
    for (int a = 0; a < 3; ++a) tmem_zero32(tmem + ((unsigned)(warp * 32) << 16) + (unsigned)(a * HC));
  let_next_start();
  wait_previous();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  if (warp == WG_TMA_WARP) {
    /* ---- row loads: input rows r0 - 1 .. r0 + rows, after input row j the
     * gradient row j (the last it meets); a tail item is one input box in two
     * ring slots, the first one even, and one gradient box */
    if (lane == 0) {
      int L = 0, G = 0;
      bool ok = true;
      auto xslot = [&](int l) {
        return bar_wait(&xempty[l % WG_NX], ((l / WG_NX) & 1) ^ 1) && !*(volatile int*)&abort_flag &&
               (saddr(xrows + (l % WG_NX) * ROW_BYTES) & 1023u) == 0;
      };
      auto gload = [&](const CUtensorMap* map, int x, int y, int b) {
        const int q = G % WG_NG;
        unsigned char* dst = grows + q * WG_G_BYTES;
        if (!bar_wait(&gempty[q], ((G / WG_NG) & 1) ^ 1) || *(volatile int*)&abort_flag || (saddr(dst) & 1023u))
          return false;
        bar_expect_tx(&gfull[q], WG_G_BYTES);
        tma_row(dst, map, x, y, b, &gfull[q]);
        gl_issued = ++G;
        return true;
      };
      for (int t = blockIdx.x; t < n.total && ok; t += gridDim.x) {
        const Item it = item_at(t, n);
        if (it.tail) {
          if (L & 1) {
            if (!(ok = xslot(L))) break;
            bar_arrive(&xfull[L % WG_NX]);
            xl_issued = ++L;
          }
          if (!(ok = xslot(L) && xslot(L + 1))) break;
          bar_expect_tx(&xfull[L % WG_NX], TAIL_TX);
          tma_row(xrows + (L % WG_NX) * ROW_BYTES, &xtail, it.x0 - 1, it.r0 - 1, it.b, &xfull[L % WG_NX]);
          bar_arrive(&xfull[(L + 1) % WG_NX]);
          xl_issued = L += 2;
          ok = gload(&gtail, it.x0, it.r0, it.b);
          continue;
        }
        for (int j = 0; j < it.rows + 2 && ok; ++j) {
          if (!(ok = xslot(L))) break;
          bar_expect_tx(&xfull[L % WG_NX], TX_BYTES);
          tma_row(xrows + (L % WG_NX) * ROW_BYTES, &xmap, it.x0 - 1, it.r0 - 1 + j, it.b, &xfull[L % WG_NX]);
          xl_issued = ++L;
          if (j < it.rows) ok = gload(&gmap, it.x0, it.r0 + j, it.b);
        }
      }
      if (!ok) atomicExch(&abort_flag, 1);
    }
  } else if (warp == WG_MMA_WARP) {
    /* ---- MMA issuer */
    if (lane == 0) {
      int L = 0, G = 0;
      bool ok = true;
      auto xlanded = [&](int l) {
        if (!bar_wait(&xfull[l % WG_NX], (l / WG_NX) & 1)) return false;
        xl_waited = l + 1;
        return !*(volatile int*)&abort_flag;
      };
      auto glanded = [&](int l) {
        if (!bar_wait(&gfull[l % WG_NG], (l / WG_NG) & 1)) return false;
        gl_waited = l + 1;
        return true;
      };
      const unsigned xbase = saddr(xrows), gbase = saddr(grows);
      /* accumulators [blk, blk + cnt) += A B */
      auto mma = [&](unsigned long long ad, unsigned gr, int blk, int cnt) {
        mma_f16(tmem + (unsigned)(blk * HC), ad, smem_desc_mn_sw64(gr, WG_G_BYTES), idesc(cnt) | kMnMajor, 1u);
      };
      /* only MMAs of one shape and accumulator are pipelined in order: where
       * the accumulators' split changes, the MMAs of the last input row come
       * first (its slot's release) */
      int split = 0, last = 0; /* the last ring slot released by a commit */
      auto same_split = [&](int s) {
        const bool wait = split != 0 && split != s;
        split = s;
        return !wait || bar_wait(&xempty[last % WG_NX], (last / WG_NX) & 1);
      };
      for (int t = blockIdx.x; t < n.total && ok; t += gridDim.x) {
        const Item it = item_at(t, n);
        if (it.tail) {
          if (L & 1) {
            if (!(ok = xlanded(L))) break;
            bar_arrive(&xempty[L % WG_NX]);
            ++L;
          }
          if (!(ok = xlanded(L) && xlanded(L + 1) && glanded(G) && same_split(1 << 8))) break;
          tc_fence_after();
          const unsigned xr = xbase + (unsigned)((L % WG_NX) * ROW_BYTES);
          const unsigned gr = gbase + (unsigned)((G % WG_NG) * WG_G_BYTES);
          for (int dy = 0; dy < 3; ++dy)
            for (int k = 0; k < BAND / 2; ++k) /* two rows of 8 pixels per K of 16 */
              mma(smem_desc_mn_sw64(xr + (unsigned)((2 * k + dy) * TAIL_PITCH), PIX_BYTES, TAIL_PITCH),
                  gr + (unsigned)(2 * k * TAIL_W * PIX_BYTES), 2 - dy, 1);
          mma_commit(&xempty[L % WG_NX]);
          mma_commit(&xempty[(L + 1) % WG_NX]);
          mma_commit(&gempty[G % WG_NG]);
          last = L + 1;
          L += 2;
          ++G;
          continue;
        }
        /* K blocks holding pixels of the image: past it the gradient is zero */
        const int ksteps = (n.W - it.x0 >= TM) ? TM / 16 : (n.W - it.x0 + 15) / 16;
        for (int j = 0; j < it.rows + 2 && ok; ++j, ++L) {
          /* input row j meets gradient rows lo .. hi of the band, row i for kernel row j - i */
          const int lo = j > 2 ? j - 2 : 0, hi = j < it.rows ? j : it.rows - 1;
          const int room = WG_NG - (G + lo) % WG_NG, cnt = hi - lo + 1;
          const int c0 = cnt < room ? cnt : room;
          const int blk = 2 - (j - lo);
          ok = xlanded(L) && (j >= it.rows || glanded(G + j)) && same_split(1 + blk + 4 * c0 + 16 * cnt);
          if (!ok) break;
          tc_fence_after();
          const unsigned xr = xbase + (unsigned)((L % WG_NX) * ROW_BYTES);
          const unsigned g0 = gbase + (unsigned)(((G + lo) % WG_NG) * WG_G_BYTES);
          for (int k = 0; k < ksteps; ++k) {
            const unsigned off = (unsigned)(k * 16 * PIX_BYTES);
            const unsigned long long ad = smem_desc_mn_sw64(xr + off, PIX_BYTES);
            mma(ad, g0 + off, blk, c0);
            if (c0 < cnt) mma(ad, gbase + off, blk + c0, cnt - c0); /* the ring of gradient rows wraps */
          }
          mma_commit(&xempty[L % WG_NX]);
          last = L;
          if (j >= 2) mma_commit(&gempty[(G + j - 2) % WG_NG]); /* read for the last time */
        }
        G += it.rows;
      }
      if (!ok) atomicExch(&abort_flag, 1);
      mma_commit(done); /* arrives once every MMA issued above has completed */
    }
  } else {
    /* ---- bias sums: thread = 16-byte chunk (8 channels) of every 32nd pixel
     * of each staged gradient row (zero outside the image) */
    float sum[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) sum[k] = 0.f;
    const int chunk = tid & 3;
    int G = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < n.total && ok; t += gridDim.x) {
      const int count = item_at(t, n).tiles();
      for (int i = 0; i < count; ++i, ++G) {
        ok = bar_wait(&gfull[G % WG_NG], (G / WG_NG) & 1) && !*(volatile int*)&abort_flag;
        ok = !__any_sync(0xffffffffu, !ok);
        if (!ok) break;
        const unsigned char* row = grows + (G % WG_NG) * WG_G_BYTES;
#pragma unroll
        for (int r = 0; r < TM / 32; ++r) {
          const int px = (tid >> 2) + 32 * r;
          const uint4 v = *reinterpret_cast<const uint4*>(row + px * PIX_BYTES + ((chunk ^ ((px >> 1) & 3)) << 4));
          const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float2 f = __bfloat1622float2(h[k]);
            sum[2 * k] += f.x;
            sum[2 * k + 1] += f.y;
          }
        }
        __syncwarp();
        if (lane == 0) bar_arrive(&gempty[G % WG_NG]);
      }
    }
    if (!ok) atomicExch(&abort_flag, 1);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], o);
      if (lane < 4) bias_sum[warp][chunk * 8 + k] = sum[k];
    }
    /* ---- epilogue: warp w reads TMEM lanes 32 w .. (shift j = w, channel
     * ci = lane) of each kernel row's accumulator */
    const bool fin = bar_wait(done, 0);
    if (__any_sync(0xffffffffu, !fin)) atomicExch(&abort_flag, 1);
    asm volatile("bar.sync 1, 128;" ::: "memory"); /* the bias sums of the four warps */
    if (!__any_sync(0xffffffffu, !fin || *(volatile int*)&abort_flag)) {
      /* the grid never exceeds the items, so every CTA accumulated rows */
      float* out = partial + (long long)blockIdx.x * WG_PART;
      if (warp < 3) {
#pragma unroll
        for (int dy = 0; dy < 3; ++dy) {
          float v[32];
          tc_fence_after();
          tmem_ld32(tmem + ((unsigned)(warp * 32) << 16) + (unsigned)((2 - dy) * HC), v);
          const int tap = dy * 3 + warp;
#pragma unroll
          for (int co = 0; co < HC; ++co) out[(tap * HC + co) * HC + lane] = v[co];
        }
      } else {
        out[9 * HC * HC + lane] = (bias_sum[0][lane] + bias_sum[1][lane]) + (bias_sum[2][lane] + bias_sum[3][lane]);
      }
    }
  }

  /* ---- drain (bounded) and free tensor memory */
  __syncthreads();
  if (abort_flag) {
    if (tid == 0) atomicExch(&g_cnn_tc_status, 1);
    if (warp == WG_TMA_WARP && lane == 0) {
      for (int j = xl_waited; j < xl_issued; ++j) bar_wait(&xfull[j % WG_NX], (j / WG_NX) & 1);
      for (int j = gl_waited; j < gl_issued; ++j) bar_wait(&gfull[j % WG_NG], (j / WG_NG) & 1);
    }
    if (warp == WG_MMA_WARP && lane == 0) bar_wait(done, 0);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(WG_TMEM_COLS) : "memory");
}

int g_tc_path = 1;

template <int MODE>
int launch(const void* x, const void* w, const float* bias, const void* mask, void* y, int B, int H, int W,
           void* stream) {
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(mid_conv_tc<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    if (e != cudaSuccess) return prml_set_error(PRML_ERR_CUDA, std::string("mid_conv_tc attribute: ") + cudaGetErrorString(e));
    attr_set = true;
  }
  if ((reinterpret_cast<unsigned long long>(x) & 15ull) || (reinterpret_cast<unsigned long long>(w) & 15ull) ||
      (reinterpret_cast<unsigned long long>(y) & 15ull) || (mask && (reinterpret_cast<unsigned long long>(mask) & 15ull)))
    return prml_set_error(PRML_ERR_ARG, "mid_conv_tc: buffers must be 16-byte aligned");
  /* x as [B][H][W][32]: dims innermost first */
  const unsigned long long dims[4] = {32, (unsigned long long)W, (unsigned long long)H, (unsigned long long)B};
  const unsigned long long strides[3] = {64, 64ull * W, 64ull * W * H};
  const unsigned box[4] = {32, SEG, 1, 1}, tail[4] = {32, TAIL_SEG, BAND + 2, 1};
  CUtensorMap map, tmap;
  int rc = prml_tensor_map_tiled(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, x, dims, strides, box, 64);
  if (!rc) rc = prml_tensor_map_tiled(&tmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, x, dims, strides, tail, 64);
  if (rc) return rc;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if ((long long)B * H * ((W + TM - 1) / TM) > 0x7fffffffLL)
    return prml_set_error(PRML_ERR_ARG, "mid_conv_tc: too many work items");
  const Items n = make_items(B, H, W, band_rows(B, H, W, 2 * sms));
  const int grid = n.total < 2 * sms ? n.total : 2 * sms;
  const cudaError_t e = prml_launch_overlapped(mid_conv_tc<MODE>, grid, dim3(THREADS), SMEM_BYTES, stream, map, tmap,
                                               static_cast<const bf16*>(w), bias, static_cast<const bf16*>(mask),
                                               static_cast<bf16*>(y), n);
  if (e != cudaSuccess) return prml_set_error(PRML_ERR_CUDA, std::string("mid_conv_tc: ") + cudaGetErrorString(e));
  return PRML_OK;
}

int launch_wgrad(const void* x, const void* g, float* partial, int parts, int* used, int B, int H, int W,
                 void* stream) {
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(mid_wgrad_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, WG_SMEM);
    if (e != cudaSuccess) return prml_set_error(PRML_ERR_CUDA, std::string("mid_wgrad_tc attribute: ") + cudaGetErrorString(e));
    attr_set = true;
  }
  if ((reinterpret_cast<unsigned long long>(x) & 15ull) || (reinterpret_cast<unsigned long long>(g) & 15ull))
    return prml_set_error(PRML_ERR_ARG, "mid_wgrad_tc: buffers must be 16-byte aligned");
  const unsigned long long dims[4] = {32, (unsigned long long)W, (unsigned long long)H, (unsigned long long)B};
  const unsigned long long strides[3] = {64, 64ull * W, 64ull * W * H};
  const unsigned xbox[4] = {32, SEG, 1, 1};
  const unsigned gbox[4] = {32, TM, 1, 1};
  const unsigned xtbox[4] = {32, TAIL_SEG, BAND + 2, 1}, gtbox[4] = {32, TAIL_W, BAND, 1};
  CUtensorMap xmap, gmap, xtail, gtail;
  int rc = prml_tensor_map_tiled(&xmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, x, dims, strides, xbox, 64);
  if (!rc) rc = prml_tensor_map_tiled(&gmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, g, dims, strides, gbox, 64);
  if (!rc) rc = prml_tensor_map_tiled(&xtail, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, x, dims, strides, xtbox, 64);
  if (!rc) rc = prml_tensor_map_tiled(&gtail, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, g, dims, strides, gtbox, 64);
  if (rc) return rc;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if ((long long)B * H * ((W + TM - 1) / TM) > 0x7fffffffLL)
    return prml_set_error(PRML_ERR_ARG, "mid_wgrad_tc: too many work items");
  int grid = parts < 2 * sms ? parts : 2 * sms;
  const Items n = make_items(B, H, W, band_rows(B, H, W, grid));
  if (grid > n.total) grid = n.total;
  *used = grid;
  const cudaError_t e = prml_launch_overlapped(mid_wgrad_tc, grid, dim3(WG_THREADS), WG_SMEM, stream, xmap, gmap, xtail,
                                               gtail, partial, n);
  if (e != cudaSuccess) return prml_set_error(PRML_ERR_CUDA, std::string("mid_wgrad_tc: ") + cudaGetErrorString(e));
  return PRML_OK;
}

}  // namespace

int prml_cnn_tc_enabled() { return g_tc_path; }

int prml_cnn_mid_wgrad_tc(const void* x, const void* g, float* partial, int parts, int* used, int B, int H, int W,
                          void* stream) {
  return launch_wgrad(x, g, partial, parts, used, B, H, W, stream);
}

int prml_cnn_mid_conv_tc(int mode, const void* x, const void* w, const float* bias, const void* mask, void* y,
                         int B, int H, int W, void* stream) {
  return mode == 0 ? launch<0>(x, w, bias, mask, y, B, H, W, stream)
                   : launch<1>(x, w, bias, mask, y, B, H, W, stream);
}

extern "C" {

int prml_cnn_set_tensor_path(int tcgen05) {
  const int prev = g_tc_path;
  g_tc_path = tcgen05 ? 1 : 0;
  return prev;
}

int prml_cnn_status(void) {
  int flag = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&flag, g_cnn_tc_status, sizeof(int));
  if (e != cudaSuccess) return prml_set_error(PRML_ERR_CUDA, std::string("prml_cnn_status: ") + cudaGetErrorString(e));
  if (flag) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_cnn_tc_status, &zero, sizeof(int));
    return prml_set_error(PRML_ERR_CUDA, "a tensor-core convolution timed out waiting on its pipeline");
  }
  return PRML_OK;
}

}  // extern "C"
