// Tensor-core path of the ball expansion: BF16 hi+lo split GEMM on tcgen05 (sm_100a).
//
// The 8 octant-parity GEMMs of fle.cu, C_p = A_p * B_p (A: folded volumes, B: basis
// columns), run here as BF16 x BF16 -> FP32 products with a split correction:
//     A B ~= A_hi B_hi + A_lo B_hi + A_hi B_lo,   A_hi = bf16(A), A_lo = bf16(A - A_hi)
// (the dropped A_lo B_lo term is ~2^-16 relative).  Two orders of the products, by the basis:
//   segmented    one GEMM over a K axis three times as long: step j of [0, 3 KB) selects (A_hi,
//                B_hi), (A_lo, B_hi) or (A_hi, B_lo), so a pipeline stage moves one tile of each,
//                64 along K.
//   interleaved  a stage holds the hi and lo tiles of both operands, 32 along K, for all three
//                products: the same bytes per stage, two thirds of the bytes per product, and B_hi
//                read once instead of twice.  (With stages of 64 along K only two fit, which was
//                1242 against 1187 us for 100 of 96^3 and 2.2x slower for 1000 of 64^3.)
// The second is for a basis past 1 GB (80^3: 2 GB).  That line is not where it stops being the faster:
// at 64^3 (500 MB) it would save 15 to 30 % of the GEMM too (1000 subtomograms 550 against 648 us).
// It is drawn for last bits.  The orientation search's choice between equal scores (the angles at
// beta = 0, alpha at 0 or 2 pi) follows them, and up to 64^3 the coefficients keep those of the
// segmented order; past it, where that order's loads take twice the products' time, they got others.
// Times of the GEMM, before (segmented, one CTA per tile) and now: 100 of 96^3 1397 -> 1105 us (5.5 TB/s
// of basis), 128 of 80^3 647 -> 381 us, 1000 of 64^3 679 -> 648 us, 256 of 64^3 321 -> 237 us, one of
// 64^3 291 -> 144 us, 128 of 48^3 138 -> 66 us, one of 48^3 118 -> 38 us.
//
// Accumulation: the tensor core adds each K=16 product into the FP32 accumulator with a
// truncating alignment, an error of about one unit in the last place of the accumulator per
// instruction.  Over the full K (15 216 octant representatives at 64^3, 2 856 instructions)
// that biases coefficients whose terms share a sign (the low degrees of a positive-mean
// volume) by ~2e-4 relative.  So the K axis is cut into chunks of kChunkKB blocks (240
// instructions, ~2e-5): each chunk accumulates into one of two tensor-memory buffers, and the
// epilogue warps add the finished buffer into running sums in registers (FP32 round-to-nearest,
// chunks in order, so the result is deterministic) while the MMAs of the next chunk run into
// the other buffer; C is written once at the end.  (Adding each chunk into C in global memory
// instead measured 2.4x slower: one row per lane makes every access a 32-way scatter.)
//
// Layout: both operands K-major bf16, tiles with 128-byte (interleaved: 64-byte) swizzle staged by
// TMA (cp.async.bulk.tensor.2d), tile M = 128 (a batch block), N = 256 or less (the basis columns of
// a class cut evenly, to 16).  One thread issues tcgen05.mma (kind::f16, M128 K16);
// eight warps read the accumulators back with tcgen05.ld, two per 32-lane quarter of tensor
// memory, each keeping 128 columns of its row.  A has rows (class * 2 + part) * Mpad + m; B is
// stored tile by tile, [class][part][N tile][K block][column][64], so that a stage's tile is one
// contiguous run of DRAM (with a K row per column instead, 1266 against 1242 us for 100
// subtomograms of 96^3).
//
// Work units: the tiles that fill whole rounds of the 148 SMs are one CTA each; the rest are cut
// along K into parts of q chunks (gemm_plan).  The first part of a tile leaves its sums in a slab,
// the others theirs in more (one per chunk, or one per part in the interleaved order), and the
// part that arrives last adds them in order.  With a slab per chunk the additions are
// those of a whole tile, so a coefficient does not depend on the split, nor on the batch it is in.
// In the interleaved order (tiles of 40 chunks at 96^3: a slab each would be 0.6 GB) a part is a group
// of chunks whose size belongs to the basis, whatever the batch, and a whole tile adds its groups'
// sums in the same order, so there too the batch does not matter.
//
// Every mbarrier wait is bounded; on expiry the kernel records an error code, stops
// issuing, waits (bounded) for the MMAs it issued, and frees its tensor memory before
// returning.
#include <cuda.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include <string.h>
#include "common.cuh"
#include "fle_tc.cuh"
#include "tc_common.cuh"

namespace {

using namespace tc;

constexpr int TM = 128, TN = 256, TK = 64;
constexpr int kMaxStages = 8;
constexpr int A_TILE = TM * TK * 2;  // 16 KB
constexpr int TKI = 32;              // K of a stage in the interleaved order
constexpr int AI_TILE = TM * TKI * 2;
constexpr size_t kSmemCap = kSmemOptIn - 1024;  // dynamic shared memory: the opt-in limit less the
                                                // static barriers
constexpr int kThreads = 320;        // warp 0: TMA, warp 1: MMA, warps 2-9: epilogue
constexpr int kEpiThreads = 256;
constexpr uint32_t kTmemCols = 512;  // two 256-column FP32 accumulators
constexpr int kChunkMma = 240;       // MMAs of an accumulator chunk

struct TcParams {
  int Mpad, KB;         // padded batch rows per (class, part), K blocks of 64
  int brow[8];          // first row of the class in B's map (64 K entries a row)
  int M;                // valid batch rows
  int mt;               // batch blocks
  int ncols[8];         // valid columns per class
  int coff[8];          // column offset of the class inside C
  int tn[8], first[9];  // columns of a tile of the class; the class's first tile / mt
  int ldc;              // row stride of C (floats)
  int stages, stage_bytes;
  int stall;            // test hook: no loads are issued, and waits give up after kStallPolls
  int ntn;              // row length of split
  const int* split;     // (8, ntn): 1 = hi+lo split (three products), 0 = plain BF16 (one)
  int whole;            // tiles below this are one unit each
  int parts, q;         // units of the others: parts of q chunks
  int group;            // interleaved: chunks whose sums are formed before they meet the others'
  int slots;            // slabs of a split tile
  float* slab;          // [split tile][slot][column][row], 256 x 128 floats each
  float* run;           // [tile that is one unit][column][row]: sums of its groups so far
  int* count;           // parts of each split tile that have arrived (zero before the launch)
};

struct BMaps {
  CUtensorMap m[8];     // per class: its tile's rows, TK (or, interleaved, TKI) of a row
};

// Poll limit of every wait while the stall hook is on: at most kStallPolls x kSuspendNs (20 ms).
constexpr long long kStallPolls = 1 << 10;

__device__ __forceinline__ void mbar_arrive_cta(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// INTERLEAVED: the order of the products (see above); it takes split tiles only.
template <bool INTERLEAVED>
__global__ void __launch_bounds__(kThreads, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ BMaps mapB,
               const __grid_constant__ TcParams P, float* __restrict__ C, int* __restrict__ err) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // 1024-byte alignment for the swizzled tiles
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t full_bar[kMaxStages];
  __shared__ __align__(8) uint64_t empty_bar[kMaxStages];
  __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2], drain_bar;
  __shared__ uint32_t tmem_base;
  __shared__ int last_part;
  __shared__ volatile int abort_flag;

  // this CTA's unit: a tile and the chunks [c0, c1) of its K steps.  M tiles vary fastest, so that
  // the CTAs of one basis N-tile run together and read its B slab from L2 rather than once per M
  // tile from DRAM
  const int unit = blockIdx.x;
  const bool is_split = unit >= P.whole;
  const int tile = is_split ? P.whole + (unit - P.whole) / P.parts : unit;
  const int part = is_split ? (unit - P.whole) % P.parts : 0;
  const int nt = tile / P.mt;
  int cls = 0;
  while (nt >= P.first[cls + 1]) ++cls;
  const int n = nt - P.first[cls], tn = P.tn[cls];
  const int m0 = (tile - nt * P.mt) * TM, n0 = n * tn;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // K steps: the three segments' blocks, or the (hi, hi) segment alone for a plain BF16 tile
  const int steps = INTERLEAVED ? P.KB * (TK / TKI) : (__ldg(&P.split[cls * P.ntn + n]) ? 3 : 1) * P.KB;
  constexpr int kSteps = INTERLEAVED ? kChunkMma / (3 * TKI / 16) : kChunkMma / 4;  // of a chunk
  const int nchunks = (steps + kSteps - 1) / kSteps;
  const int c0 = part * P.q, c1 = is_split ? min(nchunks, c0 + P.q) : nchunks;
  if (c0 >= nchunks) return;  // a part past the end of a plain BF16 tile's steps; uniform per CTA
  const int j0 = c0 * kSteps, j1 = min(steps, c1 * kSteps);
  const int S = P.stages, b_tile = tn * (INTERLEAVED ? TKI : TK) * 2;
  const long long polls = P.stall ? kStallPolls : kSpinLimit;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], kEpiThreads);
    }
    mbar_init(&drain_bar, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base;

  if (warp == 0 && lane == 0) {
    // ---- TMA producer (the stall hook issues nothing, so the MMA thread's first wait runs out)
    int s = 0, seg = INTERLEAVED ? 0 : j0 / P.KB, kb = INTERLEAVED ? j0 : j0 - seg * P.KB;
    const int ntc = P.first[cls + 1] - P.first[cls], brow = P.brow[cls] + n * P.KB * tn;
    uint32_t phase = 1;  // of the stage's release before this use (none before the first)
    for (int j = j0; j < j1 && !abort_flag && !P.stall; ++j) {
      if (j - j0 >= S && !mbar_wait_n(&empty_bar[s], phase, polls)) {
        atomicCAS(err, 0, 1);
        abort_flag = 1;
        break;
      }
      uint8_t* sa = smem + s * P.stage_bytes;
      if (INTERLEAVED) {  // A_hi, A_lo, B_hi, B_lo
        mbar_expect_tx(&full_bar[s], 2 * (AI_TILE + b_tile));
        const int blk = kb / (TK / TKI), x = (kb % (TK / TKI)) * TKI;
        for (int h = 0; h < 2; ++h) {
          tma_load_2d(sa + h * AI_TILE, &mapA, kb * TKI, (cls * 2 + h) * P.Mpad + m0, &full_bar[s]);
          tma_load_2d(sa + 2 * AI_TILE + h * b_tile, &mapB.m[cls], x, brow + (h * ntc * P.KB + blk) * tn, &full_bar[s]);
        }
      } else {
        // segment 0: (hi, hi), 1: (lo, hi), 2: (hi, lo)
        const int apart = (seg == 1) ? 1 : 0, bpart = (seg == 2) ? 1 : 0;
        mbar_expect_tx(&full_bar[s], A_TILE + b_tile);
        tma_load_2d(sa, &mapA, kb * TK, (cls * 2 + apart) * P.Mpad + m0, &full_bar[s]);
        tma_load_2d(sa + A_TILE, &mapB.m[cls], 0, brow + (bpart * ntc * P.KB + kb) * tn, &full_bar[s]);
      }
      if (++kb == P.KB && !INTERLEAVED) {
        kb = 0;
        ++seg;
      }
      if (++s == S) {
        s = 0;
        phase ^= 1;
      }
    }
  } else if (warp == 1 && lane == 0) {
    // ---- MMA issuer: this unit's chunk i into accumulator i & 1
    const uint32_t idesc = idesc_bf16(TM, tn);
    bool ok = true;
    int issued = 0, s = 0;
    uint32_t phase = 0;
    for (int c = c0; c < c1 && ok; ++c) {
      const int i = c - c0, buf = i & 1;
      if (i >= 2 && !mbar_wait_n(&acc_empty[buf], ((i >> 1) - 1) & 1, polls)) {
        atomicCAS(err, 0, 4);
        abort_flag = 1;
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t d = tmem + (uint32_t)(buf * TN);
      const int je = min(j1, (c + 1) * kSteps);
      for (int j = c * kSteps; j < je; ++j) {
        if (abort_flag || !mbar_wait_n(&full_bar[s], phase, polls)) {
          atomicCAS(err, 0, 2);
          abort_flag = 1;
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint8_t* sa = smem + s * P.stage_bytes;
        const bool fresh = j == c * kSteps;
        if (INTERLEAVED) {
          const uint64_t ah = smem_desc64(sa), alo = smem_desc64(sa + AI_TILE), bh = smem_desc64(sa + 2 * AI_TILE),
                         blo = smem_desc64(sa + 2 * AI_TILE + b_tile);
#pragma unroll
          for (int kk = 0; kk < TKI / 16; ++kk) {
            const uint64_t o = (uint64_t)(kk * 2);
            mma_bf16_id(d, ah + o, bh + o, idesc, (!fresh || kk > 0) ? 1u : 0u);
            mma_bf16_id(d, alo + o, bh + o, idesc, 1u);
            mma_bf16_id(d, ah + o, blo + o, idesc, 1u);
          }
        } else {
          const uint64_t ad = smem_desc(sa), bd = smem_desc(sa + A_TILE);
#pragma unroll
          for (int kk = 0; kk < TK / 16; ++kk) {
            // 16 bf16 = 32 bytes further along K inside the swizzle atom: +2 in the >>4 address field
            mma_bf16_id(d, ad + (uint64_t)(kk * 2), bd + (uint64_t)(kk * 2), idesc, (!fresh || kk > 0) ? 1u : 0u);
          }
        }
        mma_commit_to(&empty_bar[s]);
        ++issued;
        if (++s == S) {
          s = 0;
          phase ^= 1;
        }
      }
      if (ok) mma_commit_to(&acc_full[buf]);
    }
    if (!ok && issued > 0) {
      // let the MMAs already issued finish before the tensor memory is freed
      mma_commit_to(&drain_bar);
      mbar_wait_n(&drain_bar, 0, polls);
    }
  } else if (warp >= 2) {
    // ---- epilogue: warp w reads TMEM lanes 32*(w%4) .. +31 (rows m0 + that range), columns
    // h*128 .. +127 with h = (w-2)/4, and keeps their running sums over the chunks
    const int q = warp & 3, h = (warp - 2) >> 2;
    const int row = q * 32 + lane;
    const bool valid = m0 + row < P.M;
    const int ncol = min(tn, P.ncols[cls] - n0);  // valid columns of the tile
    // slab column 0 of this thread's row and half; slot 0 takes the first part, 1 + c - q chunk c
    // of a later one, or slot part the whole later part
    float* slab = P.slab + ((int64_t)(tile - P.whole) * P.slots * TN + h * (TN / 2)) * TM + row;
    float acc[TN / 2];
#pragma unroll
    for (int t = 0; t < TN / 2; ++t) acc[t] = 0.f;
    bool done = true;
    auto add_chunks = [&](int from, int to) {
      for (int c = from; c < to; ++c) {
        const int i = c - c0, buf = i & 1;
        if (abort_flag || !mbar_wait_n(&acc_full[buf], (i >> 1) & 1, polls)) {
          atomicCAS(err, 0, 3);
          abort_flag = 1;
          done = false;
          return;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * TN + h * (TN / 2));
        const bool to_slab = !INTERLEAVED && part > 0;
        float* out = slab + (int64_t)(1 + c - P.q) * TN * TM;
#pragma unroll
        for (int cb = 0; cb < TN / 2; cb += 32) {
          uint32_t v[32];
          asm volatile(
              "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
              "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
              : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
                "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]),
                "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]),
                "=r"(v[30]), "=r"(v[31])
              : "r"(taddr + (uint32_t)cb));
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (to_slab) {
            if (valid) {
#pragma unroll
              for (int t = 0; t < 32; ++t)
                if (h * (TN / 2) + cb + t < ncol) out[(cb + t) * TM] = __uint_as_float(v[t]);
            }
          } else {
#pragma unroll
            for (int t = 0; t < 32; ++t) acc[cb + t] += __uint_as_float(v[t]);
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        mbar_arrive_cta(&acc_empty[buf]);
      }
    };
    // interleaved, a whole tile of several groups: the sums of those before the current one
    const bool grouped = INTERLEAVED && (!is_split || P.parts == 1);
    float* run = P.run + ((int64_t)tile * TN + h * (TN / 2)) * TM + row;
    if (grouped) {
      const int n_cols = valid ? ncol - h * (TN / 2) : 0;
      for (int from = c0; from < c1 && done; from += P.group) {
        add_chunks(from, min(c1, from + P.group));
        if (from + P.group >= c1 || !done) break;
        // a group's end: the sums that the parts of a cut tile leave in their slots (U loads in flight)
        constexpr int U = 16;
#pragma unroll
        for (int t = 0; t < TN / 2; t += U) {
          float v[U];
#pragma unroll
          for (int u = 0; u < U; ++u) v[u] = from > c0 && t + u < n_cols ? __ldcg(run + (t + u) * TM) : 0.f;
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (t + u < n_cols) __stcg(run + (t + u) * TM, from > c0 ? v[u] + acc[t + u] : acc[t + u]);
            acc[t + u] = 0.f;
          }
        }
      }
    } else {
      add_chunks(c0, c1);
    }
    float* crow = C + (int64_t)(m0 + row) * P.ldc + P.coff[cls] + n0 + h * (TN / 2);
    const int w = min(TN / 2, ncol - h * (TN / 2));  // valid columns of this half (may be < 0)
    if (done && valid && (part == 0 || INTERLEAVED)) {
      const bool direct = !is_split || P.parts == 1;
      float* out = direct ? crow : slab + (int64_t)part * TN * TM;
      const int step = direct ? 1 : TM;
      const bool more = grouped && c1 - c0 > P.group;
      if (more) {
        constexpr int U = 16;
#pragma unroll
        for (int t = 0; t < TN / 2; t += U) {
          float v[U];
#pragma unroll
          for (int u = 0; u < U; ++u) v[u] = t + u < w ? __ldcg(run + (t + u) * TM) : 0.f;
#pragma unroll
          for (int u = 0; u < U; ++u) acc[t + u] = v[u] + acc[t + u];
        }
      }
#pragma unroll
      for (int t = 0; t < TN / 2; ++t)
        if (t < w) out[t * step] = acc[t];
    }
    if (is_split && P.parts > 1) {
      // the part that arrives last adds the slots in order (a part that gave up does not arrive: the
      // call has failed then)
      __threadfence();
      asm volatile("bar.sync 1, %0;" ::"n"(kEpiThreads) : "memory");
      const int arrivals = (nchunks + P.q - 1) / P.q;
      if (threadIdx.x == 64)
        last_part = !abort_flag && atomicAdd(&P.count[tile - P.whole], 1) == arrivals - 1;
      asm volatile("bar.sync 1, %0;" ::"n"(kEpiThreads) : "memory");
      if (last_part) __threadfence();
      const int slots = INTERLEAVED ? arrivals : 1 + max(0, nchunks - P.q);
      const int rows = min(TM, P.M - m0);
      constexpr int V = 4;  // slots in flight
      if (last_part && rows <= 32) {
        // few rows (one of 48^3: 37 us, against 52 with a row per thread): elements over the threads
        constexpr int U = 4;
        const float* slab0 = P.slab + (int64_t)(tile - P.whole) * P.slots * TN * TM;
        const int total = rows * ncol;
        for (int e = (int)threadIdx.x - 64; e < total; e += U * kEpiThreads) {
          float v[U];
          int at[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int i = min(e + u * kEpiThreads, total - 1), col = i / rows;
            at[u] = col * TM + i - col * rows;
            v[u] = __ldcg(slab0 + at[u]);
          }
#pragma unroll V
          for (int k = 1; k < slots; ++k)
#pragma unroll
            for (int u = 0; u < U; ++u) v[u] += __ldcg(slab0 + (int64_t)k * TN * TM + at[u]);
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (e + u * kEpiThreads < total)
              C[(int64_t)(m0 + at[u] % TM) * P.ldc + P.coff[cls] + n0 + at[u] / TM] = v[u];
        }
      } else if (last_part && valid) {
        // a row per thread, so that a warp reads 32 rows of a column together
        constexpr int U = 16;  // columns in flight
        for (int t = 0; t < w; t += U) {
          float v[U];
#pragma unroll
          for (int u = 0; u < U; ++u) v[u] = t + u < w ? __ldcg(slab + (t + u) * TM) : 0.f;
          for (int k = 1; k < slots; k += V) {
            float x[V][U];
#pragma unroll
            for (int j = 0; j < V; ++j)
#pragma unroll
              for (int u = 0; u < U; ++u)
                x[j][u] = k + j < slots && t + u < w ? __ldcg(slab + ((int64_t)(k + j) * TN + t + u) * TM) : 0.f;
#pragma unroll
            for (int j = 0; j < V; ++j)
              if (k + j < slots)
#pragma unroll
                for (int u = 0; u < U; ++u) v[u] += x[j][u];
          }
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (t + u < w) crow[t + u] = v[u];
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
  }
}

// ---------------------------------------------------------------- operand preparation
// Folded channels, split into bf16 hi/lo: Aall[((cls*2 + part) * Mpad + b) * Kpad + rep].
__global__ void fold_split_kernel(const float* __restrict__ vol, int64_t vol_stride, int B, int n_rep, int Mpad,
                                  int Kpad, const int* __restrict__ rep_img, __nv_bfloat16* __restrict__ A,
                                  int* __restrict__ count, int n_count) {
  const int rep = blockIdx.x * blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (blockIdx.x == 0 && b == 0)  // the arrival counts of the GEMM that follows
    for (int i = threadIdx.x; i < n_count; i += blockDim.x) count[i] = 0;
  if (rep >= Kpad || b >= B) return;
  float f[8];
#pragma unroll
  for (int s = 0; s < 8; ++s) {
    const int idx = rep < n_rep ? __ldg(&rep_img[rep * 8 + s]) : -1;
    f[s] = idx >= 0 ? __ldg(&vol[(int64_t)b * vol_stride + idx]) : 0.f;
  }
#pragma unroll
  for (int bit = 1; bit < 8; bit <<= 1)
#pragma unroll
    for (int s = 0; s < 8; ++s)
      if (!(s & bit)) {
        const float u = f[s], w = f[s | bit];
        f[s] = u + w;
        f[s | bit] = u - w;
      }
#pragma unroll
  for (int p = 0; p < 8; ++p) {
    uint32_t hi, lo;
    split_bf16(f[p], hi, lo);
    A[((int64_t)(p * 2 + 0) * Mpad + b) * Kpad + rep] = __ushort_as_bfloat16((unsigned short)hi);
    A[((int64_t)(p * 2 + 1) * Mpad + b) * Kpad + rep] = __ushort_as_bfloat16((unsigned short)lo);
  }
}

// Basis (K x n_p, row-major FP32 per class) -> the class's tiles [part][n / tn][k / 64][n % tn][k % 64] at Bm.
__global__ void basis_split_kernel(const float* __restrict__ basis, int n_rep, int ncls, int nt, int tn, int Kpad,
                                   __nv_bfloat16* __restrict__ Bm) {
  __shared__ float tile[32][33];
  const int k0 = blockIdx.x * 32, n0 = blockIdx.y * 32;
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int k = k0 + i, n = n0 + threadIdx.x;
    tile[i][threadIdx.x] = (k < n_rep && n < ncls) ? basis[(int64_t)k * ncls + n] : 0.f;
  }
  __syncthreads();
  const int KB = Kpad / TK;
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int n = n0 + i, k = k0 + threadIdx.x;
    if (n >= nt * tn || k >= Kpad) continue;
    const float v = tile[threadIdx.x][i];
    uint32_t hi, lo;
    split_bf16(v, hi, lo);
    const int64_t at = (((int64_t)(n / tn) * KB + k / TK) * tn + n % tn) * TK + k % TK;
    Bm[at] = __ushort_as_bfloat16((unsigned short)hi);
    Bm[(int64_t)nt * KB * tn * TK + at] = __ushort_as_bfloat16((unsigned short)lo);
  }
}

typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

int make_map(CUtensorMap* map, void* base, uint64_t inner, uint64_t rows, uint32_t box_rows, uint32_t box_k) {
  static EncodeTiled fn = nullptr;
  if (!fn) {
    cudaDriverEntryPointQueryResult q;
    void* p = nullptr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !p)
      return MTB_ERR_CUDA;
    fn = reinterpret_cast<EncodeTiled>(p);
  }
  const cuuint64_t dims[2] = {inner, rows};
  const cuuint64_t strides[1] = {inner * 2};
  const cuuint32_t box[2] = {box_k, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE,
                        box_k == TKI ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? MTB_OK : MTB_ERR_CUDA;
}

constexpr int kSMs = 148;
constexpr size_t kSlabCap = (size_t)128 << 20;  // bytes of slabs a plan may take
constexpr size_t kInterleaveBytes = (size_t)1 << 30;  // see the top

// How a GEMM of mt batch blocks is cut into units.
struct GemmPlan {
  bool interleaved;
  int tiles, whole, parts, q, slots, units;
  int runs;  // tiles that add the sums of several groups on their own
};

// Tiles beyond the whole rounds of the SMs are cut into parts of q chunks; q minimises the rounds
// times their length (a chunk's loads at the 110 GB/s an SM takes in, 5 us for a unit's start and
// end), the adding of the slots and the slabs' way to memory and back.  One batch block of 48^3 (16
// tiles of 5 chunks) runs as 80 units instead of 16, 100 subtomograms of 96^3 (117 tiles of 40) as
// 585 instead of 117.  The interleaved order is for a basis past kInterleaveBytes; see the top.  There
// the best q of one batch block is the group of every batch (t->group; 0 while it is being
// chosen), and larger batches only choose whether to cut by it.
GemmPlan gemm_plan(const FleTc* t, int mt) {
  GemmPlan p;
  const int KB = t->Kpad / TK;
  int nt = 0;
  size_t cols = 0;
  for (int k = 0; k < 8; ++k) {
    nt += t->nt[k];
    cols += t->ncols[k];
  }
  const bool all_split = t->n_split_tiles == t->n_tiles;
  p.interleaved = all_split && cols * t->Kpad * 4 > kInterleaveBytes;
  const int nchunks = (KB * 12 + kChunkMma - 1) / kChunkMma;
  p.tiles = nt * mt;
  p.whole = p.tiles / kSMs * kSMs;
  const int rest = p.tiles - p.whole;
  p.parts = 1;
  p.q = nchunks;
  p.slots = 0;
  int tn = 16;
  for (int k = 0; k < 8; ++k) tn = t->nt[k] && t->tn[k] > tn ? t->tn[k] : tn;
  const double chunk = (p.interleaved ? 40 : 60) * (A_TILE + 128.0 * tn) / 110e3;  // us
  double best = 1e30;
  for (int q = nchunks; q >= 1 && rest > 0; --q) {
    if (p.interleaved && t->group && q != t->group && q != nchunks) continue;
    const int parts = (nchunks + q - 1) / q;
    const int slots = parts == 1 ? 0 : (p.interleaved ? parts : 1 + nchunks - q);
    const size_t bytes = (size_t)rest * slots * TN * TM * sizeof(float);
    if (bytes > kSlabCap) continue;
    const int rounds = (rest * parts + kSMs - 1) / kSMs;
    const double cost = rounds * (q * chunk + 5.0) + (parts > 1 ? 6.0 + 1.5 * slots : 0.0) + 2.0 * bytes / 6.5e6;
    if (cost < best - 1e-9) {
      best = cost;
      p.parts = parts;
      p.q = q;
      p.slots = slots;
    }
  }
  p.units = p.whole + rest * p.parts;
  p.runs = p.interleaved && t->group < nchunks ? (p.parts == 1 ? p.tiles : p.whole) : 0;
  return p;
}

}  // namespace

size_t fle_tc_a_elems(int max_batch, int n_rep) {
  const int Mpad = (max_batch + TM - 1) / TM * TM;
  const int Kpad = (n_rep + TK - 1) / TK * TK;
  return (size_t)16 * Mpad * Kpad;
}

int fle_tc_prepare(FleTc* t, float* const* basis, const int* class_cols, const int* class_off, int n_rep,
                   int max_batch, int n_cols, const std::vector<std::vector<int>>& col_deg, int split_degree) {
  memset(t, 0, sizeof(*t));
  t->Mpad = (max_batch + TM - 1) / TM * TM;
  t->Kpad = (n_rep + TK - 1) / TK * TK;
  int maxc = 0;
  for (int k = 0; k < 8; ++k) maxc = class_cols[k] > maxc ? class_cols[k] : maxc;
  t->n_rep = n_rep;
  t->n_cols = n_cols;
  for (int k = 0; k < 8; ++k) {
    t->ncols[k] = class_cols[k];
    t->coff[k] = class_off[k];
    // the class's columns cut evenly into the fewest tiles, in steps of 16 (with a degree
    // schedule, which is by tiles of 256, they stay 256)
    t->nt[k] = (class_cols[k] + TN - 1) / TN;
    t->tn[k] = TN;
    if (t->nt[k] && split_degree < 0) t->tn[k] = ((class_cols[k] + t->nt[k] - 1) / t->nt[k] + 15) / 16 * 16;
  }
  int64_t rows = 0;  // of 64 K entries
  for (int k = 0; k < 8; ++k) {
    t->brow[k] = (int)rows;
    rows += (int64_t)2 * t->nt[k] * (t->Kpad / TK) * t->tn[k];
  }
  if (rows > 0x7fffffff) return MTB_ERR_ARG;  // TMA coordinates
  const size_t asz = (size_t)16 * t->Mpad * t->Kpad, bsz = (size_t)rows * TK;
  if (cudaMalloc(&t->A, asz * 2) != cudaSuccess) return MTB_ERR_OOM;
  if (cudaMalloc(&t->B, bsz * 2) != cudaSuccess) return MTB_ERR_OOM;
  if (cudaMalloc(&t->err, sizeof(int)) != cudaSuccess) return MTB_ERR_OOM;
  // which tiles take the split: those holding a column of degree above split_degree
  t->ntn = (maxc + TN - 1) / TN;
  {
    std::vector<int> flags((size_t)8 * t->ntn, 1);
    for (int k = 0; k < 8; ++k)
      for (int n = 0; n < t->ntn; ++n) {
        const int c0 = n * TN;
        if (c0 >= class_cols[k]) continue;
        const int c1 = (c0 + TN < class_cols[k] ? c0 + TN : class_cols[k]) - 1;
        const int top = (size_t)k < col_deg.size() && (size_t)c1 < col_deg[k].size() ? col_deg[k][c1] : 1 << 30;
        flags[(size_t)k * t->ntn + n] = (split_degree < 0 || top > split_degree) ? 1 : 0;
        t->n_tiles += 1;
        t->n_split_tiles += flags[(size_t)k * t->ntn + n];
      }
    if (cudaMalloc(&t->split, flags.size() * sizeof(int)) != cudaSuccess) return MTB_ERR_OOM;
    if (cudaMemcpy(t->split, flags.data(), flags.size() * sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess)
      return MTB_ERR_CUDA;
  }
  if (cudaMemset(t->B, 0, bsz * 2) != cudaSuccess || cudaMemset(t->A, 0, asz * 2) != cudaSuccess ||
      cudaMemset(t->err, 0, sizeof(int)) != cudaSuccess)
    return MTB_ERR_CUDA;
  for (int k = 0; k < 8; ++k) {
    if (!class_cols[k]) continue;
    dim3 g((t->Kpad + 31) / 32, (t->nt[k] * t->tn[k] + 31) / 32);
    basis_split_kernel<<<g, dim3(32, 8)>>>(basis[k], n_rep, class_cols[k], t->nt[k], t->tn[k], t->Kpad,
                                           reinterpret_cast<__nv_bfloat16*>(t->B) + (int64_t)t->brow[k] * TK);
    if (cudaGetLastError() != cudaSuccess) return MTB_ERR_CUDA;
  }
  if (cudaDeviceSynchronize() != cudaSuccess) return MTB_ERR_CUDA;
  int rc = MTB_OK;
  for (int i = 0; i < 2 && !rc; ++i) {  // stages of TK, of TKI
    const uint32_t k = i ? TKI : TK;
    rc = make_map(reinterpret_cast<CUtensorMap*>(t->mapA[i]), t->A, (uint64_t)t->Kpad, (uint64_t)16 * t->Mpad, TM, k);
    for (int c = 0; c < 8 && !rc; ++c)
      rc = make_map(reinterpret_cast<CUtensorMap*>(t->mapB[i][c]), t->B, TK, (uint64_t)rows, (uint32_t)t->tn[c], k);
  }
  if (rc) return rc;
  // slabs, running sums and arrival counts of every batch up to max_batch
  t->group = gemm_plan(t, 1).q;
  size_t slab = 0, run = 0;
  for (int mt = 1; mt <= t->Mpad / TM; ++mt) {
    const GemmPlan p = gemm_plan(t, mt);
    run = p.runs > (int64_t)run ? p.runs : run;
    const size_t n = (size_t)(p.tiles - p.whole) * p.slots * TN * TM * sizeof(float);
    slab = n > slab ? n : slab;
    if (p.parts > 1 && p.tiles - p.whole > t->n_count) t->n_count = p.tiles - p.whole;
  }
  if (slab && cudaMalloc(&t->slab, slab) != cudaSuccess) return MTB_ERR_OOM;
  if (run && cudaMalloc(&t->run, run * TN * TM * sizeof(float)) != cudaSuccess) return MTB_ERR_OOM;
  if (t->n_count && cudaMalloc(&t->count, t->n_count * sizeof(int)) != cudaSuccess) return MTB_ERR_OOM;
  return MTB_OK;
}

void fle_tc_release(FleTc* t) {
  if (t->A) cudaFree(t->A);
  if (t->B) cudaFree(t->B);
  if (t->err) cudaFree(t->err);
  if (t->split) cudaFree(t->split);
  if (t->slab) cudaFree(t->slab);
  if (t->run) cudaFree(t->run);
  if (t->count) cudaFree(t->count);
  memset(t, 0, sizeof(*t));
}

int fle_tc_forward(FleTc* t, const float* vol, int64_t vol_stride, int B, const int* rep_img, float* C,
                   cudaStream_t st) {
  dim3 fg((t->Kpad + 255) / 256, B);
  mtb_prof_begin(st);
  fold_split_kernel<<<fg, 256, 0, st>>>(vol, vol_stride, B, t->n_rep, t->Mpad, t->Kpad, rep_img,
                                        reinterpret_cast<__nv_bfloat16*>(t->A), t->count, t->n_count);
  mtb_prof_end(st, "fold_split_kernel");
  MTB_LAUNCH_CHECK();
  TcParams P;
  P.Mpad = t->Mpad;
  P.KB = t->Kpad / TK;
  P.M = B;
  P.mt = (B + TM - 1) / TM;
  const GemmPlan plan = gemm_plan(t, P.mt);
  int tn_max = 16;
  P.first[0] = 0;
  for (int k = 0; k < 8; ++k) {
    P.ncols[k] = t->ncols[k];
    P.coff[k] = t->coff[k];
    P.tn[k] = t->tn[k];
    P.brow[k] = t->brow[k];
    P.first[k + 1] = P.first[k] + t->nt[k];
    if (t->nt[k] && t->tn[k] > tn_max) tn_max = t->tn[k];
  }
  P.ldc = t->n_cols;
  // stages on 1024-byte boundaries (a B tile of 16 rows is 2 KB)
  P.stage_bytes = A_TILE + tn_max * TK * 2;  // the same for both orders
  P.stages = (int)((kSmemCap - 1024) / P.stage_bytes);
  if (P.stages > kMaxStages) P.stages = kMaxStages;
  P.stall = t->stall;
  P.ntn = t->ntn;
  P.split = t->split;
  P.whole = plan.whole;
  P.parts = plan.parts;
  P.q = plan.q;
  P.group = t->group;
  P.slots = plan.slots;
  P.slab = t->slab;
  P.run = t->run;
  P.count = t->count;
  const size_t smem = (size_t)P.stages * P.stage_bytes + 1024;
  const auto kernel = plan.interleaved ? gemm_tc_kernel<true> : gemm_tc_kernel<false>;
  MTB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemCap));
  mtb_prof_begin(st);
  kernel<<<plan.units, kThreads, smem, st>>>(*reinterpret_cast<const CUtensorMap*>(t->mapA[plan.interleaved]),
                                             *reinterpret_cast<const BMaps*>(t->mapB[plan.interleaved]), P, C, t->err);
  mtb_prof_end(st, "gemm_tc_kernel");
  MTB_LAUNCH_CHECK();
  return MTB_OK;
}

int fle_tc_check(FleTc* t, cudaStream_t st) {
  int h = 0;
  MTB_CUDA_TRY(cudaMemcpyAsync(&h, t->err, sizeof(int), cudaMemcpyDeviceToHost, st));
  MTB_CUDA_TRY(cudaStreamSynchronize(st));
  if (h) MTB_CUDA_TRY(cudaMemsetAsync(t->err, 0, sizeof(int), st));  // reported once
  return h ? MTB_ERR_TIMEOUT : MTB_OK;
}
