// Prefill form of the grouped 4-bit experts: a grouped GEMM on the tcgen05 tensor cores.
//
// A CTA owns one unit = (plan item of <= 192 pairs, 128 weight rows).  The roles are swapped against the usual GEMM:
// the WEIGHTS are the MMA's A operand (M = 128 rows: 128 output columns of one matrix, or 64 columns of gate and the
// same 64 of up), the item's PAIRS the B operand (N = pairs rounded up to 16, <= 192), so an expert with 140 pairs
// costs 144 / 128 of a full tile instead of two.  Per group of 64 inputs (one pipeline stage):
//   warps 0-7    turn nibbles into the prefill form's bf16 weights (w = bf16(q * s + b), one rounding) and store them
//                straight into TENSOR MEMORY, a weight row a lane (tcgen05.st): two sets of four warps take the even and
//                the odd stages, each set with an A stage of its own;
//   gathering    warps (8-11, or 8-9 in the build for small items): the pairs' input rows with 16-byte cp.async into the
//                128-byte-swizzled B tile;
//   MMA          warp (the next): one lane issues tcgen05.mma (cta_group::1, kind::f16, M = 128, K = 16; A from tensor
//                memory, B from shared memory) into fp32 accumulators in tensor memory, and commits each stage back;
//   copying      warp (the last): bulk copies of the packed blocks into a deep staging ring, a lane a column block.
// After the last group two or three warps a lane quarter read the accumulators (tcgen05.ld), apply the epilogue and store
// rows by pair id.
// One fp32 chain over K in group order: a pair's bits do not depend on its item, its chunk or the call.
//
// What bounds it: instruction issue of the dequantisation.  On a B200 at 2048 tokens of 128 experts (2048 x 768, top 8) the
// schedulers issue in 0.74 of the cycles of gate/up (down 0.67), the ALU pipe is 0.59 (0.50) busy, the multiply pipe 0.47
// (0.41), tcgen05 0.34 (0.25), shared memory 0.32, DRAM 0.19; about 1000 of the dequantising warps' instructions a stage
// stand against 256 cycles of MMA.  The build for small items at 317 tokens with a shared expert: issue 0.73 (0.66), ALU
// 0.60 (0.52), tcgen05 0.13 (0.10), and more warps that wait for their inputs.
// With the A tiles in shared memory a stage of gate/up moved 154 KB through it at 192 pairs (of it 64 KB A written and
// read) and one CTA filled an SM; without them two or three CTAs share it, and one unit's start, epilogue and waits run
// under the others' K loops.  gate/up 220 -> 158 us, down 182 -> 110 us at 2048 tokens; 172 -> 93 and 143 -> 65 us at 317.
// (Replaces src/tensorfold/cuda/experts_prefill.cu:31-195: prefill_kernel and its launch.)

#include "api.h"
#include "common.cuh"

namespace tfb {

constexpr int PF_ROWS = 128;            // weight rows a unit (MMA M)
constexpr int PF_MAXP = 192;            // pairs an item may hold (MMA N)
constexpr int PF_SMALL_MAXP = 64;       // the same in the build for plans of small items
constexpr int PF_DQ_WARPS = 8;          // warps 0-7: dequantise (two sets of four), then the epilogue

// What the two builds differ in.  Items of up to 192 pairs: two CTAs an SM.  Items of up to 64: a third of the accumulators
// and of the B ring, two gathering warps - three CTAs, because a unit of few pairs is mostly start, latency and epilogue.
// (317 tokens, top 8 of 128 and a shared expert: gate/up 119 us in the large build, 93 in this one, down 84 and 65.)
template <int MAXP>
struct PrefillShape {
  static constexpr int CTAS = MAXP > PF_SMALL_MAXP ? 2 : 3;                    // an SM
  static constexpr int GA_WARPS = MAXP > PF_SMALL_MAXP ? 4 : 2;               // warps 8 ..: gather the pairs' input rows
  static constexpr int MMA_WARP = PF_DQ_WARPS + GA_WARPS, COPY_WARP = MMA_WARP + 1;
  static constexpr int THREADS = (COPY_WARP + 1) * 32;
  static constexpr int GA_ROWS = GA_WARPS * 4;                                 // rows a pass of the gathering warps
  static constexpr int EPI_PARTS = MAXP > PF_SMALL_MAXP ? 3 : 2;              // warps a lane quarter in the epilogue
  static constexpr int A_COL = MAXP;                                           // tensor memory: accumulators, two A stages
  static constexpr int TMEM_COLS = MAXP + 64;
};

template <int M>
constexpr int PF_CB = PF_ROWS / COLS / M;   // packed column blocks a unit

// Two rings in shared memory: the B tiles (whole tiles of the item's own height, so items of fewer pairs get more
// stages) and the packed blocks as they come from HBM.
template <int MAXP>
struct PrefillSmem {
  static constexpr int SP = 8;
  static constexpr int B_BYTES = 3 * MAXP * 128;
  static constexpr int SB_MAX = 6;
  static constexpr int PACKED_BYTES = PF_ROWS / COLS * BLOCK_BYTES;
  static constexpr int PACKED_OFFSET = B_BYTES;
  static constexpr int TABLE_OFFSET = PACKED_OFFSET + SP * PACKED_BYTES;   // int out_row[MAXP]
  static constexpr int BAR_OFFSET = (TABLE_OFFSET + MAXP * 4 + 15) / 16 * 16;
  static constexpr int NBARS = 2 * SP + 2 * 2 + 2 * SB_MAX + 1;
  static constexpr int TMEM_OFFSET = BAR_OFFSET + NBARS * 8;
  static constexpr int TOTAL = TMEM_OFFSET + 16 + 1024;         // + slack to align the tiles to 1024 bytes
  static_assert(PrefillShape<MAXP>::CTAS * (TOTAL + 1024) <= 228 * 1024, "the CTAs share an SM's shared memory");
  static_assert(PrefillShape<MAXP>::CTAS * PrefillShape<MAXP>::TMEM_COLS <= 512, "and its tensor memory");
};

// ---- tcgen05 wrappers ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_addr(dst_smem)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

// K-major operand tile of rows x 64 bf16 (128 bytes a row), 128-byte swizzle, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);            // start address
  d |= (uint64_t)1 << 16;                              // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;                    // stride byte offset: the next 8-row group
  d |= (uint64_t)1 << 46;                              // descriptor version (sm_100)
  d |= (uint64_t)2 << 61;                              // SWIZZLE_128B
  return d;
}
// kind::f16: D fp32, A and B bf16, both K-major, M = 128, N = n
__device__ __forceinline__ uint32_t umma_idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(PF_ROWS >> 4) << 24);
}
// A from tensor memory: lane = row, a 32-bit column = two consecutive inputs (K = 16: eight columns)
__device__ __forceinline__ void umma_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d_tmem),
      "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accum)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smem_addr(bar))
               : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16};\n" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// The prefill form's weight pair from the bf16 pair (128 + q0, 128 + q1) and the column's (scale, bias) word.
// bf16 scales: bf16(q * s + b) with one rounding (a bf16 fma), as src/tensorfold/cuda/experts_prefill.cu:25-29;
// fp16 scales: the fp32 fma rounded to bf16.
template <int SB>
__device__ __forceinline__ uint32_t prefill_pair(uint32_t v, uint32_t sb) {
  if constexpr (SB == SB_BF16) {
    const uint32_t k128 = BF16_128, s2 = __byte_perm(sb, sb, 0x1010), b2 = __byte_perm(sb, sb, 0x3232);
    __nv_bfloat162 q = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&v),
                               *reinterpret_cast<const __nv_bfloat162*>(&k128));
    __nv_bfloat162 r = __hfma2(q, *reinterpret_cast<const __nv_bfloat162*>(&s2),
                               *reinterpret_cast<const __nv_bfloat162*>(&b2));
    return *reinterpret_cast<uint32_t*>(&r);
  } else {
    const float2 f = sb_pair<SB>(sb);
    const uint32_t k128 = BF16_128;
    const __nv_bfloat162 q = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&v),
                                     *reinterpret_cast<const __nv_bfloat162*>(&k128));   // exact
    const uint32_t qv = *reinterpret_cast<const uint32_t*>(&q);
    const float2 w = ffma2(make_float2(bf16_lo(qv), bf16_hi(qv)), make_float2(f.x, f.x), make_float2(f.y, f.y));
    __nv_bfloat162 r = __floats2bfloat162_rn(w.x, w.y);
    return *reinterpret_cast<uint32_t*>(&r);
  }
}

template <int M, int EPI, int SB, int MAXP>
__global__ void __launch_bounds__(PrefillShape<MAXP>::THREADS, PrefillShape<MAXP>::CTAS)
prefill_kernel(const __nv_bfloat16* __restrict__ X, int64_t x_stride, int slots, const uint8_t* __restrict__ W, int KG,
               int NB, const int* __restrict__ items, const int* __restrict__ counts, const int* __restrict__ members,
               void* __restrict__ out, int N, float limit) {
  using SM = PrefillSmem<MAXP>;
  using SH = PrefillShape<MAXP>;
  constexpr int SP = SM::SP, CB = PF_CB<M>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  int* out_row = reinterpret_cast<int*>(smem + SM::TABLE_OFFSET);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SM::BAR_OFFSET);
  uint64_t* packed_full = bars;                  // [SP] the bulk copy landed
  uint64_t* packed_free = bars + SP;             // [SP] the four warps of the stage's set have read it
  uint64_t* a_ready = bars + 2 * SP;             // [2] the four warps of the set stored their rows of the A stage
  uint64_t* a_free = a_ready + 2;                // [2] the MMAs that read the A stage retired
  uint64_t* b_ready = a_free + 2;                // [SB_MAX] the pairs' input rows landed
  uint64_t* b_free = b_ready + SM::SB_MAX;       // [SB_MAX] the MMAs that read the B stage retired
  uint64_t* acc_ready = b_free + SM::SB_MAX;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + SM::TMEM_OFFSET);

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nct = (NB + CB - 1) / CB;
  const int it = blockIdx.x / nct, ct = blockIdx.x - it * nct;

  if (tid == 0) {
    for (int s = 0; s < SP; ++s) {
      mbar_init(packed_full + s, 1);
      mbar_init(packed_free + s, PF_DQ_WARPS / 2);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(a_ready + s, PF_DQ_WARPS / 2);
      mbar_init(a_free + s, 1);
    }
    for (int s = 0; s < SM::SB_MAX; ++s) {
      mbar_init(b_ready + s, SH::GA_WARPS * 32);
      mbar_init(b_free + s, 1);
    }
    mbar_init(acc_ready, 1);
    mbar_fence_init();
    fence_async_smem();
  }
  pdl_wait();
  after_wait(X, items, counts, members);
  const bool live = it < ld_dep(counts);          // uniform over the CTA
  if (live && warp == SH::MMA_WARP) tmem_alloc(tmem_slot, SH::TMEM_COLS);
  int e = 0, first = 0, cnt = 0;
  if (live) {
    e = ld_dep(items + 3 * it);
    first = ld_dep(items + 3 * it + 1);
    cnt = min(ld_dep(items + 3 * it + 2), MAXP);
    for (int i = tid; i < MAXP; i += SH::THREADS) out_row[i] = i < cnt ? ld_dep(members + first + i) : -1;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (!live) return;
  const uint32_t tmem_base = *tmem_slot;
  const int nmma = max(16, (cnt + 15) & ~15);
  const int sb = min(SM::SB_MAX, SM::B_BYTES / (nmma * 128));    // B stages: 3 (192 pairs) to 6
  const int b_bytes = nmma * 128;                                // a multiple of 1024: 8-row swizzle groups stay aligned
  const int cb0 = ct * CB, ncb = min(CB, NB - cb0);              // packed column blocks of this unit
  bool ok = true;

  if (warp == SH::COPY_WARP) {
    // ---------------- packed weights: HBM -> the packed ring, a lane a column block, as far ahead as the ring allows
    const size_t cb_stride = (size_t)KG * (M * BLOCK_BYTES);
    const uint8_t* wsrc = W + (size_t)e * NB * cb_stride + (size_t)(cb0 + lane) * cb_stride;
    int g = 0;
    for (; g < KG; ++g, wsrc += M * BLOCK_BYTES) {
      const int s = g % SP, round = g / SP;
      if (round > 0) ok = mbar_wait_warp(packed_free + s, (round - 1) & 1);
      if (!ok) break;
      if (lane == 0) mbar_expect_tx(packed_full + s, (uint32_t)ncb * (M * BLOCK_BYTES));
      __syncwarp();
      if (lane < ncb)
        bulk_g2s(smem + SM::PACKED_OFFSET + s * SM::PACKED_BYTES + lane * (M * BLOCK_BYTES), wsrc, M * BLOCK_BYTES,
                 packed_full + s);
    }
    if (!ok && lane == 0)                            // give the copies in flight a while to land
      for (int f = max(0, g - SP); f < g; ++f) mbar_wait_for(packed_full + f % SP, (f / SP) & 1, 10000000ull);
    __syncwarp();
  } else if (warp == SH::MMA_WARP) {
    // ---------------- MMA issue: one lane ----------------
    if (lane == 0) {
      const uint32_t idesc = umma_idesc(nmma);
      const uint64_t desc0 = umma_desc(smem_addr(smem));       // addresses count 16 bytes
      int s = 0, ph = 0;
      for (int g = 0; g < KG && ok; ++g) {
        ok = mbar_wait(b_ready + s, ph) && mbar_wait(a_ready + (g & 1), (g >> 1) & 1);
        if (!ok) break;
        tc_fence_after();
        const uint64_t desc = desc0 + (uint32_t)(s * (b_bytes >> 4));
        const uint32_t a = tmem_base + SH::A_COL + (g & 1) * 32;
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) umma_ta(tmem_base, a + ks * 8, desc + 2 * ks, idesc, (g | ks) ? 1u : 0u);
        umma_commit(a_free + (g & 1));
        umma_commit(b_free + s);
        if (++s == sb) {
          s = 0;
          ph ^= 1;
        }
      }
      if (ok) umma_commit(acc_ready);
    }
    __syncwarp();
  } else if (warp >= PF_DQ_WARPS) {
    // ---------------- the gathering warps: the pairs' input rows into the swizzled B tiles ----------------
    // thread -> chunk c of rows r0, r0 + GA_ROWS, ...: the row pointers stay in registers for the whole K loop
    constexpr int GA_PER = MAXP / SH::GA_ROWS;       // 16-byte chunks a thread a stage
    const int gt = tid - PF_DQ_WARPS * 32, c = gt & 7, r0 = gt >> 3;
    const __nv_bfloat16* rowp[GA_PER];
#pragma unroll
    for (int j = 0; j < GA_PER; ++j) {
      const int p = out_row[min(r0 + SH::GA_ROWS * j, cnt - 1)];   // rows past the last repeat it: their columns are never stored
      rowp[j] = X + (size_t)(slots ? p / slots : p) * x_stride + c * 8;
    }
    const uint32_t boff = (uint32_t)(r0 * 128 + ((c ^ (r0 & 7)) << 4));      // rows GA_ROWS apart share r & 7
    int s = 0, ph = 1, back = 0;                     // ph: a ring's first round finds every stage free
    for (int g = 0; g < KG && ok; ++g) {
      if (g >= sb) ok = mbar_wait_warp(b_free + s, ph);
      if (!ok) break;
      uint8_t* btile = smem + s * b_bytes + boff;
#pragma unroll
      for (int j = 0; j < GA_PER; ++j) {
        if (SH::GA_ROWS * j >= cnt) break;
        cp_async16(btile + j * (SH::GA_ROWS * 128), rowp[j]);
        rowp[j] += GS;
      }
      cp_async_commit();
      if (++s == sb) {
        s = 0;
        ph ^= 1;
      }
      if (g >= 1) {                                  // the stage before this one has landed: publish it
        cp_async_wait<1>();
        fence_async_smem();
        mbar_arrive(b_ready + back);
        if (++back == sb) back = 0;
      }
    }
    cp_async_wait<0>();
    fence_async_smem();
    if (ok) mbar_arrive(b_ready + back);
  } else {
    // ---------------- warps 0-7: dequantise into the A stages ----------------
    // A lane holds one weight row: tensor-memory lanes 32 q .. 32 q + 31 belong to warps q and q + 4.  Lane 4 gq + t
    // takes column 8 (t & 1) + gq of a 16-column tile; t >> 1 picks the tile (one matrix: of the two of column block
    // q) or the matrix (gate / up: of tile q & 1 of column block q >> 1).
    // A row's 64 nibbles are four 8-byte pieces, 16 bytes apart; the lanes read them in rotated orders so that a half
    // warp's loads touch every bank once (in the same order they were a four-way conflict), and the rotation is
    // undone in registers.
    const int gq = lane >> 2, t = lane & 3, q = warp & 3, set = warp >> 2;
    const int cbw = M == 1 ? q : q >> 1, tt = M == 1 ? t >> 1 : q & 1, mm = M == 1 ? 0 : t >> 1, hi = t & 1;
    const int rot = (t >> 1) * 2 + ((gq >> 1) & 1);
    const int at = cbw * (M * BLOCK_BYTES) + mm * BLOCK_BYTES;
    const int w_at = at + tt * TILE_BYTES + gq * 64 + hi * 8, sb_at = at + SB_OFFSET + gq * 16 + (2 * tt + hi) * 4;
    const uint32_t a_dst = tmem_base + ((uint32_t)(q * 32) << 16) + SH::A_COL + set * 32;
    for (int g = set; g < KG && ok; g += 2) {
      const int sp = g % SP;
      ok = mbar_wait_warp(packed_full + sp, (g / SP) & 1);
      if (!ok) break;
      const uint8_t* blk = smem + SM::PACKED_OFFSET + sp * SM::PACKED_BYTES;
      uint2 w[4];
      // (a block that the unit lacks: whatever the slot holds, its columns are never stored)
      const uint32_t sbw = *reinterpret_cast<const uint32_t*>(blk + sb_at);
#pragma unroll
      for (int u = 0; u < 4; ++u) w[u] = *reinterpret_cast<const uint2*>(blk + w_at + (((u + rot) & 3) << 4));
      __syncwarp();
      mbar_arrive_if(packed_free + sp, lane == 0);
      uint2 v[4], x[4];                              // piece k = w[(k - rot) & 3]
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = (rot & 1) ? w[(k + 3) & 3] : w[k];
#pragma unroll
      for (int k = 0; k < 4; ++k) x[k] = (rot & 2) ? v[(k + 2) & 3] : v[k];
#pragma unroll
      for (int h = 0; h < 2; ++h) {                  // half a row: 32 inputs, 16 columns
        uint32_t o[16];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t word = i & 1 ? x[2 * h + (i >> 1)].y : x[2 * h + (i >> 1)].x;
#pragma unroll
          for (int j = 0; j < 4; ++j) o[4 * i + j] = prefill_pair<SB>(nib_pair(word, 4 * j), sbw);
        }
        if (h == 0 && g >= 2) {
          ok = mbar_wait_warp(a_free + set, ((g >> 1) - 1) & 1);
          if (!ok) break;
          tc_fence_after();
        }
        tmem_st16(a_dst + 16 * h, o);
      }
      if (!ok) break;
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      mbar_arrive_if(a_ready + set, lane == 0);
    }
  }
  // ---------------- epilogue: the dequantising warps, and the four gathering warps of the large build ----------------
  // TMEM lane quarter warp & 3, a weight row a lane (numbered as the dequantising warps do); the two or three warps
  // of a quarter take a part of the pairs each, 16 pairs a load.  Gate and up rows of a column sit in lanes 2 apart: of
  // two neighbouring pairs the gate lane forms the first and the up lane the second, one exchange for both.
  if (warp < 4 * SH::EPI_PARTS) {
    if (ok) ok = mbar_wait_warp(acc_ready, 0);
    if (ok) {
      tc_fence_after();
      const int q = warp & 3, part = warp >> 2, gq = lane >> 2, t = lane & 3;
      const int col = M == 1 ? ct * PF_ROWS + q * 32 + (t >> 1) * 16 + (t & 1) * 8 + gq
                             : ct * (PF_ROWS / 2) + q * 16 + (t & 1) * 8 + gq;
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16);
      const int blocks = nmma / 16, per = (blocks + SH::EPI_PARTS - 1) / SH::EPI_PARTS;
      const int jb = min(blocks, part * per) * 16, je = min(blocks, (part + 1) * per) * 16;
      for (int j0 = jb; j0 < je; j0 += 16) {
        uint32_t a[16];
        tmem_ld16(taddr + j0, a);
        tmem_ld_wait();
        // the values first (independent chains the compiler can interleave: one after the other, each behind its own
        // row lookup and branch, they took 2 us a block), then their rows and the stores
        if constexpr (M == 2) {
          static_assert(EPI == EPI_SWIGLU, "two matrices: gate and up");
          const bool up_lane = (t & 2) != 0;
          float r[8];
          int rows[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float give = __uint_as_float(up_lane ? a[2 * j] : a[2 * j + 1]);
            const float keep = __uint_as_float(up_lane ? a[2 * j + 1] : a[2 * j]);
            const float got = __shfl_xor_sync(0xffffffffu, give, 2);
            rows[j] = out_row[j0 + 2 * j + (up_lane ? 1 : 0)];
            r[j] = swiglu_fast(up_lane ? got : keep, up_lane ? keep : got, limit);
          }
          if (col < N) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (rows[j] >= 0)
                static_cast<__nv_bfloat16*>(out)[(size_t)rows[j] * N + col] = __float2bfloat16_rn(r[j]);
          }
        } else if (col < N) {
          float r[16];
          int rows[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float v = __uint_as_float(a[j]);
            rows[j] = out_row[j0 + j];
            r[j] = EPI == EPI_RELU2 ? relu2(v) : v;
          }
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            if (rows[j] < 0) continue;
            const size_t at = (size_t)rows[j] * N + col;
            if constexpr (EPI == EPI_F32) {
              static_cast<float*>(out)[at] = r[j];
            } else {
              static_cast<__nv_bfloat16*>(out)[at] = __float2bfloat16_rn(r[j]);
            }
          }
        }
      }
    }
  }
  pdl_launch_dependents();
  tc_fence_before();
  __syncthreads();
  if (warp == SH::MMA_WARP) tmem_dealloc(tmem_base, SH::TMEM_COLS);
}

template <int M, int EPI, int SB, int MAXP>
int launch_prefill(const void* x, int64_t x_stride, int slots, const void* w, int kg, int nb, const int* items,
                   const int* counts, const int* members, void* out, int n, float limit, int64_t max_items,
                   cudaStream_t stream) {
  using SM = PrefillSmem<MAXP>;
  auto* kern = prefill_kernel<M, EPI, SB, MAXP>;
  static bool configured[64] = {false};
  int dev = 0;
  TFB_CUDA(cudaGetDevice(&dev), "experts_prefill: cudaGetDevice");
  if (dev < 0 || dev >= 64) return fail(TFB_ERR_ARG, "experts_prefill: device index %d out of range", dev);
  if (!configured[dev]) {
    TFB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SM::TOTAL),
             "experts_prefill: shared memory opt-in");
    configured[dev] = true;
  }
  const int64_t grid = max_items * ((nb + PF_CB<M> - 1) / PF_CB<M>);
  if (grid >= (int64_t(1) << 31)) return fail(TFB_ERR_ARG, "experts_prefill: too many units");
  return check_cuda(launch(kern, dim3((unsigned)grid), dim3(PrefillShape<MAXP>::THREADS), (size_t)SM::TOTAL, stream,
                           static_cast<const __nv_bfloat16*>(x), x_stride, slots, static_cast<const uint8_t*>(w), kg,
                           nb, items, counts, members, out, n, limit),
                    "experts_prefill");
}

}  // namespace tfb

using namespace tfb;

static int experts_prefill(int gs, int epi, const void* x, int64_t x_stride, int slots, const void* w, int kg, int nb,
                           const int32_t* items, const int32_t* counts, const int32_t* members, void* out, int n,
                           float limit, int64_t max_items, int sb_type, int tile, void* stream) {
  TFB_REQUIRE(gs == GS, "experts_prefill: groups of %d inputs only, not %d", GS, gs);
  TFB_REQUIRE(x && w && items && counts && members && out, "experts_prefill: null pointer");
  TFB_REQUIRE(kg >= 1 && nb >= 1 && n == nb * COLS, "experts_prefill: n must be the column blocks times %d", COLS);
  TFB_REQUIRE(aligned16(x) && x_stride % 8 == 0 && x_stride >= (int64_t)kg * GS,
              "experts_prefill: x rows of K = groups * group size inputs, 16-byte aligned");
  TFB_REQUIRE(aligned16(w), "experts_prefill: w must be 16-byte aligned");
  TFB_REQUIRE(slots >= 0 && max_items >= 0, "experts_prefill: bad slots or item count");
  TFB_REQUIRE(sb_type == SB_BF16 || sb_type == SB_FP16, "experts_prefill: scales are bf16 (0) or fp16 (1), not %d",
              sb_type);
  TFB_REQUIRE(tile >= 1 && tile <= PF_MAXP, "experts_prefill: items of 1..%d pairs, not %d", PF_MAXP, tile);
  if (max_items == 0) return TFB_OK;
  auto st = static_cast<cudaStream_t>(stream);
#define TFB_PRE2(EPI_, M_, SB_)                                                                                        \
  return tile <= PF_SMALL_MAXP                                                                                         \
             ? launch_prefill<M_, EPI_, SB_, PF_SMALL_MAXP>(x, x_stride, slots, w, kg, nb, items, counts, members, out, \
                                                            n, limit, max_items, st)                                   \
             : launch_prefill<M_, EPI_, SB_, PF_MAXP>(x, x_stride, slots, w, kg, nb, items, counts, members, out, n,    \
                                                      limit, max_items, st)
#define TFB_PRE(EPI_, M_)                              \
  if (epi == EPI_) {                                   \
    if (sb_type == SB_BF16) TFB_PRE2(EPI_, M_, SB_BF16); \
    TFB_PRE2(EPI_, M_, SB_FP16);                       \
  }
  TFB_PRE(EPI_F32, 1) TFB_PRE(EPI_RELU2, 1) TFB_PRE(EPI_SWIGLU, 2) TFB_PRE(EPI_BF16, 1)
#undef TFB_PRE
#undef TFB_PRE2
  return fail(TFB_ERR_ARG, "experts_prefill: no kernel for epilogue %d", epi);
}

// Grouped 4-bit expert matmul, prefill form, over a plan whose items hold at most 192 pairs.  Arguments as the
// reference extension's `prefill` (src/tensorfold/cuda/experts.cpp:50-56); max_items = an upper bound of the items.
extern "C" int tfb_experts_prefill(int gs, int epi, const void* x, int64_t x_stride, int slots, const void* w, int kg,
                                   int nb, const int32_t* items, const int32_t* counts, const int32_t* members,
                                   void* out, int n, float limit, int64_t max_items, int sb_type, void* stream) {
  return experts_prefill(gs, epi, x, x_stride, slots, w, kg, nb, items, counts, members, out, n, limit, max_items, sb_type,
                         PF_MAXP, stream);
}

// The same over a plan whose items hold at most `tile` pairs (1..192): with 64 or fewer a build with less of an SM to a
// CTA, three of them an SM.  A pair's bits do not depend on the tile.
extern "C" int tfb_experts_prefill_tile(int gs, int epi, const void* x, int64_t x_stride, int slots, const void* w, int kg,
                                        int nb, const int32_t* items, const int32_t* counts, const int32_t* members,
                                        void* out, int n, float limit, int64_t max_items, int sb_type, int tile,
                                        void* stream) {
  return experts_prefill(gs, epi, x, x_stride, slots, w, kg, nb, items, counts, members, out, n, limit, max_items, sb_type,
                         tile, stream);
}
