// Routed experts on EXL3 trellis-coded weights (ExLlamaV3's format), any codebook, a width per expert matrix.
//
// A 16 x 16 tile is a circular MSB-first bitstream of 256 values; value p's 16-bit state is the window ending at
// E(p) = (p >> 1) K2 + (p odd ? K2 : K2 >> 1) (K2 = half-bits a value); a codebook turns a state into an fp16 value;
// value p sits at row 2 (l % 4) + (j & 1) + 8 ((j >> 1) & 1), column l / 4 + 8 (j >> 2) of its tile (l = p / 8,
// j = p % 8) - so lane l's eight values are exactly its mma.m16n8k16 fragment of the tile.  Here the tile
// (transposed) is the A operand (16 output columns x 16 inputs) and the pairs' rotated inputs the B operand.
// The layer is y = (((x * suh) H) W_q) H * svh per 128-block, H = 128-point Hadamard / sqrt(128).
//
// Three launches a layer call (src/tensorfold/cuda/exl3/experts.py:173-202 needs seven):
//   prologue  one block sorts the (row, slot) pairs by expert into items of <= 16 or 32 pairs (the affine plan's sort),
//             the others rotate every routed pair's input for gate and up (x * suh, 128-point transform, fp16);
//   gate/up   CTA = (item, 64 columns, matrix): the four warps split K, each pulls its rows of tiles through a private
//             shared-memory ring with bulk async copies, decodes from shared memory and multiplies; the K slices meet
//             in warp order; the LAST of the four CTAs that share (item, 128 columns) - counted with an atomic - runs
//             the epilogue (rotate, svh, SwiGLU, suh_d, rotate) for the block and stores the down projection's input;
//   down      the same kernel with the output rotation (and svh) as its epilogue; y fp32 per pair.
// Calls with many pairs an expert sort into items of <= 32 pairs, which a second form of the kernel takes
// (grouped_tc_kernel: 128 columns a CTA, decoded tiles go to tensor memory, tcgen05.mma multiplies): the same sums.
// Fixed-order reductions everywhere: a pair's bits never depend on the other rows of the call.
// (Replaces src/tensorfold/cuda/exl3/experts.cu and experts_grouped.cuh; the trellises are read in place.)

#include <type_traits>

#include "api.h"
#include "common.cuh"

namespace tfb {
namespace exl3 {

constexpr float HAD_SCALE = 0.08838834764831845f;   // 1 / sqrt(128)
constexpr int GR_WARPS = 4;                         // K slices a CTA (part of the arithmetic: they meet in warp order)
constexpr int GR_NTB = 4;                           // 16-column tiles a CTA: 64 columns (2: the narrow CTAs, 32 columns)
constexpr int GR_NARROW_NTB = 2;
constexpr int GR_PT = 2;                            // mma tiles of 8 pairs an item: 16 pairs
constexpr int GR_PAIRS = 8 * GR_PT;
constexpr int GR_SLOT_BYTES = 2048;                 // a ring slot: whole rows of the CTA's four tiles
constexpr int GR_STAGES = 3;

// the tensor-memory kernel (the wide items)
constexpr int TC_SETS = 4;                          // sets of four decoding warps; a set takes every fourth step
constexpr int TC_DEC_WARPS = 4 * TC_SETS;           // warps 0-15: decode, then the epilogue
constexpr int TC_LOAD_WARP = TC_DEC_WARPS, TC_MMA_WARP = TC_DEC_WARPS + 1;
constexpr int TC_THREADS = (TC_DEC_WARPS + 2) * 32;
constexpr int TC_COLS = 128;                        // output columns a CTA (MMA M), one rotation block
constexpr int TC_PAIRS = 32;                        // the most pairs an item holds (MMA N)
constexpr int TC_STEP = 64;                         // inputs a step; a stage of the rings: two steps
constexpr int TC_PARTS = 4;                         // parts of K, an accumulator each (part of the arithmetic)
constexpr int TC_A_COL = TC_PARTS * TC_PAIRS;  // tensor memory: the accumulators, then an A stage a set
constexpr int TC_TMEM_COLS = TC_A_COL + 32 * TC_SETS;

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) { return __byte_perm(a, b, sel); }

// ---- codebooks: two states -> two fp16 values (src/tensorfold/cuda/exl3/format.py:31-48) ------------------------
template <int CB>
__device__ __forceinline__ uint32_t cb_pair(uint32_t s0, uint32_t s1) {
  if constexpr (CB == 2) {                            // mul1: fma(1024 + sum of the bytes of s * M, scale, bias) in fp16
    const uint32_t h0 = __dp4a(s0 * 0x83DCD12Du, 0x01010101u, 0x6400u);
    const uint32_t h1 = __dp4a(s1 * 0x83DCD12Du, 0x01010101u, 0x6400u);
    const uint32_t hv = prmt(h0, h1, 0x5410);
    const __half2 r = __hfma2(*reinterpret_cast<const __half2*>(&hv), __half2half2(__ushort_as_half(0x1EEE)),
                              __half2half2(__ushort_as_half(0xC931)));
    return *reinterpret_cast<const uint32_t*>(&r);
  } else {                                            // 3inst / mcg: the two fp16 halves of the masked product, added
    uint32_t x0 = CB == 1 ? s0 * 0xCBAC1FEDu : s0 * 89226354u + 64248484u;
    uint32_t x1 = CB == 1 ? s1 * 0xCBAC1FEDu : s1 * 89226354u + 64248484u;
    asm("lop3.b32 %0, %1, %2, %3, 0x6A;\n" : "=r"(x0) : "r"(x0), "r"(0x8FFF8FFFu), "r"(0x3B603B60u));   // (x & M) ^ F
    asm("lop3.b32 %0, %1, %2, %3, 0x6A;\n" : "=r"(x1) : "r"(x1), "r"(0x8FFF8FFFu), "r"(0x3B603B60u));
    // each value = low half + high half of its own word: the fp16 adds take the halves straight from the register
    // (no permute), one permute packs the two results
    uint32_t r;
    asm("{\n.reg .b16 a, b, c, d;\n"
        "mov.b32 {a, b}, %1;\n"
        "mov.b32 {c, d}, %2;\n"
        "add.rn.f16 a, a, b;\n"
        "add.rn.f16 c, c, d;\n"
        "mov.b32 %0, {a, c};\n}\n"
        : "=r"(r)
        : "r"(x0), "r"(x1));
    return r;
  }
}

// ---- a lane's eight states of a tile ----------------------------------------------------------------------------
// delta(j): first bit of value 8 l + j's window relative to value 8 l's (the same for every lane)
template <int K2>
__host__ __device__ constexpr int delta(int j) {
  return ((j + 1) * K2 - ((K2 & 1) ? ((j + 1) & 1) : 0)) / 2 - (K2 >> 1);
}
template <int K2>
struct Win {
  static constexpr int TW = 4 * K2;                                 // 32-bit words a tile
  static constexpr int SPAN = delta<K2>(7) + 16;                    // stream bits a lane's windows cover
  static constexpr int NW = K2 == 8 ? 2 : (31 + SPAN + 31) / 32;    // words a lane reads (worst offset; <= 4)
  static constexpr int NV = (SPAN + 31) / 32;                       // 32-bit chunks of the lane's span
};

// The words of a tile a lane needs: NW consecutive words (cyclically) from the one holding the first bit of value
// 8 lane's window.  4 bits a value (K2 = 8): exactly words lane - 1 and lane.  GLOBAL: the tile is in global memory
// (read-only path); else in shared memory.
template <int K2, bool GLOBAL>
__device__ __forceinline__ void lane_words(const uint32_t* __restrict__ tile, int lane, uint32_t (&w)[Win<K2>::NW]) {
  constexpr int TW = Win<K2>::TW, NW = Win<K2>::NW;
  const int first = 4 * lane * K2 + (K2 >> 1) - 16 + 32 * TW;       // E(8 lane) - 16, made non-negative
  int wi = (first >> 5) % TW;
#pragma unroll
  for (int i = 0; i < NW; ++i) {
    w[i] = GLOBAL ? __ldg(tile + wi) : tile[wi];
    wi = wi + 1 == TW ? 0 : wi + 1;
  }
}

// A 16-bit half of a word, zero-extended.  MUL: by a two-way dot product (times 1 and 0), which runs on the multiply
// pipe; else by a byte permute on the ALU pipe.  Both pipes take one instruction every two cycles a scheduler and the
// decode is bound by the fuller one, so the states' extraction is split between them: 4.00 bits 23 ALU + 16 multiply ->
// 19 + 20 (61 -> 54 cycles a tile in a loop of its own), the other widths 28-30 + 16 -> 22 + 24 (71 -> 64).
template <bool MUL>
__device__ __forceinline__ uint32_t half_hi(uint32_t w) {
  return MUL ? __dp2a_lo(w, 0x0100u, 0u) : prmt(w, 0u, 0x4432);
}
template <bool MUL>
__device__ __forceinline__ uint32_t half_lo(uint32_t w) {
  return MUL ? __dp2a_lo(w, 0x0001u, 0u) : prmt(w, 0u, 0x4410);
}

// st[j] = state of value 8 lane + j from the lane's words.  MUL: the multiply pipe has room (not with a codebook that
// uses it for a byte sum).
template <int K2, bool MUL>
__device__ __forceinline__ void lane_states(const uint32_t (&w)[Win<K2>::NW], int lane, uint32_t (&st)[8]) {
  constexpr int NW = Win<K2>::NW, NV = Win<K2>::NV;
  if constexpr (K2 == 8) {
    // 16-bit windows ending 4 (j + 1) bits into the lane's own word w[1], the stream running on from w[0]: a word that
    // starts with window j ends with window j + 4
    const uint32_t t[4] = {__funnelshift_l(w[1], w[0], 20), __funnelshift_l(w[1], w[0], 24),
                           __funnelshift_l(w[1], w[0], 28), w[1]};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      st[j] = half_hi<false>(t[j]);
      st[j + 4] = half_lo<MUL>(t[j]);
    }
  } else {
    const int off = (4 * lane * K2 + (K2 >> 1) - 16 + 32 * Win<K2>::TW) & 31;
    uint32_t v[NV];                                   // v[i] = stream bits [first + 32 i, first + 32 i + 32)
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] = __funnelshift_l(i + 1 < NW ? w[i + 1] : 0u, w[i], off);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int d = delta<K2>(j), i = d >> 5, o = d & 31;
      const uint32_t next = v[i + 1 < NV ? i + 1 : i];   // o > 16: the window runs into it (d + 16 <= SPAN: it exists)
      if (o == 0) {
        st[j] = half_hi<MUL>(v[i]);
      } else if (o == 16) {
        st[j] = half_lo<MUL>(v[i]);
      } else if (o == 8) {                            // on a byte boundary: one permute cuts it out
        st[j] = prmt(v[i], 0u, 0x4421);
      } else if (o < 16) {
        st[j] = half_lo<MUL>(v[i] >> (16 - o));
      } else {
        st[j] = half_hi<MUL>(__funnelshift_l(next, v[i], o));
      }
    }
  }
}

// The lane's tile values as the mma A fragment of the transposed tile (rows = output columns, k = inputs):
// a0 = (col g, k 2t, 2t+1) = values 0, 1; a1 = (col g + 8, same k) = values 4, 5; a2 = (col g, k + 8) = values 2, 3;
// a3 = (col g + 8, k + 8) = values 6, 7.
template <int CB, int K2>
__device__ __forceinline__ void decode_words(const uint32_t (&w)[Win<K2>::NW], int lane, uint32_t (&a)[4]) {
  uint32_t st[8];
  lane_states<K2, CB != 2>(w, lane, st);
  a[0] = cb_pair<CB>(st[0], st[1]);
  a[2] = cb_pair<CB>(st[2], st[3]);
  a[1] = cb_pair<CB>(st[4], st[5]);
  a[3] = cb_pair<CB>(st[6], st[7]);
}

__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// One warp's k-tile rows [kt0, kt0 + nkt) of the CTA's four column tiles into acc.  The rows travel through the warp's
// ring: a slot holds ROWS whole rows (one bulk copy a row: the four tiles of a row are contiguous in the trellis), the
// elected lane refills a slot as soon as the warp has decoded it.  The rows of a slot are unrolled in blocks of up to
// four, whose inputs are loaded before the block's tiles are decoded.  x[pt]: the lane's pair (B column lane / 4 of
// tile pt) at input 16 kt0 + 2 (lane % 4).  NPT: the mma tiles of eight pairs that are live (one decode feeds them all).
// Returns false when a copy never landed.
template <int CB, int K2, int PT, int NPT, int NTB, bool COMPACT, bool INLINE_WAIT>
__device__ __forceinline__ bool warp_rows(const uint8_t* __restrict__ T, int ntiles, int kt0, int nkt, int nt0,
                                          const __half* const (&x)[PT], uint8_t* ring, uint64_t* bars, int lane,
                                          float (&acc)[NTB][PT][4]) {
  constexpr int TW = Win<K2>::TW, NW = Win<K2>::NW;
  constexpr int TILE_B = 16 * K2, SEG = NTB * TILE_B;                 // bytes a tile / a row of the CTA's tiles
  constexpr int ROWS = GR_SLOT_BYTES / SEG < 1 ? 1 : (GR_SLOT_BYTES / SEG > 16 ? 16 : GR_SLOT_BYTES / SEG);
  // rows a block (their inputs sit in registers; 4 was 3 % slower).  COMPACT: one row a block and the blocks of a slot
  // walked by a loop - a fifth of the code, for layers of mixed widths, where blocks that decode different widths
  // share an SM and the unrolled loops of five or seven widths miss the instruction cache all the time
  constexpr int RBMAX = COMPACT ? 1 : 2;
  constexpr int RB = ROWS < RBMAX ? ROWS : RBMAX;
  static_assert(ROWS * SEG <= GR_SLOT_BYTES, "a slot holds whole rows");
  const int nslot = (nkt + ROWS - 1) / ROWS;
  const uint8_t* src = T + ((size_t)kt0 * ntiles + nt0) * TILE_B;
  const size_t row_stride = (size_t)ntiles * TILE_B;
  auto issue = [&](int f) {
    const int rows = min(ROWS, nkt - f * ROWS);
    uint64_t* bar = bars + f % GR_STAGES;
    uint8_t* dst = ring + (f % GR_STAGES) * GR_SLOT_BYTES;
    mbar_expect_tx(bar, (uint32_t)(rows * SEG));
    for (int r = 0; r < rows; ++r) bulk_g2s(dst + r * SEG, src + (size_t)(f * ROWS + r) * row_stride, SEG, bar);
  };
  if (lane == 0)
    for (int f = 0; f < GR_STAGES && f < nslot; ++f) issue(f);
  // where the lane's words sit inside a tile: NW consecutive words (cyclically) from the one that holds the first bit
  // of value 8 lane's window
  int word[NW];
  {
    int wi = ((4 * lane * K2 + (K2 >> 1) - 16 + 32 * TW) >> 5) % TW;
#pragma unroll
    for (int j = 0; j < NW; ++j) {
      word[j] = wi;
      wi = wi + 1 == TW ? 0 : wi + 1;
    }
  }
  const __half* xp[PT];
#pragma unroll
  for (int pt = 0; pt < PT; ++pt) xp[pt] = x[pt];
  int stage = 0;
  uint32_t phase = 0;
  for (int f = 0; f < nslot; ++f) {
    const int rows = min(ROWS, nkt - f * ROWS);
    const uint32_t* slot = reinterpret_cast<const uint32_t*>(ring + stage * GR_SLOT_BYTES);
#pragma unroll(COMPACT ? 1 : 16)
    for (int r0 = 0; r0 < ROWS; r0 += RB) {
      if (r0 < rows) {
        uint32_t b[RB][NPT][2];
#pragma unroll
        for (int r = 0; r < RB; ++r)
#pragma unroll
          for (int pt = 0; pt < NPT; ++pt) {
            b[r][pt][0] = b[r][pt][1] = 0u;
            if (r0 + r < rows) {
              b[r][pt][0] = *reinterpret_cast<const uint32_t*>(xp[pt] + (r0 + r) * 16);
              b[r][pt][1] = *reinterpret_cast<const uint32_t*>(xp[pt] + (r0 + r) * 16 + 8);
            }
          }
        if (r0 == 0 && !(INLINE_WAIT ? mbar_wait_warp_inline(bars + stage, phase) : mbar_wait_warp(bars + stage, phase))) {
          for (int g = f + 1; g < nslot && g < f + GR_STAGES; ++g)    // give the other copies in flight a while to land
            mbar_wait_for(bars + g % GR_STAGES, (g / GR_STAGES) & 1, 10000000ull);
          return false;
        }
#pragma unroll
        for (int r = 0; r < RB; ++r) {
          if (r0 + r < rows) {
#pragma unroll
            for (int i = 0; i < NTB; ++i) {
              const uint32_t* tile = slot + (r0 + r) * (SEG / 4) + i * TW;
              uint32_t w[NW], a[4];
#pragma unroll
              for (int j = 0; j < NW; ++j) w[j] = tile[word[j]];
              decode_words<CB, K2>(w, lane, a);
#pragma unroll
              for (int pt = 0; pt < NPT; ++pt) mma_f16(acc[i][pt], a, b[r][pt][0], b[r][pt][1]);   // one decode, every pair tile
            }
          }
        }
      }
    }
#pragma unroll
    for (int pt = 0; pt < PT; ++pt) xp[pt] += ROWS * 16;
    __syncwarp();
    if (lane == 0 && f + GR_STAGES < nslot) issue(f + GR_STAGES);
    if (++stage == GR_STAGES) {
      stage = 0;
      phase ^= 1u;
    }
  }
  return true;
}

// Two k-tiles of a 16-column tile go to tensor memory as the MMA's A operand: 16 lanes (columns) x 128
// bits a repeat, register 2 r = (lane g, 32-bit column 4 r + t), 2 r + 1 = (lane g + 8, the same) - which is where a
// decoded tile's four registers already are.
__device__ __forceinline__ void tmem_st_16x128b_x4(uint32_t taddr, const uint32_t (&a)[2][4]) {
  asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"r"(taddr),
               "r"(a[0][0]), "r"(a[0][1]), "r"(a[0][2]), "r"(a[0][3]), "r"(a[1][0]), "r"(a[1][1]), "r"(a[1][2]),
               "r"(a[1][3])
               : "memory");
}

// Shared memory of a CTA: the trellis ring (stages of 128 inputs x 128 columns: 1024 K2 bytes), the B ring (32 pairs x
// 128 inputs a stage, two 128-byte-swizzled tiles), the pair table, barriers.  After the main loop the trellis ring's
// memory takes the sums ([32][128] fp32).
struct TrellisSmem {
  static constexpr int RING_BYTES = 65536, SP_MAX = 8;
  static constexpr int B_TILE = TC_PAIRS * 128, SB = 4;
  static constexpr int B_OFFSET = RING_BYTES;
  static constexpr int PAIR_OFFSET = B_OFFSET + SB * 2 * B_TILE;
  static constexpr int BAR_OFFSET = PAIR_OFFSET + TC_PAIRS * 4;
  static constexpr int NBARS = 2 * SP_MAX + 2 * TC_SETS + 2 * SB + 1;
  static constexpr int FLAG_OFFSET = BAR_OFFSET + NBARS * 8;     // tensor-memory address, last-arrival flag
  static constexpr int TOTAL = FLAG_OFFSET + 16 + 1024;          // + slack to align the tiles to 1024 bytes
};
static_assert(TC_PARTS * TC_PAIRS * TC_COLS * 4 <= TrellisSmem::RING_BYTES, "every part's accumulators fit the ring");
static_assert(2 * (TrellisSmem::TOTAL + 1024) <= 228 * 1024 && 2 * TC_TMEM_COLS <= 512, "two CTAs share an SM");

template <int K2>
struct Ring {
  static constexpr int STAGE_BYTES = 2 * TC_STEP / 16 * (TC_COLS / 16) * 16 * K2;
  static constexpr int SP = K2 <= 8 ? 8 : 4;
  static_assert(SP * STAGE_BYTES <= TrellisSmem::RING_BYTES && SP <= TrellisSmem::SP_MAX, "the ring holds its stages");
};

// One decoding warp's share of the CTA's steps of 64 inputs: warp q of a set takes the column tiles 2 q and 2 q + 1
// (tensor-memory lanes 32 q ..) of the set's steps.  Returns false when a wait ran out.
template <int CB, int K2>
__device__ __forceinline__ bool decode_stages(const uint8_t* ring, uint64_t* packed_full, uint64_t* packed_free,
                                              uint64_t* a_ready, uint64_t* a_free, uint32_t a_dst, int set, int q,
                                              int steps, int lane) {
  constexpr int TW = Win<K2>::TW, NW = Win<K2>::NW, SP = Ring<K2>::SP;
  // where the lane's words sit inside a tile: NW consecutive words (cyclically) from the one that holds the first bit
  // of value 8 lane's window
  int word[NW];
  {
    int wi = ((4 * lane * K2 + (K2 >> 1) - 16 + 32 * TW) >> 5) % TW;
#pragma unroll
    for (int j = 0; j < NW; ++j) {
      word[j] = wi + ((set & 1) * (TC_STEP / 16) * (TC_COLS / 16) + 2 * q) * TW;   // odd sets: a stage's second step
      wi = wi + 1 == TW ? 0 : wi + 1;
    }
  }
  for (int g = set, use = 0; g < steps; g += TC_SETS, ++use) {
    const int p = g >> 1, sp = p % SP;
    if (!mbar_wait_warp(packed_full + sp, (p / SP) & 1)) return false;
    if (use > 0) {
      if (!mbar_wait_warp(a_free + set, (use - 1) & 1)) return false;
      tc_fence_after();
    }
    const uint32_t* stage = reinterpret_cast<const uint32_t*>(ring + sp * Ring<K2>::STAGE_BYTES);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t a[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint32_t* tile = stage + ((2 * h + i) * (TC_COLS / 16) + c) * TW;
          uint32_t w[NW];
#pragma unroll
          for (int j = 0; j < NW; ++j) w[j] = tile[word[j]];
          uint32_t v[4];
          decode_words<CB, K2>(w, lane, v);
#pragma unroll
          for (int j = 0; j < 4; ++j) a[i][j] = v[j];
        }
        tmem_st_16x128b_x4(a_dst + ((uint32_t)(16 * c) << 16) + 16 * h, a);
      }
    }
    __syncwarp();
    mbar_arrive_if(packed_free + sp, lane == 0);
    tmem_st_wait();
    tc_fence_before();
    __syncwarp();
    mbar_arrive_if(a_ready + set, lane == 0);
  }
  return true;
}

// ---- 128-point Walsh-Hadamard transform by 16 lanes, 8 consecutive values a lane ---------------------------------
// Strides 1, 2, 4 inside the lane, 8 .. 64 across the 16 lanes of a half warp (sub = lane % 16); a warp transforms two
// blocks at once.  Not scaled.  FMA: o + v or o - v across the lanes as one fma with the lane's sign (the product is exact:
// the same bits) instead of two adds and a select - for the kernels that do little else (the prologue at 512 tokens of a
// 4096-wide layer 43 -> 38 us); inside grouped_kernel the extra live values cost its main loop 5 %.
template <bool FMA>
__device__ __forceinline__ void hadamard128(float (&v)[8], int sub) {
#pragma unroll
  for (int h = 1; h < 8; h <<= 1)
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if ((i & h) == 0) {
        const float a = v[i], b = v[i + h];
        v[i] = a + b;
        v[i + h] = a - b;
      }
#pragma unroll
  for (int m = 1; m < 16; m <<= 1) {
    const float sign = (sub & m) ? -1.f : 1.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float o = __shfl_xor_sync(0xffffffffu, v[i], m);
      if constexpr (FMA)
        v[i] = fmaf(sign, v[i], o);
      else
        v[i] = (sub & m) ? o - v[i] : v[i] + o;
    }
  }
}

// The same by 8 lanes, 16 consecutive values a lane (a warp transforms four blocks at once): a quarter fewer shuffles a
// block, and the strides in the same order, so the same bits.
__device__ __forceinline__ void hadamard128_wide(float (&v)[16], int sub) {
#pragma unroll
  for (int h = 1; h < 16; h <<= 1)
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if ((i & h) == 0) {
        const float a = v[i], b = v[i + h];
        v[i] = a + b;
        v[i + h] = a - b;
      }
#pragma unroll
  for (int m = 1; m < 8; m <<= 1) {
    const float sign = (sub & m) ? -1.f : 1.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = fmaf(sign, v[i], __shfl_xor_sync(0xffffffffu, v[i], m));
  }
}

__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&f)[8]) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  f[0] = bf16_lo(u.x); f[1] = bf16_hi(u.x); f[2] = bf16_lo(u.y); f[3] = bf16_hi(u.y);
  f[4] = bf16_lo(u.z); f[5] = bf16_hi(u.z); f[6] = bf16_lo(u.w); f[7] = bf16_hi(u.w);
}
__device__ __forceinline__ void load8(const __half* p, float (&f)[8]) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const __half2* h = reinterpret_cast<const __half2*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __half22float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ void load8(const float* p, float (&f)[8]) {   // another CTA of this launch wrote it: L2
  const float4 a = __ldcg(reinterpret_cast<const float4*>(p)), b = __ldcg(reinterpret_cast<const float4*>(p) + 1);
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
__device__ __forceinline__ void load8_shared(const float* p, float (&f)[8]) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
__device__ __forceinline__ void store8(__half* p, const float (&f)[8], float scale) {
  uint4 u;
  __half2* h = reinterpret_cast<__half2*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(f[2 * i] * scale, f[2 * i + 1] * scale);
  *reinterpret_cast<uint4*>(p) = u;
}

// ---- epilogues of one pair and one 128-block, by a half warp ------------------------------------------------------
// gate/up: rotate both, * svh, SwiGLU (act_mode 0: the GLM family's bf16 roundings; 1: fp32), * suh_d, rotate, fp16.
// (arithmetic of src/tensorfold/cuda/exl3/experts.cu:116-158)
__device__ __forceinline__ void gateup_block(float (&g)[8], float (&u)[8], const __half* svh_g, const __half* svh_u,
                                             const __half* suh_d, __half* xd, int sub, float limit, int act_mode,
                                             bool store) {
  float sg[8], su[8], sd[8];
  load8(svh_g + 8 * sub, sg);
  load8(svh_u + 8 * sub, su);
  load8(suh_d + 8 * sub, sd);
  hadamard128<false>(g, sub);
  hadamard128<false>(u, sub);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float act;
    if (act_mode == 0) {
      const float gv = fminf(round_bf16(g[i] * HAD_SCALE * sg[i]), limit);
      const float uv = fminf(fmaxf(round_bf16(u[i] * HAD_SCALE * su[i]), -limit), limit);
      act = round_bf16(round_bf16(gv / (1.f + expf(-gv))) * uv);
    } else {
      const float gv = fminf(g[i] * HAD_SCALE * sg[i], limit);
      const float uv = fminf(fmaxf(u[i] * HAD_SCALE * su[i], -limit), limit);
      act = gv / (1.f + expf(-gv)) * uv;
    }
    g[i] = act * sd[i];
  }
  hadamard128<false>(g, sub);
  if (store) store8(xd + 8 * sub, g, HAD_SCALE);
}

// down: y = rotate(z) * svh, fp32.  (src/tensorfold/cuda/exl3/experts.cu:161-180)
__device__ __forceinline__ void down_block(float (&v)[8], const __half* svh, float* y, int sub, bool store) {
  float s[8];
  load8(svh + 8 * sub, s);
  hadamard128<false>(v, sub);
  if (!store) return;
  float4 a, b;
  a.x = v[0] * HAD_SCALE * s[0]; a.y = v[1] * HAD_SCALE * s[1]; a.z = v[2] * HAD_SCALE * s[2]; a.w = v[3] * HAD_SCALE * s[3];
  b.x = v[4] * HAD_SCALE * s[4]; b.y = v[5] * HAD_SCALE * s[5]; b.z = v[6] * HAD_SCALE * s[6]; b.w = v[7] * HAD_SCALE * s[7];
  reinterpret_cast<float4*>(y + 8 * sub)[0] = a;
  reinterpret_cast<float4*>(y + 8 * sub)[1] = b;
}

// What the prologue needs to lay the items out by width: the three matrices' width tables [E] and the table it fills,
// [3, stride, 4] (gate, up, down order).
struct WidthOrder {
  const int* k2[3];
  int* sorted;
  int stride;
};

struct GroupedArgs {
  const __half* x[2];            // rotated inputs [P, K] fp16 of matrix 0 / 1
  const int64_t* tp[2];          // trellis pointers [E]
  const int* k2[2];              // half-bit widths [E]
  const int* items;              // [., 3] (expert, first, count <= 32)
  const int* sorted[2];          // or null: the items in the order their CTAs should run, [., 4] = (expert, first, count, index)
  const int* counts;             // [0] = items
  const int* members;            // pair ids p = row * slots + slot, grouped by expert
  float* z;                      // [mats, P, N] fp32
  int* arrive;                   // [max items * N / 128] zero between launches
  const __half* sv[2];           // svh [E, N] of matrix 0 / 1
  const __half* suh_next;        // gate/up: suh of the down projection [E, N]
  void* out;                     // gate/up: xd [P, N] fp16; down: y [P, N] fp32
  int K, N, P, mats, epi, act_mode;
  int k2_all;                    // 8: every tensor has 4.00 bits (a promise); else 0
  float limit;
};

enum GroupedEpilogue : int { GE_NONE = 0, GE_GATEUP = 1, GE_DOWN = 2 };

// CTA (item, 64 columns, matrix), items of up to 16 pairs.
// K2F: 0, or the one width every tensor of the launch has (the host knows it): the kernel then holds that width's loop
// alone - a tenth of the code, which matters where a CTA's life is short (one token: the dominant stall of the
// all-widths kernel was the instruction fetch).
// NTB: 16-column tiles a CTA (4, or 2 where the launch would otherwise have too few CTAs to fill the GPU).
// INLINE_WAIT: a slot's wait without a call, for launches that leave a scheduler one to three warps (exl3_grouped_launch).
template <int CB, int K2F, int NTB, bool COMPACT, bool INLINE_WAIT>
__global__ void __launch_bounds__(GR_WARPS * 32)
grouped_kernel(const GroupedArgs a) {
  constexpr int PT = GR_PT, PAIRS = GR_PAIRS, GR_RED_STRIDE = NTB * 16 + 1;
  constexpr int RING_BYTES = GR_WARPS * GR_STAGES * GR_SLOT_BYTES, RED_BYTES = GR_WARPS * PAIRS * GR_RED_STRIDE * 4;
  // the K slices meet in the ring's memory (free by then)
  __shared__ __align__(128) uint8_t ring[RING_BYTES > RED_BYTES ? RING_BYTES : RED_BYTES];
  __shared__ uint64_t bars[GR_WARPS * GR_STAGES];
  __shared__ int pair_sh[PAIRS];
  __shared__ int last_sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int nt0 = blockIdx.x * NTB, mat = blockIdx.z;
  if (lane == 0) {
#pragma unroll
    for (int s = 0; s < GR_STAGES; ++s) mbar_init(bars + warp * GR_STAGES + s, 1);
    mbar_fence_init();
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  }
  __syncwarp();
  pdl_wait();
  const int *items = a.items, *counts = a.counts, *members = a.members, *sorted = a.sorted[mat];
  const __half* xin = a.x[mat];
  after_wait(items, counts, members, xin, sorted);
  // the item is read together with the count that says whether it exists (its slot is always inside the table)
  const int n_items = ld_dep(counts);
  int it = blockIdx.y, e, first, cnt;
  if (sorted != nullptr) {                            // the CTA's place in the launch is not the item's index
    const int4 s4 = ld_dep4(sorted + 4 * blockIdx.y);
    e = s4.x, first = s4.y, cnt = min(s4.z, PAIRS), it = s4.w;
  } else {
    e = ld_dep(items + 3 * it), first = ld_dep(items + 3 * it + 1), cnt = min(ld_dep(items + 3 * it + 2), PAIRS);
  }
  if ((int)blockIdx.y >= n_items) return;
  if (tid < PAIRS) pair_sh[tid] = tid < cnt ? ld_dep(members + first + tid) : -1;
  const uint8_t* T = reinterpret_cast<const uint8_t*>(a.tp[mat][e]);
  const int k2 = a.k2[mat][e];
  const int live = (cnt + 7) >> 3;                   // mma tiles of pairs in use
  // lanes past the item's last pair read its first pair's row: an mma column depends on its own inputs only
  const int KT = a.K >> 4, per_warp = (KT + GR_WARPS - 1) / GR_WARPS;
  const int kt0 = min(KT, warp * per_warp), nkt = min(KT, kt0 + per_warp) - kt0;
  const __half* x[PT];
#pragma unroll
  for (int pt = 0; pt < PT; ++pt) {
    const int p = ld_dep(members + first + (8 * pt + g < cnt ? 8 * pt + g : 0));
    x[pt] = xin + (size_t)p * a.K + kt0 * 16 + 2 * t;
  }
  float acc[NTB][PT][4];
#pragma unroll
  for (int i = 0; i < NTB; ++i)
#pragma unroll
    for (int pt = 0; pt < PT; ++pt) acc[i][pt][0] = acc[i][pt][1] = acc[i][pt][2] = acc[i][pt][3] = 0.f;
  bool ok = true;
  uint8_t* my_ring = ring + warp * (GR_STAGES * GR_SLOT_BYTES);
  uint64_t* my_bars = bars + warp * GR_STAGES;
#define TFB_K2_BODY(K2_)                                                                                         \
    ok = live > 1 ? warp_rows<CB, K2_, PT, PT, NTB, COMPACT, INLINE_WAIT>(T, a.N >> 4, kt0, nkt, nt0, x, my_ring,  \
                                                                          my_bars, lane, acc)                     \
                  : warp_rows<CB, K2_, PT, 1, NTB, COMPACT, INLINE_WAIT>(T, a.N >> 4, kt0, nkt, nt0, x, my_ring,   \
                                                                         my_bars, lane, acc);
#define TFB_K2(K2_) \
  case K2_:         \
    TFB_K2_BODY(K2_) \
    break;
  if constexpr (K2F != 0) {
    if (k2 == K2F) {
      TFB_K2_BODY(K2F)
    } else {
      atomicCAS(&g_kernel_status, 0, ST_BAD_INDEX);   // not the width the host promised
      ok = false;
    }
  } else {
    switch (k2) {
      TFB_K2(2) TFB_K2(3) TFB_K2(4) TFB_K2(5) TFB_K2(6) TFB_K2(7) TFB_K2(8) TFB_K2(9) TFB_K2(10) TFB_K2(11) TFB_K2(12)
      TFB_K2(13) TFB_K2(14) TFB_K2(15) TFB_K2(16)
      default:
        atomicCAS(&g_kernel_status, 0, ST_BAD_INDEX);   // a width the host should have refused
        ok = false;
        break;
    }
  }
#undef TFB_K2
#undef TFB_K2_BODY
  pdl_launch_dependents();
  if (__syncthreads_or(ok ? 0 : 1)) return;           // a copy never landed (recorded): store nothing
  // the K slices meet in warp order (the ring's memory is free: every warp is past its loop)
  // acc[i][pt]: d0 = (col g, pair 2t), d1 = (col g, pair 2t + 1), d2 = (col g + 8, pair 2t), d3 = (col g + 8, 2t + 1)
  float* red = reinterpret_cast<float*>(ring);
#pragma unroll
  for (int i = 0; i < NTB; ++i)
#pragma unroll
    for (int pt = 0; pt < PT; ++pt) {
      float* base = red + (warp * PAIRS + 8 * pt + 2 * t) * GR_RED_STRIDE + i * 16 + g;
      base[0] = acc[i][pt][0];
      base[GR_RED_STRIDE] = acc[i][pt][1];
      base[8] = acc[i][pt][2];
      base[GR_RED_STRIDE + 8] = acc[i][pt][3];
    }
  __syncthreads();
  for (int o = tid; o < PAIRS * NTB * 16; o += GR_WARPS * 32) {
    const int pi = o / (NTB * 16), col = o % (NTB * 16);
    const int p = pair_sh[pi];
    if (p < 0) continue;
    float s = red[pi * GR_RED_STRIDE + col];
#pragma unroll
    for (int w = 1; w < GR_WARPS; ++w) s += red[(w * PAIRS + pi) * GR_RED_STRIDE + col];
    a.z[((size_t)mat * a.P + p) * a.N + nt0 * 16 + col] = s;
  }
  if (a.epi == GE_NONE) return;
  // Whoever finishes last among the CTAs that share (item, 128 columns) - two column halves, times the matrices -
  // finds every part of the block in z and runs the block's epilogue.
  constexpr int PER_BLOCK = 128 / (16 * NTB);          // CTAs that share a 128-column block of one matrix
  const int blk = blockIdx.x / PER_BLOCK;
  int* counter = a.arrive + (size_t)it * (a.N >> 7) + blk;
  __syncthreads();
  if (tid == 0) {
    const int need = PER_BLOCK * a.mats;
    const int seen = arrive_count(counter);
    last_sh = seen == need - 1;
    if (seen == need - 1) *counter = 0;               // nobody else touches it before the next launch
  }
  __syncthreads();
  if (!last_sh) return;
  // a half warp a pair (the transform's shuffles need every lane of the warp: a half without a pair repeats the item's
  // first pair and stores nothing); pairs fill an item from the front, so a warp whose first pair is missing is done
  const int sub = lane & 15, half = lane >> 4;
  for (int p0 = 2 * warp; p0 < PAIRS && pair_sh[p0] >= 0; p0 += 2 * GR_WARPS) {
    const int p = pair_sh[p0 + half];
    const int q = p < 0 ? pair_sh[0] : p;
    const size_t at = (size_t)q * a.N + blk * 128, sc = (size_t)e * a.N + blk * 128;
    float g[8], u[8];
    load8(a.z + at + 8 * sub, g);
    if (a.epi == GE_GATEUP) {
      load8(a.z + (size_t)a.P * a.N + at + 8 * sub, u);
      gateup_block(g, u, a.sv[0] + sc, a.sv[1] + sc, a.suh_next + sc, static_cast<__half*>(a.out) + at, sub, a.limit,
                   a.act_mode, p >= 0);
    } else {
      down_block(g, a.sv[0] + sc, static_cast<float*>(a.out) + at, sub, p >= 0);
    }
  }
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
// kind::f16: D fp32, A and B fp16, both K-major, M = 128, N = n
__device__ __forceinline__ uint32_t umma_idesc_f16(int n) {
  return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TC_COLS >> 4) << 24);
}

// CTA (item, 128 columns, matrix), eighteen warps.  Per stage of 128 inputs: a warp copies the trellis rows into the ring
// and gathers the pairs' rotated inputs into swizzled B tiles, the decoding warps turn the 64 tiles into fp16 and store
// them in tensor memory, one lane of the last warp multiplies (A from tensor memory: a tile is decoded once for up to
// 32 pairs and touches neither shared memory nor further registers).
// The four parts of K are four accumulators, added in order: the sums of grouped_kernel's four warps, bit for bit.
//
// What bounds it: latency in the decoding warps' pipeline, at about 60 instructions a tile and lane.  A B200 at 4.00 bits, 128
// experts of 2048 x 768, 20 pairs an expert: the schedulers issue in 0.58 of the cycles (down 0.52), the ALU pipe is 0.48
// (0.40) busy, the multiply pipe 0.41 (0.33), DRAM 0.16; of 13 cycles from one of a warp's instructions to the next, 8 wait for
// a long-latency result, the pipeline's barriers among them (a set has one A stage and waits for it before it decodes).
// Two CTAs of sixteen decoding warps fill an SM's tensor memory.
// The layer takes 310 us, with the register kernel 374; 160 experts of 4096 x 1536 with widths of 2 to 8 bits at 512 tokens
// 1655 us with an mma.sync form, 1315 with this one.
template <int CB>
__global__ void __launch_bounds__(TC_THREADS, 2)
grouped_tc_kernel(const GroupedArgs a) {
  using SM = TrellisSmem;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  int* pair_sh = reinterpret_cast<int*>(smem + SM::PAIR_OFFSET);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SM::BAR_OFFSET);
  uint64_t* packed_full = bars;                       // [SP] the trellis rows of the stage landed
  uint64_t* packed_free = packed_full + SM::SP_MAX;   // [SP] the decoding warps have read it
  uint64_t* a_ready = packed_free + SM::SP_MAX;       // [sets] the set's four warps stored their tiles
  uint64_t* a_free = a_ready + TC_SETS;               // [sets] the MMAs that read the A stage retired
  uint64_t* b_ready = a_free + TC_SETS;                     // [SB] the pairs' inputs landed
  uint64_t* b_free = b_ready + SM::SB;                // [SB] the MMAs that read the B stage retired
  uint64_t* acc_ready = b_free + SM::SB;
  uint32_t* flags = reinterpret_cast<uint32_t*>(smem + SM::FLAG_OFFSET);   // [0] tensor memory, [1] last
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int blk = blockIdx.x, mat = blockIdx.z;
  if (tid == 0) {
    for (int s = 0; s < SM::SP_MAX; ++s) {
      mbar_init(packed_full + s, 1);
      mbar_init(packed_free + s, 8);                  // the two sets whose steps the stage holds
    }
    for (int s = 0; s < TC_SETS; ++s) {
      mbar_init(a_ready + s, 4);
      mbar_init(a_free + s, 1);
    }
    for (int s = 0; s < SM::SB; ++s) {
      mbar_init(b_ready + s, 32);
      mbar_init(b_free + s, 1);
    }
    mbar_init(acc_ready, 1);
    mbar_fence_init();
    fence_async_smem();
  }
  pdl_wait();
  const int *items = a.items, *counts = a.counts, *members = a.members, *sorted = a.sorted[mat];
  const __half* xin = a.x[mat];
  after_wait(items, counts, members, xin, sorted);
  // the item is read together with the count that says whether it exists (its slot is always inside the table)
  const int n_items = ld_dep(counts);
  int it = blockIdx.y, e, first, cnt;
  if (sorted != nullptr) {                            // the CTA's place in the launch is not the item's index
    const int4 s4 = ld_dep4(sorted + 4 * blockIdx.y);
    e = s4.x, first = s4.y, cnt = min(s4.z, TC_PAIRS), it = s4.w;
  } else {
    e = ld_dep(items + 3 * it), first = ld_dep(items + 3 * it + 1), cnt = min(ld_dep(items + 3 * it + 2), TC_PAIRS);
  }
  if ((int)blockIdx.y >= n_items) return;
  const uint8_t* T = reinterpret_cast<const uint8_t*>(a.tp[mat][e]);
  const int k2 = a.k2[mat][e];
  // a width the host should have refused, or not the one it promised
  if (k2 < 2 || k2 > 16 || (a.k2_all == 8 && k2 != 8)) {
    if (tid == 0) atomicCAS(&g_kernel_status, 0, ST_BAD_INDEX);
    return;
  }
  if (warp == TC_MMA_WARP) tmem_alloc(flags, TC_TMEM_COLS);
  if (tid < TC_PAIRS) pair_sh[tid] = tid < cnt ? ld_dep(members + first + tid) : -1;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = flags[0];
  const int nmma = cnt > 16 ? 32 : 16;
  // the parts of K: `part` k-tiles of 16 inputs each, as grouped_kernel's warps take them (K / 16 is a multiple of 8)
  const int steps = a.K / TC_STEP, part = (a.K / 16) / TC_PARTS;
  const int stages = steps / 2;
  const int sp_n = k2 <= 8 ? 8 : 4, stage_bytes = 2 * TC_STEP / 16 * (TC_COLS / 16) * 16 * k2;   // Ring<k2>
  bool ok = true;

  if (warp == TC_LOAD_WARP) {
    // Trellis: a lane a row of tiles.  Inputs: lane -> 16-byte chunk c of pairs r0, r0 + 4, ..; pairs past the item's
    // last are left as they are (an MMA column depends on its own pair only, and theirs are never stored).
    constexpr int PER = TC_PAIRS / 4, LAG = 2;
    const uint32_t row_bytes = (uint32_t)(TC_COLS / 16) * 16 * k2;
    const size_t row_stride = (size_t)(a.N >> 4) * 16 * k2, stage_stride = (2 * TC_STEP / 16) * row_stride;
    const uint8_t* src = T + (size_t)lane * row_stride + (size_t)blk * row_bytes;
    const int c = lane & 7, r0 = lane >> 3;
    const __half* xk = xin + c * 8;
    uint32_t row[PER];                                // in 128 inputs (K is a multiple): 32 bits hold 2^39 inputs
#pragma unroll
    for (int j = 0; j < PER; ++j) row[j] = (uint32_t)max(pair_sh[r0 + 4 * j], 0) * (uint32_t)(a.K >> 7);
    int s = 0, ph = 1, back = 0, sp = 0, pph = 1;     // ph, pph: a ring's first round finds every stage free
    constexpr int rows = 2 * TC_STEP / 16;            // K is a multiple of 128: whole stages
    int p = 0;
    for (; p < stages; ++p) {
      if (p >= sp_n) ok = mbar_wait_warp(packed_free + sp, pph);
      if (!ok) break;
      if (lane == 0) mbar_expect_tx(packed_full + sp, (uint32_t)rows * row_bytes);
      __syncwarp();
      if (lane < rows) bulk_g2s(smem + sp * stage_bytes + lane * row_bytes, src, row_bytes, packed_full + sp);
      src += stage_stride;
      if (++sp == sp_n) {
        sp = 0;
        pph ^= 1;
      }
      if (p >= SM::SB) ok = mbar_wait_warp(b_free + s, ph);
      if (!ok) {
        ++p;
        break;
      }
      uint8_t* btile = smem + SM::B_OFFSET + s * (2 * SM::B_TILE) + r0 * 128;
#pragma unroll
      for (int j = 0; j < PER; ++j) {
        if (4 * j >= cnt) break;
        const int r = r0 + 4 * j;
        if (r < cnt) {
          uint8_t* dst = btile + 4 * j * 128 + ((c ^ (r & 7)) << 4);
          const __half* from = xk + (size_t)row[j] * 128;
          cp_async16(dst, from);
          cp_async16(dst + SM::B_TILE, from + TC_STEP);
        }
      }
      xk += 2 * TC_STEP;
      cp_async_commit();
      if (++s == SM::SB) {
        s = 0;
        ph ^= 1;
      }
      if (p >= LAG) {                                 // the stage LAG back has landed: publish it
        cp_async_wait<LAG>();
        fence_async_smem();
        mbar_arrive(b_ready + back);
        if (++back == SM::SB) back = 0;
      }
    }
    cp_async_wait<0>();
    fence_async_smem();
    if (ok)
      for (int f = max(0, stages - LAG); f < stages; ++f) {
        mbar_arrive(b_ready + back);
        if (++back == SM::SB) back = 0;
      }
    else if (lane == 0)                                // give the trellis copies in flight a while to land
      for (int f = max(0, p - sp_n); f < p; ++f) mbar_wait_for(packed_full + (f & (sp_n - 1)), (f / sp_n) & 1, 10000000ull);
    __syncwarp();
  } else if (warp == TC_MMA_WARP) {
    if (lane == 0) {
      const uint32_t idesc = umma_idesc_f16(nmma);
      const uint64_t desc0 = umma_desc(smem_addr(smem + SM::B_OFFSET));     // addresses count 16 bytes
      int s = 0, ph = 0, done = 0;                    // k-tiles done of the part
      uint32_t d = tmem;                              // its accumulator
      for (int g = 0; g < steps; ++g) {
        const int t = g & 1, set = g & (TC_SETS - 1);
        if (t == 0) ok = mbar_wait(b_ready + s, ph);
        ok = ok && mbar_wait(a_ready + set, (g / TC_SETS) & 1);
        if (!ok) break;
        tc_fence_after();
        const uint32_t at = tmem + TC_A_COL + set * 32;
        const uint64_t desc = desc0 + (uint32_t)((2 * s + t) * (SM::B_TILE >> 4));
#pragma unroll
        for (int ks = 0; ks < TC_STEP / 16; ++ks) {
          umma_ta(d, at + ks * 8, desc + ks * 2, idesc, done > 0 ? 1u : 0u);   // a part's first k-tile starts its accumulator
          if (++done == part) {
            done = 0;
            d += TC_PAIRS;
          }
        }
        umma_commit(a_free + set);
        if (t == 1) {
          umma_commit(b_free + s);
          if (++s == SM::SB) {
            s = 0;
            ph ^= 1;
          }
        }
      }
      if (ok) umma_commit(acc_ready);
    }
    __syncwarp();
  } else {
    const int q = warp & 3, set = warp >> 2;
    const uint32_t a_dst = tmem + ((uint32_t)(32 * q) << 16) + TC_A_COL + set * 32;
#define TFB_K2(K2_)                                                                                                    \
  case K2_:                                                                                                            \
    ok = decode_stages<CB, K2_>(smem, packed_full, packed_free, a_ready, a_free, a_dst, set, q, steps, lane);          \
    break;
    switch (k2) {
      TFB_K2(2) TFB_K2(3) TFB_K2(4) TFB_K2(5) TFB_K2(6) TFB_K2(7) TFB_K2(8) TFB_K2(9) TFB_K2(10) TFB_K2(11) TFB_K2(12)
      TFB_K2(13) TFB_K2(14) TFB_K2(15) TFB_K2(16)
    }
#undef TFB_K2
    if (ok) ok = mbar_wait_warp(acc_ready, 0);
  }
  pdl_launch_dependents();
  tc_fence_after();
  bool good = !__syncthreads_or(ok ? 0 : 1);          // a wait ran out (recorded): store nothing
  // The accumulators, the parts added in order, as [pair][column] in the ring's memory (every copy has landed and been
  // read).  Warp -> lane quarter q (columns 32 q + lane) and 8 of the pairs.
  float* acc_sh = reinterpret_cast<float*>(smem);
  constexpr int EP = TC_PAIRS / TC_SETS;
  const int q = warp & 3, j0 = (warp >> 2) * EP;
  if (good && warp < TC_DEC_WARPS && j0 < cnt) {
    float v[EP];
    uint32_t r[EP];
    const uint32_t from = tmem + ((uint32_t)(32 * q) << 16) + j0;
    tmem_ld8(from, r);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < EP; ++j) v[j] = __uint_as_float(r[j]);
    for (int i = 1; i < TC_PARTS; ++i) {
      tmem_ld8(from + i * TC_PAIRS, r);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < EP; ++j) v[j] += __uint_as_float(r[j]);
    }
    float* z = a.z + (size_t)mat * a.P * a.N + blk * TC_COLS + 32 * q + lane;
#pragma unroll
    for (int j = 0; j < EP; ++j) {
      if (j0 + j >= cnt) continue;
      acc_sh[(j0 + j) * TC_COLS + 32 * q + lane] = v[j];
      if (a.epi != GE_DOWN) z[(size_t)pair_sh[j0 + j] * a.N] = v[j];
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == TC_MMA_WARP) tmem_dealloc(tmem, TC_TMEM_COLS);
  if (!good || a.epi == GE_NONE) return;
  if (a.epi == GE_GATEUP) {
    // whoever finishes last of the two matrices' CTAs finds the other's part of the block in z and runs the epilogue
    int* counter = a.arrive + (size_t)it * (a.N >> 7) + blk;
    if (tid == 0) {
      const int seen = arrive_count(counter);
      flags[1] = seen == a.mats - 1;
      if (seen == a.mats - 1) *counter = 0;           // nobody else touches it before the next launch
    }
    __syncthreads();
    if (!flags[1]) return;
  }
  // a half warp a pair (the transform's shuffles need every lane of the warp: a half without a pair repeats the warp's
  // first pair and stores nothing); pairs fill an item from the front, so a warp whose first pair is missing is done
  const int sub = lane & 15, half = lane >> 4;
  for (int p0 = 2 * warp; p0 < cnt; p0 += 2 * (TC_THREADS / 32)) {
    const bool have = p0 + half < cnt;
    const int i = have ? p0 + half : p0, p = pair_sh[i];
    const size_t at = (size_t)p * a.N + blk * TC_COLS, sc = (size_t)e * a.N + blk * TC_COLS;
    float own[8];
    load8_shared(acc_sh + i * TC_COLS + 8 * sub, own);
    if (a.epi == GE_GATEUP) {
      float other[8];
      load8(a.z + (size_t)(1 - mat) * a.P * a.N + at + 8 * sub, other);
      float(&g)[8] = mat == 0 ? own : other;
      float(&u)[8] = mat == 0 ? other : own;
      gateup_block(g, u, a.sv[0] + sc, a.sv[1] + sc, a.suh_next + sc, static_cast<__half*>(a.out) + at, sub, a.limit,
                   a.act_mode, have);
    } else {
      down_block(own, a.sv[0] + sc, static_cast<float*>(a.out) + at, sub, have);
    }
  }
}

}  // namespace exl3
}  // namespace tfb

namespace tfb {
namespace exl3 {

// W_q [K, N] fp16 of one matrix through the same lane decode (the bit-exactness hook, and the prompt form's weights).  A
// warp takes a row of eight tiles: all their words in flight, decoded, transposed through shared memory (the fragments hold
// pairs of inputs, the rows want pairs of columns) and stored as whole rows of 256 bytes.  vec: out is 16-byte aligned.
// Bound by the write of W_q; with one tile a block and 2-byte stores a 4096 x 4096 matrix
// at 4.00 bits took 35 us, this one 8.3 (42 MB: 5.0 TB/s).
constexpr int DQ_WARPS = 8, DQ_TILES = 8, DQ_STRIDE = 16 * DQ_TILES + 8;   // halves a staged row: rows 16 bytes apart mod 128

template <int CB, int K2>
__global__ void __launch_bounds__(DQ_WARPS * 32)
dequant_kernel(const uint32_t* __restrict__ T, __half* __restrict__ out, int K, int N, int vec) {
  constexpr int NW = Win<K2>::NW;
  __shared__ __align__(16) __half rows[DQ_WARPS][16 * DQ_STRIDE];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, ntiles = N >> 4, nblk = (ntiles + DQ_TILES - 1) / DQ_TILES;
  const int64_t u = (int64_t)blockIdx.x * DQ_WARPS + warp;
  const int kt = (int)(u / nblk), nt0 = (int)(u - (int64_t)kt * nblk) * DQ_TILES;
  pdl_wait();
  after_wait(T);
  if (kt >= (K >> 4)) return;
  const int live = min(DQ_TILES, ntiles - nt0);
  const uint32_t* src = T + ((size_t)kt * ntiles + nt0) * Win<K2>::TW;
  uint32_t w[DQ_TILES][NW];
#pragma unroll
  for (int i = 0; i < DQ_TILES; ++i) lane_words<K2, true>(src + (size_t)(i < live ? i : 0) * Win<K2>::TW, lane, w[i]);
  __half* stage = rows[warp];
  // the transposing store: lane 8 m + r gives the address of input row r of matrix m = (columns 8 (m & 1), inputs 8 (m >> 1))
  const uint32_t to = smem_addr(stage + ((lane >> 4) * 8 + (lane & 7)) * DQ_STRIDE + ((lane >> 3) & 1) * 8);
#pragma unroll
  for (int i = 0; i < DQ_TILES; ++i) {
    uint32_t a[4];
    decode_words<CB, K2>(w[i], lane, a);
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};\n" ::"r"(to + i * 32), "r"(a[0]),
                 "r"(a[1]), "r"(a[2]), "r"(a[3])
                 : "memory");
  }
  __syncwarp();
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int row = 2 * r + (lane >> 4), c = (lane & 15) * 8;
    if (c >= live * 16) continue;
    const uint4 v = *reinterpret_cast<const uint4*>(stage + row * DQ_STRIDE + c);
    __half* dst = out + (size_t)(kt * 16 + row) * N + nt0 * 16 + c;
    if (vec) {
      *reinterpret_cast<uint4*>(dst) = v;
    } else {
      const __half* h = reinterpret_cast<const __half*>(&v);
#pragma unroll
      for (int j = 0; j < 8; ++j) dst[j] = h[j];
    }
  }
}

}  // namespace exl3

// The first launch of a layer call.  Block 0 (when `sort`): the plan's stable sort of the pairs by expert, items of at
// most 16 pairs (ids outside [0, E) are left out), and the number of distinct experts into ucount.  The other blocks:
// out_m[p, :] = fp16(((x[row of p] * suh_m[expert of p]) H) / sqrt(128)) for every routed pair and 128-block, a half
// warp a block, both matrices from one read of x.  suh1 == nullptr: one matrix.
// (src/tensorfold/cuda/exl3/experts.cu:19-111: `group` and `rot_in`)
template <typename TIN>
__global__ void __launch_bounds__(PLAN_THREADS)
exl3_prologue_kernel(const int* __restrict__ picks, int P, int E, int slots, int sort, int* __restrict__ members,
                     int* __restrict__ items, int* __restrict__ counts, int* __restrict__ ucount,
                     const TIN* __restrict__ x, int64_t x_stride, const __half* __restrict__ suh0,
                     const __half* __restrict__ suh1, __half* __restrict__ out0, __half* __restrict__ out1, int K,
                     exl3::WidthOrder wo) {
  extern __shared__ int whist[];
  __shared__ int first[PLAN_EMAX];
  __shared__ uint64_t tot2[2][PLAN_THREADS / 32];
  __shared__ int bucket[3][16];
  pdl_wait();
  after_wait(picks, x);
  if (blockIdx.x == 0) {
    if (sort) {
      plan_block<PLAN_THREADS>(picks, P, E, sort, members, items, counts, whist, first, tot2);
      if (threadIdx.x == 0) ucount[0] = counts[1];    // written by this thread inside plan_block
      if (wo.sorted != nullptr) {
        // The items once more for each matrix, widest trellis first: blocks that run at the same time then decode the
        // same width, i.e. run the same code (every width is its own unrolled loop; seven of them at once on an SM
        // miss the instruction cache all the time).  The order inside a width is whatever the atomics give: no
        // result depends on it.
        if (threadIdx.x < 48) bucket[threadIdx.x / 16][threadIdx.x % 16] = 0;
        __threadfence_block();
        __syncthreads();
        const int n = counts[0];
        for (int i = threadIdx.x; i < n; i += PLAN_THREADS) {
          const int e = items[3 * i];
#pragma unroll
          for (int m = 0; m < 3; ++m) atomicAdd(&bucket[m][16 - min(max(wo.k2[m][e], 1), 16)], 1);
        }
        __syncthreads();
        if (threadIdx.x < 3) {
          int run = 0;
          for (int b = 0; b < 16; ++b) {
            const int c = bucket[threadIdx.x][b];
            bucket[threadIdx.x][b] = run;
            run += c;
          }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += PLAN_THREADS) {
          const int4 item = make_int4(items[3 * i], items[3 * i + 1], items[3 * i + 2], i);
#pragma unroll
          for (int m = 0; m < 3; ++m) {
            const int at = atomicAdd(&bucket[m][16 - min(max(wo.k2[m][item.x], 1), 16)], 1);
            reinterpret_cast<int4*>(wo.sorted + (size_t)m * wo.stride * 4)[at] = item;
          }
        }
      }
    }
    pdl_launch_dependents();
    return;
  }
  const int lane = threadIdx.x & 31, sub = lane & 15, half = lane >> 4;
  const int nblk = K >> 7;
  const int64_t units = (int64_t)P * nblk;
  const int64_t warps = (int64_t)(gridDim.x - 1) * (PLAN_THREADS / 32);
  for (int64_t u0 = 2 * ((int64_t)(blockIdx.x - 1) * (PLAN_THREADS / 32) + (threadIdx.x >> 5)); u0 < units;
       u0 += 2 * warps) {
    const bool have = u0 + half < units;              // the transform's shuffles need every lane: an idle half repeats u0
    const int64_t u = have ? u0 + half : u0;
    const int p = (int)(u / nblk), blk = (int)(u - (int64_t)p * nblk);
    const int e = picks[p];
    const bool routed = have && e >= 0 && e < E;
    const int es = routed ? e : 0;
    float xv[8], s[2][8];
    exl3::load8(x + (size_t)(p / slots) * x_stride + blk * 128 + 8 * sub, xv);
#pragma unroll
    for (int m = 0; m < 2; ++m)
      if ((m ? suh1 : suh0) != nullptr) exl3::load8((m ? suh1 : suh0) + (size_t)es * K + blk * 128 + 8 * sub, s[m]);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      if ((m ? suh1 : suh0) == nullptr) continue;
      float v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = xv[i] * s[m][i];
      exl3::hadamard128<true>(v, sub);
      if (routed) exl3::store8((m ? out1 : out0) + (size_t)p * K + blk * 128 + 8 * sub, v, exl3::HAD_SCALE);
    }
  }
  pdl_launch_dependents();
}

// The prompt form's epilogue: out[m, block] = rotate(z[m, block]) / sqrt(128) * svh + bias for every row and
// 128-column block of a product z [M, N] fp32, eight lanes a block.  vec: the rows of out are 16-byte aligned.
// (the epilogue of src/tensorfold/cuda/exl3/prefill.py:15-44 `_gemm`)
template <typename TOUT>
__global__ void __launch_bounds__(256)
exl3_rot_out_kernel(const float* __restrict__ z, const __half* __restrict__ svh, const __half* __restrict__ bias,
                    TOUT* __restrict__ out, int64_t out_stride, int M, int N, int vec) {
  const int lane = threadIdx.x & 31, sub = lane & 7, quad = lane >> 3;
  const int nblk = N >> 7;
  const int64_t units = (int64_t)M * nblk;
  const int64_t warps = (int64_t)gridDim.x * 8;
  pdl_wait();
  after_wait(z, svh, bias);
  for (int64_t u0 = 4 * ((int64_t)blockIdx.x * 8 + (threadIdx.x >> 5)); u0 < units; u0 += 4 * warps) {
    const bool have = u0 + quad < units;              // the transform's shuffles need every lane: an idle one repeats u0
    const int64_t u = have ? u0 + quad : u0;
    const int m = (int)(u / nblk), blk = (int)(u - (int64_t)m * nblk);
    float v[16], s[2][8], b[2][8];
    const float4* src = reinterpret_cast<const float4*>(z + (size_t)m * N + blk * 128 + 16 * sub);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 t = src[i];
      v[4 * i] = t.x; v[4 * i + 1] = t.y; v[4 * i + 2] = t.z; v[4 * i + 3] = t.w;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      exl3::load8(svh + blk * 128 + 16 * sub + 8 * h, s[h]);
#pragma unroll
      for (int i = 0; i < 8; ++i) b[h][i] = 0.f;
      if (bias != nullptr) exl3::load8(bias + blk * 128 + 16 * sub + 8 * h, b[h]);
    }
    exl3::hadamard128_wide(v, sub);
    if (!have) continue;
    __align__(16) TOUT y[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float f = fmaf(v[i] * exl3::HAD_SCALE, s[i >> 3][i & 7], b[i >> 3][i & 7]);
      if constexpr (sizeof(TOUT) == 4) y[i] = f;
      else if constexpr (std::is_same<TOUT, __half>::value) y[i] = __float2half_rn(f);
      else y[i] = __float2bfloat16_rn(f);
    }
    TOUT* dst = out + (size_t)m * out_stride + blk * 128 + 16 * sub;
    if (vec) {
#pragma unroll
      for (int i = 0; i < (int)sizeof(TOUT); ++i) reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(y)[i];
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i) dst[i] = y[i];
    }
  }
  pdl_launch_dependents();
}

// Grouping for callers of the `group` operator, in one block: the plan's stable sort (one item an expert), then the
// reference's tables: uids = distinct routed experts (< E) ascending, members[u][<= maxm] = row * 32 + slot in row
// order, -1 after the last.  (src/tensorfold/cuda/exl3/experts.cu:19-72)
__global__ void __launch_bounds__(PLAN_THREADS)
exl3_group_kernel(const int* __restrict__ picks, int P, int E, int slots, int* __restrict__ tmp_members,
                  int* __restrict__ tmp_items, int* __restrict__ tmp_counts, int* __restrict__ uids,
                  int* __restrict__ ucount, int* __restrict__ members, int maxm, int maxu) {
  extern __shared__ int whist[];
  __shared__ int first[PLAN_EMAX];
  __shared__ uint64_t tot2[2][PLAN_THREADS / 32];
  pdl_wait();
  after_wait(picks);
  plan_block<PLAN_THREADS>(picks, P, E, P + 1, tmp_members, tmp_items, tmp_counts, whist, first, tot2);
  __threadfence_block();
  __syncthreads();
  const int n = min(tmp_counts[0], maxu);
  if (threadIdx.x == 0) ucount[0] = n;
  for (int u = threadIdx.x; u < n; u += PLAN_THREADS) uids[u] = tmp_items[3 * u];
  for (int64_t i = threadIdx.x; i < (int64_t)n * maxm; i += PLAN_THREADS) {
    const int u = (int)(i / maxm), j = (int)(i - (int64_t)u * maxm);
    const int f = tmp_items[3 * u + 1], c = tmp_items[3 * u + 2];
    int code = -1;
    if (j < c) {
      const int p = tmp_members[f + j];
      code = (p / slots) * 32 + p % slots;
    }
    members[i] = code;
  }
  pdl_launch_dependents();
}

}  // namespace tfb

using namespace tfb;

static int exl3_check_k2(const char* who, int k2) {
  TFB_REQUIRE(k2 >= 2 && k2 <= 16, "%s: half-bit width %d outside 2..16", who, k2);
  return TFB_OK;
}

// W_q [K, N] fp16 of one trellis [K/16, N/16, 8 * k2] int16.  (exl3/experts.py:205-213 `dequant`)
extern "C" int tfb_exl3_dequant(const void* trellis, void* out, int K, int N, int k2, int cb, void* stream) {
  TFB_REQUIRE(trellis && out, "exl3_dequant: null pointer");
  TFB_REQUIRE(K > 0 && N > 0 && K % 16 == 0 && N % 16 == 0, "exl3_dequant: K and N must be multiples of 16");
  TFB_REQUIRE(cb >= 0 && cb <= 2, "exl3_dequant: codebook must be 0 (3inst), 1 (mcg) or 2 (mul1)");
  if (int rc = exl3_check_k2("exl3_dequant", k2)) return rc;
  const int64_t warps = (int64_t)(K / 16) * ((N / 16 + exl3::DQ_TILES - 1) / exl3::DQ_TILES);
  const int64_t blocks = (warps + exl3::DQ_WARPS - 1) / exl3::DQ_WARPS;
  TFB_REQUIRE(blocks < (int64_t(1) << 31), "exl3_dequant: too many tiles");
  const dim3 grid((unsigned)blocks);
  auto st = static_cast<cudaStream_t>(stream);
  auto* t = static_cast<const uint32_t*>(trellis);
  auto* o = static_cast<__half*>(out);
  const int vec = aligned16(out) ? 1 : 0;             // rows are multiples of 32 bytes
  cudaError_t e = cudaSuccess;
#define TFB_DQ(CB_, K2_)                                               \
  case K2_:                                                            \
    e = launch(exl3::dequant_kernel<CB_, K2_>, grid, dim3(exl3::DQ_WARPS * 32), 0, st, t, o, K, N, vec); \
    break;
#define TFB_DQ_ALL(CB_)                                                                                          \
  switch (k2) {                                                                                                  \
    TFB_DQ(CB_, 2) TFB_DQ(CB_, 3) TFB_DQ(CB_, 4) TFB_DQ(CB_, 5) TFB_DQ(CB_, 6) TFB_DQ(CB_, 7) TFB_DQ(CB_, 8)     \
    TFB_DQ(CB_, 9) TFB_DQ(CB_, 10) TFB_DQ(CB_, 11) TFB_DQ(CB_, 12) TFB_DQ(CB_, 13) TFB_DQ(CB_, 14)               \
    TFB_DQ(CB_, 15) TFB_DQ(CB_, 16)                                                                              \
  }
  if (cb == 0) { TFB_DQ_ALL(0) } else if (cb == 1) { TFB_DQ_ALL(1) } else { TFB_DQ_ALL(2) }
#undef TFB_DQ_ALL
#undef TFB_DQ
  return check_cuda(e, "exl3_dequant");
}

// Opts a plan-sized kernel into the dynamic shared memory of PLAN_EMAX experts, once a device.
template <typename Kernel>
static int plan_smem_opt_in(Kernel kernel, int* configured, const char* what) {
  int dev = 0;
  TFB_CUDA(cudaGetDevice(&dev), what);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    TFB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(sizeof(int) * 32 * PLAN_EMAX)),
             what);
    configured[dev] = 1;
  }
  return TFB_OK;
}

// pick [R, slots] -> uids [maxu], ucount [1], members [maxu, maxm]; tmp_members [R * slots], tmp_items
// [3 * min(R * slots, E)], tmp_counts [2] are caller scratch.  (exl3/experts.cpp `group`)
extern "C" int tfb_exl3_group(const int32_t* pick, int32_t* uids, int32_t* ucount, int32_t* members,
                              int32_t* tmp_members, int32_t* tmp_items, int32_t* tmp_counts, int R, int slots, int E,
                              int maxu, int maxm, void* stream) {
  TFB_REQUIRE(pick && uids && ucount && members && tmp_members && tmp_items && tmp_counts, "exl3_group: null pointer");
  TFB_REQUIRE(E >= 1 && E <= PLAN_EMAX, "exl3_group: at most %d experts, not %d", PLAN_EMAX, E);
  TFB_REQUIRE(slots >= 1 && slots <= 32, "exl3_group: 1..32 slots, not %d", slots);
  TFB_REQUIRE(R >= 0 && maxu >= 0 && maxm >= 0, "exl3_group: bad sizes");
  static int configured[64] = {0};
  if (int rc = plan_smem_opt_in(exl3_group_kernel, configured, "exl3_group: shared memory opt-in")) return rc;
  return check_cuda(launch(exl3_group_kernel, dim3(1), dim3(PLAN_THREADS), sizeof(int) * 32 * (size_t)E,
                           static_cast<cudaStream_t>(stream), pick, R * slots, E, slots, tmp_members, tmp_items,
                           tmp_counts, uids, ucount, members, maxm, maxu),
                    "exl3_group");
}

// ---- grouping without caller scratch ---------------------------------------------------------------------------
// For hosts that cannot give this library device memory at call time: a serving process that handed every free byte
// of HBM to its own pools at start-up (so a later cudaMalloc fails), or a decode loop where allocation calls are
// banned because they stall the whole device.  The sort's temporaries live in the array below, which every GPU that
// loads the library carries until the process ends (about 140 KB).
constexpr int GROUP_STATIC_MAX_PAIRS = 32768;         // R * slots a call may sort
constexpr int GROUP_STATIC_WORDS = GROUP_STATIC_MAX_PAIRS + 3 * tfb::PLAN_EMAX + 64;
static __device__ __align__(256) int g_group_scratch[GROUP_STATIC_WORDS];
static int* g_group_scratch_ptr[64] = {nullptr};      // the array's device address, per device (host code cannot use the symbol itself)

// Same result as tfb_exl3_group, with no scratch arguments.  Limits: R * slots <= 32768, E <= 1024, slots <= 32.
// The first call on a device looks up the array's device address (cudaGetSymbolAddress) and opts the kernel into its
// shared-memory size; make that first call before starting any stream capture.  All calls on a device share the one
// array: two calls whose kernels may run at the same time on that GPU (different streams) would corrupt each other -
// keep them on one stream or order them with events.  Nothing in the array has to start at zero; a call overwrites
// what it reads.  Calls no allocating routine.
extern "C" int tfb_exl3_group_static(const int32_t* pick, int32_t* uids, int32_t* ucount, int32_t* members, int R,
                                     int slots, int E, int maxu, int maxm, void* stream) {
  TFB_REQUIRE(pick && uids && ucount && members, "exl3_group_static: null pointer");
  TFB_REQUIRE(E >= 1 && E <= PLAN_EMAX, "exl3_group_static: at most %d experts, not %d", PLAN_EMAX, E);
  TFB_REQUIRE(slots >= 1 && slots <= 32, "exl3_group_static: 1..32 slots, not %d", slots);
  TFB_REQUIRE(R >= 0 && maxu >= 0 && maxm >= 0, "exl3_group_static: bad sizes");
  TFB_REQUIRE((int64_t)R * slots <= GROUP_STATIC_MAX_PAIRS,
              "exl3_group_static: %lld pairs exceed the built-in scratch (%d pairs); use tfb_exl3_group with caller "
              "scratch", (long long)R * slots, GROUP_STATIC_MAX_PAIRS);
  int dev = 0;
  TFB_CUDA(cudaGetDevice(&dev), "exl3_group_static: cudaGetDevice");
  TFB_REQUIRE(dev >= 0 && dev < 64, "exl3_group_static: device index %d out of range", dev);
  if (g_group_scratch_ptr[dev] == nullptr) {
    int* ptr = nullptr;
    TFB_CUDA(cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_group_scratch),
             "exl3_group_static: cudaGetSymbolAddress");
    TFB_CUDA(cudaFuncSetAttribute(exl3_group_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(sizeof(int) * 32 * PLAN_EMAX)),
             "exl3_group_static: shared memory opt-in");
    g_group_scratch_ptr[dev] = ptr;
  }
  int* base = g_group_scratch_ptr[dev];
  int* tmp_counts = base;                             // [2] (+ padding to keep the next arrays 256-byte aligned)
  int* tmp_items = base + 64;                         // [3 * min(pairs, E)]
  int* tmp_members = base + 64 + 3 * PLAN_EMAX;       // [pairs]
  return check_cuda(launch(exl3_group_kernel, dim3(1), dim3(PLAN_THREADS), sizeof(int) * 32 * (size_t)E,
                           static_cast<cudaStream_t>(stream), pick, R * slots, E, slots, tmp_members, tmp_items,
                           tmp_counts, uids, ucount, members, maxm, maxu),
                    "exl3_group_static");
}

// The first launch of a routed call: sorts the pairs by expert (when `sort`, which is then the pairs an item holds, 16
// or 32: members [R * slots], items [(min(R * slots, E) + R * slots / sort), 3] = (expert, first, count <= sort),
// counts [2], ucount [1] = distinct experts)
// and rotates the inputs: out0 / out1 [R * slots, K] fp16 for the two matrices (suh1 / out1 null: one matrix).
// sorted (or null): int32 [3, sorted_stride, 4], filled with the items as (expert, first, count, index), once in the
// order of each matrix's widths k2_g / k2_u / k2_d [E] (widest first), for tfb_exl3_gateup / tfb_exl3_down of a layer
// whose tensors differ in width; sorted_stride >= the sort's items.
extern "C" int tfb_exl3_prologue(const void* x, int64_t x_stride, int x_is_fp16, const int32_t* pick, const void* suh0,
                                 const void* suh1, void* out0, void* out1, int R, int K, int slots, int E, int sort,
                                 int32_t* members, int32_t* items, int32_t* counts, int32_t* ucount,
                                 const int32_t* k2_g, const int32_t* k2_u, const int32_t* k2_d, int32_t* sorted,
                                 int sorted_stride, void* stream) {
  TFB_REQUIRE(x && pick && suh0 && out0, "exl3_prologue: null pointer");
  TFB_REQUIRE(sorted == nullptr || (sort && k2_g && k2_u && k2_d && sorted_stride >= 1 && aligned16(sorted)),
              "exl3_prologue: the width order needs the sort, the three width tables and a 16-byte aligned table");
  const exl3::WidthOrder wo = {{k2_g, k2_u, k2_d}, sorted, sorted_stride};
  TFB_REQUIRE((suh1 == nullptr) == (out1 == nullptr), "exl3_prologue: the second matrix's scales and output come together");
  TFB_REQUIRE(!sort || (members && items && counts && ucount), "exl3_prologue: null sort table");
  TFB_REQUIRE(sort == 0 || sort == exl3::GR_PAIRS || sort == exl3::TC_PAIRS,
              "exl3_prologue: sort is 0 (the caller sorted), %d or %d (pairs an item)", exl3::GR_PAIRS, exl3::TC_PAIRS);
  TFB_REQUIRE(K > 0 && K % 128 == 0, "exl3_prologue: K must be a multiple of 128");
  TFB_REQUIRE(slots >= 1 && slots <= 32 && x_stride >= K && x_stride % 8 == 0, "exl3_prologue: bad slots or stride");
  TFB_REQUIRE(aligned16(x) && aligned16(suh0) && aligned16(out0) && aligned16(suh1) && aligned16(out1),
              "exl3_prologue: 16-byte aligned rows");
  TFB_REQUIRE(E >= 1 && E <= PLAN_EMAX, "exl3_prologue: at most %d experts, not %d", PLAN_EMAX, E);
  if (R <= 0) return TFB_OK;
  const int64_t units = (int64_t)R * slots * (K / 128);
  const int64_t want = (units + 2 * (PLAN_THREADS / 32) - 1) / (2 * (PLAN_THREADS / 32));
  const int rot_blocks = (int)(want < 2 * sm_count() ? want : 2 * sm_count());
  const dim3 grid(1 + rot_blocks);
  const size_t smem = sort ? sizeof(int) * 32 * (size_t)E : 0;
  auto st = static_cast<cudaStream_t>(stream);
  cudaError_t e;
  if (x_is_fp16) {
    static int configured[64] = {0};
    if (int rc = plan_smem_opt_in(exl3_prologue_kernel<__half>, configured, "exl3_prologue: shared memory opt-in")) return rc;
    e = launch(exl3_prologue_kernel<__half>, grid, dim3(PLAN_THREADS), smem, st, pick, R * slots, E, slots, sort, members,
               items, counts, ucount, static_cast<const __half*>(x), x_stride, static_cast<const __half*>(suh0),
               static_cast<const __half*>(suh1), static_cast<__half*>(out0), static_cast<__half*>(out1), K, wo);
  } else {
    static int configured[64] = {0};
    if (int rc = plan_smem_opt_in(exl3_prologue_kernel<__nv_bfloat16>, configured, "exl3_prologue: shared memory opt-in"))
      return rc;
    e = launch(exl3_prologue_kernel<__nv_bfloat16>, grid, dim3(PLAN_THREADS), smem, st, pick, R * slots, E, slots, sort,
               members, items, counts, ucount, static_cast<const __nv_bfloat16*>(x), x_stride,
               static_cast<const __half*>(suh0), static_cast<const __half*>(suh1), static_cast<__half*>(out0),
               static_cast<__half*>(out1), K, wo);
  }
  return check_cuda(e, "exl3_prologue");
}

static int exl3_grouped_launch(const char* who, exl3::GroupedArgs a, int cb, int max_items, int item_pairs,
                               int k2_all, int col_tiles, void* stream) {
  TFB_REQUIRE(col_tiles == exl3::GR_NTB || col_tiles == exl3::GR_NARROW_NTB, "%s: %d or %d column tiles a block, not %d",
              who, exl3::GR_NTB, exl3::GR_NARROW_NTB, col_tiles);
  TFB_REQUIRE(k2_all == 0 || k2_all == -1 || (k2_all >= 2 && k2_all <= 16),
              "%s: k2_all is 0, -1 (the widths differ) or the one width of every tensor", who);
  TFB_REQUIRE(k2_all == 8 || col_tiles == exl3::GR_NTB, "%s: only a launch of 4.00-bit tensors (k2_all 8) takes blocks of %d "
              "column tiles", who, exl3::GR_NARROW_NTB);
  TFB_REQUIRE(item_pairs == exl3::GR_PAIRS || item_pairs == exl3::TC_PAIRS, "%s: items of %d or %d pairs, not %d",
              who, exl3::GR_PAIRS, exl3::TC_PAIRS, item_pairs);
  TFB_REQUIRE(a.K > 0 && a.N > 0 && a.K % 128 == 0 && a.N % 128 == 0, "%s: K and N must be multiples of 128", who);
  TFB_REQUIRE(cb >= 0 && cb <= 2, "%s: codebook must be 0 (3inst), 1 (mcg) or 2 (mul1)", who);
  TFB_REQUIRE(max_items >= 0 && a.P >= 0, "%s: bad sizes", who);
  if (max_items == 0 || a.P == 0) return TFB_OK;
  TFB_REQUIRE(max_items <= 65535, "%s: too many items for one launch", who);
  auto st = static_cast<cudaStream_t>(stream);
  cudaError_t e;
  if (item_pairs == exl3::TC_PAIRS) {
    a.k2_all = k2_all == 8 ? 8 : 0;
    using Kernel = void (*)(exl3::GroupedArgs);
    const Kernel kern = cb == 0   ? Kernel(exl3::grouped_tc_kernel<0>)
                        : cb == 1 ? Kernel(exl3::grouped_tc_kernel<1>)
                                  : Kernel(exl3::grouped_tc_kernel<2>);
    static bool configured[3][64] = {};
    int dev = 0;
    TFB_CUDA(cudaGetDevice(&dev), who);
    if (dev < 0 || dev >= 64) return fail(TFB_ERR_ARG, "%s: device index %d out of range", who, dev);
    if (!configured[cb][dev]) {
      TFB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, exl3::TrellisSmem::TOTAL), who);
      configured[cb][dev] = true;
    }
    return check_cuda(launch(kern, dim3(a.N / exl3::TC_COLS, max_items, a.mats), dim3(exl3::TC_THREADS),
                             (size_t)exl3::TrellisSmem::TOTAL, st, a),
                      who);
  }
  const dim3 grid(a.N / (16 * col_tiles), max_items, a.mats);          // an item's column blocks run together
  const dim3 block(exl3::GR_WARPS * 32);
  const bool four = k2_all == 8;                      // the one width with a kernel of its own (4.00 bits a weight)
  const bool narrow = col_tiles == exl3::GR_NARROW_NTB;
  // Few items with many pairs each: a warp mostly waits for its own chain and holds two live tiles of pairs, and the call
  // behind a slot's wait costs it registers (one tensor of 6144 x 1024, 3 bits, 16 rows: 60.7 us with the call, 53.1 without;
  // 20 experts of 4096 x 1536, 8 pairs each: 167.6 and 162.3).  Else the shorter code of the call is the faster (one row of
  // 4096 x 4096: 33.5 and 34.7; 128 experts of 2048 x 768, 5 rows: 73.4 and 75.7, 64 rows: 210.7 and 214.8).  By what both
  // launches of a layer share: with gate/up in one build and down in the other they miss the instruction cache (20 experts,
  // 8 rows: 141.8 -> 150.7 us).  The build for 4.00 bits gains nothing either way.
  constexpr int INLINE_WAIT_ITEMS = 64;
  const bool few = max_items <= INLINE_WAIT_ITEMS && a.P > 4 * max_items;
#define TFB_GR4(CB_, K2F_, NTB_, COMPACT_, INLINE_) \
  launch(exl3::grouped_kernel<CB_, K2F_, NTB_, COMPACT_, INLINE_>, grid, block, 0, st, a)
#define TFB_GR(CB_)                                                      \
  e = k2_all == -1 ? TFB_GR4(CB_, 0, exl3::GR_NTB, true, false)          \
      : narrow     ? TFB_GR4(CB_, 8, exl3::GR_NARROW_NTB, false, false)  \
      : four       ? TFB_GR4(CB_, 8, exl3::GR_NTB, false, false)         \
      : few        ? TFB_GR4(CB_, 0, exl3::GR_NTB, false, true)          \
                   : TFB_GR4(CB_, 0, exl3::GR_NTB, false, false)
  if (cb == 0) {
    TFB_GR(0);
  } else if (cb == 1) {
    TFB_GR(1);
  } else {
    TFB_GR(2);
  }
#undef TFB_GR
#undef TFB_GR4
  return check_cuda(e, who);
}

// xd [P, N] fp16 = the down projection's rotated input of every routed pair: gate and up (trellis GEMV over the rotated
// inputs xg, xu [P, K] fp16), output rotation, svh, SwiGLU (act_mode 0: bf16 roundings, 1: fp32; clipped at limit),
// suh_d, rotation - one launch.  tp_*: int64 trellis pointers [E] (16-byte aligned trellises), k2_*: int32 [E];
// items / counts / members: the prologue's sort; z: fp32 scratch [2, P, N]; arrive: int scratch
// [max_items * N / 128], zero before the first call (every call leaves it zero); max_items >= the sort's items.
// sorted_g / sorted_u (or null): the prologue's width orders of the two matrices ([., 4] each).  item_pairs: 16 or 32,
// the most pairs an item of the sort holds (32: the tensor-memory kernel, in which one decode of a weight tile serves up to
// 32 pairs - for calls with many pairs an expert); a pair's bits do not depend on it.  k2_all: 0, or the width that
// every k2_g and k2_u entry has (a promise: the launch may then use a kernel built for that width alone; a tensor of
// another width sets the status word and stores nothing); -1: the widths differ (a build of the kernel with short
// loops: blocks of different widths then share an SM's instruction cache).  col_tiles: 4 or 2, the 16-column tiles a block takes - 2
// doubles the blocks of a launch that would otherwise not fill the GPU (few experts in use; built for k2_all = 8 only);
// no result depends on it.
// (exl3/experts.cpp `grouped` + `gateup_epilogue`: src/tensorfold/cuda/exl3/experts_grouped.cuh:190-284,
// src/tensorfold/cuda/exl3/experts.cu:116-158)
extern "C" int tfb_exl3_gateup(const void* xg, const void* xu, const int64_t* tp_g, const int64_t* tp_u,
                               const int32_t* k2_g, const int32_t* k2_u, const int32_t* items, const int32_t* counts,
                               const int32_t* members, float* z, int32_t* arrive, const void* svh_g, const void* svh_u,
                               const void* suh_d, void* xd, int K, int N, int P, int cb, int max_items, float limit,
                               int act_mode, const int32_t* sorted_g, const int32_t* sorted_u, int item_pairs,
                               int k2_all, int col_tiles, void* stream) {
  TFB_REQUIRE((sorted_g == nullptr) == (sorted_u == nullptr) && aligned16(sorted_g) && aligned16(sorted_u),
              "exl3_gateup: the two width orders come together, 16-byte aligned");
  TFB_REQUIRE(xg && xu && tp_g && tp_u && k2_g && k2_u && items && counts && members && z && arrive && svh_g && svh_u &&
                  suh_d && xd,
              "exl3_gateup: null pointer");
  TFB_REQUIRE(act_mode == 0 || act_mode == 1, "exl3_gateup: act_mode 0 (bf16 roundings) or 1 (fp32)");
  TFB_REQUIRE(aligned16(z) && aligned16(svh_g) && aligned16(svh_u) && aligned16(suh_d) && aligned16(xd),
              "exl3_gateup: 16-byte aligned rows");
  exl3::GroupedArgs a = {};
  a.x[0] = static_cast<const __half*>(xg);
  a.x[1] = static_cast<const __half*>(xu);
  a.tp[0] = tp_g;
  a.tp[1] = tp_u;
  a.k2[0] = k2_g;
  a.k2[1] = k2_u;
  a.items = items;
  a.sorted[0] = sorted_g;
  a.sorted[1] = sorted_u;
  a.counts = counts;
  a.members = members;
  a.z = z;
  a.arrive = arrive;
  a.sv[0] = static_cast<const __half*>(svh_g);
  a.sv[1] = static_cast<const __half*>(svh_u);
  a.suh_next = static_cast<const __half*>(suh_d);
  a.out = xd;
  a.K = K;
  a.N = N;
  a.P = P;
  a.mats = 2;
  a.epi = exl3::GE_GATEUP;
  a.act_mode = act_mode;
  a.limit = limit;
  return exl3_grouped_launch("exl3_gateup", a, cb, max_items, item_pairs, k2_all, col_tiles, stream);
}

// y [P, N] fp32 = rotate(x [P, K] fp16 times W_q of each pair's expert) * svh of every routed pair (rows of other
// pairs are left as they are) - one launch; z: fp32 scratch [P, N]; the other arguments as tfb_exl3_gateup
// (sorted: the prologue's width order of the down matrices, or null).
// (exl3/experts.cpp `grouped` + `down_epilogue`: src/tensorfold/cuda/exl3/experts.cu:161-180)
extern "C" int tfb_exl3_down(const void* x, const int64_t* tp, const int32_t* k2, const int32_t* items,
                             const int32_t* counts, const int32_t* members, float* z, int32_t* arrive, const void* svh,
                             float* y, int K, int N, int P, int cb, int max_items, const int32_t* sorted,
                             int item_pairs, int k2_all, int col_tiles, void* stream) {
  TFB_REQUIRE(x && tp && k2 && items && counts && members && z && arrive && svh && y, "exl3_down: null pointer");
  TFB_REQUIRE(aligned16(sorted), "exl3_down: the width order must be 16-byte aligned");
  TFB_REQUIRE(aligned16(z) && aligned16(svh) && aligned16(y), "exl3_down: 16-byte aligned rows");
  exl3::GroupedArgs a = {};
  a.x[0] = a.x[1] = static_cast<const __half*>(x);
  a.tp[0] = a.tp[1] = tp;
  a.k2[0] = a.k2[1] = k2;
  a.items = items;
  a.sorted[0] = a.sorted[1] = sorted;
  a.counts = counts;
  a.members = members;
  a.z = z;
  a.arrive = arrive;
  a.sv[0] = a.sv[1] = static_cast<const __half*>(svh);
  a.suh_next = nullptr;
  a.out = y;
  a.K = K;
  a.N = N;
  a.P = P;
  a.mats = 1;
  a.epi = exl3::GE_DOWN;
  a.act_mode = 1;
  a.limit = 0.f;
  return exl3_grouped_launch("exl3_down", a, cb, max_items, item_pairs, k2_all, col_tiles, stream);
}

// out [M, N] (fp32: out_type 0, fp16: 1, bf16: 2; rows out_stride elements apart) = rotate(z) / sqrt(128) * svh + bias
// for every 128-column block of z [M, N] fp32 (bias fp16 [N] or null): the output side of an EXL3 product formed
// elsewhere (a dense GEMM over the decoded W_q for prompts).
// (src/tensorfold/cuda/exl3/prefill.py:15-44: the rotation epilogue of `_gemm`)
extern "C" int tfb_exl3_rot_out(const float* z, const void* svh, const void* bias, void* out, int64_t out_stride,
                                int out_type, int M, int N, void* stream) {
  TFB_REQUIRE(z && svh && out, "exl3_rot_out: null pointer");
  TFB_REQUIRE(N > 0 && N % 128 == 0 && out_stride >= N, "exl3_rot_out: N must be a multiple of 128, rows at least N apart");
  TFB_REQUIRE(out_type >= 0 && out_type <= 2, "exl3_rot_out: out_type 0 (fp32), 1 (fp16) or 2 (bf16)");
  TFB_REQUIRE(aligned16(z) && aligned16(svh) && aligned16(bias), "exl3_rot_out: 16-byte aligned rows");
  if (M <= 0) return TFB_OK;
  const int64_t units = (int64_t)M * (N / 128);
  const int64_t want = (units + 31) / 32;
  const dim3 grid((unsigned)(want < 16 * sm_count() ? want : 16 * sm_count()));
  auto st = static_cast<cudaStream_t>(stream);
  auto* sv = static_cast<const __half*>(svh);
  auto* bi = static_cast<const __half*>(bias);
  const int vec = aligned16(out) && (out_stride * (out_type == 0 ? 4 : 2)) % 16 == 0 ? 1 : 0;
  cudaError_t e;
  if (out_type == 0)
    e = launch(exl3_rot_out_kernel<float>, grid, dim3(256), 0, st, z, sv, bi, static_cast<float*>(out), out_stride, M, N, vec);
  else if (out_type == 1)
    e = launch(exl3_rot_out_kernel<__half>, grid, dim3(256), 0, st, z, sv, bi, static_cast<__half*>(out), out_stride, M, N,
               vec);
  else
    e = launch(exl3_rot_out_kernel<__nv_bfloat16>, grid, dim3(256), 0, st, z, sv, bi, static_cast<__nv_bfloat16*>(out),
               out_stride, M, N, vec);
  return check_cuda(e, "exl3_rot_out");
}
