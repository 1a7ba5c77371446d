// QMatMul::forward on the 5th-generation tensor cores (tcgen05 / TMEM) for decode batches, up to 64 activation rows, and for those
// short prompts (up to 1024 rows) that leave most of the prefill kernel's pairs without work (plan_batch_tile, launch_plan.h).
//
//   y[m, n] = sum_k x[m, k] * W[n, k]      W quantized (device fragment tiles), x f32 or bf16
//
// Step 1 (prep kernel, gemm_tc.cu): x -> f16 with a power-of-two scale per row, written as the shared-memory
// image of the B operand: 64-k blocks of bn rows x 128 bytes, 128B-swizzled, the blocks of a 256-k unit one behind the other; in
// the k order that all types share, in one of Q6_K's own (a lane then finds all that it converts in its own words), or both.
// Step 2 (this kernel): a cluster of C CTAs computes 128 weight rows at a time, each CTA a share of the K loop. A unit is 256 k:
//   * warps 0, 23   stream the raw quantized tiles of the unit (contiguous bytes per row-tile) into a ring with cp.async.bulk;
//   * warp 1        one bulk copy of the unit's activation image (no tensor map, no multicast);
//   * warps 7..22   dequantize from the raw ring to f16 with packed half arithmetic into TMEM (tcgen05.st): the A operand;
//   * warp 2        issues tcgen05.mma M=128, N=bn, K=16 (f16 x f16 -> f32, A from TMEM, B from shared memory), sixteen per
//                   unit, and commits the stage back. One barrier per stage collects the dequantize warps and the copy, one
//                   commit frees both operands;
//   * warps 3..6    epilogue: tcgen05.ld, exchange of the partial sums, row scale, bias, store; double-buffered accumulators.
//                   The dequantize warps help with a CTA's last one.
// The partial sums cross through distributed shared memory: the columns are dealt out over the cluster in chunks of eight,
// a CTA sends its sums of the others' chunks (st.async, completing on the receiver's barrier) and adds those of its own in
// rank order (fixed order, no float atomics). Clusters have nothing to do with one another.
// All weights of a call (q|k|v, gate|up; any mix of types) go out as one launch over their 128-row tiles, dealt out round robin
// to the clusters that fit the GPU. C is a function of the weight's shape alone (launch_plan.h), so a row's bits depend on
// neither the batch, the other weights of the call, nor the device; weights that want another C go out as a launch of their own.
//
// More than 64 rows go in tiles of up to 128 (a tile and 128 weight rows are an item; accumulators of 64 or 128 columns), a launch per
// weight, side by side. K is not cut then: the sums, and their bits, are those of the prefill kernel. A layer of 4096-wide
// Q4_K / Q6_K linears at 96 / 128 / 256 / 512 rows: 147 / 150 / 167 / 223 -> 115 / 123 / 149 / 207 us; 2560-wide Q8_0 at 96 / 256: 113 / 125 ->
// 71 / 84; 1024-wide Q8_0 at 96 / 256 / 512: 64 / 70 / 75 -> 40 / 49 / 58. A unit takes 0.67 us with 16 rows, 0.72 with 64 (dequantize), 0.9 with 96
// and 1.05 with 128: 64 KB of activations a unit, 9 TB/s from L2 over all CTAs, where a pair of the prefill kernel shares its rows.
//
// What bounds it. Small weights: the chain conversion (1.0 us) - its completion (0.7) - first activation image (0.6) - MMAs of
// the share - exchange (0.6) - stores and exit, some 5 us. Large ones: the issue slots and the ALU pipe of the dequantize warps
// (about 1250 cycles a unit at 32 rows against 790 that its bytes need at the measured copy rate). At 64 rows the MMAs take
// 610 cycles of a unit; with a CTA per SM (cta_group::1) and A in TMEM an MMA of 32 / 64 columns takes 20 / 33 cycles, with A in
// shared memory 41 / 49.
// Measured with graph replay, conversion included, against pairs of CTAs (cta_group::2) with one launch per weight and partial
// sums through global memory, us a call:
//   attn_q|k|v 2560 + 640 + 640 x 2560 Q5_K, Q6_K, 32 rows 16.7 -> 7.6    ffn_gate|up 2 x 8192 x 2560 Q5_K, 32 rows 23.1 -> 12.8
//   attn_q|k|v 8192 + 1024 + 1024 x 5120 Q4_K, Q6_K, 64 rows 32.2 -> 20.0   ffn_gate|up 2 x 25600 x 5120 Q4_K, 64 rows 68.4 -> 50.4
//   attn_output 4096 x 4096 Q4_K, 32 rows 11.1 -> 8.1                      ffn_down 5120 x 25600 Q6_K, 64 rows 52.1 -> 40.6
// Q6_K in a k order of its own (5120 x 25600, 32 / 64 rows): 38.3 / 43.0 -> 34.8 / 40.6 us; a call that needs both images (the q|k|v
// above at 64 rows): 19.5 -> 20.0.
// Every wait is bounded; on expiry the CTA records TURQ_E_TIMEOUT, releases its TMEM and returns.
#include <atomic>

#include "launch_plan.h"
#include "tc_common.cuh"
#include "turq_internal.h"

namespace turq {

namespace {

constexpr int MAX_RAW = 10;        // raw ring slots
constexpr int A_COLS = 32;         // TMEM columns of a 64-k block of the weight operand
constexpr int CH = 8;              // columns of a chunk: what a CTA of the cluster adds up as a whole
constexpr int CH_BYTES = BM * CH * 4;
constexpr int EP_WARPS = 4;
constexpr int DQ_WARP0 = 7;        // first dequantize warp; warps 3..6 are the epilogue, one per TMEM lane quarter (warp & 3)
constexpr int DQ_WARPS = 16;       // two groups of eight, one row-tile each, which take turns at the units
constexpr int HELPERS = 1 + DQ_WARPS / 4;  // warps per TMEM lane quarter that share a CTA's last epilogue
constexpr int RAW_WARP2 = DQ_WARP0 + DQ_WARPS;  // the second raw producer
constexpr int THREADS = (RAW_WARP2 + 1) * 32;
// Register bound (72) of the kernel: leaves a CTA of the conversion kernel room beside it on an SM.
constexpr int REG_THREADS = 896;
constexpr int TMEM_COLS = 512;     // two accumulators, the stages of the weight operand
constexpr int MAX_PARTS = 4;
// The forms of the kernel. COLS: columns of an accumulator. 64 leaves TMEM for three operand stages of a unit each; 128 for eight
// blocks, as four stages of half a unit, so that a group of dequantize warps makes one half while the MMAs read the other; the
// activations then have stages of their own, three. TILED: more than 64 rows, in tiles of up to COLS rows; K is not cut.
template <int COLS, bool TILED> struct Form {
  static constexpr bool WIDE = COLS > 64;
  static constexpr int HALVES = WIDE ? 2 : 1;       // stages of a unit
  static constexpr int BPS = 4 / HALVES;            // 64-k blocks of a stage
  static constexpr int ST = WIDE ? 4 : 3;           // stages: of the weight operand, or of both
  static constexpr int BST = 3;                     // stages of the activations, bn * BPS * 128 bytes each
  static constexpr int A_COL0 = 2 * COLS;
};

// Sub-block scales of a unit (Q4_K / Q5_K): lane 2r + h holds, for row r of the row-tile, the f16 scales and negated mins of
// sub-blocks 4h, 4h + 1 (dl[0], ml[0]) and 4h + 2, 4h + 3 (dl[1], ml[1]). Worked out once per unit and row instead of by
// every lane that needs them.
struct RowScales { uint32_t dl[2], ml[2]; };
template <int DT>
__device__ __forceinline__ RowScales row_scales(const uint8_t* t, int lane) {
  RowScales u{};
  if constexpr (DT == TQ_Q4_K || DT == TQ_Q5_K) {
    const __half2 off = __float2half2_rn(1024.f);
    const uint4 hd = lds_v4(t + 16 * (lane >> 1));
    // Half arithmetic only (no int->float / float->half conversions, which share one narrow pipe):
    // d * sc is exact in f32, so one f16 multiply rounds it the same way.
    const __half2 dd = u2h2(__byte_perm(hd.x, 0u, 0x1010)), mm = __hneg2(u2h2(__byte_perm(hd.x, 0u, 0x3232)));
    // 6-bit scales / mins of sub-blocks 0..3 or 4..7, one per byte
    const bool hi = lane & 1;
    const uint32_t scw = hi ? ((hd.w & 0x0F0F0F0Fu) | ((hd.y >> 2) & 0x30303030u)) : (hd.y & 0x3F3F3F3Fu);
    const uint32_t mnw = hi ? (((hd.w >> 4) & 0x0F0F0F0Fu) | ((hd.z >> 2) & 0x30303030u)) : (hd.z & 0x3F3F3F3Fu);
    u.dl[0] = h22u(__hmul2(dd, __hsub2(pair01(scw), off)));
    u.dl[1] = h22u(__hmul2(dd, __hsub2(pair23(scw), off)));
    u.ml[0] = h22u(__hmul2(mm, __hsub2(pair01(mnw), off)));
    u.ml[1] = h22u(__hmul2(mm, __hsub2(pair23(mnw), off)));
  }
  return u;
}

// 64-k block i of a unit (t: the row-tile's raw bytes in shared memory) as registers of a tcgen05.st 16x256b.x4:
// register 4j + 2h + e of lane 4g + c holds columns 8j + 2c + e of row g + 8h, two f16 each, so
// chunk j (16 k, one MMA) has from this lane the elements 32 (j / 2) + 8c + 4 (j % 2) + {0, 2, 1, 3}; in Q6_K's own order
// (OWN) 16j + 4c + {0, 2, 1, 3}.
template <int DT, bool OWN>
__device__ __forceinline__ void dequant_frag(const uint8_t* t, const RowScales& us, int i, int lane, uint32_t (&o)[16]) {
  const int g = lane >> 2, c = lane & 3;
  if constexpr (DT == TQ_Q8_0) {
    const __half2 off = __float2half2_rn(1152.f);  // 1024 + 128: bytes are biased by xor 0x80
#pragma unroll
    for (int s = 0; s < 2; s++) {
      const uint8_t* tt = t + (2 * i + s) * 544;
      const uint4 q = lds_v4(tt + TQ_Q8_0_QS + 16 * lane);
      const uint32_t w[2][2] = {{q.x ^ 0x80808080u, q.y ^ 0x80808080u}, {q.z ^ 0x80808080u, q.w ^ 0x80808080u}};
#pragma unroll
      for (int hr = 0; hr < 2; hr++) {
        const __half2 d2 = __half2half2(__ushort_as_half((unsigned short)lds_u16(tt + 2 * (g + 8 * hr))));
#pragma unroll
        for (int b = 0; b < 2; b++) {
          o[4 * (2 * s + b) + 2 * hr] = h22u(__hmul2(__hsub2(pair02(w[hr][b]), off), d2));
          o[4 * (2 * s + b) + 2 * hr + 1] = h22u(__hmul2(__hsub2(pair13(w[hr][b]), off), d2));
        }
      }
    }
  } else if constexpr (DT == TQ_Q4_K || DT == TQ_Q5_K) {
    constexpr int QS = DT == TQ_Q4_K ? TQ_Q4K_QS : TQ_Q5K_QS;
    const uint4 q = lds_v4(t + QS + 512 * i + 16 * lane);
    const uint32_t w[2][2] = {{q.x, q.y}, {q.z, q.w}};
    uint32_t qh[2][2] = {{0, 0}, {0, 0}};
    if constexpr (DT == TQ_Q5_K) {
      const uint4 h4 = lds_v4(t + TQ_Q5K_QH + 16 * lane);
      qh[0][0] = h4.x; qh[0][1] = h4.y; qh[1][0] = h4.z; qh[1][1] = h4.w;
    }
#pragma unroll
    for (int hr = 0; hr < 2; hr++) {
      const int src = 2 * (g + 8 * hr) + (i >> 1);
      const __half2 dl2 = u2h2(__shfl_sync(0xFFFFFFFFu, us.dl[i & 1], src)), ml2 = u2h2(__shfl_sync(0xFFFFFFFFu, us.ml[i & 1], src));
      // sub-blocks 2i (low nibbles) and 2i + 1 (high nibbles)
      const __half2 dlo = __low2half2(dl2), dhi = __high2half2(dl2), mlo = __low2half2(ml2), mhi = __high2half2(ml2);
#pragma unroll
      for (int b = 0; b < 2; b++) {
        __half2 v[2][2];  // [nibble][bytes 0, 2 | 1, 3]
        if constexpr (DT == TQ_Q4_K) {
          // A nibble becomes a half without being moved: under the exponent of 1024 the low nibble counts ones, under
          // that of 64 the high nibble (16 units of 1/16) does; the offset subtracts exactly. Bytes 1 and 3 are brought
          // down once, as halves 1024 + byte; their low nibble is what is left without 16 times (64 + high nibble).
          const uint32_t x = w[hr][b];
          const __half2 k64 = u2h2(0x54005400u), k1024 = u2h2(0x64006400u), m16 = __float2half2_rn(-16.f);
          const __half2 p = pair13(x);
          const __half2 h02 = u2h2((x & 0x00F000F0u) | 0x54005400u), h13 = u2h2((h22u(p) & 0x00F000F0u) | 0x54005400u);
          v[0][0] = __hsub2(u2h2((x & 0x000F000Fu) | 0x64006400u), k1024);
          v[0][1] = __hfma2(h13, m16, p);
          v[1][0] = __hsub2(h02, k64);
          v[1][1] = __hsub2(h13, k64);
        } else {
          const __half2 off = __float2half2_rn(1024.f);
#pragma unroll
          for (int s = 0; s < 2; s++) {
            // the sub-block's bit, brought to bit 4 of every byte
            const uint32_t m = ((w[hr][b] >> (4 * s)) & 0x0F0F0F0Fu) |
                               (__funnelshift_l(qh[hr][b], qh[hr][b], 4 - (2 * i + s)) & 0x10101010u);
            v[s][0] = __hsub2(pair02(m), off);
            v[s][1] = __hsub2(pair13(m), off);
          }
        }
        o[4 * b + 2 * hr] = h22u(__hfma2(v[0][0], dlo, mlo));
        o[4 * b + 2 * hr + 1] = h22u(__hfma2(v[0][1], dlo, mlo));
        o[4 * (2 + b) + 2 * hr] = h22u(__hfma2(v[1][0], dhi, mhi));
        o[4 * (2 + b) + 2 * hr + 1] = h22u(__hfma2(v[1][1], dhi, mhi));
      }
    }
  } else if constexpr (OWN) {  // chunk j is the block's 16-element sub-block j
    const uint4 ql = lds_v4(t + TQ_Q6K_QL + 512 * i + 16 * lane), qv = lds_v4(t + TQ_Q6K_QH + 512 * (i >> 1) + 16 * lane);
    const __half2 off = __float2half2_rn(1056.f);     // 1024 + 32
    const __half2 off_sc = __float2half2_rn(1152.f);  // 1024 + 128: the int8 scales are biased by xor 0x80
#pragma unroll
    for (int hr = 0; hr < 2; hr++) {
      const uint32_t qh = (i & 1) ? (hr ? qv.w : qv.y) : (hr ? qv.z : qv.x);
      // d * scale of the four sub-blocks in half arithmetic (exact product, one rounding)
      const __half2 dd = __half2half2(__ushort_as_half((unsigned short)lds_u16(t + TQ_Q6K_D + 2 * (g + 8 * hr))));
      const uint32_t scb = ld_u32(t + 16 * (g + 8 * hr) + 4 * i) ^ 0x80808080u;
      const __half2 d01 = __hmul2(dd, __hsub2(pair01(scb), off_sc)), d23 = __hmul2(dd, __hsub2(pair23(scb), off_sc));
#pragma unroll
      for (int jj = 0; jj < 4; jj++) {
        const __half2 dl = jj == 0 ? __low2half2(d01) : jj == 1 ? __high2half2(d01) : jj == 2 ? __low2half2(d23) : __high2half2(d23);
        const uint32_t w = jj < 2 ? (hr ? ql.z : ql.x) : (hr ? ql.w : ql.y);
        const int sh = 2 * jj;  // 2-bit field jj of the qh word moved to bits 4..5 of every byte
        const uint32_t m = (((jj & 1) ? w >> 4 : w) & 0x0F0F0F0Fu) | ((sh <= 4 ? qh << (4 - sh) : qh >> (sh - 4)) & 0x30303030u);
        o[4 * jj + 2 * hr] = h22u(__hmul2(__hsub2(pair02(m), off), dl));
        o[4 * jj + 2 * hr + 1] = h22u(__hmul2(__hsub2(pair13(m), off), dl));
      }
    }
  } else {  // Q6_K: a lane takes its eight elements of every 32 from the two lanes that hold them in the tile
    const int nib = c >> 1, la = 4 * g + 2 * (c & 1);
    const uint8_t* const qhp = t + TQ_Q6K_QH + 512 * (i >> 1) + 4 * (i & 1) + 16 * la;
    const uint4 qa = lds_v4(t + TQ_Q6K_QL + 512 * i + 16 * la), qb = lds_v4(t + TQ_Q6K_QL + 512 * i + 16 * la + 16);
    const __half2 off = __float2half2_rn(1056.f);     // 1024 + 32
    const __half2 off_sc = __float2half2_rn(1152.f);  // 1024 + 128: the int8 scales are biased by xor 0x80
#pragma unroll
    for (int hr = 0; hr < 2; hr++) {
      const uint32_t ql[2][2] = {{hr ? qa.z : qa.x, hr ? qb.z : qb.x}, {hr ? qa.w : qa.y, hr ? qb.w : qb.y}};
      const uint32_t qh[2] = {ld_u32(qhp + 8 * hr), ld_u32(qhp + 16 + 8 * hr)};
      // d * scale of sub-blocks 4i + nib and 4i + 2 + nib in half arithmetic (exact product, one rounding)
      const __half2 dd = __half2half2(__ushort_as_half((unsigned short)lds_u16(t + TQ_Q6K_D + 2 * (g + 8 * hr))));
      const uint32_t scb = ld_u32(t + 16 * (g + 8 * hr) + 4 * i) ^ 0x80808080u;
      const __half2 dl2 = __hmul2(dd, __hsub2(pair02(scb >> (8 * nib)), off_sc));
#pragma unroll
      for (int s = 0; s < 2; s++) {
        const __half2 dl = s ? __high2half2(dl2) : __low2half2(dl2);
#pragma unroll
        for (int b = 0; b < 2; b++) {
          // 2-bit field 2s + nib of the qh word, brought to bits 4..5 of every byte
          const uint32_t m = ((ql[s][b] >> (4 * nib)) & 0x0F0F0F0Fu) |
                             (__funnelshift_l(qh[b], qh[b], 4 - 4 * s - 2 * nib) & 0x30303030u);
          o[4 * (2 * s + b) + 2 * hr] = h22u(__hmul2(__hsub2(pair02(m), off), dl));
          o[4 * (2 * s + b) + 2 * hr + 1] = h22u(__hmul2(__hsub2(pair13(m), off), dl));
        }
      }
    }
  }
}
__device__ __forceinline__ void tmem_store_block(uint32_t taddr, const uint32_t (&o)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]), "r"(o[8]), "r"(o[9]), "r"(o[10]),
      "r"(o[11]), "r"(o[12]), "r"(o[13]), "r"(o[14]), "r"(o[15])
      : "memory");
}


// Whether a weight is multiplied in the k order of its own tiles. Only where the K loop is cut: a sum that one CTA adds up
// keeps the MMAs of the prefill kernel, and with them its bits.
__host__ __device__ __forceinline__ bool own_order(int dtype, int csize) { return dtype == TQ_Q6_K && csize > 1; }

struct BatchPart {
  const uint8_t* tiles;
  const uint8_t* xh;   // B operand image in the weight's k order: [mt][kblocks][bn][128 bytes]
  float* y;            // [m, n_rows]
  float* y_alt;
  const float* bias;
  int64_t n_rows;
  int row_tiles;       // 16-row tiles of the weight
  int ktiles;          // device tiles per row-tile
  int dtype;
  int item0;           // the first of the weight's items (128 weight rows by a tile of activation rows)
};

struct BatchArgs {
  BatchPart part[MAX_PARTS];
  int nparts;
  int items;            // of all weights
  int kblocks;          // k / 64
  int KU;               // units of 256 k per row (the last one of a Q8_0 weight may hold fewer blocks)
  int m;                // activation rows
  int bn;               // rows of a tile, a multiple of 16
  int mt;               // tiles of bn rows (1 up to 64 rows)
  int raw_slots, slot_bytes;
  int red_bytes;        // exchange buffer of a CTA
  const float* rscale;  // [m] factor undoing the f16 row scaling
  int* status;
  // tiled form (tc_common.cuh): the preceding launch belongs to the same call and reads the same x; go-ahead words [CTA] of this
  // launch and of the one behind it, which has next_ctas CTAs (0: none follows)
  int sibling;
  int *go, *next_go;
  int next_ctas;
  // exchange slots (tp.cu): with y_toggle set, the result goes to y_alt instead of y when the
  // word it points to, plus one, is odd - read after the preceding kernels have completed
  const unsigned* y_toggle;
};

// The items a cluster works on, in order; every role of all its CTAs walks the same list.
template <bool TILED> struct Walk {
  int item, part, step;
  __device__ __forceinline__ void init(int first, int clusters) {
    item = first - clusters;
    step = clusters;
    part = 0;
  }
  __device__ __forceinline__ bool next(const BatchArgs& a) {
    item += step;
    if (item >= a.items) return false;
    while (part + 1 < a.nparts && item >= a.part[part + 1].item0) part++;
    return true;
  }
  __device__ __forceinline__ bool last(const BatchArgs& a) const { return item + step >= a.items; }
  __device__ __forceinline__ int row_tile(const BatchArgs& a) const {
    const int i = item - a.part[part].item0;
    return (TILED ? i / a.mt : i) * (BM / TQ_TILE_ROWS);
  }
  __device__ __forceinline__ int m0(const BatchArgs& a) const {  // the first activation row
    const int i = item - a.part[part].item0;
    return TILED ? i % a.mt * a.bn : 0;
  }
  __device__ __forceinline__ int rows(const BatchArgs& a) const {
    const int left = a.m - m0(a);
    return TILED && left > a.bn ? a.bn : left;
  }
};

__device__ __forceinline__ void commit_to(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s_u32(bar)) : "memory");
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(s_u32(dst)), "l"(src),
               "r"(bytes), "r"(s_u32(bar))
               : "memory");
}
// Walks chunks of columns; which CTA of the cluster adds one up, and which of that CTA's chunks it is. No divisions on the way.
struct Chunk {
  int ch, owner, index;
  __device__ __forceinline__ Chunk(int first, int csize) : ch(0), owner(0), index(0) { advance(first, csize); }
  __device__ __forceinline__ void advance(int by, int csize) {
    ch += by;
    owner += by;
    while (owner >= csize) { owner -= csize; index++; }
  }
};

// Epilogue of one item for one TMEM lane quarter (32 weight rows): of the chunks h0, h0 + hstep, ... those that other CTAs
// add up are sent to them, then those of this CTA (chunk % cluster size == rank) are added and stored.
// Exchange buffer of a CTA: [its chunks][other ranks][CH / 4][BM] of four columns.
template <bool TILED>
__device__ __forceinline__ void epilogue(const BatchArgs& a, const Walk<TILED>& w, int rank, int csize, int quarter, int lane, uint32_t tmem,
                                         int h0, int hstep, const float* scale, uint8_t* red, uint64_t* red_full, uint32_t parity, volatile int* abort_flag) {
  const int m0 = w.m0(a), rows = w.rows(a), nchunks = (rows + CH - 1) / CH;
  const uint32_t taddr = tmem + ((uint32_t)(32 * quarter) << 16);
  const int row = 32 * quarter + lane;
  float v[CH];
  auto load_acc = [&](int ch) {
    uint32_t u[CH];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
                 : "r"(taddr + (uint32_t)(ch * CH))
                 : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < CH; j++) v[j] = __uint_as_float(u[j]);
  };
  if (csize > 1) {
    Chunk c(h0, csize);
    for (; c.ch < nchunks; c.advance(hstep, csize)) {
      const int to = c.owner;
      if (to == rank) continue;
      load_acc(c.ch);
      const uint32_t slot = (uint32_t)(c.index * (csize - 1) + (rank < to ? rank : rank - 1));
      const uint32_t dst = map_to_rank(s_u32(red) + slot * CH_BYTES + (uint32_t)row * 16, (uint32_t)to);
      const uint32_t bar = map_to_rank(s_u32(red_full), (uint32_t)to);
#pragma unroll
      for (int j = 0; j < CH / 4; j++)
        asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                         dst + (uint32_t)(j * BM * 16)),
                     "f"(v[4 * j]), "f"(v[4 * j + 1]), "f"(v[4 * j + 2]), "f"(v[4 * j + 3]), "r"(bar)
                     : "memory");
    }
  }
  const BatchPart& p = a.part[w.part];
  const int64_t n = (int64_t)w.row_tile(a) * TQ_TILE_ROWS + row;
  const bool live = n < p.n_rows;
  const float bv = (p.bias && live) ? p.bias[n] : 0.f;
  float* ybase = p.y;
  if (a.y_toggle && ((*reinterpret_cast<const volatile unsigned*>(a.y_toggle) + 1u) & 1u)) ybase = p.y_alt;
  float* const yp = ybase + (TILED ? (int64_t)m0 * p.n_rows : 0) + n;
  scale += m0;
  bool waited = csize == 1;
  for (Chunk c(h0, csize); c.ch < nchunks; c.advance(hstep, csize)) {
    if (c.owner != rank) continue;
    const int ch = c.ch;
    load_acc(ch);
    if (csize > 1) {
      if (!waited) {
        bar_pass(red_full, parity, abort_flag);
        waited = true;
      }
      const uint8_t* const in = red + (c.index * (csize - 1)) * CH_BYTES + row * 16;
      float s[CH];
#pragma unroll
      for (int j = 0; j < CH; j++) s[j] = rank == 0 ? v[j] : 0.f;
      for (int o = 0; o < csize; o++) {  // rank order
        if (o == rank) {
          if (o > 0) {
#pragma unroll
            for (int j = 0; j < CH; j++) s[j] += v[j];
          }
        } else {
          const uint8_t* const from = in + (o < rank ? o : o - 1) * CH_BYTES;
#pragma unroll
          for (int j = 0; j < CH / 4; j++) {
            const float4 q = *reinterpret_cast<const float4*>(from + j * BM * 16);
            s[4 * j] += q.x;
            s[4 * j + 1] += q.y;
            s[4 * j + 2] += q.z;
            s[4 * j + 3] += q.w;
          }
        }
      }
#pragma unroll
      for (int j = 0; j < CH; j++) v[j] = s[j];
    }
    if (live) {
      const float4 r0 = *reinterpret_cast<const float4*>(scale + ch * CH), r1 = *reinterpret_cast<const float4*>(scale + ch * CH + 4);
      const float r[CH] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
      float* yc = yp + (int64_t)(ch * CH) * p.n_rows;
      const int cols = rows - ch * CH;
#pragma unroll
      for (int j = 0; j < CH; j++) {
        if (j < cols) *yc = v[j] * r[j] + bv;
        yc += p.n_rows;
      }
    }
  }
}

// The rings as the dequantize warps walk them.
struct DequantPos {
  int use, s, turn;
  uint32_t rph, ph;
};

// A warp's share of an item: one 16-row tile (`dq` of the CTA's eight) of every other unit. Whole units, so that what a
// unit costs beside the conversion itself (barriers, scales, addresses) is spread over four blocks.
template <class F, int DT, bool OWN = false>
__device__ __forceinline__ void dequant_units(const BatchArgs& a, int ka, int kb, bool live, int dq, int grp, int lane, uint8_t* raw0,
                                              uint64_t* raw_full, uint64_t* raw_empty, uint64_t* full, uint64_t* empty, uint32_t tmem,
                                              DequantPos& pos, volatile int* abort_flag) {
  for (int ku = ka; ku < kb; ku++) {
    if (pos.turn == grp) {
      bar_pass(&raw_full[pos.use], pos.rph, abort_flag);
      const int slot = pos.use >= a.raw_slots ? pos.use - a.raw_slots : pos.use;
      const uint8_t* raw = raw0 + slot * a.slot_bytes + dq * UnitGeom<DT>::BYTES;
      const int nb = a.kblocks - 4 * ku;
      const RowScales us = row_scales<DT>(raw, lane);
#pragma unroll
      for (int h = 0; h < F::HALVES; h++) {
        bar_pass(&empty[pos.s + h], pos.ph ^ 1u, abort_flag);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t dst = tmem + ((uint32_t)(16 * dq) << 16) + (uint32_t)(F::A_COL0 + (pos.s + h) * F::BPS * A_COLS);
        if (live) {
#pragma unroll
          for (int e = 0; e < F::BPS; e++) {
            const int b = h * F::BPS + e;
            if (b == 0 || DT != TQ_Q8_0 || b < nb) {
              uint32_t o[16];
              dequant_frag<DT, OWN>(raw, us, b, lane, o);
              tmem_store_block(dst + (uint32_t)(e * A_COLS), o);
            }
          }
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) bar_arrive(&full[pos.s + h]);
      }
      if (lane == 0) bar_arrive(&raw_empty[pos.use]);
    }
    pos.turn ^= 1;
    pos.s += F::HALVES;
    if (pos.s == F::ST) { pos.s = 0; pos.ph ^= 1u; }
    if (++pos.use == 2 * a.raw_slots) { pos.use = 0; pos.rph ^= 1u; }
  }
}

template <int COLS, bool TILED>
__global__ void __launch_bounds__(REG_THREADS, 1) gemm_batch_kernel(const __grid_constant__ BatchArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // 1024-byte alignment for the swizzled operand; the same offsets in all CTAs of the cluster
  uint8_t* const smem = smem_raw + ((1024u - (s_u32(smem_raw) & 1023u)) & 1023u);
  using F = Form<COLS, TILED>;
  constexpr int ST = F::ST, BST = F::BST;
  const int b_stage = a.bn * F::BPS * 128;
  uint8_t* const sB = smem;
  uint8_t* const sRaw = sB + BST * b_stage;
  uint8_t* const sRed = sRaw + a.raw_slots * a.slot_bytes;
  float* const sScale = reinterpret_cast<float*>(sRed + a.red_bytes);  // row scales
  uint64_t* const full = reinterpret_cast<uint64_t*>(sScale + (TILED ? a.mt * a.bn : GEMM_BATCH_ROWS));  // both operands of a stage (wide: the weights)
  uint64_t* const empty = full + ST;
  uint64_t* const b_full = F::WIDE ? empty + ST : full;      // the activations' stages
  uint64_t* const b_empty = F::WIDE ? b_full + BST : empty;
  uint64_t* const raw_full = F::WIDE ? b_empty + BST : empty + ST;
  uint64_t* const raw_empty = raw_full + 2 * MAX_RAW;
  uint64_t* const acc_full = raw_empty + 2 * MAX_RAW;
  uint64_t* const acc_empty = acc_full + 2;
  uint64_t* const last_full = acc_empty + 2;  // the CTA's last accumulator is complete
  uint64_t* const red_full = last_full + 1;   // the other CTAs' sums of an item are here; of the last item
  uint64_t* const red_last = red_full + 1;
  uint64_t* const red_free = red_last + 1;    // the other CTAs have read what this one sent them of an item
  uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(red_free + 1);
  volatile int* const abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = TILED ? 0 : (int)cluster_rank(), csize = TILED ? 1 : (int)cluster_size();

  // Siblings: beside the set-up, whose barrier then orders every warp of the CTA behind the word's acquire.
  bool go = true;
  if (TILED && a.sibling && warp == 1 && lane == 0) go = take_go(a.go + blockIdx.x);
  if (warp == 0) {
    // one barrier per lane
    if (lane < ST) {
      bar_init(&full[lane], DQ_WARPS / 2 + (F::WIDE ? 0 : 1));
      bar_init(&empty[lane], 1);
    }
    if (F::WIDE && lane < BST) {
      bar_init(&b_full[lane], 1);
      bar_init(&b_empty[lane], 1);
    }
    if (lane < 2 * a.raw_slots) {
      bar_init(&raw_full[lane], 1);
      bar_init(&raw_empty[lane], DQ_WARPS / 2);
    }
    if (lane < 2) {
      bar_init(&acc_full[lane], 1);
      bar_init(&acc_empty[lane], EP_WARPS);
    }
    if (lane == 0) {
      bar_init(last_full, 1);
      bar_init(red_full, 1);
      bar_init(red_last, 1);
      bar_init(red_free, (uint32_t)(EP_WARPS * (csize > 1 ? csize - 1 : 1)));
      *abort_flag = 0;
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_u32(tmem_slot)), "n"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (csize > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");  // the others' barriers: waited for below
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  // this CTA's share of the K loop, the same for every item
  const int ka = a.KU * rank / csize, kb = a.KU * (rank + 1) / csize;

  Walk<TILED> walk;
  walk.init((int)blockIdx.x / csize, (int)gridDim.x / csize);
  if (warp == 0 || warp == RAW_WARP2) {
    // ------------------------------------------------------------ raw weight bytes -> ring (lane r: row-tile r)
    // Two warps take turns at the units: a warp needs some 70 cycles to issue a copy, 600 for the eight of a unit.
    // A slot has two sets of barriers for its alternate uses, so that one set always belongs to the same producer and the same
    // group of dequantize warps, also where the number of slots is odd: whoever skipped a phase of a barrier could ask for the
    // next but one while the barrier is two behind, which its parity does not tell apart.
    int use = 0, turn = warp == 0 ? 0 : 1;
    uint32_t ph = 0;
    bool ok = true;
    while (ok && walk.next(a)) {
      const BatchPart& p = a.part[walk.part];
      const int tiles_u = p.dtype == TQ_Q8_0 ? UnitGeom<TQ_Q8_0>::TILES : 1;
      const int tb = tq_tile_bytes(p.dtype), ub = tiles_u * tb;
      const int rt0 = walk.row_tile(a);
      const int nlive = p.row_tiles - rt0 > 8 ? 8 : p.row_tiles - rt0;
      const uint8_t* const row = p.tiles + (int64_t)(rt0 + lane) * p.ktiles * tb;
      for (int ku = ka; ku < kb; ku++) {
        if (turn == 0) {
          // the use before this one went by the slot's other set
          const bool second = use >= a.raw_slots;
          const int slot = second ? use - a.raw_slots : use;
          ok = __all_sync(0xFFFFFFFFu, bar_wait(&raw_empty[second ? slot : use + a.raw_slots], second ? ph : ph ^ 1u, abort_flag));
          if (!ok) break;
          int nt = p.ktiles - ku * tiles_u;
          if (nt > tiles_u) nt = tiles_u;
          const uint32_t bytes = (uint32_t)(nt * tb);
          if (lane == 0) bar_expect_tx(&raw_full[use], bytes * (uint32_t)nlive);
          __syncwarp();
          if (lane < nlive) bulk_load(sRaw + slot * a.slot_bytes + lane * ub, row + (int64_t)ku * ub, bytes, &raw_full[use]);
        }
        turn ^= 1;
        if (++use == 2 * a.raw_slots) { use = 0; ph ^= 1u; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ activation image -> stages
    if (lane == 0) {
      // Programmatic stream serialization: the image comes from the conversion launch before this one (the
      // weight side starts without waiting). A sibling's go-ahead word stands for that wait; the proxy fence carries what
      // its acquire made visible over to the bulk copies.
      if (TILED && a.sibling) {
        if (!go) *abort_flag = 1;
        asm volatile("fence.proxy.async.global;" ::: "memory");
      } else {
        asm volatile("griddepcontrol.wait;" ::: "memory");
      }
      asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      while (ok && walk.next(a)) {
        const uint8_t* xh = a.part[walk.part].xh;
        if (TILED) xh += (int64_t)walk.m0(a) * a.kblocks * 128;
        for (int ku = F::HALVES * ka; ok && ku < F::HALVES * kb; ku++) {
          ok = bar_wait(&b_empty[s], ph ^ 1u, abort_flag);
          if (!ok) break;
          const int left = a.kblocks - F::BPS * ku, nb = left < 0 ? 0 : left < F::BPS ? left : F::BPS;
          const uint32_t bytes = (uint32_t)(nb * a.bn * 128);
          bar_expect_tx(&b_full[s], bytes);
          if (!F::WIDE || nb > 0) bulk_load(sB + s * b_stage, xh + (int64_t)ku * b_stage, bytes, &b_full[s]);
          if (++s == BST) { s = 0; ph ^= 1u; }
        }
      }
    }
  } else if (warp == 2) {
    // ------------------------------------------------------------ MMA issuer
    // The whole warp walks the loop and one elected lane issues: control flow and descriptors stay warp-uniform.
    // instruction descriptor: f32 accumulate, f16 x f16, both K-major, N = bn, M = 128
    const uint32_t idesc = (1u << 4) | ((uint32_t)(a.bn >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
    // K-major, 128-byte swizzle matrix descriptor (8-row groups 1024 B apart): a constant high
    // half plus a low half that advances by 2 (32 bytes >> 4) per 16-element K step
    constexpr uint64_t desc_hi = (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
    const uint32_t b_lo0 = (s_u32(sB) & 0x3FFFFu) >> 4, b_step = (uint32_t)(a.bn * 128) >> 4;
    const bool issuer = elect_one();
    int s = 0, sb = 0, nitem = 0;
    uint32_t ph = 0, bph = 0;
    while (walk.next(a)) {
      const int acc = nitem & 1;
      const uint32_t aph = (uint32_t)(nitem >> 1) & 1u;
      nitem++;
      bar_pass(&acc_empty[acc], aph ^ 1u, abort_flag);
      const uint32_t d = tmem_base + (uint32_t)(acc * COLS);
      uint32_t accumulate = 0;  // the first MMA of the item overwrites the accumulator
      for (int ku = F::HALVES * ka; ku < F::HALVES * kb; ku++) {
        const int nb = a.kblocks - F::BPS * ku;
        if (!F::WIDE) sb = s;
        bar_pass(&full[s], ph, abort_flag);
        if (F::WIDE) bar_pass(&b_full[sb], bph, abort_flag);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (issuer) {
#pragma unroll
          for (int b = 0; b < F::BPS; b++) {
            if ((!F::WIDE && b == 0) || b < nb) {
              const uint64_t db = desc_hi | (uint64_t)(b_lo0 + (uint32_t)(sb * F::BPS + b) * b_step);
#pragma unroll
              for (int kk = 0; kk < BK / 16; kk++)
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
                    "r"(tmem_base + (uint32_t)(F::A_COL0 + (s * F::BPS + b) * A_COLS + 8 * kk)), "l"(db + (uint64_t)(2 * kk)), "r"(idesc),
                    "r"(b + kk > 0 ? 1u : accumulate)
                    : "memory");
            }
          }
          commit_to(&empty[s]);  // frees the operands once these MMAs have read them
          if (F::WIDE) commit_to(&b_empty[sb]);
        }
        __syncwarp();
        accumulate = 1u;
        if (++s == ST) { s = 0; ph ^= 1u; }
        if (F::WIDE && ++sb == BST) { sb = 0; bph ^= 1u; }
      }
      if (issuer) commit_to(walk.last(a) ? last_full : &acc_full[acc]);
      __syncwarp();
    }
  } else if (warp < DQ_WARP0) {
    // ------------------------------------------------------------ epilogue
    if (!TILED || !a.sibling) asm volatile("griddepcontrol.wait;" ::: "memory");  // y may still be read, the row scales still written
    if (TILED && warp == 3)  // what this launch has waited for, a sibling behind it need not wait for again
      for (int i = (int)(blockIdx.x + lane * gridDim.x); i < a.next_ctas; i += 32 * (int)gridDim.x) st_release(a.next_go + i, 1);
    if (csize > 1) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");  // before anything is sent
    const int quarter = warp & 3;
    // In shared memory, where no store to y keeps a load of the next scale behind it (every load on its own: 2800 cycles a chunk)
    for (int i = (warp - 3) * 32 + lane; i < (TILED ? a.mt * a.bn : GEMM_BATCH_ROWS); i += EP_WARPS * 32) sScale[i] = i < a.m ? a.rscale[i] : 0.f;
    asm volatile("bar.sync 2, %0;" ::"n"(EP_WARPS * 32) : "memory");
    // bytes an item's exchange brings this CTA
    const int nchunks = (a.m + CH - 1) / CH, mine = (nchunks - rank + csize - 1) / csize;
    const uint32_t incoming = TILED ? 0u : (uint32_t)(mine * (csize - 1) * CH_BYTES);
    int nitem = 0;
    while (walk.next(a)) {
      const int acc = nitem & 1;
      const uint32_t aph = (uint32_t)(nitem >> 1) & 1u;
      const bool last = walk.last(a);
      if (warp == 3 && lane == 0 && incoming) bar_expect_tx(last ? red_last : red_full, incoming);
      bar_pass(last ? last_full : &acc_full[acc], last ? 0u : aph, abort_flag);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (nitem > 0 && csize > 1) bar_pass(red_free, (uint32_t)(nitem - 1) & 1u, abort_flag);
      // the last epilogue is shared with the dequantize warps, which have nothing left to do
      if (last) asm volatile("bar.sync 1, %0;" ::"n"((EP_WARPS + DQ_WARPS) * 32) : "memory");
      epilogue(a, walk, rank, csize, quarter, lane, tmem_base + (uint32_t)(acc * COLS), 0, last ? HELPERS : 1, sScale, sRed,
               last ? red_last : red_full, last ? 0u : (uint32_t)nitem & 1u, abort_flag);
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (!last) {
        if (lane == 0) bar_arrive(&acc_empty[acc]);
        if (lane < csize && lane != rank)
          asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(map_to_rank(s_u32(red_free), (uint32_t)lane)) : "memory");
      }
      nitem++;
    }
  } else {
    // ------------------------------------------------------------ dequantize
    // A warp reaches one quarter of TMEM's lanes (warp & 3), 32 rows: two of the four warps of a quarter
    // take one 16-row tile each in one unit, the other two in the next.
    const int dqw = (warp - DQ_WARP0) >> 2;  // 0..3 within the quarter
    const int grp = dqw >> 1;
    const int dq = 2 * (warp & 3) + (dqw & 1);  // row-tile of 16 rows inside the CTA's 128 rows
    DequantPos pos{0, 0, 0, 0u, 0u};
    int nitem = 0;
    Walk<TILED> lw = walk;
    while (walk.next(a)) {
      lw = walk;
      nitem++;
      const BatchPart& p = a.part[walk.part];
      const bool live = walk.row_tile(a) + dq < p.row_tiles;  // rows beyond the weight are never stored
      switch (p.dtype) {
        case TQ_Q8_0: dequant_units<F, TQ_Q8_0>(a, ka, kb, live, dq, grp, lane, sRaw, raw_full, raw_empty, full, empty, tmem_base, pos, abort_flag); break;
        case TQ_Q4_K: dequant_units<F, TQ_Q4_K>(a, ka, kb, live, dq, grp, lane, sRaw, raw_full, raw_empty, full, empty, tmem_base, pos, abort_flag); break;
        case TQ_Q5_K: dequant_units<F, TQ_Q5_K>(a, ka, kb, live, dq, grp, lane, sRaw, raw_full, raw_empty, full, empty, tmem_base, pos, abort_flag); break;
        default:
          if (own_order(p.dtype, csize))
            dequant_units<F, TQ_Q6_K, true>(a, ka, kb, live, dq, grp, lane, sRaw, raw_full, raw_empty, full, empty, tmem_base, pos, abort_flag);
          else
            dequant_units<F, TQ_Q6_K>(a, ka, kb, live, dq, grp, lane, sRaw, raw_full, raw_empty, full, empty, tmem_base, pos, abort_flag);
          break;
      }
    }
    // nothing left to dequantize: help with the epilogue of the last item
    if (!TILED || !a.sibling) asm volatile("griddepcontrol.wait;" ::: "memory");
    if (csize > 1) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    const int acc = (nitem - 1) & 1;
    bar_pass(last_full, 0, abort_flag);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("bar.sync 1, %0;" ::"n"((EP_WARPS + DQ_WARPS) * 32) : "memory");
    epilogue(a, lw, rank, csize, warp & 3, lane, tmem_base + (uint32_t)(acc * COLS), dqw + 1, HELPERS, sScale, sRed, red_last, 0u, abort_flag);
  }
  // (every thread waits for the cluster's set-up before it arrives for its end)
  if (csize > 1 && (warp < 3 || warp == RAW_WARP2)) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*abort_flag) {
    // a wait ran out: give copies still in flight time to land in this CTA's shared memory
    for (int i = 0; i < 64; i++) __nanosleep(2000);
    if (threadIdx.x == 0) {
      *reinterpret_cast<volatile int*>(a.status) = 7;  // TURQ_E_TIMEOUT; the word may be mapped host memory
      __threadfence_system();
    }
  }
  // no CTA leaves while another may still send to it
  if (csize > 1) {
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(TMEM_COLS) : "memory");
  }
  // whoever waits for this launch has then waited for all of the call
  if (TILED && a.sibling && threadIdx.x == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Barriers and row scales.
template <int COLS, bool TILED> constexpr int bar_bytes(int scales) {
  using F = Form<COLS, TILED>;
  return scales * 4 + (2 * F::ST + (F::WIDE ? 2 * F::BST : 0) + 4 * MAX_RAW + 8) * 8 + 8;
}

int part_slot_bytes(int dtype) { return 8 * (dtype == TQ_Q8_0 ? UnitGeom<TQ_Q8_0>::TILES : 1) * tq_tile_bytes(dtype); }

// Allows the kernel all of an SM's shared memory, once per device: before it is launched, and before its occupancy is asked for.
template <int COLS, bool TILED>
cudaError_t configure() {
  static PerDeviceOnce configured;
  int dev = 0;
  cudaGetDevice(&dev);
  if (configured.done(dev)) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(gemm_batch_kernel<COLS, TILED>, cudaFuncAttributeMaxDynamicSharedMemorySize, device_smem_optin());
  if (e == cudaSuccess) configured.set(dev);
  return e;
}

// Clusters of `c` > 1 CTAs that are resident at once (one CTA per SM; SMs at the edge of a GPC stay empty), looked up once per
// device and size. Sizes the grid; what a cluster computes does not depend on it.
cudaError_t resident_clusters(int c, int* out) {
  static std::atomic<int> known[64][BATCH_MAX_CLUSTER + 1];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::atomic<int> unkept{0};
  return static_cast<cudaError_t>(ask_once(dev >= 0 && dev < 64 ? known[dev][c] : unkept, [&](int* n) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)c);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = (size_t)device_smem_optin();
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)c;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t a = configure<64, false>();
    if (a == cudaSuccess) a = cudaOccupancyMaxActiveClusters(n, gemm_batch_kernel<64, false>, &cfg);
    if (a != cudaSuccess) cudaGetLastError();  // reported by the call; not left for the next check
    return (int)a;
  }, out));
}

// Exchange buffer of a CTA: the sums of its share of the columns from the others of the cluster.
int exchange_bytes(int bn, int c) { return (bn / CH + c - 1) / c * (c - 1) * CH_BYTES; }

template <int COLS, bool TILED>
cudaError_t launch_form(BatchArgs& a, int c, int clusters, cudaStream_t s) {
  using F = Form<COLS, TILED>;
  a.red_bytes = exchange_bytes(a.bn, c);
  // 4 KB stay free for a CTA of the next call's conversion kernel.
  const int fixed = F::BST * F::BPS * a.bn * 128 + a.red_bytes + bar_bytes<COLS, TILED>(TILED ? a.mt * a.bn : GEMM_BATCH_ROWS) + 1024;
  const int room = device_smem_optin() - 4096 - fixed;
  a.raw_slots = room / a.slot_bytes < MAX_RAW ? room / a.slot_bytes : MAX_RAW;
  if (room < 0 || a.raw_slots < 2) return cudaErrorInvalidConfiguration;
  cudaError_t e = configure<COLS, TILED>();
  if (e != cudaSuccess) return e;
  return launch_pdl_cluster(gemm_batch_kernel<COLS, TILED>, (unsigned)c, dim3((unsigned)(clusters * c)), dim3(THREADS),
                            (size_t)(fixed + a.raw_slots * a.slot_bytes), s, a);
}

}  // namespace

bool gemm_batch_takes(const GemvPart* parts, int nparts, int64_t m, int sm_count) {
  if (m <= GEMM_BATCH_ROWS) return true;
  int64_t tiles = 0, call_tiles = 0;  // of 128 and of 256 rows
  for (int i = 0; i < nparts; i++) {
    tiles += (parts[i].n_rows + BM - 1) / BM;
    call_tiles += (parts[i].n_rows + 2 * BM - 1) / (2 * BM);
  }
  return plan_batch_tile(tiles, call_tiles, m, sm_count) > 0;
}

cudaError_t launch_gemm_batch(const GemvPart* parts, int nparts, int64_t k, const void* x, int x_dtype, int64_t m, uint8_t* scratch,
                              cudaStream_t s, uint8_t* workspace, int sm_count, int* launches, int* dev_status_word,
                              const unsigned* y_toggle) {
  if (k % BK != 0 || k > INT32_MAX || m <= 0 || m > GEMM_TILED_ROWS || nparts < 1 || nparts > MAX_PARTS) return cudaErrorInvalidValue;
  const int KU = (int)((k + UNIT_K - 1) / UNIT_K);
  const bool tiled = m > GEMM_BATCH_ROWS;
  int resident[BATCH_MAX_CLUSTER + 1] = {0, sm_count}, cluster[MAX_PARTS];  // a CTA of its own has an SM
  int64_t tiles = 0, call_tiles = 0;
  for (int i = 0; i < nparts; i++) {
    if (!tq_is_weight_type(parts[i].dtype) || k % tq_block_elems(parts[i].dtype) != 0) return cudaErrorInvalidValue;
    const int64_t t = (parts[i].n_rows + BM - 1) / BM;
    if (t > (1 << 24)) return cudaErrorInvalidValue;
    tiles += t;
    call_tiles += (parts[i].n_rows + 2 * BM - 1) / (2 * BM);
    // beyond 64 rows no sum is cut: all larger calls, this kernel's and the prefill kernel's, have the same bits
    cluster[i] = tiled ? 1 : plan_batch_cluster((int)t, KU);
    if (!resident[cluster[i]]) {
      cudaError_t e = resident_clusters(cluster[i], &resident[cluster[i]]);
      if (e != cudaSuccess) return e;
    }
  }
  const int bn = tiled ? plan_batch_tile(tiles, call_tiles, m, sm_count) : (int)(m + 15) / 16 * 16;
  if (bn <= 0) return cudaErrorInvalidValue;
  const int mt = (int)((m + bn - 1) / bn);
  // images of both k orders where a call needs both, the row scales behind them
  bool own = false, common = false;
  for (int i = 0; i < nparts; i++) (own_order(parts[i].dtype, cluster[i]) ? own : common) = true;
  const size_t image = gemm_operand_bytes((int64_t)mt * bn, k);
  uint8_t* const xh16 = scratch + (common ? image : 0);
  float* rscale = reinterpret_cast<float*>(scratch + ((int)own + (int)common) * image);
  cudaError_t e = launch_prep_image(x, x_dtype, m, k, bn, common ? scratch : nullptr, own ? xh16 : nullptr, rscale, s);
  if (launches) (*launches)++;
  if (e != cudaSuccess) return e;

  bool done[MAX_PARTS] = {};
  for (int i0 = 0; i0 < nparts; i0++) {
    if (done[i0]) continue;
    const int c = cluster[i0];
    auto items = [&](int i) { return (int)((parts[i].n_rows + BM - 1) / BM) * mt; };
    BatchArgs a{};
    a.kblocks = (int)(k / BK);
    a.KU = KU;
    a.m = (int)m;
    a.bn = bn;
    a.mt = mt;
    a.rscale = rscale;
    a.status = dev_status_word;
    a.y_toggle = y_toggle;
    for (int i = i0; i < nparts; i++) {
      if (tiled ? i != i0 : cluster[i] != c) continue;
      done[i] = true;
      BatchPart& p = a.part[a.nparts++];
      p.tiles = parts[i].tiles;
      p.xh = own_order(parts[i].dtype, c) ? xh16 : scratch;
      p.y = parts[i].y;
      p.y_alt = parts[i].y_alt;
      p.bias = parts[i].bias;
      p.n_rows = parts[i].n_rows;
      p.dtype = parts[i].dtype;
      p.row_tiles = (int)((p.n_rows + TQ_TILE_ROWS - 1) / TQ_TILE_ROWS);
      p.ktiles = (int)(k / tq_block_elems(p.dtype));
      p.item0 = a.items;
      a.items += items(i);
      if (part_slot_bytes(p.dtype) > a.slot_bytes) a.slot_bytes = part_slot_bytes(p.dtype);
    }
    int clusters = resident[c];
    if (clusters > a.items) clusters = a.items;
    if (tiled) {  // the weights of the call one launch each, side by side
      a.sibling = i0 > 0;
      a.go = reinterpret_cast<int*>(workspace) + (size_t)i0 * sm_count;
      a.next_go = a.go + sm_count;
      a.next_ctas = i0 + 1 == nparts ? 0 : items(i0 + 1) < sm_count ? items(i0 + 1) : sm_count;
    }
    e = !tiled ? launch_form<64, false>(a, c, clusters, s) : bn <= 64 ? launch_form<64, true>(a, c, clusters, s) : launch_form<128, true>(a, c, clusters, s);
    if (launches) (*launches)++;
    if (e != cudaSuccess) {
      if (a.sibling) cudaMemsetAsync(workspace, 0, gemm_workspace_bytes(sm_count), s);  // go-ahead words that nobody takes
      return e;
    }
  }
  return cudaSuccess;
}

}  // namespace turq
