// Per-warp arithmetic of the integer-scheme GEMV: one device tile (16 weight rows x one wire
// block) held in shared memory against up to 8*MG quantized activation rows, with integer
// MMAs.
//
// Lane l = 4g + c holds weight rows g and g+8 (A fragment) and, as B fragment, the bytes of
// activation row g for the elements lane column c owns (8c..8c+7 of every 32-element
// sub-block; 4c..4c+3 of every 16-element one). Its C fragment is
//   c0 = (row g, act 2c)  c1 = (row g, act 2c+1)  c2 = (row g+8, act 2c)  c3 = (row g+8, act 2c+1).
// Sub-block scales stay integers; one f32 multiply per (super-)block and output element.
// Fragment chunks are read from shared memory where they are needed (128-bit loads), which
// keeps the live register set small (96 registers, two CTAs per SM; one group of rows spills nothing, or 4 bytes
// with planes in global memory, two groups up to 24 bytes, 52 in the wide mixed Q5_K launch, four groups 210 to 360).
#pragma once
#include "device_utils.cuh"
#include "layout.h"

namespace turq {

template <int DT> struct TileGeom;
template <> struct TileGeom<TQ_Q8_0> { static constexpr int BYTES = 544, ELEMS = 32, GROUP = 4; };
template <> struct TileGeom<TQ_Q4_K> { static constexpr int BYTES = 2304, ELEMS = 256, GROUP = 1; };
template <> struct TileGeom<TQ_Q5_K> { static constexpr int BYTES = 2816, ELEMS = 256, GROUP = 1; };
template <> struct TileGeom<TQ_Q6_K> { static constexpr int BYTES = 3360, ELEMS = 256, GROUP = 1; };

// Quantized activation planes (global scratch or shared memory) of R rows, in the order in which the MMA loop reads them: a
// lane finds what it needs in as few and as wide words as there are, neighbouring rows lie next to each other (no bank
// conflicts, whole sectors from global memory), and a run of k-tiles is one contiguous range. With row-major planes more than
// half of the shared-memory wavefronts of a 16-row tile were conflicts (the block sums of four rows in the same banks) and a
// Q6_K tile read its quants in sixteen words a row. Row-major against this order, us a call, 8 / 16 rows:
//   2 x 12288 x 4096 Q4_K 19.8 -> 17.5, 33.4 -> 23.6   4096 x 12288 Q6_K 15.8 -> 13.7, 30.6 -> 18.9
//   2 x 8192 x 2560 Q5_K 11.7 -> 11.3, 16.6 -> 15.4    5120 x 25600 Q6_K (planes in global memory) 35.8 -> 27.0, 61.9 -> 38.9
//   2 x 8192 x 2560 Q8_0 13.7 -> 12.2, 17.1 -> 16.3
//   qs    K-quants: [k/64][R][64 bytes], the 64 bytes in one of two orders (ActOrder)
//         Q8_0:     [k/32][R][32 bytes], element order
//   dsc   f32   [k/bs][R]          bs = 256 (Q8_K) or 32 (Q8_0; the f16-rounded scale)
//   bs16  int16 [k/256][2][R][8]   Q8_K: sums of 16 consecutive qs
//   bs32  int16 [k/256][R][8]      Q8_K: sums of 32 consecutive qs
struct ActPack {
  const int8_t* qs;
  const float* dsc;
  const int16_t* bs16;
  const int16_t* bs32;
  int R;
};

// Byte offset of element e (0..63) of row r inside the row's 64 bytes of a chunk.
//   order32 (Q4_K, Q5_K, mixed launches): lane column c's eight bytes of both 32-element sub-blocks, 16 bytes together. The
//     columns of rows 2, 3, 6, 7 change places pairwise, so that Q6_K tiles of a mixed launch, which read four-byte words,
//     meet in a bank twice and not four times.
//   order16 (Q6_K): lane column c's four bytes of all four 16-element sub-blocks, 16 bytes together.
enum class ActOrder { order32, order16 };
__host__ __device__ __forceinline__ int act_offset(ActOrder o, int r, int e) {
  if (o == ActOrder::order32) return 16 * (((e & 31) >> 3) ^ (r & 2)) + 8 * (e >> 5) + (e & 7);
  return 16 * ((e & 15) >> 2) + 4 * (e >> 4) + (e & 3);
}

// What a lane needs to find its rows in the planes; the same for every tile. Rows beyond the valid ones are clamped to the last
// one: their columns of the MMA are not stored. GUARD: their quants are not read at all. That pays where reads are what a
// tile waits for and costs a test per read: Q8_0 with four groups of rows (us a call without / with, 17 / 24 / 32 rows: 128 x 25600 60.9 / 49.5,
// 67.9 / 54.1, 70.5 / 52.7; 2560 x 2560 12.0 / 10.5, 13.5 / 11.5, 14.0 / 12.4; 5120 x 25600 68.7 / 64.9, 70.0 / 66.6, 73.6 / 68.2) and
// Q4_K with two (9 rows: 512 x 8192 10.8 / 9.9, 1536 x 8960 11.7 / 10.8; all shapes 2 %). Elsewhere with up to two groups it loses
// 1 to 6 %, and K-quants with four are even.
template <int MG, bool GUARD>
struct LaneAct {
  int q[MG];        // offset of row 8 mg + g inside a chunk of qs; GUARD: -1 beyond the valid rows
  int r0[MG], r1[MG];  // rows 8 mg + 2 c, 8 mg + 2 c + 1
  __device__ __forceinline__ void init(int lane, int rows, int row_bytes) {
    const int g = lane >> 2, c = lane & 3;
#pragma unroll
    for (int mg = 0; mg < MG; mg++) {
      const int b = 8 * mg + g, m0 = 8 * mg + 2 * c;
      q[mg] = b < rows ? b * row_bytes : GUARD ? -1 : (rows - 1) * row_bytes;
      r0[mg] = m0 < rows ? m0 : rows - 1;
      r1[mg] = m0 + 1 < rows ? m0 + 1 : rows - 1;
    }
  }
};

__device__ __forceinline__ int sext_byte(uint32_t w, int b) { return (int)(int8_t)((w >> (8 * b)) & 0xFFu); }
__device__ __forceinline__ uint4 lds_v4(const uint8_t* p) { return *reinterpret_cast<const uint4*>(p); }
__device__ __forceinline__ uint32_t lds_u16(const uint8_t* p) { return *reinterpret_cast<const uint16_t*>(p); }

// One tile (or GROUP consecutive Q8_0 tiles) at shared-memory address t, tile index kt of its
// row, against the activation rows of the pass; adds into acc[mg][0..3]. ORDER: the order of the planes' qs.
template <int DT, int MG, ActOrder ORDER, bool GUARD>
__device__ __forceinline__ void tile_mma(const uint8_t* __restrict__ t, int lane, const ActPack& act, const LaneAct<MG, GUARD>& la, int kt,
                                         int ntiles_left, float (&acc)[MG][4]) {
  static_assert(DT == TQ_Q8_0 || DT == TQ_Q6_K || ORDER == ActOrder::order32, "Q4_K and Q5_K tiles read order32");
  static_assert(DT != TQ_Q6_K || !GUARD, "Q6_K tiles read clamped rows");
  const int g = lane >> 2, c = lane & 3;
  if constexpr (DT == TQ_Q8_0) {
    auto one = [&](int u) {
      const uint8_t* tu = t + 544 * u;
      const uint4 q = lds_v4(tu + TQ_Q8_0_QS + 16 * lane);
      const uint32_t a[4] = {q.x, q.z, q.y, q.w};
      const float dw0 = f16_bits_to_f32(lds_u16(tu + 2 * g)), dw1 = f16_bits_to_f32(lds_u16(tu + 2 * (g + 8)));
      const int kb = kt + u;
#pragma unroll
      for (int mg = 0; mg < MG; mg++) {
        uint2 b = make_uint2(0, 0);
        if (!GUARD || la.q[mg] >= 0) b = ld_v2(act.qs + (int64_t)kb * act.R * 32 + la.q[mg] + 8 * c);
        int cc[4] = {0, 0, 0, 0};
        mma_16832<false>(cc, a, b.x, b.y);
        const float* const dsc = act.dsc + (int64_t)kb * act.R;
        const float dx0 = dsc[la.r0[mg]], dx1 = dsc[la.r1[mg]];
        acc[mg][0] += (float)cc[0] * (dw0 * dx0);
        acc[mg][1] += (float)cc[1] * (dw0 * dx1);
        acc[mg][2] += (float)cc[2] * (dw1 * dx0);
        acc[mg][3] += (float)cc[3] * (dw1 * dx1);
      }
    };
    // A whole group without a question between its tiles, so that the loads of all four are under way together: asked tile by
    // tile, every tile waits for its own quants and scales. us a call so / asked, 8 and 16 rows: 128 x 25600 19.2 / 39.1 and
    // 24.5 / 42.5 (planes in global memory), 4096 x 12288 12.7 / 13.1 and 18.7 / 25.5, 2560 x 8192 12.2 / 12.6 and 13.8 / 15.5.
    // Four groups of rows have loads enough, and no registers for more (5120 x 25600, 32 rows 80.4 / 73.4).
    if (MG <= 2 && ntiles_left >= 4) {
#pragma unroll
      for (int u = 0; u < 4; u++) one(u);
    } else {
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (u < ntiles_left) one(u);
    }
  } else if constexpr (DT == TQ_Q4_K || DT == TQ_Q5_K) {
    constexpr int QS = DT == TQ_Q4_K ? TQ_Q4K_QS : TQ_Q5K_QS;
    // Integer accumulators per C-fragment element: even sub-blocks (low nibbles), odd
    // sub-blocks (Q4_K: high nibbles kept in place, i.e. 16 x the dot product) and mins.
    int aE[MG][4], aO[MG][4], aM[MG][4];
    const uint4 h0 = lds_v4(t + 16 * g), h1 = lds_v4(t + 16 * (g + 8));
    // 6-bit scales / mins of both rows, four per word, decoded with byte-parallel ops
    uint32_t scl[2], sch[2];
    {
      const uint4 hh[2] = {h0, h1};
#pragma unroll
      for (int hr = 0; hr < 2; hr++) {
        const uint32_t s0 = hh[hr].y, s1 = hh[hr].z, s2 = hh[hr].w;
        scl[hr] = s0 & 0x3F3F3F3Fu;
        sch[hr] = (s2 & 0x0F0F0F0Fu) | ((s0 >> 2) & 0x30303030u);
        const int mnl = (int)(s1 & 0x3F3F3F3Fu);
        const int mnh = (int)(((s2 >> 4) & 0x0F0F0F0Fu) | ((s1 >> 2) & 0x30303030u));
#pragma unroll
        for (int mg = 0; mg < MG; mg++) {
          const int16_t* const bs = act.bs32 + (int64_t)kt * act.R * 8;
          const uint4 bs0 = ld_v4(bs + la.r0[mg] * 8), bs1 = ld_v4(bs + la.r1[mg] * 8);
          // mins: sum_j mn_j * bsum_j, two 16-bit x 8-bit products per instruction
          aM[mg][2 * hr] = __dp2a_hi((int)bs0.w, mnh, __dp2a_lo((int)bs0.z, mnh, __dp2a_hi((int)bs0.y, mnl, __dp2a_lo((int)bs0.x, mnl, 0))));
          aM[mg][2 * hr + 1] = __dp2a_hi((int)bs1.w, mnh, __dp2a_lo((int)bs1.z, mnh, __dp2a_hi((int)bs1.y, mnl, __dp2a_lo((int)bs1.x, mnl, 0))));
        }
      }
    }
#pragma unroll
    for (int mg = 0; mg < MG; mg++)
#pragma unroll
      for (int e = 0; e < 4; e++) aE[mg][e] = aO[mg][e] = 0;
    uint4 qh = make_uint4(0, 0, 0, 0);
    if constexpr (DT == TQ_Q5_K) qh = lds_v4(t + TQ_Q5K_QH + 16 * lane);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint4 q = lds_v4(t + QS + 512 * i + 16 * lane);
      uint32_t alo[4] = {q.x & 0x0F0F0F0Fu, q.z & 0x0F0F0F0Fu, q.y & 0x0F0F0F0Fu, q.w & 0x0F0F0F0Fu};
      uint32_t ahi[4] = {q.x & 0xF0F0F0F0u, q.z & 0xF0F0F0F0u, q.y & 0xF0F0F0F0u, q.w & 0xF0F0F0F0u};
      if constexpr (DT == TQ_Q5_K) {
        // the fifth bit would be worth 256 in place, so the odd sub-block is shifted down
        const uint32_t hw[4] = {qh.x, qh.z, qh.y, qh.w};
#pragma unroll
        for (int e = 0; e < 4; e++) {
          alo[e] |= ((hw[e] >> (2 * i)) << 4) & 0x10101010u;
          ahi[e] = (ahi[e] >> 4) | (((hw[e] >> (2 * i + 1)) << 4) & 0x10101010u);
        }
      }
      // sub-blocks 2i and 2i+1 are bytes (2i & 3), (2i+1 & 3) of the low or high scale word
      int se[2], so[2];
#pragma unroll
      for (int hr = 0; hr < 2; hr++) {
        const uint32_t sw = i < 2 ? scl[hr] : sch[hr];
        se[hr] = (int)__byte_perm(sw, 0, 0x4440 + ((2 * i) & 3));
        so[hr] = (int)__byte_perm(sw, 0, 0x4440 + ((2 * i + 1) & 3));
      }
#pragma unroll
      for (int mg = 0; mg < MG; mg++) {
        uint4 bx = make_uint4(0, 0, 0, 0);
        if (!GUARD || la.q[mg] >= 0) bx = ld_v4(act.qs + (int64_t)(4 * kt + i) * act.R * 64 + la.q[mg] + 16 * (c ^ ((la.q[mg] >> 6) & 2)));
        int clo[4] = {0, 0, 0, 0}, chi[4] = {0, 0, 0, 0};
        mma_16832<true>(clo, alo, bx.x, bx.y);
        mma_16832<true>(chi, ahi, bx.z, bx.w);
#pragma unroll
        for (int hr = 0; hr < 2; hr++) {
          aE[mg][2 * hr] += se[hr] * clo[2 * hr];
          aE[mg][2 * hr + 1] += se[hr] * clo[2 * hr + 1];
          aO[mg][2 * hr] += so[hr] * chi[2 * hr];
          aO[mg][2 * hr + 1] += so[hr] * chi[2 * hr + 1];
        }
      }
    }
    const float d[2] = {f16_bits_to_f32(h0.x), f16_bits_to_f32(h1.x)};
    const float dmin[2] = {f16_bits_to_f32(h0.x >> 16), f16_bits_to_f32(h1.x >> 16)};
#pragma unroll
    for (int mg = 0; mg < MG; mg++) {
      const float* const dsc = act.dsc + (int64_t)kt * act.R;
      const float dx0 = dsc[la.r0[mg]], dx1 = dsc[la.r1[mg]];
#pragma unroll
      for (int hr = 0; hr < 2; hr++) {
        constexpr int SH = DT == TQ_Q4_K ? 4 : 0;
        const int i0 = aE[mg][2 * hr] + (aO[mg][2 * hr] >> SH), i1 = aE[mg][2 * hr + 1] + (aO[mg][2 * hr + 1] >> SH);
        acc[mg][2 * hr] += (dx0 * d[hr]) * (float)i0 - (dx0 * dmin[hr]) * (float)aM[mg][2 * hr];
        acc[mg][2 * hr + 1] += (dx1 * d[hr]) * (float)i1 - (dx1 * dmin[hr]) * (float)aM[mg][2 * hr + 1];
      }
    }
  } else {  // Q6_K: sum_j sc_j * (dot_j(q) - 32 * bsum_j), q unsigned 0..63
    int aI[MG][4];
    const uint4 s0v = lds_v4(t + 16 * g), s1v = lds_v4(t + 16 * (g + 8));
    const uint32_t scw[2][4] = {{s0v.x, s0v.y, s0v.z, s0v.w}, {s1v.x, s1v.y, s1v.z, s1v.w}};
#pragma unroll
    for (int mg = 0; mg < MG; mg++) {
      // the -32 offset: sum_j sc_j * bsum16_j, two products per instruction
      const int16_t* const bs = act.bs16 + (int64_t)kt * act.R * 16;
      const int16_t* const bh = bs + act.R * 8;
      const uint4 p0 = ld_v4(bs + la.r0[mg] * 8), p1 = ld_v4(bh + la.r0[mg] * 8);
      const uint4 q0 = ld_v4(bs + la.r1[mg] * 8), q1 = ld_v4(bh + la.r1[mg] * 8);
      const uint32_t bw0[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
      const uint32_t bw1[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
      for (int hr = 0; hr < 2; hr++) {
        int o0 = 0, o1 = 0;
#pragma unroll
        for (int w = 0; w < 4; w++) {
          o0 = __dp2a_hi((int)bw0[2 * w + 1], (int)scw[hr][w], __dp2a_lo((int)bw0[2 * w], (int)scw[hr][w], o0));
          o1 = __dp2a_hi((int)bw1[2 * w + 1], (int)scw[hr][w], __dp2a_lo((int)bw1[2 * w], (int)scw[hr][w], o1));
        }
        aI[mg][2 * hr] = -32 * o0;
        aI[mg][2 * hr + 1] = -32 * o1;
      }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint4 ql = lds_v4(t + TQ_Q6K_QL + 512 * i + 16 * lane);
      const uint4 qh = lds_v4(t + TQ_Q6K_QH + 512 * (i >> 1) + 16 * lane);
      uint4 bx[MG];  // order16: this lane's words of the chunk's four sub-blocks
      if constexpr (ORDER == ActOrder::order16) {
#pragma unroll
        for (int mg = 0; mg < MG; mg++) bx[mg] = ld_v4(act.qs + (int64_t)(4 * kt + i) * act.R * 64 + la.q[mg] + 16 * c);
      }
      // qh word of this chunk's four sub-blocks: chunk i of ql pairs with qh word (i & 1) of each row
      const uint32_t qh0 = (i & 1) ? qh.y : qh.x, qh1 = (i & 1) ? qh.w : qh.z;
#pragma unroll
      for (int jj = 0; jj < 4; jj++) {
        const int tw = jj >> 1, nib = jj & 1;
        const uint32_t w0 = tw ? ql.y : ql.x, w1 = tw ? ql.w : ql.z;
        uint32_t a0 = (nib ? (w0 >> 4) : w0) & 0x0F0F0F0Fu, a1 = (nib ? (w1 >> 4) : w1) & 0x0F0F0F0Fu;
        // 2-bit field jj of the qh word moved to bits 4..5 of every byte
        const int sh = 2 * jj;
        a0 |= (sh <= 4 ? (qh0 << (4 - sh)) : (qh0 >> (sh - 4))) & 0x30303030u;
        a1 |= (sh <= 4 ? (qh1 << (4 - sh)) : (qh1 >> (sh - 4))) & 0x30303030u;
        const int sc0 = sext_byte(scw[0][i], jj), sc1 = sext_byte(scw[1][i], jj);
#pragma unroll
        for (int mg = 0; mg < MG; mg++) {
          uint32_t b;
          if constexpr (ORDER == ActOrder::order16) {
            b = jj == 0 ? bx[mg].x : jj == 1 ? bx[mg].y : jj == 2 ? bx[mg].z : bx[mg].w;
          } else {  // elements 16 jj + 4 c ...: column 2 (jj & 1) + c / 2 of sub-block jj / 2, word c & 1
            b = ld_u32(act.qs + (int64_t)(4 * kt + i) * act.R * 64 + la.q[mg] +
                       16 * ((2 * (jj & 1) + (c >> 1)) ^ ((la.q[mg] >> 6) & 2)) + 8 * (jj >> 1) + 4 * (c & 1));
          }
          int cc[4] = {0, 0, 0, 0};
          mma_16816_u8s8(cc, a0, a1, b);
          aI[mg][0] += sc0 * cc[0];
          aI[mg][1] += sc0 * cc[1];
          aI[mg][2] += sc1 * cc[2];
          aI[mg][3] += sc1 * cc[3];
        }
      }
    }
    const float d0 = f16_bits_to_f32(lds_u16(t + TQ_Q6K_D + 2 * g)), d1 = f16_bits_to_f32(lds_u16(t + TQ_Q6K_D + 2 * (g + 8)));
#pragma unroll
    for (int mg = 0; mg < MG; mg++) {
      const float* const dsc = act.dsc + (int64_t)kt * act.R;
      const float dx0 = dsc[la.r0[mg]], dx1 = dsc[la.r1[mg]];
      acc[mg][0] += (dx0 * d0) * (float)aI[mg][0];
      acc[mg][1] += (dx1 * d0) * (float)aI[mg][1];
      acc[mg][2] += (dx0 * d1) * (float)aI[mg][2];
      acc[mg][3] += (dx1 * d1) * (float)aI[mg][3];
    }
  }
}

// The same tile against ONE activation row (decode, M = 1), K-quant types. With a single row the
// 8-wide activation operand of the MMA would carry seven rows of zeros and every lane would
// still apply the sub-block scales to all four of its C elements. Here the eight B columns carry
// the eight 32-element sub-blocks instead (16-element ones for Q6_K, in two accumulator sets):
// the MMA of sub-block s gets the activation bytes in column s only, so after the tile's MMAs
// C[row][j] is the integer dot of `row` with sub-block j. A lane then scales just its own two
// (four) sub-blocks, the four lanes of a row add their integers with two shuffles, and the
// float step is the one of the general function - same integers, same float operations, so
// the result has the bits of tile_mma<DT, 1> with rows = 1. Each lane loads one 8-byte (two
// 4-byte) activation fragment per tile instead of eight (sixteen).
template <int DT, ActOrder ORDER>
__device__ __forceinline__ void tile_mma_row1(const uint8_t* __restrict__ t, int lane, const ActPack& act, int kt, float (&acc)[1][4]) {
  static_assert(DT == TQ_Q6_K || ORDER == ActOrder::order32, "Q4_K and Q5_K tiles read order32");
  static_assert(DT == TQ_Q4_K || DT == TQ_Q5_K || DT == TQ_Q6_K, "single-row variant exists for the K-quants");
  const int g = lane >> 2, c = lane & 3;
  const float dx0 = act.dsc[(int64_t)kt * act.R];
  if constexpr (DT == TQ_Q4_K || DT == TQ_Q5_K) {
    constexpr int QS = DT == TQ_Q4_K ? TQ_Q4K_QS : TQ_Q5K_QS;
    constexpr int SH = DT == TQ_Q4_K ? 4 : 0;
    const uint4 h0 = lds_v4(t + 16 * g), h1 = lds_v4(t + 16 * (g + 8));
    const uint4 hh[2] = {h0, h1};
    const uint4 bs0 = ld_v4(act.bs32 + (int64_t)kt * act.R * 8);
    uint32_t scl[2], sch[2];
    int aM[2];
#pragma unroll
    for (int hr = 0; hr < 2; hr++) {
      const uint32_t s0 = hh[hr].y, s1 = hh[hr].z, s2 = hh[hr].w;
      scl[hr] = s0 & 0x3F3F3F3Fu;
      sch[hr] = (s2 & 0x0F0F0F0Fu) | ((s0 >> 2) & 0x30303030u);
      const int mnl = (int)(s1 & 0x3F3F3F3Fu);
      const int mnh = (int)(((s2 >> 4) & 0x0F0F0F0Fu) | ((s1 >> 2) & 0x30303030u));
      aM[hr] = __dp2a_hi((int)bs0.w, mnh, __dp2a_lo((int)bs0.z, mnh, __dp2a_hi((int)bs0.y, mnl, __dp2a_lo((int)bs0.x, mnl, 0))));
    }
    // this lane's activation fragment: elements 8c .. 8c+7 of sub-block g
    const uint2 frag = ld_v2(act.qs + (int64_t)(4 * kt + (g >> 1)) * act.R * 64 + 16 * c + 8 * (g & 1));
    int cc[4] = {0, 0, 0, 0};
    uint4 qh = make_uint4(0, 0, 0, 0);
    if constexpr (DT == TQ_Q5_K) qh = lds_v4(t + TQ_Q5K_QH + 16 * lane);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint4 q = lds_v4(t + QS + 512 * i + 16 * lane);
      uint32_t alo[4] = {q.x & 0x0F0F0F0Fu, q.z & 0x0F0F0F0Fu, q.y & 0x0F0F0F0Fu, q.w & 0x0F0F0F0Fu};
      uint32_t ahi[4] = {q.x & 0xF0F0F0F0u, q.z & 0xF0F0F0F0u, q.y & 0xF0F0F0F0u, q.w & 0xF0F0F0F0u};
      if constexpr (DT == TQ_Q5_K) {
        const uint32_t hw[4] = {qh.x, qh.z, qh.y, qh.w};
#pragma unroll
        for (int e = 0; e < 4; e++) {
          alo[e] |= ((hw[e] >> (2 * i)) << 4) & 0x10101010u;
          ahi[e] = (ahi[e] >> 4) | (((hw[e] >> (2 * i + 1)) << 4) & 0x10101010u);
        }
      }
      const bool lo_mine = g == 2 * i, hi_mine = g == 2 * i + 1;
      mma_16832<true>(cc, alo, lo_mine ? frag.x : 0u, lo_mine ? frag.y : 0u);
      mma_16832<true>(cc, ahi, hi_mine ? frag.x : 0u, hi_mine ? frag.y : 0u);
    }
    // cc[0] = (row g, sub-block 2c), cc[1] = (row g, 2c+1), cc[2] = (row g+8, 2c), cc[3] = (row g+8, 2c+1)
    const int sh_even = 8 * ((2 * c) & 3), sh_odd = sh_even + 8;
    int p[2];
#pragma unroll
    for (int hr = 0; hr < 2; hr++) {
      const uint32_t sw = c < 2 ? scl[hr] : sch[hr];
      const int s_even = (int)((sw >> sh_even) & 0xFFu), s_odd = (int)((sw >> sh_odd) & 0xFFu);
      p[hr] = s_even * cc[2 * hr] + ((s_odd * cc[2 * hr + 1]) >> SH);
      p[hr] += __shfl_xor_sync(0xFFFFFFFFu, p[hr], 1);
      p[hr] += __shfl_xor_sync(0xFFFFFFFFu, p[hr], 2);
    }
    const float d[2] = {f16_bits_to_f32(h0.x), f16_bits_to_f32(h1.x)};
    const float dmin[2] = {f16_bits_to_f32(h0.x >> 16), f16_bits_to_f32(h1.x >> 16)};
    acc[0][0] += (dx0 * d[0]) * (float)p[0] - (dx0 * dmin[0]) * (float)aM[0];
    acc[0][2] += (dx0 * d[1]) * (float)p[1] - (dx0 * dmin[1]) * (float)aM[1];
  } else {  // Q6_K: 16 sub-blocks of 16 elements -> two accumulator sets of 8 columns
    const uint4 s0v = lds_v4(t + 16 * g), s1v = lds_v4(t + 16 * (g + 8));
    const uint32_t scw[2][4] = {{s0v.x, s0v.y, s0v.z, s0v.w}, {s1v.x, s1v.y, s1v.z, s1v.w}};
    const int16_t* b0p = act.bs16 + (int64_t)kt * act.R * 16;
    const uint4 p0 = ld_v4(b0p), p1 = ld_v4(b0p + act.R * 8);
    const uint32_t bw0[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
    int off32[2];
#pragma unroll
    for (int hr = 0; hr < 2; hr++) {
      int o0 = 0;
#pragma unroll
      for (int w = 0; w < 4; w++) o0 = __dp2a_hi((int)bw0[2 * w + 1], (int)scw[hr][w], __dp2a_lo((int)bw0[2 * w], (int)scw[hr][w], o0));
      off32[hr] = -32 * o0;
    }
    // this lane's activation fragments: elements 4c .. 4c+3 of sub-blocks g and g + 8
    const int8_t* const qp = act.qs + (int64_t)(4 * kt + (g >> 2)) * act.R * 64 +
                             (ORDER == ActOrder::order16 ? 16 * c + 4 * (g & 3) : 16 * (2 * (g & 1) + (c >> 1)) + 8 * ((g >> 1) & 1) + 4 * (c & 1));
    const uint32_t fa = ld_u32(qp), fb = ld_u32(qp + act.R * 128);
    int ca[4] = {0, 0, 0, 0}, cb[4] = {0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint4 ql = lds_v4(t + TQ_Q6K_QL + 512 * i + 16 * lane);
      const uint4 qh = lds_v4(t + TQ_Q6K_QH + 512 * (i >> 1) + 16 * lane);
      const uint32_t qh0 = (i & 1) ? qh.y : qh.x, qh1 = (i & 1) ? qh.w : qh.z;
#pragma unroll
      for (int jj = 0; jj < 4; jj++) {
        const int j = 4 * i + jj;
        const int tw = jj >> 1, nib = jj & 1;
        const uint32_t w0 = tw ? ql.y : ql.x, w1 = tw ? ql.w : ql.z;
        uint32_t a0 = (nib ? (w0 >> 4) : w0) & 0x0F0F0F0Fu, a1 = (nib ? (w1 >> 4) : w1) & 0x0F0F0F0Fu;
        const int sh = 2 * jj;
        a0 |= (sh <= 4 ? (qh0 << (4 - sh)) : (qh0 >> (sh - 4))) & 0x30303030u;
        a1 |= (sh <= 4 ? (qh1 << (4 - sh)) : (qh1 >> (sh - 4))) & 0x30303030u;
        if (j < 8) {
          mma_16816_u8s8(ca, a0, a1, g == j ? fa : 0u);
        } else {
          mma_16816_u8s8(cb, a0, a1, g == j - 8 ? fb : 0u);
        }
      }
    }
    // ca: sub-blocks 2c, 2c+1 (rows g | g+8); cb: sub-blocks 8+2c, 9+2c
    const int b_even = (2 * c) & 3, b_odd = b_even + 1;
    int p[2];
#pragma unroll
    for (int hr = 0; hr < 2; hr++) {
      const uint32_t wa = (c >> 1) ? scw[hr][1] : scw[hr][0];
      const uint32_t wb = (c >> 1) ? scw[hr][3] : scw[hr][2];
      p[hr] = sext_byte(wa, b_even) * ca[2 * hr] + sext_byte(wa, b_odd) * ca[2 * hr + 1] + sext_byte(wb, b_even) * cb[2 * hr] +
              sext_byte(wb, b_odd) * cb[2 * hr + 1];
      p[hr] += __shfl_xor_sync(0xFFFFFFFFu, p[hr], 1);
      p[hr] += __shfl_xor_sync(0xFFFFFFFFu, p[hr], 2);
      p[hr] += off32[hr];
    }
    const float d0 = f16_bits_to_f32(lds_u16(t + TQ_Q6K_D + 2 * g)), d1 = f16_bits_to_f32(lds_u16(t + TQ_Q6K_D + 2 * (g + 8)));
    acc[0][0] += (dx0 * d0) * (float)p[0];
    acc[0][2] += (dx0 * d1) * (float)p[1];
  }
}

}  // namespace turq
