// QMatMul::forward on the 5th-generation tensor cores (tcgen05 / TMEM) for prefill: more than 64
// activation rows (up to 64: gemm_batch.cu).
//
//   y[m, n] = sum_k x[m, k] * W[n, k]      W quantized (device fragment tiles), x f32 or bf16
//
// Step 1 (prep kernel): x -> f16 [M, K], each row scaled by a power of two that puts its largest
// magnitude just below the top of the f16 range (the scale is undone exactly in the epilogue).
// Step 2 (this kernel): pairs of CTAs (a cluster of two, cta_group::2) produce output tiles of 256
// weight rows x `bn` <= 256 activation rows. Each CTA holds its 128 weight rows as the A operand and
// half of the activation rows as its part of the B operand, so an activation byte crosses from L2
// into shared memory once per 256 weight rows.
//   * warp 0        streams the raw quantized tiles of the CTA's 128 weight rows (units of 256 k,
//                   contiguous bytes per row-tile) into a ring with cp.async.bulk: how far the
//                   weights run ahead is set by shared memory, not by registers;
//   * warp 1        TMA of the activation tile (bn/2 rows x 64 k, f16, 128B swizzle, no multicast),
//                   completing on the leader CTA's barrier;
//   * warp 2        (leader CTA) one thread issues tcgen05.mma M=256, N=bn, K=16, f16 x f16 -> f32,
//                   four per stage, and commits the stage back to the producers of both CTAs;
//   * warps 3..6    epilogue: tcgen05.ld the accumulator, undo the row scale, add bias, store. The
//                   accumulator is double buffered (2 x 256 TMEM columns), so the next tile's MMAs
//                   run meanwhile;
//   * warps 7..22   dequantize (two groups of eight, each two 64-k blocks of a unit) from the raw ring
//                   to f16 with packed half arithmetic into shared memory, K-major 128B-swizzled, and
//                   arrive on the leader's barrier.
// MMA roles: A = weights (rows = TMEM lanes), B = activations (columns).
// Work: whole tiles, dealt out to persistent pairs.
//
// What bounds it: the tensor pipe (90 % of active cycles at 12288 x 4096 Q4_K, 2048 rows), the
// power limit and the last wave of tiles.
// Measured with graph replay, conversion included, against one CTA per 128 rows with weights prefetched
// into registers and one ring for both operands: Q4_K 12288 x 4096, 2048 rows  231 -> 161 us (1280 TFLOP/s).
// Steps on the way: an MMA loop walked by the whole warp, one lane issuing, instead of by one divergent
// thread (2048 rows: 210 -> 173 us); remote arrivals without a cluster-scope release (270 -> 210 us; the
// proxy fence already orders the operand tile).
// Every wait is bounded; on expiry the CTA records TURQ_E_TIMEOUT, releases its TMEM and returns.
#include <cstdlib>
#include <cuda.h>
#include <cuda_fp16.h>

#include <cstdio>

#include "actquant.cuh"
#include "launch_plan.h"
#include "tc_common.cuh"
#include "turq_internal.h"

namespace turq {

namespace {

constexpr int MAX_ST = 8;    // operand stages
constexpr int MAX_RAW = 8;   // raw ring slots
constexpr int A_BYTES = BM * BK * 2;  // 16 KB per block
constexpr int DQ_WARP0 = 7;        // first dequantize warp; warps 3..6 are the epilogue, one per TMEM lane quarter (warp & 3)
constexpr int DQ_WARPS = 8;        // warps that together produce one stage of the weight operand
constexpr int DQ_GROUPS = 2;       // groups of DQ_WARPS warps working on alternate stages
constexpr int HELPERS = 1 + DQ_WARPS * DQ_GROUPS / 4;  // warps per TMEM lane quarter that share a pair's last epilogue
constexpr int TC_THREADS = (DQ_WARP0 + DQ_WARPS * DQ_GROUPS) * 32;
// Register bound (72) of the kernel: leaves a CTA of the conversion kernel room beside it on an SM.
constexpr int TC_REG_THREADS = 896;
constexpr int TMEM_COLS = 512;     // two accumulators of 256 columns

// The barriers of a pair's leader collect arrivals of both CTAs.
__device__ __forceinline__ void bar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void commit_to_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(s_u32(bar)),
               "h"((unsigned short)3)
               : "memory");
}

// Dequantizes 64-k block i of a unit (not Q6_K; t: the row-tile's raw bytes in shared memory), block e of the
// warp's two, to f16 and stores it in the swizzled operand tile; `a_rows` points at the row-tile's 16
// rows there. Odd rows store their two 64-byte halves in the other order than even ones: with the
// same order rows g and g + 1 of a quarter-warp meet in the same banks and every store takes two passes.
template <int DT>
__device__ __forceinline__ void dequant_block(const uint8_t* t, const UnitScales& us, int i, int e, int lane, uint8_t* a_rows) {
  const int g = lane >> 2, c = lane & 3, odd = g & 1;
  uint8_t* const row = a_rows + g * 128;
  const uint32_t o0 = (uint32_t)((((4 * odd) ^ (c >> 1) ^ g) << 4) + 8 * (c & 1));
  auto store = [&](int hr, int h, const uint4& o) {  // the eight elements of sub-block h ^ odd
    *reinterpret_cast<uint2*>(row + hr * 1024 + (o0 ^ (h << 6))) = make_uint2(o.x, o.y);
    *reinterpret_cast<uint2*>(row + hr * 1024 + (o0 ^ (h << 6) ^ 32u)) = make_uint2(o.z, o.w);
  };
  if constexpr (DT == TQ_Q8_0) {
    const __half2 off = __float2half2_rn(1152.f);  // 1024 + 128: bytes are biased by xor 0x80
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint8_t* tt = t + (2 * i + (h ^ odd)) * 544;
      const uint4 q = lds_v4(tt + TQ_Q8_0_QS + 16 * lane);
      const uint32_t dd = lds_u16(tt + 2 * g) | (lds_u16(tt + 2 * (g + 8)) << 16);
      const uint32_t w[2][2] = {{q.x ^ 0x80808080u, q.y ^ 0x80808080u}, {q.z ^ 0x80808080u, q.w ^ 0x80808080u}};
#pragma unroll
      for (int hr = 0; hr < 2; hr++) {
        const __half2 d2 = u2h2(__byte_perm(dd, 0u, hr ? 0x3232 : 0x1010));
        uint4 o;
        o.x = h22u(__hmul2(__hsub2(pair02(w[hr][0]), off), d2));
        o.y = h22u(__hmul2(__hsub2(pair13(w[hr][0]), off), d2));
        o.z = h22u(__hmul2(__hsub2(pair02(w[hr][1]), off), d2));
        o.w = h22u(__hmul2(__hsub2(pair13(w[hr][1]), off), d2));
        store(hr, h, o);
      }
    }
  } else if constexpr (DT == TQ_Q4_K || DT == TQ_Q5_K) {
    constexpr int QS = DT == TQ_Q4_K ? TQ_Q4K_QS : TQ_Q5K_QS;
    const uint4 q = lds_v4(t + QS + 512 * i + 16 * lane);
    const uint32_t w[2][2] = {{q.x, q.y}, {q.z, q.w}};
    uint32_t dl2[2], ml2[2];
#pragma unroll
    for (int hr = 0; hr < 2; hr++) {
      const int src = 2 * (g + 8 * hr) + e;
      dl2[hr] = __shfl_sync(0xFFFFFFFFu, us.dl, src);
      ml2[hr] = __shfl_sync(0xFFFFFFFFu, us.ml, src);
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int nib = h ^ odd;  // 0: sub-block 2i (low nibbles), 1: sub-block 2i + 1
      const uint32_t sel = nib ? 0x3232u : 0x1010u;
      if constexpr (DT == TQ_Q4_K) {
        // A nibble becomes a half without being moved: under the exponent of 1024 the low nibble counts
        // ones, under that of 64 the high nibble (16 units of 1/16) does; the offset subtracts exactly.
        const uint32_t mask = nib ? 0x00F000F0u : 0x000F000Fu, magic = nib ? 0x54005400u : 0x64006400u;
        const __half2 off = u2h2(magic);
#pragma unroll
        for (int hr = 0; hr < 2; hr++) {
          const __half2 dl = u2h2(__byte_perm(dl2[hr], 0u, sel)), ml = u2h2(__byte_perm(ml2[hr], 0u, sel));
          uint4 o;
          o.x = h22u(__hfma2(__hsub2(u2h2((w[hr][0] & mask) | magic), off), dl, ml));
          o.y = h22u(__hfma2(__hsub2(u2h2(((w[hr][0] >> 8) & mask) | magic), off), dl, ml));
          o.z = h22u(__hfma2(__hsub2(u2h2((w[hr][1] & mask) | magic), off), dl, ml));
          o.w = h22u(__hfma2(__hsub2(u2h2(((w[hr][1] >> 8) & mask) | magic), off), dl, ml));
          store(hr, h, o);
        }
      } else {
        const __half2 off = __float2half2_rn(1024.f);
        const uint4 h4 = lds_v4(t + TQ_Q5K_QH + 16 * lane);
        const uint32_t qh[2][2] = {{h4.x, h4.y}, {h4.z, h4.w}};
        const int rot = 4 - (2 * i + nib);  // brings the sub-block's bit to bit 4 of every byte
#pragma unroll
        for (int hr = 0; hr < 2; hr++) {
          const __half2 dl = u2h2(__byte_perm(dl2[hr], 0u, sel)), ml = u2h2(__byte_perm(ml2[hr], 0u, sel));
          const uint32_t m0 = ((w[hr][0] >> (4 * nib)) & 0x0F0F0F0Fu) | (__funnelshift_l(qh[hr][0], qh[hr][0], rot) & 0x10101010u);
          const uint32_t m1 = ((w[hr][1] >> (4 * nib)) & 0x0F0F0F0Fu) | (__funnelshift_l(qh[hr][1], qh[hr][1], rot) & 0x10101010u);
          uint4 o;
          o.x = h22u(__hfma2(__hsub2(pair02(m0), off), dl, ml));
          o.y = h22u(__hfma2(__hsub2(pair13(m0), off), dl, ml));
          o.z = h22u(__hfma2(__hsub2(pair02(m1), off), dl, ml));
          o.w = h22u(__hfma2(__hsub2(pair13(m1), off), dl, ml));
          store(hr, h, o);
        }
      }
    }
  }
}

// The group's two blocks of a Q6_K unit. A lane converts the words that it holds in the tile (16-element sub-blocks, four
// elements a lane) and stores every four where the common k order wants them; rows with bit 1 of their number set store their
// two 64-byte halves in the other order (see above). Fetched from the lanes that hold them, eight elements a store as for the
// other types, a block takes 28 shared-memory wavefronts of loads instead of 11 and more variable shifts. 4096 x 12288,
// 512 / 2048 rows, conversion included: 77 / 218 -> 65 / 197 us; 12288 x 4096: 58 / 205 -> 52 / 181 us.
__device__ __forceinline__ void dequant_q6k(const uint8_t* t, int grp, int lane, uint8_t* a_rows) {
  const int g = lane >> 2, c = lane & 3, flip = (g >> 1) & 1;
  uint8_t* const row = a_rows + g * 128;
  const uint32_t o0 = (uint32_t)((((4 * flip) | (2 * (c & 1))) ^ g) << 4) + 8 * (c >> 1);
  const __half2 off = __float2half2_rn(1056.f);     // 1024 + 32
  const __half2 off_sc = __float2half2_rn(1152.f);  // 1024 + 128: the int8 scales are biased by xor 0x80
  const uint4 qv = lds_v4(t + TQ_Q6K_QH + 512 * grp + 16 * lane);
  uint2 sc[2];
  __half2 dd[2];
#pragma unroll
  for (int hr = 0; hr < 2; hr++) {
    sc[hr] = *reinterpret_cast<const uint2*>(t + 16 * (g + 8 * hr) + 8 * grp);
    dd[hr] = __half2half2(__ushort_as_half((unsigned short)lds_u16(t + TQ_Q6K_D + 2 * (g + 8 * hr))));
  }
#pragma unroll
  for (int e = 0; e < 2; e++) {
    const uint4 q = lds_v4(t + TQ_Q6K_QL + 512 * (2 * grp + e) + 16 * lane);
#pragma unroll
    for (int hr = 0; hr < 2; hr++) {
      const uint32_t qh = e ? (hr ? qv.w : qv.y) : (hr ? qv.z : qv.x);
      // d * scale of the block's four sub-blocks in half arithmetic (exact product, one rounding)
      const uint32_t scb = (e ? sc[hr].y : sc[hr].x) ^ 0x80808080u;
      const uint32_t d01 = h22u(__hmul2(dd[hr], __hsub2(pair01(scb), off_sc))), d23 = h22u(__hmul2(dd[hr], __hsub2(pair23(scb), off_sc)));
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int s = h ^ flip;  // sub-blocks 2s (low nibbles) and 2s + 1
        const uint32_t w = s ? (hr ? q.w : q.y) : (hr ? q.z : q.x);
        const uint32_t hi = qh << (4 - 4 * s);  // their 2-bit fields at bits 4..5 and 6..7 of every byte
        const __half2 dl = u2h2(s ? d23 : d01);
        const uint32_t m0 = (w & 0x0F0F0F0Fu) | (hi & 0x30303030u), m1 = ((w >> 4) & 0x0F0F0F0Fu) | ((hi >> 2) & 0x30303030u);
        uint8_t* const p = row + e * A_BYTES + hr * 1024;
        *reinterpret_cast<uint2*>(p + (o0 ^ (h << 6))) =
            make_uint2(h22u(__hmul2(__hsub2(pair02(m0), off), __low2half2(dl))), h22u(__hmul2(__hsub2(pair13(m0), off), __low2half2(dl))));
        *reinterpret_cast<uint2*>(p + (o0 ^ (h << 6) ^ 16u)) =
            make_uint2(h22u(__hmul2(__hsub2(pair02(m1), off), __high2half2(dl))), h22u(__hmul2(__hsub2(pair13(m1), off), __high2half2(dl))));
      }
    }
  }
}

struct GemmArgs {
  const uint8_t* tiles;
  int64_t n_rows;   // weight rows (output features)
  int row_tiles;    // 16-row tiles of the weight
  int ktiles;       // device tiles per row-tile
  int kblocks;      // k / 64
  int KU;           // units of 256 k per row (the last one of a Q8_0 weight may hold fewer blocks)
  int m;            // activation rows
  int bn;           // activation rows per pair tile: a multiple of 16, at most 256
  int mt;           // activation tiles
  int total;        // tiles
  int sibling;      // the preceding launch belongs to the same call and reads the same x (see the kernel)
  int* go;          // [CTA] a sibling's go-ahead words, zero between launches
  int* next_go;     // those of the launch behind this one, which has next_ctas CTAs (0: no sibling follows)
  int next_ctas;
  int a_stages, b_stages, raw_slots;
  const float* rscale;  // [m] factor undoing the f16 row scaling
  float* y;             // [m, n_rows]
  const float* bias;
  int* status;
  // exchange slots (tp.cu): with y_toggle set, the result goes to y_alt instead of y when the
  // word it points to, plus one, is odd - read after the preceding kernels have completed
  const unsigned* y_toggle;
  float* y_alt;
};

// The tiles a pair works on, in order; every role of both CTAs walks the same list.
struct Tiles {
  int u, total, step;
  __device__ __forceinline__ void init(const GemmArgs& a, int pair, int pairs) {
    u = pair;
    total = a.total;
    step = pairs;
  }
  __device__ __forceinline__ bool last() const { return u >= total; }  // after next(): nothing follows
  __device__ __forceinline__ bool next(int& t) {
    if (u >= total) return false;
    t = u;
    u += step;
    return true;
  }
};

// Epilogue of one tile for one TMEM lane quarter (32 weight rows): columns in chunks of 16, the
// chunks h0, h0 + hstep, ...
__device__ __forceinline__ void epilogue(const GemmArgs& a, float* ybase, int t, int rank, int quarter, int lane, uint32_t tmem, int h0, int hstep) {
  constexpr int CH = 16;
  const int m0 = (t % a.mt) * a.bn;
  const int cols = a.m - m0 < a.bn ? a.m - m0 : a.bn;
  const int nchunks = (cols + CH - 1) / CH;
  const int64_t n = (int64_t)(t / a.mt) * (2 * BM) + rank * BM + 32 * quarter + lane;
  const float bv = (a.bias && n < a.n_rows) ? a.bias[n] : 0.f;
  float* const yp = ybase + (int64_t)m0 * a.n_rows + n;
  for (int ch = h0; ch < nchunks; ch += hstep) {
    const int col0 = ch * CH;
    uint32_t v[CH];
    const uint32_t taddr = tmem + ((uint32_t)(32 * quarter) << 16) + (uint32_t)col0;
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    if (n < a.n_rows) {
#pragma unroll
      for (int j = 0; j < CH; j++)
        if (col0 + j < cols) yp[(int64_t)(col0 + j) * a.n_rows] = __uint_as_float(v[j]) * a.rscale[m0 + col0 + j] + bv;
    }
  }
}

template <int DT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TC_REG_THREADS, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ GemmArgs a) {
  constexpr int TB = TileGeom<DT>::BYTES;
  constexpr int UB = UnitGeom<DT>::BYTES;
  constexpr int SLOT_BYTES = 8 * UB;
  constexpr int KA = 2;          // 64-k blocks per stage of the weight operand (one per stage of the activation operand)
  constexpr int ACC_COLS = 256;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // 1024-byte alignment for the swizzled tiles; the same offsets in both CTAs of the pair
  uint8_t* smem = smem_raw + ((1024u - (s_u32(smem_raw) & 1023u)) & 1023u);
  const int SA = a.a_stages, SB = a.b_stages, RS = a.raw_slots;
  const int b_bytes = a.bn * (BK * 2 / 2);  // this CTA's half of the activation tile, per block
  uint8_t* sA = smem;
  uint8_t* sB = sA + SA * KA * A_BYTES;
  uint8_t* sRaw = sB + SB * b_bytes;
  // The two operands have rings of their own: an activation tile is a trip to L2 away and needs many
  // stages in flight, a weight tile comes from this SM's raw ring and needs few.
  // a_full[s] (leader only): both CTAs' weight tiles, one arrival per dequantize warp
  // b_full[s] (leader only): both halves of the activation tile (transaction bytes of both CTAs)
  uint64_t* a_full = reinterpret_cast<uint64_t*>(sRaw + RS * SLOT_BYTES);
  uint64_t* a_empty = a_full + MAX_ST;
  uint64_t* b_full = a_empty + MAX_ST;
  uint64_t* b_empty = b_full + MAX_ST;
  uint64_t* raw_full = b_empty + MAX_ST;
  uint64_t* raw_empty = raw_full + MAX_RAW;
  uint64_t* acc_full = raw_empty + MAX_RAW;
  uint64_t* acc_empty = acc_full + 2;  // leader only
  uint64_t* last_full = acc_empty + 2;  // the pair's last accumulator is complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(last_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = blockIdx.x & 1u;  // rank in the cluster of two
  const int pair = (int)(blockIdx.x >> 1), pairs = (int)(gridDim.x >> 1);

  // Siblings: beside the set-up, whose barrier then orders every warp of the CTA behind the word's acquire.
  bool go = true;
  if (a.sibling && warp == 1 && lane == 0) go = take_go(a.go + blockIdx.x);
  if (threadIdx.x == 0) {
    for (int s = 0; s < SA; s++) {
      bar_init(&a_full[s], 2 * DQ_WARPS);
      bar_init(&a_empty[s], 1);
    }
    for (int s = 0; s < SB; s++) {
      bar_init(&b_full[s], 1);
      bar_init(&b_empty[s], 1);
    }
    for (int s = 0; s < RS; s++) {
      bar_init(&raw_full[s], 1);
      bar_init(&raw_empty[s], DQ_WARPS * DQ_GROUPS);
    }
    for (int s = 0; s < 2; s++) {
      bar_init(&acc_full[s], 1);
      bar_init(&acc_empty[s], 8);
    }
    bar_init(last_full, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_u32(tmem_slot)), "n"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_all();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;

  Tiles seg;
  seg.init(a, pair, pairs);
  int t;
  if (warp == 0) {
    // ------------------------------------------------------------ raw weight bytes -> ring
    // Lane r < 8 copies row-tile r's share of the unit: issued by one lane, the eight copies of a unit
    // took 600 ns one after the other, half of what the unit lasts.
    int slot = 0;
    uint32_t ph = 0;
    bool ok = true;
    while (ok && seg.next(t)) {
      const int rt0 = (t / a.mt) * 16 + (int)rank * 8;
      int nlive = a.row_tiles - rt0;
      nlive = nlive < 0 ? 0 : nlive > 8 ? 8 : nlive;
      const uint8_t* const row = a.tiles + (int64_t)(rt0 + lane) * a.ktiles * TB;
      for (int ku = 0; ku < a.KU; ku++) {
        ok = __all_sync(0xFFFFFFFFu, bar_wait(&raw_empty[slot], ph ^ 1u, abort_flag));
        if (!ok) break;
        int nt = a.ktiles - ku * UnitGeom<DT>::TILES;
        if (nt > UnitGeom<DT>::TILES) nt = UnitGeom<DT>::TILES;
        const uint32_t bytes = (uint32_t)(nt * TB);
        if (lane == 0) bar_expect_tx(&raw_full[slot], bytes * (uint32_t)nlive);
        __syncwarp();
        if (lane < nlive)
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                           s_u32(sRaw + slot * SLOT_BYTES + lane * UB)),
                       "l"(row + (int64_t)ku * UB), "r"(bytes), "r"(s_u32(&raw_full[slot]))
                       : "memory");
        if (++slot == RS) { slot = 0; ph ^= 1u; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ TMA producer (activations)
    if (lane == 0) {
      // Programmatic stream serialization: the f16 operand comes from the conversion launch before
      // this one (the weight side starts without waiting). A sibling launch (the next weight of a
      // call, same x) has a GEMM before it, beside which it runs: its go-ahead word stands for that
      // wait, and before it ends (below) it waits for that GEMM's end, so that whoever waits for it has
      // waited for all of the call. The proxy fence carries what the word's acquire made visible over
      // to the tensor copies.
      asm volatile("prefetch.tensormap [%0];" ::"l"(&xmap) : "memory");
      if (a.sibling) {
        if (!go) *abort_flag = 1;
        asm volatile("fence.proxy.async.global;" ::: "memory");
      } else {
        asm volatile("griddepcontrol.wait;" ::: "memory");
      }
      asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      while (ok && seg.next(t)) {
        const int row = (t % a.mt) * a.bn + (int)rank * (a.bn >> 1);
        for (int k = 0; k < a.kblocks; k++) {
          ok = bar_wait(&b_empty[s], ph ^ 1u, abort_flag);
          if (!ok) break;
          if (rank == 0) bar_expect_tx(&b_full[s], 2u * (uint32_t)b_bytes);
          asm volatile(
              "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                  s_u32(sB + s * b_bytes)),
              "l"(&xmap), "r"(k * BK), "r"(row), "r"(map_to_rank(s_u32(&b_full[s]), 0))
              : "memory");
          if (++s == SB) { s = 0; ph ^= 1u; }
        }
      }
    }
  } else if (warp == 2) {
    // ------------------------------------------------------------ MMA issuer
    // The whole warp walks the loop and one elected lane issues: control flow and descriptors stay
    // warp-uniform. This loop's own instructions are what separates the MMAs of consecutive stages when
    // there are few activation rows.
    if (rank == 0) {
      // instruction descriptor: f32 accumulate, f16 x f16, both K-major, N = bn, M = 256
      const uint32_t idesc = (1u << 4) | ((uint32_t)(a.bn >> 3) << 17) | ((uint32_t)(2 * BM >> 4) << 24);
      // K-major, 128-byte swizzle matrix descriptors (8-row groups 1024 B apart): a constant high
      // half plus a low half that advances by 2 (32 bytes >> 4) per 16-element K step
      constexpr uint64_t desc_hi = (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
      const uint32_t a_lo0 = (s_u32(sA) & 0x3FFFFu) >> 4, b_lo0 = (s_u32(sB) & 0x3FFFFu) >> 4;
      const uint32_t b_step = (uint32_t)b_bytes >> 4;
      const bool issuer = elect_one();
      int s = 0, sb = 0, nseg = 0;
      uint32_t ph = 0, bph = 0;
      while (seg.next(t)) {
        const int acc = nseg & 1;
        const uint32_t aph = (uint32_t)(nseg >> 1) & 1u;
        nseg++;
        bar_pass(&acc_empty[acc], aph ^ 1u, abort_flag);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t d = tmem_base + (uint32_t)(acc * ACC_COLS);
        uint32_t accumulate = 0;  // the first MMA of the tile overwrites the accumulator
        for (int k = 0; k < a.kblocks; k += KA) {
          const uint64_t da0 = desc_hi | (uint64_t)(a_lo0 + (uint32_t)(s * KA) * (A_BYTES >> 4));
          bar_pass(&a_full[s], ph, abort_flag);
#pragma unroll
          for (int b = 0; b < KA; b++) {
            if (b == 0 || k + b < a.kblocks) {
              const bool last = b == KA - 1 || k + b + 1 >= a.kblocks;
              bar_pass(&b_full[sb], bph, abort_flag);
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              const uint64_t db0 = desc_hi | (uint64_t)(b_lo0 + (uint32_t)sb * b_step);
              if (issuer) {
#pragma unroll
                for (int kk = 0; kk < BK / 16; kk++) {
                  asm volatile(
                      "{\n\t.reg .pred p;\n\t"
                      "setp.ne.b32 p, %4, 0;\n\t"
                      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
                      "l"(da0 + (uint64_t)(b * (A_BYTES >> 4) + 2 * kk)), "l"(db0 + (uint64_t)(2 * kk)), "r"(idesc),
                      "r"(b + kk > 0 ? 1u : accumulate)
                      : "memory");
                }
                // release the stages to both CTAs' producers once these MMAs have read them
                commit_to_pair(&b_empty[sb]);
                if (last) commit_to_pair(&a_empty[s]);
              }
              if (++sb == SB) { sb = 0; bph ^= 1u; }
            }
          }
          accumulate = 1u;
          if (++s == SA) { s = 0; ph ^= 1u; }
        }
        if (issuer) commit_to_pair(seg.last() ? last_full : &acc_full[acc]);
      }
      __syncwarp();
    }
  } else if (warp < DQ_WARP0) {
    // ------------------------------------------------------------ epilogue
    if (!a.sibling) asm volatile("griddepcontrol.wait;" ::: "memory");  // y may still be read, the row scales still written
    if (warp == 3)  // what this launch has waited for, a sibling behind it need not wait for again
      for (int c = (int)(blockIdx.x + lane * gridDim.x); c < a.next_ctas; c += 32 * (int)gridDim.x) st_release(a.next_go + c, 1);
    float* ybase = a.y;
    if (a.y_toggle && ((*reinterpret_cast<const volatile unsigned*>(a.y_toggle) + 1u) & 1u)) ybase = a.y_alt;
    const int quarter = warp & 3;
    const uint32_t empty0 = map_to_rank(s_u32(&acc_empty[0]), 0);
    int nseg = 0;
    while (seg.next(t)) {
      const int acc = nseg & 1;
      const uint32_t aph = (uint32_t)(nseg >> 1) & 1u;
      nseg++;
      if (!(seg.last() ? bar_wait(last_full, 0, abort_flag) : bar_wait(&acc_full[acc], aph, abort_flag))) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // the last epilogue is shared with the dequantize warps, which have nothing left to do
      epilogue(a, ybase, t, (int)rank, quarter, lane, tmem_base + (uint32_t)(acc * ACC_COLS), 0, seg.last() ? HELPERS : 1);
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive_cluster(empty0 + 8u * (uint32_t)acc);
    }
  } else {
    // ------------------------------------------------------------ dequantize
    // A warp reaches one quarter of TMEM's lanes (warp & 3), 32 rows: two of the four warps of a quarter
    // take one 16-row tile each for one group, two for the other. A group makes blocks 2 grp, 2 grp + 1.
    const int dqw = (warp - DQ_WARP0) >> 2;  // 0..3 within the quarter
    const int grp = dqw >> 1;
    const int dq = 2 * (warp & 3) + (dqw & 1);  // row-tile of 16 rows inside the CTA's 128 rows
    const uint32_t a_full0 = map_to_rank(s_u32(&a_full[0]), 0);
    int slot = 0, s = 0, nseg = 0;
    uint32_t rph = 0, ph = 0;
    int lt = 0;  // the last tile
    while (seg.next(t)) {
      lt = t;
      nseg++;
      const bool live = (t / a.mt) * 16 + (int)rank * 8 + dq < a.row_tiles;  // rows beyond the weight are never stored
      for (int ku = 0; ku < a.KU; ku++) {
        bar_pass(&raw_full[slot], rph, abort_flag);
        const uint8_t* raw = sRaw + slot * SLOT_BYTES + dq * UB;
        int nb = a.kblocks - 4 * ku;
        if (nb > 4) nb = 4;
        nb -= 2 * grp;  // this group makes the unit's blocks 2 grp, 2 grp + 1
        if (nb > 0) {
          const UnitScales us = unit_scales<DT>(raw, 2 * grp + (lane & 1), lane);
          int si = s + grp;
          uint32_t phi = ph;
          if (si >= SA) { si -= SA; phi ^= 1u; }
          bar_pass(&a_empty[si], phi ^ 1u, abort_flag);
          uint8_t* const dst = sA + si * KA * A_BYTES + dq * 16 * 128;
          if constexpr (DT == TQ_Q6_K) {
            if (live) dequant_q6k(raw, grp, lane, dst);
          } else {
#pragma unroll
            for (int b = 0; b < 2; b++)
              if (live && b < nb) dequant_block<DT>(raw, us, 2 * grp + b, b, lane, dst + b * A_BYTES);
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic-proxy stores -> visible to the MMA
          __syncwarp();
          if (lane == 0) bar_arrive_cluster(a_full0 + 8u * (uint32_t)si);
        }
        s += a.kblocks - 4 * ku > KA ? 2 : 1;
        if (s >= SA) { s -= SA; ph ^= 1u; }
        __syncwarp();
        if (lane == 0) bar_arrive(&raw_empty[slot]);
        if (++slot == RS) { slot = 0; rph ^= 1u; }
      }
    }
    // nothing left to dequantize: help with the epilogue of the last tile
    if (nseg > 0) {
      if (!a.sibling) asm volatile("griddepcontrol.wait;" ::: "memory");
      float* ybase = a.y;
      if (a.y_toggle && ((*reinterpret_cast<const volatile unsigned*>(a.y_toggle) + 1u) & 1u)) ybase = a.y_alt;
      const int acc = (nseg - 1) & 1;
      if (bar_wait(last_full, 0, abort_flag)) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        epilogue(a, ybase, lt, (int)rank, warp & 3, lane, tmem_base + (uint32_t)(acc * ACC_COLS), (warp - DQ_WARP0) / 4 + 1, HELPERS);
      }
    }
  }
  __syncthreads();
  if (*abort_flag) {
    // a wait ran out: give copies still in flight time to land in this CTA's shared memory
    for (int i = 0; i < 64; i++) __nanosleep(2000);
    if (threadIdx.x == 0) {
      *reinterpret_cast<volatile int*>(a.status) = 7;  // TURQ_E_TIMEOUT; the word may be mapped host memory
      __threadfence_system();
    }
  }
  // neither CTA leaves while the other may still arrive on its barriers or have its operands read
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  // (execution only: nothing but barriers and operand tiles is shared between the two)
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  if (warp == 2) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(TMEM_COLS) : "memory");
  }
  if (a.sibling && threadIdx.x == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
}

// x [m, k] (f32 / bf16) -> f16 with a per-row power-of-two scale that brings the row's
// largest magnitude into [8192, 16384): rows of large values do not overflow f16 and rows of
// tiny values do not sink into its subnormals. rscale[m] undoes the scale exactly in the
// epilogue. Rows that are all zero, or hold an infinity or NaN, are converted as they are.
// The row is written in the operands' k order (tc_common.cuh): as a row of [m, k] (prefill),
// or as a row of the operand's shared-memory images [tile of image_rows rows][k / 64][image_rows][128 bytes], 128B-swizzled,
// which gemm_batch.cu copies in whole. One CTA per row; up to 4096 values stay in registers between the search for the largest
// magnitude and the conversion. CLUSTER (few long rows, plan_prep_cluster): a cluster of CTAs a row, 4096 values each (beyond
// 8 x 4096 the rest is read again), whose maxima meet in distributed shared memory.
// At 48 registers a thread (40 where the GEMM behind has a warp more; the cluster form spills 32 bytes there) a CTA fits beside a CTA of the GEMM, so the conversion
// of the next call is resident before this call ends.
constexpr int PREP_THREADS = 256, PREP_KEEP = 2;
static_assert(PREP_VALUES == PREP_THREADS * 8 * PREP_KEEP, "what the plan counts a CTA to keep");
template <bool IMAGE, bool CLUSTER>
__global__ void __launch_bounds__(PREP_THREADS, IMAGE ? 6 : 5) prep_act_kernel(const void* __restrict__ x, int is_bf16, uint32_t k, int image_rows,
                                                                               __half* __restrict__ xh, __half* __restrict__ xh16,
                                                                               float* __restrict__ rscale) {
  __shared__ float wmax[8];
  __shared__ float cta_max;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");  // the GEMM behind may start on its weights
  asm volatile("griddepcontrol.wait;" ::: "memory");               // x may still be written, the operand buffer still read
  const int csize = CLUSTER ? (int)cluster_size() : 1, rank = CLUSTER ? (int)cluster_rank() : 0;
  const uint32_t row = blockIdx.x / csize;
  // this CTA's columns, in whole 64-k blocks (k < 2^31: no sum below leaves 32 bits)
  const uint32_t per = CLUSTER ? (k / 64 + csize - 1) / csize * 64 : k, c0 = rank * per, c1 = c0 + per < k ? c0 + per : k;
  const int64_t row0 = (int64_t)row * k;
  float v[PREP_KEEP][8];
  float amax = 0.f;
#pragma unroll
  for (int j = 0; j < PREP_KEEP; j++) {
    const uint32_t i = c0 + (j * PREP_THREADS + threadIdx.x) * 8;
    if (i < c1) {
      load8(x, is_bf16, row0 + i, v[j]);
#pragma unroll
      for (int e = 0; e < 8; e++) amax = fmaxf(amax, fabsf(v[j][e]));
    }
  }
#pragma unroll 2
  for (uint32_t i = c0 + PREP_VALUES + threadIdx.x * 8; i < c1; i += PREP_THREADS * 8) {
    float u[8];
    load8(x, is_bf16, row0 + i, u);
#pragma unroll
    for (int e = 0; e < 8; e++) amax = fmaxf(amax, fabsf(u[e]));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
  if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = wmax[0];
#pragma unroll
  for (int w = 1; w < 8; w++) amax = fmaxf(amax, wmax[w]);
  if constexpr (CLUSTER) {
    if (threadIdx.x == 0) cta_max = amax;
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    for (int r = 0; r < csize; r++) {
      float other;
      asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(other) : "r"(map_to_rank(s_u32(&cta_max), (uint32_t)r)));
      amax = fmaxf(amax, other);
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");  // read: waited for before the CTA ends
  }
  float s = 1.f;
  if (amax > 0.f && amax < 3.0e38f) {  // also false for NaN
    int e;
    frexpf(amax, &e);           // amax = f * 2^e, f in [0.5, 1)
    int se = 14 - e;            // scaled row maximum lands in [8192, 16384)
    if (se > 126) se = 126;     // keep the scale and its reciprocal normal numbers
    s = ldexpf(1.f, se);
  }
  if (threadIdx.x == 0 && rank == 0) rscale[row] = 1.f / s;
  // the row in the image of its tile of image_rows rows (a multiple of 16)
  const uint32_t tile = IMAGE ? row / (uint32_t)image_rows : 0;
  const uint32_t image_row = IMAGE ? (tile * (k / 64) - tile) * (uint32_t)image_rows + row : 0;  // in rows of 128 bytes
  auto store8 = [&](uint32_t i, const float (&u)[8]) {
    uint32_t o[4];
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int e = 0; e < 2; e++) o[2 * h + e] = h22u(__floats2half2_rn(u[4 * h + e] * s, u[4 * h + e + 2] * s));
    // the two fours of an eight belong to two 16-k chunks
    const int in_block = (int)(i & 32) + (int)(i & 31) / 2;  // inside the 64-k block
    if constexpr (IMAGE) {  // in the common order, in Q6_K's own, or in both
      const size_t block = (size_t)((i >> 6) * (uint32_t)image_rows + image_row) * 128;
      const int swz = (int)(row & 7) << 4;  // 16-byte chunks exchanged by the row's low bits
      if (xh) {
        uint8_t* const p = reinterpret_cast<uint8_t*>(xh) + block;
        const int off = (2 * in_block) ^ swz;
        *reinterpret_cast<uint2*>(p + off) = make_uint2(o[0], o[1]);
        *reinterpret_cast<uint2*>(p + (off ^ 32)) = make_uint2(o[2], o[3]);
      }
      if (xh16)
        *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(xh16) + block + ((2 * (int)(i & 63)) ^ swz)) = make_uint4(o[0], o[1], o[2], o[3]);
    } else {
      __half* const p = xh + row0 + (i & ~63u) + in_block;
      *reinterpret_cast<uint2*>(p) = make_uint2(o[0], o[1]);
      *reinterpret_cast<uint2*>(p + 16) = make_uint2(o[2], o[3]);
    }
  };
#pragma unroll
  for (int j = 0; j < PREP_KEEP; j++) {
    const uint32_t i = c0 + (j * PREP_THREADS + threadIdx.x) * 8;
    if (i < c1) store8(i, v[j]);
  }
#pragma unroll 2
  for (uint32_t i = c0 + PREP_VALUES + threadIdx.x * 8; i < c1; i += PREP_THREADS * 8) {
    float u[8];
    load8(x, is_bf16, row0 + i, u);
    store8(i, u);
  }
  if constexpr (CLUSTER) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

template <int DT>
cudaError_t launch_tc_dt(const CUtensorMap& map, GemmArgs a, int pairs, cudaStream_t s) {
  constexpr int SLOT_BYTES = 8 * UnitGeom<DT>::BYTES;
  constexpr int BAR_BYTES = (4 * MAX_ST + 2 * MAX_RAW + 5) * 8 + 8;
  // Shared memory: three raw slots and three weight stages, two where that leaves no room for
  // four activation blocks in flight, the rest for activation stages and raw slots.
  // (A dequantize warp only waits on the stages it fills itself. Behind a unit of one stage - an
  // in-feature count that is no multiple of 256 - it is three stages on from its last wait; with two
  // stages it could then wait two phases ahead of the barrier, which the parity does not tell apart.)
  // 4 KB stay free for a CTA of the next call's conversion kernel.
  const int budget = device_smem_optin() - 1024 - BAR_BYTES - 4096;
  const int a_stage = 2 * A_BYTES, b_stage = a.bn * BK;
  int sa = 3, sb = 4, rs = 3;
  auto left = [&]() { return budget - sa * a_stage - sb * b_stage - rs * SLOT_BYTES; };
  if (left() < 0 && a.kblocks % 4 == 0) sa = 2;
  if (left() < 0) rs = 2;
  if (left() < 0) sb = 3;
  if (left() < 0) return cudaErrorInvalidConfiguration;
  while (sb < MAX_ST && left() >= b_stage) sb++;
  while (rs < MAX_RAW && left() >= SLOT_BYTES) rs++;
  a.a_stages = sa;
  a.b_stages = sb;
  a.raw_slots = rs;
  static PerDeviceOnce configured;
  int dev = 0;
  cudaGetDevice(&dev);
  if (!configured.done(dev)) {
    cudaError_t e = cudaFuncSetAttribute(gemm_tc_kernel<DT>, cudaFuncAttributeMaxDynamicSharedMemorySize, device_smem_optin());
    if (e != cudaSuccess) return e;
    configured.set(dev);
  }
  const size_t smem = (size_t)(sa * a_stage + sb * b_stage + rs * SLOT_BYTES) + BAR_BYTES + 1024;
  return launch_pdl(gemm_tc_kernel<DT>, dim3((unsigned)(2 * pairs)), dim3(TC_THREADS), smem, s, map, a);
}

}  // namespace

// The f16 operand: rows up to a multiple of 16 for the image of a decode batch.
size_t gemm_operand_bytes(int64_t m, int64_t k) { return ((size_t)((m + 15) / 16 * 16) * (size_t)k * 2 + 255) & ~(size_t)255; }
// One operand, two images of a decode batch, or the image of a short prompt, whose last tile of up to GEMM_TILE_ROWS rows is
// held whole; never less for more rows (a reservation stands for all smaller calls).
size_t gemm_tc_scratch_bytes(int64_t m, int64_t k) {
  const size_t rows = gemm_operand_bytes(m <= GEMM_BATCH_ROWS ? m : m + GEMM_TILE_ROWS, k);
  const size_t images = 2 * gemm_operand_bytes(m < GEMM_BATCH_ROWS ? m : GEMM_BATCH_ROWS, k);
  return (rows > images ? rows : images) + (((size_t)m * 4 + 255) & ~(size_t)255) + 256;
}

// Go-ahead words [weight of the call][CTA].
size_t gemm_workspace_bytes(int sms) { return (size_t)GEMM_SIBLINGS * sms * 4; }

template <bool IMAGE, bool CLUSTER>
static cudaError_t launch_prep(unsigned c, const void* x, int x_dtype, int64_t m, int64_t k, int image_rows, uint8_t* xh, uint8_t* xh16, float* rscale,
                               cudaStream_t s) {
  cudaError_t e = prefer_matmul_carveout<prep_act_kernel<IMAGE, CLUSTER>>();
  if (e != cudaSuccess) return e;
  return launch_pdl_cluster(prep_act_kernel<IMAGE, CLUSTER>, CLUSTER ? c : 0, dim3((unsigned)m * c), dim3(PREP_THREADS), 0, s, x, (int)(x_dtype == TQ_BF16), (uint32_t)k,
                            image_rows, reinterpret_cast<__half*>(xh), reinterpret_cast<__half*>(xh16), rscale);
}
cudaError_t launch_prep_image(const void* x, int x_dtype, int64_t m, int64_t k, int image_rows, uint8_t* xh, uint8_t* xh16, float* rscale, cudaStream_t s) {
  const unsigned c = (unsigned)plan_prep_cluster(m, k, device_sm_count());
  return c > 1 ? launch_prep<true, true>(c, x, x_dtype, m, k, image_rows, xh, xh16, rscale, s)
               : launch_prep<true, false>(c, x, x_dtype, m, k, image_rows, xh, xh16, rscale, s);
}
static cudaError_t launch_prep_rows(const void* x, int x_dtype, int64_t m, int64_t k, uint8_t* xh, float* rscale, cudaStream_t s) {
  const unsigned c = (unsigned)plan_prep_cluster(m, k, device_sm_count());
  return c > 1 ? launch_prep<false, true>(c, x, x_dtype, m, k, 0, xh, nullptr, rscale, s) : launch_prep<false, false>(c, x, x_dtype, m, k, 0, xh, nullptr, rscale, s);
}

// Activation rows per pair tile, activation tiles and pairs of a launch; call_tiles: 256-row tiles of all weights of the call.
struct TcShape { int bn, mt, pairs; };
static TcShape tc_shape(int64_t n_rows, int64_t call_tiles, int64_t m, int sm_count) {
  TcShape p;
  p.bn = plan_gemm_rows(call_tiles, m, sm_count);
  p.mt = (int)((m + p.bn - 1) / p.bn);
  p.pairs = plan_gemm_pairs((n_rows + 2 * BM - 1) / (2 * BM) * p.mt, sm_count);
  return p;
}

cudaError_t launch_gemm_tc(int dtype, const uint8_t* tiles, int64_t n_rows, int64_t k, const void* x, int x_dtype,
                           int64_t m, float* y, const float* bias, uint8_t* scratch, uint8_t* workspace, int sm_count, cudaStream_t s,
                           int* launches, int* dev_status_word, int64_t call_tiles, int sibling, int64_t next_rows, const unsigned* y_toggle,
                           float* y_alt) {
  if (k % BK != 0 || m <= GEMM_BATCH_ROWS || m > INT32_MAX || k > INT32_MAX || sibling < 0 ||
      sibling + (next_rows > 0 ? 1 : 0) >= GEMM_SIBLINGS) return cudaErrorInvalidValue;
  EncodeTiledFn enc = encode_fn();
  if (!enc) return cudaErrorNotSupported;
  float* rscale = reinterpret_cast<float*>(scratch + gemm_operand_bytes(m, k));
  cudaError_t e = cudaSuccess;
  if (sibling == 0) {  // several weights that read the same x share one conversion
    e = launch_prep_rows(x, x_dtype, m, k, scratch, rscale, s);
    if (launches) (*launches)++;
    if (e != cudaSuccess) return e;
  }

  const int64_t n_tiles = (n_rows + 2 * BM - 1) / (2 * BM);
  const TcShape shape = tc_shape(n_rows, call_tiles > 0 ? call_tiles : n_tiles, m, sm_count);
  const int bn = shape.bn;
  CUtensorMap map;
  const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)m};
  const cuuint64_t strides[1] = {(cuuint64_t)k * 2};
  const cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)bn / 2};
  const cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, scratch, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;

  GemmArgs a{};
  a.tiles = tiles;
  a.n_rows = n_rows;
  a.row_tiles = (int)((n_rows + TQ_TILE_ROWS - 1) / TQ_TILE_ROWS);
  a.ktiles = (int)(k / tq_block_elems(dtype));
  a.kblocks = (int)(k / BK);
  a.KU = (int)((k + UNIT_K - 1) / UNIT_K);
  a.m = (int)m;
  a.bn = bn;
  a.mt = shape.mt;
  const int64_t total = n_tiles * a.mt;
  if (total > (int64_t)1 << 30) return cudaErrorInvalidValue;
  a.total = (int)total;
  a.sibling = sibling > 0;
  a.rscale = rscale;
  a.y = y;
  a.bias = bias;
  a.go = reinterpret_cast<int*>(workspace) + (size_t)sibling * sm_count;
  a.next_go = a.go + sm_count;
  a.next_ctas = next_rows > 0 ? 2 * tc_shape(next_rows, call_tiles, m, sm_count).pairs : 0;
  a.status = dev_status_word;
  a.y_toggle = y_toggle;
  a.y_alt = y_alt;
  switch (dtype) {
    case TQ_Q8_0: e = launch_tc_dt<TQ_Q8_0>(map, a, shape.pairs, s); break;
    case TQ_Q4_K: e = launch_tc_dt<TQ_Q4_K>(map, a, shape.pairs, s); break;
    case TQ_Q5_K: e = launch_tc_dt<TQ_Q5_K>(map, a, shape.pairs, s); break;
    case TQ_Q6_K: e = launch_tc_dt<TQ_Q6_K>(map, a, shape.pairs, s); break;
    default: return cudaErrorInvalidValue;
  }
  if (launches) (*launches)++;
  return e;
}

}  // namespace turq
