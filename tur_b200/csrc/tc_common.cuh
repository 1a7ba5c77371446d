// Device code that the prefill GEMM (gemm_tc.cu) and the GEMM of decode batches (gemm_batch.cu) share:
// bounded barrier waits, the f16 operand's k order, the raw units of a weight and their sub-block scales.
#pragma once
#include <cuda_fp16.h>

#include "device_utils.cuh"
#include "gemv_tile.cuh"
#include "layout.h"

namespace turq {

constexpr int BM = 128;      // weight rows per CTA
constexpr int BK = 64;       // k per operand block (one 128-byte swizzle row of f16)
constexpr int UNIT_K = 256;  // k per unit of raw weight bytes (four blocks)
constexpr long long TC_WAIT_CYCLES = 4000000000ll;

__device__ __forceinline__ uint32_t s_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void bar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s_u32(bar)), "r"(count));
}
__device__ __forceinline__ void bar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(s_u32(bar)) : "memory");
}
__device__ __forceinline__ void bar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(s_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_try(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(s_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool bar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  if (bar_try(bar, parity)) return true;  // the common case costs one poll, no clock read
  const long long t0 = clock64();
  for (uint32_t i = 0;; i++) {
    if (bar_try(bar, parity)) return true;
    if ((i & 255u) == 255u && (*abort_flag || clock64() - t0 > TC_WAIT_CYCLES)) break;
  }
  *abort_flag = 1;
  return false;
}
// The same for loops that do not look at the result: after an expiry the abort flag makes every further
// wait return soon, and what such a loop then does stays within its buffers. Without the way out the
// loop's control flow is the same for the whole warp.
static __device__ __noinline__ void bar_wait_slow(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  bar_wait(bar, parity, abort_flag);
}
__device__ __forceinline__ void bar_pass(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  if (!bar_try(bar, parity)) bar_wait_slow(bar, parity, abort_flag);
}
// An address of this CTA's shared memory -> the same in the CTA of the cluster with that rank.
__device__ __forceinline__ uint32_t map_to_rank(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(r));
  return r;
}
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void st_release(int* p, int v) { asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }

// ---- dequantization to f16 with packed half arithmetic (two elements per instruction).
// An integer q <= 1023 becomes the half 1024 + q by OR-ing it under the exponent 0x6400;
// subtracting the offset is exact, so the only roundings are the f16 sub-block scale / min
// and the final multiply-add. The error stays a few 1e-4 of the value, inside the 2e-3 budget
// of the tensor-core mode (the bit-exact f32 decode lives in decode.cuh).
__device__ __forceinline__ __half2 u2h2(uint32_t u) { return *reinterpret_cast<__half2*>(&u); }
__device__ __forceinline__ uint32_t h22u(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
// k order of both f16 operands: a 16-k chunk (one MMA) of an aligned 32 holds, for c = 0..3, elements
// 8c + {0, 2, 1, 3} (first chunk) or 8c + 4 + {0, 2, 1, 3} (second) - what lane column c of a fragment
// tile finds in one word, in the pairs the word gives without a shuffle. The same for prefill and decode
// batches. (Their f32 sums still associate differently: decode batches cut the K loops, prefill does not.)
// bytes (b0, b2) / (b1, b3) of a word of small integers -> half2 (1024 + b0, 1024 + b2) / ...
__device__ __forceinline__ __half2 pair02(uint32_t w) { return u2h2(__byte_perm(w, 0x64646464u, 0x5240)); }
__device__ __forceinline__ __half2 pair13(uint32_t w) { return u2h2(__byte_perm(w, 0x64646464u, 0x5341)); }
__device__ __forceinline__ __half2 pair01(uint32_t w) { return u2h2(__byte_perm(w, 0x64646464u, 0x5140)); }
__device__ __forceinline__ __half2 pair23(uint32_t w) { return u2h2(__byte_perm(w, 0x64646464u, 0x5342)); }

// Siblings (the later weights of a call) run beside their predecessor, so griddepcontrol.wait, which
// waits for its end, cannot be what makes the shared operand visible to them. Instead every CTA of a
// sibling takes one go-ahead word that the launch before it released, once that launch itself could see
// the operand and the end of everything older than the call. A word is taken by exchanging it for zero:
// an exchange follows the write that it reads immediately in the word's order of writes, so a word set
// for an earlier call, which that call's exchange has taken, cannot be read again.
// The words are there when the sibling starts or soon after: every CTA of the launch before it has then
// started and waits for nothing more before it releases them. Taken after the CTA's set-up and released
// before dependents may start, they cost up to 1.2 us a sibling (Q8_0 2560 + 640 + 640 rows x 2560, 32
// activation rows, us a call: 15.8 without, 18.2 so, 16.1 as it is; Q4_K + Q4_K + Q6_K 4096 + 1024 + 1024 x 4096,
// 300 rows: 34.1, 36.3, 35.3).
__device__ __forceinline__ bool take_go(int* p) {
  const long long t0 = clock64();
  int v;
  do {
    asm volatile("atom.acquire.gpu.global.exch.b32 %0, [%1], 0;" : "=r"(v) : "l"(p) : "memory");
  } while (v == 0 && clock64() - t0 <= TC_WAIT_CYCLES);
  return v != 0;
}

// Raw bytes of one unit (16 weight rows x 256 k) as they lie in a ring slot.
template <int DT> struct UnitGeom {
  static constexpr int TILES = UNIT_K / TileGeom<DT>::ELEMS;  // device tiles per unit: 8 (Q8_0) or 1
  static constexpr int BYTES = TILES * TileGeom<DT>::BYTES;   // per row-tile
};

// Scales of the two 64-k blocks of a unit that a warp dequantizes (Q4_K / Q5_K): lane 2r + e holds,
// for row r of the row-tile and block e of the warp's two, the f16 scale and negated min of the
// block's two sub-blocks. Worked out once per unit and row instead of by every lane that needs them.
struct UnitScales { uint32_t dl, ml; };
template <int DT>
__device__ __forceinline__ UnitScales unit_scales(const uint8_t* t, int i, int lane) {
  UnitScales u{0u, 0u};
  if constexpr (DT == TQ_Q4_K || DT == TQ_Q5_K) {
    const __half2 off = __float2half2_rn(1024.f);
    const uint4 hd = lds_v4(t + 16 * (lane >> 1));
    // Half arithmetic only (no int->float / float->half conversions, which share one narrow pipe):
    // d * sc is exact in f32, so one f16 multiply rounds it the same way.
    const __half2 dd = u2h2(__byte_perm(hd.x, 0u, 0x1010)), mm = u2h2(__byte_perm(hd.x, 0u, 0x3232));
    // 6-bit scales / mins of sub-blocks 0..3 or 4..7, one per byte; block i needs bytes 2(i&1), 2(i&1)+1
    const uint32_t scw = i >= 2 ? ((hd.w & 0x0F0F0F0Fu) | ((hd.y >> 2) & 0x30303030u)) : (hd.y & 0x3F3F3F3Fu);
    const uint32_t mnw = i >= 2 ? (((hd.w >> 4) & 0x0F0F0F0Fu) | ((hd.z >> 2) & 0x30303030u)) : (hd.z & 0x3F3F3F3Fu);
    const int sh = 16 * (i & 1);
    u.dl = h22u(__hmul2(dd, __hsub2(pair01(scw >> sh), off)));
    u.ml = h22u(__hneg2(__hmul2(mm, __hsub2(pair01(mnw >> sh), off))));
  }
  return u;
}

// Launch with programmatic stream serialization: the kernel may be scheduled while its
// predecessor in the stream still runs and orders itself with griddepcontrol.wait. In clusters of `cluster` CTAs, or as
// the kernel is declared (0).
template <class... Params, class... Args>
inline cudaError_t launch_pdl_cluster(void (*kernel)(Params...), unsigned cluster, dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}
template <class... Params, class... Args>
inline cudaError_t launch_pdl(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args... args) {
  return launch_pdl_cluster(kernel, 0, grid, block, smem, s, args...);
}

}  // namespace turq
