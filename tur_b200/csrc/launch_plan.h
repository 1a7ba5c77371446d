// Host-side launch arithmetic of the GEMV and the GEMM, free of CUDA so that it can be
// compiled and checked on a machine without a GPU: how the tiles of a weight are dealt out to
// CTAs, which launches share their activation planes, how many CTAs share the K loop of 128 weight rows in decode batches,
// which activation-tile height is used.
#pragma once
#include <atomic>
#include <cstdint>

namespace turq {

// Units = tiles (groups of 4 tiles for Q8_0); a row-tile has KU of them. CTA b owns units
// [start(b), start(b + 1)) with start(b) = min(b * split_q + min(b, split_r), total).
struct GemvSplit {
  int grid;
  int split_q, split_r;
  bool aligned;  // every CTA owns whole row-tiles: no partial sums cross CTAs
};

// Whole row-tiles per CTA when that keeps at least 70 % of the CTA slots busy or the problem is
// small (at most 24 units per slot); otherwise an even split in units, where a row-tile cut
// between CTAs is finished by the CTA holding its first unit. Depends on the shape only.
// force: -1 = choose, 0 = even split, 1 = whole row-tiles.
inline GemvSplit plan_gemv_split(int row_tiles, int KU, int slots, int force = -1) {
  GemvSplit p{};
  const int64_t T = (int64_t)row_tiles * KU;
  const int per = (row_tiles + slots - 1) / slots;
  const int ga = per > 0 ? (row_tiles + per - 1) / per : 0;
  bool aligned = (int64_t)ga * 10 >= (int64_t)slots * 7 || T <= (int64_t)slots * 24;
  if (force == 0) aligned = false;
  if (force == 1) aligned = true;
  p.aligned = aligned;
  if (aligned) {
    p.grid = ga;
    p.split_q = per * KU;
    p.split_r = 0;
  } else {
    p.grid = (int64_t)slots > T ? (int)T : slots;
    p.split_q = (int)(T / p.grid);
    p.split_r = (int)(T % p.grid);
  }
  return p;
}

inline int64_t gemv_split_start(const GemvSplit& p, int64_t total_units, int b) {
  const int64_t u = (int64_t)b * p.split_q + (b < p.split_r ? b : p.split_r);
  return u < total_units ? u : total_units;
}

// Whether a launch of up to 16 rows whose activation planes fit an SM's shared memory, but not a CTA's half
// of it, runs as wide CTAs (one copy of the planes and two sets of warps per SM) or reads the planes from
// global memory. What the wide form saves is the way to L2 per activation fragment, most for Q8_0 (an
// f32 scale per 32 values beside the quants) and Q6_K (four-byte fragments), least for Q4_K and Q5_K; a
// mixed launch also spares a launch per type. What it costs is ring stages (two to four instead of six)
// and, where there are no more shares than SMs, half of the SMs. The lines were drawn with row-major planes. Measured on B200
// with today's, global / wide, us a call ((w) or (g): the other side than the rule's is faster there):
//   Q8_0        5120 x 25600, 3 / 4 rows 27.9 / 26.7, 28.0 / 27.0   4096 x 12288, 6 / 8 rows 14.2 / 12.2, 14.1 / 12.6
//               2560 x 8192, 8 / 12 rows 10.7 / 12.1 (g), 13.5 / 13.3   512 x 8192, 12 rows 10.6 / 11.3 (g)
//   Q6_K        4096 x 12288, 4 / 6 rows 12.4 / 12.3, 12.6 / 12.2   2048 x 5120, 12 rows 10.7 / 9.1   2560 x 8192, 8 rows 9.1 / 8.8
//               640 x 6144, 8 / 12 rows 6.3 / 7.3 (g), 10.3 / 9.7
//     shares cut, shorter than two row-tiles: 5120 x 25600, 2 / 3 rows 25.1 / 23.8 (w), 25.5 / 25.1 (w)   5120 x 13312, 5 / 7 rows 17.5 / 17.3, 17.4 / 17.6
//   Q4_K, Q5_K  4096 x 12288 Q4_K, 6 / 8 rows 10.6 / 9.7, 10.5 / 10.0   25600 x 5120 Q4_K, 12 rows 34.1 / 24.1   9600 x 8192 Q4_K, 8 rows 15.7 / 14.5
//     shares cut, shorter than two row-tiles: 5120 x 8192 Q4_K, 8 / 9 / 12 rows 12.1 / 12.6, 15.5 / 14.4 (w), 15.8 / 14.9 (w)
//                                             6144 x 6144 Q4_K, 9 / 16 rows 13.3 / 13.3, 15.4 / 15.0 (w)   5120 x 25600 Q4_K, 3 rows 21.1 / 19.3 (w)
//     an SM for every share: 128 x 16384 Q4_K, 4 rows 9.5 / 9.9   640 x 8192 Q4_K, 8 / 12 rows 6.6 / 7.1, 10.3 / 9.1 (w)
//     a third of the slots idle: 2560 x 8192 Q5_K, 8 / 12 rows 8.8 / 8.2 (w), 13.1 / 10.8
//   mixed (global: a launch per type) 4096 + 1024 + 1024 x 4096, 9 / 12 rows 16.2 / 16.3, 18.7 / 12.9   8192 + 1024 + 1024 x 5120, 9 rows 23.7 / 20.1
enum class GemvPlaneReads { q8_0, q6_k /* also mixed launches */, q45_k };
inline bool plan_gemv_wide(GemvPlaneReads reads, int rows, const GemvSplit& split, int64_t total_units, int KU, int slots) {
  const bool cut_short = !split.aligned && total_units < (int64_t)2 * KU * split.grid;
  if (reads == GemvPlaneReads::q8_0) return true;
  if (reads == GemvPlaneReads::q6_k) return rows > 3 || !cut_short;
  if (cut_short || 2 * split.grid <= slots) return false;
  return rows > 8 || (int64_t)split.grid * 10 >= (int64_t)slots * 7;
}

// ---- tcgen05 GEMM (pairs of CTAs, 256 weight rows per pair), more than 64 activation rows

// Class of the activation rows per pair tile: 256, unless twice as many tiles still fit the SMs in one wave - then 128,
// which doubles the pairs at work.
inline int plan_gemm_bn(int64_t n_rows, int64_t m, int sm_count) {
  return 2 * ((n_rows + 127) / 128) * ((m + 255) / 256) <= sm_count ? 128 : 256;
}

// Activation rows per pair tile (a multiple of 16, at most 256) for a call whose weights have `call_tiles` 256-row tiles in
// all: the weights of a call run side by side, so what counts is how the tiles of all of them fill the pairs. The least
// time of a tile times what the tiles take of the pairs: a tile of b rows takes about b + 110 (units of an activation row), and
// below 90 rows the weights' dequantization holds it at 200; a last wave counts for a third by what is in it and for two thirds
// whole, since where it is nearly empty the clocks rise with the power that the idle SMs leave. The smaller number of tiles
// where two are alike. Measured on B200 at every height for 32 calls of 384 to 3000 rows, what the choice loses against the best
// height of each: 0.13 % in the geometric mean, 6 % at most (a last wave counted whole and tiles held at 260: 0.9 %, 27 %). us a call, tiles of the choice
// / of the old one: 2 x 8192 x 2560 Q8_0, 1300 rows 109 (6) / 120 (8)   2 x 12288 x 4096 Q4_K, 1700 rows 257 (7) / 269 (9)
//   25600 x 5120 Q4_K, 768 rows 149 (3) / 157 (4)   1024 x 3072 Q8_0, 1300 rows 21 (17) / 25 (10)
// A height of its own for every weight put the small ones of a call on tiles of 128 rows (a layer at 2048 rows 865 us, at one height 793).
inline int plan_gemm_rows(int64_t call_tiles, int64_t m, int sm_count) {
  const int64_t slots = sm_count / 2 > 0 ? sm_count / 2 : 1;
  auto rows_of = [&](int64_t mt) { return ((m + mt - 1) / mt + 15) / 16 * 16; };
  const int64_t cls = plan_gemm_bn(256 * call_tiles, m, sm_count), mt0 = (m + 255) / 256;
  int64_t best = rows_of((m + cls - 1) / cls), best_cost = 0;
  for (int64_t i = -1; i < 3 * mt0 && i < 24; i++) {  // the class above first, then more and more tiles
    const int64_t b = i < 0 ? best : rows_of(mt0 + i), tiles = call_tiles * ((m + b - 1) / b);
    const int64_t whole = (tiles + slots - 1) / slots * slots;  // waves
    const int64_t cost = (2 * whole + (tiles > slots ? tiles : slots)) * (b + 110 > 200 ? b + 110 : 200);
    if (i < 0 || cost < best_cost || (cost == best_cost && b > best)) {
      best = b;
      best_cost = cost;
    }
  }
  return (int)best;
}

// Persistent pairs of CTAs for a weight of `tiles` pair tiles, which are dealt out to them whole, round robin.
inline int plan_gemm_pairs(int64_t tiles, int sm_count) {
  const int64_t slots = sm_count / 2 > 0 ? sm_count / 2 : 1;
  return (int)(tiles < slots ? tiles : slots);
}

// ---- tcgen05 GEMM of decode batches (gemm_batch.cu): clusters of CTAs that share the K loop of 128 weight rows

constexpr int BATCH_MAX_CLUSTER = 6;
// Clusters of 1..6 CTAs, a CTA per SM, that are resident at once on a B200: the model by which the rule below counts rounds. It
// is not what the device in use answers: how its SMs are spread over GPCs, and a process's share of it, may size a grid, but not cut a K loop.
constexpr int BATCH_RESIDENT[BATCH_MAX_CLUSTER + 1] = {0, 148, 74, 45, 33, 26, 22};

// CTAs per cluster for a weight of `tiles` 128-row tiles and `KU` units of 256 k. A function of the weight's shape alone: it
// fixes how the f32 sums associate, so it may depend on neither the batch, the other weights of a call, nor the device or the process.
// The weights that share an x should agree all the same, or
// the call takes a launch for each size, hence a rule that goes by what a weight looks like rather than by the best size for each.
// Measured on B200 with 1 / 2 / 3 / 4 / 6 CTAs, us a call at 32 rows:
//   more than twice as many rows as columns (ffn_gate|up, heads: called in pairs or large anyway): fewest units in sequence
//     at twice the tiles, an exchange counted as one unit more
//     2 x 8192 x 2560 Q5_K 12.8 / 13.0 / 15.4 / 16.2 / 19.7   2 x 12288 x 4096 Q4_K 25.4 / 21.5 / 26.5 / 23.1 / 29.5
//     2 x 25600 x 5120 Q4_K 46.2 / 46.9 / 51.2 / 52.3 / 64.5  2 x 3072 x 1024 Q8_0 6.1 / 6.0 / 8.6 / 7.0 / 7.0
//   else up to 23 units (attn_q|k|v, attn_output): four CTAs, but no more than one per two units
//     4096 + 1024 + 1024 x 4096 15.9 / 10.8 / 14.3 / 10.8 / 12.5     8192 + 1024 + 1024 x 5120 20.6 / 20.1 / 16.9 / 17.0 / 18.2
//     4096 x 4096 13.4 / 9.2 / 8.8 / 8.1 / 9.2   2560 x 2560 10.0 / 6.7 / 6.7 / 6.8 / 6.8   2048 + 1024 + 1024 x 1024 5.9 / 5.8 / 6.2 / 6.0 / 6.0
//   else (ffn_down and wide attn_output, called alone): fewest units in sequence
//     5120 x 25600 Q6_K 88.8 / 50.8 / 40.3 / 52.3 / 40.8   5120 x 8192 Q4_K 24.6 / 15.9 / 13.8 / 16.4 / 14.4
//     2560 x 8192 Q6_K 28.3 / 16.6 / 13.3 / 11.8 / 11.2
inline int plan_batch_cluster(int tiles, int KU) {
  auto rounds = [](int t, int c) { return (t + BATCH_RESIDENT[c] - 1) / BATCH_RESIDENT[c]; };
  int best = 1;
  if (tiles > 4 * KU) {
    int64_t cost = (int64_t)rounds(2 * tiles, 1) * KU;
    for (int c = 2; c <= 4; c *= 2) {
      const int64_t n = (int64_t)rounds(2 * tiles, c) * ((KU + c - 1) / c + 1);
      if (n < cost) { best = c; cost = n; }
    }
  } else if (KU < 24) {
    best = KU < 8 ? (KU + 1) / 2 : 4;
  } else {
    int64_t cost = 0;
    for (int c = 3; c <= BATCH_MAX_CLUSTER; c++) {
      const int64_t n = (int64_t)rounds(tiles, c) * ((KU + c - 1) / c);
      if (c == 3 || n < cost) { best = c; cost = n; }
    }
  }
  return best < KU ? best : KU;
}

// A positive number that is asked for once and then known: `ask(&n)` returns an error or 0. Only an answer is kept; an error goes
// back to the caller, and the next one asks again.
template <class Ask>
inline int ask_once(std::atomic<int>& known, Ask ask, int* out) {
  int n = known.load(std::memory_order_acquire);
  if (n <= 0) {
    const int e = ask(&n);
    if (e != 0) return e;
    if (n < 1) n = 1;
    known.store(n, std::memory_order_release);
  }
  *out = n;
  return 0;
}

// Activation rows per tile (a multiple of 16, at most 128) with which gemm_batch.cu takes a call of more than 64 rows, without
// cutting K, or 0: the prefill kernel takes it. tiles, call_tiles: 128-row and 256-row tiles of all weights of the call.
// What is left idle decides: pairs of CTAs on 256 weight rows leave most of the GPU without work for a short prompt, CTAs of
// their own on 128 rows and as few activation rows as it takes fill it. Both sides by their waves times the time of a unit of
// 256 k: here (0.66 + bn / 1000) us up to 64 rows and (0.41 + bn / 200) us beyond, there, with the rows of plan_gemm_rows, (b + 110) / 218 us, at least 260 / 218; a
// twelfth has to be gained. Measured on B200, prefill kernel / this one, us a call (the prefill side with tiles of 144 rows and
// more, which its rule took then; where it takes smaller ones now it is up to 20 % faster on the small weights, and still behind there):
//   rows                  65            128           256           384           512
//   4096 x 4096 Q4_K      21.2 / 15.6   22.3 / 15.7   22.7 / 17.8   24.7 / 20.8   25.2 / 22.3   (768: 28.0 / 34.1)
//   4096 x 12288 Q4_K     50.9 / 38.5   52.7 / 39.7   56.3 / 41.8   60.8 / 50.8   61.1 / 56.0   (768: 73.3 / 92.8)
//   2560 x 8192 Q8_0      48.2 / 29.5   66.9 / 22.7   63.1 / 27.0   58.7 / 31.3   53.8 / 34.8   (768: 54.8 / 39.5)
//   12288 x 4096 Q8_0     23.1 / 19.1   29.4 / 21.2   34.2 / 35.7   56.7 / 41.3   57.8 / 55.5
//   25600 x 5120 Q4_K     46.2 / 39.2   48.8 / 43.6   62.6 / 66.9   86.6 / 101    103 / 127
//   1024 x 3072 Q8_0      17.1 / 10.6   21.9 / 11.0   22.2 / 13.2   22.3 / 12.3   22.6 / 14.0   (1000: 26.0 / 16.3)
// and calls of several weights: 4096 + 1024 + 1024 x 4096 Q4_K, Q6_K, 128 / 256 rows 27.7 / 23.6, 29.4 / 26.1; 2 x 12288 x 4096 Q4_K,
// 128 rows 44.1 / 38.0; 2560 + 640 + 640 x 2560 Q8_0, 256 rows 24.6 / 17.1.
inline int plan_batch_tile(int64_t tiles, int64_t call_tiles, int64_t m, int sm_count) {
  if (m <= 64 || m > 1024) return 0;
  const int64_t slots = sm_count / 2 > 0 ? sm_count / 2 : 1;
  const int64_t b = plan_gemm_rows(call_tiles, m, sm_count), mt = (m + b - 1) / b;
  int64_t best_cost = (call_tiles * mt + slots - 1) / slots * (b + 110 > 260 ? b + 110 : 260) * 9200 / 218;
  int best = 0;
  for (int bn = 128; bn >= 16; bn -= 16) {
    const int64_t cost = (tiles * ((m + bn - 1) / bn) + sm_count - 1) / sm_count * (bn <= 64 ? 6600 + 10 * bn : 4100 + 50 * bn);
    if (cost < best_cost) { best = bn; best_cost = cost; }
  }
  return best;
}

// ---- conversion of the activations to f16 (prep_act_kernel): a CTA per row, or a cluster of CTAs

constexpr int PREP_VALUES = 4096;      // values of a row that a CTA keeps in registers between its two passes
constexpr int PREP_MAX_CLUSTER = 8;
constexpr int PREP_CTAS_PER_SM = 5;    // that are resident at once

// CTAs that share a row of k values: one per 4096 beyond 16384 values, while the clusters of all m rows are resident at once. What
// they save is a second read of the row, one CTA's chain of it; where there are rows enough to fill the GPU that chain is hidden, and
// clusters only cost their barriers. Measured on B200 with / without, conversion and a GEMM of 128 weight rows, us a call:
//   rows        32            64            96            128           256           1200          4096
//   17408       12.3 / 13.2   13.5 / 14.1   44.3 / 44.3   44.8 / 44.3   49.0 / 45.1   98.6 / 81.7   177 / 124
//   25600       15.5 / 16.9   17.3 / 17.8   63.7 / 64.2   67.1 / 64.3   71.9 / 65.2   147 / 125     265 / 179
//   49152       28.6 / 30.0   27.4 / 30.0   119 / 122     123 / 122     128 / 124     255 / 240     423 / 372
// Up to 16384 values the cluster's barriers cost what the second pass does (12288: 17.2 / 20.0 and 18.7 / 20.0 us at 32 / 64 rows).
inline int plan_prep_cluster(int64_t m, int64_t k, int sm_count) {
  if (k <= 4 * PREP_VALUES) return 1;
  const int64_t want = (k + PREP_VALUES - 1) / PREP_VALUES, c = want < PREP_MAX_CLUSTER ? want : PREP_MAX_CLUSTER;
  return m <= (int64_t)PREP_CTAS_PER_SM * sm_count / c ? (int)c : 1;
}

}  // namespace turq
