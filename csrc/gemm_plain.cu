// The plain GEMM C[M,N] = act(A[M,K] * Bt[N,K]^T) on one GPU: what every fused op runs at world size 1
// and fused.matmul everywhere. bf16 operands, or fp32 operands multiplied as tf32; fp32 accumulation;
// bf16 or fp32 result. This file picks among three kernel families and launches:
//   tile    one wave, a tile or a K range of it per CTA or pair (gemm_tile.cu)
//   flow    persistent pairs that draw tiles in order (gemm_flow.cu)
//   flow + tile  whole waves by the one, the rest by the other in a launch that starts as SMs become free
//   single  persistent single CTAs on the shared main loop (here): narrow outputs, layouts asked for
//           explicitly, rank emulation
// Optionally warps without another role copy the row operand somewhere else while the tiles are computed
// (the all-gather GEMM at world size 1 returns its gathered operand).
#include <algorithm>
#include <cmath>
#include "kraken/gemm_host.h"
#include "kraken/gemm_hooks.cuh"

namespace kraken {

constexpr int kPlainThreads = kGemmThreads + kCopyThreads;

template <int BN, int ELT>
__device__ __forceinline__ void plain_body(const GemmParams& p, unsigned bid, unsigned nb) {
  extern __shared__ unsigned char smem_raw[];
  PlainHooks h;
  h.bn = BN;
  gemm_mainloop<BN, PlainHooks, ELT>(p, bid, nb, h, smem_raw);
}
template <int BN, int ELT>
__global__ void __launch_bounds__(kPlainThreads, 1) gemm_plain_kernel(const __grid_constant__ GemmParams p) {
  plain_body<BN, ELT>(p, blockIdx.x, gridDim.x);
}
template <int BN, int ELT>
__global__ void __launch_bounds__(kPlainThreads, 1) gemm_plain_emu_kernel(const GemmParams* ps) {
  plain_body<BN, ELT>(ps[blockIdx.y], blockIdx.x, gridDim.x);
}

// ---- plan -------------------------------------------------------------------------------------
enum PlainKind : int { PLAIN_SINGLE = 0, PLAIN_TILE = 1, PLAIN_FLOW = 2 };
struct PlainPlan {
  int kind;
  bool swap;        // the weights (Bt) are the row operand and the tile is stored transposed
  bool pair;        // TILE: CTA pairs
  int bn, rb;       // column tile; FLOW: row blocks per tile
  int splits;       // TILE
  int workers;      // CTAs, or pairs, of a persistent kernel
  // FLOW: only the first `cut` rows (cut_n: columns) of the output, the rest by the one-wave kernel in a second launch
  int cut;
  bool cut_n, rest_swap, rest_pair;
  int rest_bn, rest_splits;
};

constexpr double kFlowUs = 4.65, kEpilogueUs = 3.15;       // start and end of the persistent pairs; an epilogue that nothing hides
// Where the rows of an operand start: 0 on 128-byte lines, 1 on 32-byte sectors, 2 in the middle of sectors
// (a row length of an odd number of 16-byte units): each 128 bytes then cost a fifth sector.
static int row_class(long long ld, int elt) { return ld * elt % 128 == 0 ? 0 : ld * elt % 32 == 0 ? 1 : 2; }

// Time model, in microseconds, fitted to 6000 timings of 190 problems on a B200 (interleaved, operands out of HBM): what it
// picks is 1.5 % slower on average than the best plan measured for a problem.
//
// A K block (64 bf16 or 32 fp32 columns of K) takes the longer of its MMAs and of bringing its operand rows into shared
// memory, plus a sixth of the other. The second is no matter of L2 or HBM but of what an SM takes in: per 128-byte row 1.19
// clocks where rows start on lines, 1.62 on sectors, 2.52 in the middle of sectors (fitted; a loop of loads alone at full clock:
// 235, 139 and 94 GB/s, which are 1.07, 1.81 and 2.68).
constexpr double kClocksPerUs = 1465;
static double stage_us(double mma_clocks, double fill_clocks) {
  return (std::max({mma_clocks, fill_clocks, 255.0}) + 0.156 * std::min(mma_clocks, fill_clocks)) / kClocksPerUs;
}
static const double kFillClocks[3] = {1.19, 1.62, 2.52};
// a pair's rb x 256 rows times bn columns, `loaded` of each half of which are fetched
static double block_us(int bn, int rb, int class_r, int class_c, int loaded) {
  const double fill = 128 * rb * kFillClocks[class_r] + std::min(loaded, bn / 2) * kFillClocks[class_c];
  // Two row blocks: fewer and larger stages in flight, which costs where rows are off the lines; on the lines what they save in
  // operand traffic, and so in power, is more (2048 x 3584 x 8192 99.5 us in 512 x 208 tiles, 102.5 in 256 x 208).
  const double two = class_r == 0 && class_c == 0 ? 0.99 : 1.034;
  return stage_us(2.0 * rb * bn, fill) * (rb == 2 ? two : 1.0);
}
// A single CTA's 128 rows times bn columns. Up to 64 columns the weights' way out of HBM counts, and no power limit (60 GB/s
// a CTA where rows start mid-sector, 110 on lines).
static double single_us(int bn, int class_r, int class_c, int loaded) {
  static const double kNarrowUs[3] = {0.147, 0.17, 0.25};
  if (bn <= 64) return kNarrowUs[class_r] * (1 + 0.3 * std::min(loaded, bn) / 128);
  return stage_us(2.0 * bn, 128 * kFillClocks[class_r] + std::min(loaded, bn) * kFillClocks[class_c]);
}
constexpr double kHbmBytesPerUs = 6.45e6;

// What it takes, or, when that is not below `limit`, something that is not either.
static double flow_us(int rows, int cols, int num_kb, int bn, int rb, int pairs, int class_r, int class_c, double hbm_us, double limit,
                      PlanStats* stats) {
  const int tiles_r = (rows + 256 * rb - 1) / (256 * rb), tiles_c = (cols + bn - 1) / bn, last_cols = (cols - (tiles_c - 1) * bn + 15) / 16 * 16;
  if (tiles_c == 1) bn = last_cols;                        // every tile is that narrow
  // what is not hidden: start and last epilogue, and with one accumulator set the epilogue of every tile
  const double bubble = 2 * rb * bn <= 512 ? 0.0 : kEpilogueUs;
  const int narrow = last_cols < bn ? tiles_r : 0, T = tiles_r * tiles_c - narrow, whole = T / pairs, rest = T % pairs;
  // Three waves and more run at the power limit, where wide tiles move less per operation (4509 x 14824 x 4272: 192 columns
  // 402-464 us, 256 columns 382-441).
  const double power = whole >= 3 ? 1 + std::min(0.05, 0.05 * (256 - bn) / 64) : 1.0;
  const double full = num_kb * block_us(bn, rb, class_r, class_c, bn) * power;
  const bool halves = narrow == 0 && rb == 2 && rest && 2 * rest <= pairs;
  const double least = std::max(whole * (full + bubble) + (rest && !halves ? kBusyFloor * full : 0.0), hbm_us) + kFlowUs;
  if (least >= limit) return least;
  ++stats->timed;
  double last;
  if (narrow > 0) {
    // the narrow tiles of the last column fill the last wave
    // (few bytes in flight: the stages are cut for whole tiles)
    const double thin = std::min(full, num_kb * std::max(0.26 * rb, 1.35 * block_us(last_cols, rb, class_r, class_c, last_cols)));
    const int fit = rest ? (pairs - rest) * (int)(full / thin) : 0, left = std::max(0, narrow - fit);
    last = rest ? full * busy_factor(std::min(1.0, (rest + narrow * thin / full) / pairs)) : 0.0;
    const double then = (left + pairs - 1) / pairs * thin * busy_factor(std::min(1.0, (double)left / pairs));
    // all of them on the pairs that the last wave leaves free, or what is left of them after it
    last = rest ? std::min(last + then, std::max(last, (narrow + pairs - rest - 1) / (pairs - rest) * thin)) : then;
  } else if (halves) {
    last = num_kb * block_us(bn, 1, class_r, class_c, bn) * busy_factor(2.0 * rest / pairs);
  } else {
    last = rest ? full * busy_factor((double)rest / pairs) : 0.0;
  }
  return std::max(whole * (full + bubble) + last, hbm_us) + kFlowUs;
}

// The second launch of a problem, beside its own K blocks and sums (us)
constexpr double kRestUs = 3.6;
// The best one-wave kernel for M x N x K, splits 0 if there is none that takes less than `limit`.
struct TileChoice {
  double us;
  bool swap, pair;
  int bn, splits;
};
static TileChoice best_tile(const DeviceState* d, int M, int N, int num_kb, int elt, int class_a, int class_b, double hbm_us, bool pairs_ok,
                            PlanStats* stats, double limit = 1e30) {
  TileChoice best = {limit, false, false, 0, 0};
  for (int swap = 0; swap < 2; ++swap) {
    const int rows = swap ? N : M, cols = swap ? M : N, cr = swap ? class_b : class_a, cc = swap ? class_a : class_b;
    auto offer = [&](bool pair, int bn, double kb_us) {
      const int tiles = ((rows + (pair ? 255 : 127)) / (pair ? 256 : 128)) * ((cols + bn - 1) / bn);
      double us = best.us;
      const int s = tiles <= d->num_sms ? tile_gemm_splits(d, tiles, num_kb, bn, pair, elt, kb_us, hbm_us, &us, stats) : 0;
      if (s > 0) best = {us, swap != 0, pair, bn, s};
    };
    if (cols <= 128) {
      const int bn = pick_bn(cols);
      offer(false, bn, single_us(bn, cr, cc, cols));
    }
    // Pairs only where the second CTA has rows. Single CTAs always: one tile of both dimensions up to 128 is eight K ranges in
    // a cluster instead of one CTA that walks all of K (64 x 128 x 8192 6.6 us against 26.1, 1 x 128 x 7168 5.0 against 19.5).
    for (int bn = 128; pairs_ok && rows > 128 && bn <= 256; bn += 32)
      if (bn == 128 || bn - 32 < cols) offer(true, bn, block_us(bn, 1, cr, cc, cols));
  }
  return best;
}

static PlainPlan plain_plan(const DeviceState* d, int M, int N, int K, int elt, int swap_ab, int bn_override, int use_pair,
                            int max_ctas, int class_a, int class_b, PlanStats* stats) {
  PlainPlan pl;
  memset(&pl, 0, sizeof(pl));
  pl.rb = 1;
  const bool emu = emu_recorder().active;
  int cap = (int)grid_cap(d);
  if (max_ctas > 0 && max_ctas < cap) cap = max_ctas;
  const bool pair_ok = use_pair != 0 && pair_enabled() && !emu && cap >= 2;
  const int num_kb = (K + 128 / elt - 1) / (128 / elt), pairs = cap / 2;
  const double hbm_us = ((double)M + N) * K * elt / kHbmBytesPerUs;
  const bool whole_chip = max_ctas <= 0 && !emu;
  pl.swap = swap_ab < 0 ? (M <= 64 && N >= 128) : swap_ab != 0;
  if (bn_override >= 10000 && !emu) {
    pl.kind = PLAIN_TILE;
    pl.splits = bn_override / 10000;
    pl.pair = bn_override / 1000 % 10 != 0;
    pl.bn = bn_override % 1000;
    return pl;
  }
  if (bn_override >= 1000 && bn_override < 10000 && pair_ok) {
    pl.kind = PLAIN_FLOW;
    pl.bn = bn_override % 1000;
    pl.rb = bn_override / 1000;
    pl.workers = pairs;
    return pl;
  }
  if (swap_ab < 0 && bn_override <= 0 && pair_ok && std::min(M, N) > 64 && std::max(M, N) > 128) {
    // the whole choice is open: both orientations, every tile width, one wave with K splits or many
    double best = 1e30;
    // the rests that were asked for, no shorter than `limit` where there is no kernel: many tile shapes leave the same one
    struct Rest {
      int at;
      bool cut_n;
      double limit;
      TileChoice tile;
    } rests[2 * 11 * 2 * 2];                         // orientations, tile widths, row blocks, cuts
    int num_rests = 0;
    auto best_rest = [&](int at, bool cut_n, double rest_hbm_us, double limit) {
      Rest* r = std::find_if(rests, rests + num_rests, [&](const Rest& q) { return q.at == at && q.cut_n == cut_n; });
      if (r == rests + num_rests) {
        ++num_rests;
        *r = {at, cut_n, 0.0, {0.0, false, false, 0, 0}};
      }
      if (r->tile.splits == 0 && limit > r->limit) {
        r->limit = limit;
        r->tile = best_tile(d, cut_n ? M : M - at, cut_n ? N - at : N, num_kb, elt, class_a, class_b, rest_hbm_us, true, stats, limit);
      }
      return r->tile;
    };
    if (whole_chip) {
      const TileChoice c = best_tile(d, M, N, num_kb, elt, class_a, class_b, hbm_us, true, stats);
      if (c.splits > 0) {
        best = c.us;
        pl.kind = PLAIN_TILE; pl.swap = c.swap; pl.pair = c.pair; pl.bn = c.bn; pl.splits = c.splits;
      }
    }
    for (int swap = 0; swap < 2; ++swap) {
      const int rows = swap ? N : M, cols = swap ? M : N, cr = swap ? class_b : class_a, cc = swap ? class_a : class_b;
      if (rows <= 128) continue;
      for (int bn = 64, step; bn <= 256; bn += step) {
        step = bn >= 128 ? 16 : 32;
        if (bn > 64 && bn - step >= cols) continue;                  // wider than needed
        for (int rb = 1; rb <= 2; ++rb) {
          if (rb == 2 && rows <= 256) continue;
          // A transposed store writes shorter runs: row-major unless the other way saves something. fp32 operands: both store
          // chunk by chunk, and take longer to the end (334 x 4444 x 1312 14.8 us, the one-wave kernel 13.6).
          const double factor = !swap ? 1.0 : elt == 4 ? 1.03 : ((rows + 256 * rb - 1) / (256 * rb)) * ((cols + bn - 1) / bn) >= 2 * pairs ? 1.05 : 1.08, fp32_us = elt == 4 ? 1.0 : 0.0;
          const double us = flow_us(rows, cols, num_kb, bn, rb, pairs, cr, cc, hbm_us, (best - fp32_us) / factor, stats) * factor + fp32_us;
          if (us < best) {
            best = us;
            pl.kind = PLAIN_FLOW; pl.swap = swap != 0; pl.pair = true; pl.bn = bn; pl.rb = rb; pl.splits = 0; pl.workers = pairs;
            pl.cut = 0;
          }
          if (!whole_chip) continue;
          // Whole waves here, and what is left, cut along K, in a second launch: with 512 x 208 tiles 84 of them on 74
          // pairs (582 x 13976 x 9512, 166 us), or 72 and then 21 tiles of three K ranges each (138 us).
          const int tiles_r = (rows + 256 * rb - 1) / (256 * rb), tiles_c = (cols + bn - 1) / bn, whole = tiles_r * tiles_c / pairs;
          if (whole == 0 || whole > 8) continue;
          const double power = whole >= 3 ? 1 + std::min(0.05, 0.05 * (256 - bn) / 64) : 1.0;
          const double main_us = whole * (num_kb * block_us(bn, rb, cr, cc, bn) * power + (2 * rb * bn <= 512 ? 0.0 : kEpilogueUs)) * factor + kFlowUs;
          if (main_us + kRestUs >= best) continue;
          for (int by_col = 0; by_col < 2; ++by_col) {
            const int strips = whole * pairs / (by_col ? tiles_r : tiles_c);
            if (strips < 1 || strips >= (by_col ? tiles_c : tiles_r)) continue;
            const int at = strips * (by_col ? bn : 256 * rb);
            const bool cut_n = (by_col != 0) != (swap != 0);
            const int m = cut_n ? M : M - at, n = cut_n ? N - at : N;
            // The rest's MMAs on every SM, and its operands' way out of HBM, are the least that it takes.
            const double rest_hbm_us = ((double)m + n) * K * elt / kHbmBytesPerUs;
            const double least = std::max(kBusyFloor * 2 / (kBM * kClocksPerUs) / d->num_sms * m * n * num_kb, rest_hbm_us);
            if (std::max(main_us + least + kRestUs, hbm_us + kFlowUs) * 1.02 >= best) continue;
            const TileChoice c = best_rest(at, cut_n, rest_hbm_us, best / 1.02 - main_us - kRestUs + kTilePairUs);
            const double both = std::max(main_us + c.us - (c.pair ? kTilePairUs : kTileSingleUs) + kRestUs, hbm_us + kFlowUs);
            if (c.splits == 0 || both * 1.02 >= best) continue;      // not for what the model cannot tell
            best = both;
            pl.kind = PLAIN_FLOW; pl.swap = swap != 0; pl.pair = true; pl.bn = bn; pl.rb = rb; pl.splits = 0; pl.workers = pairs;
            pl.cut = at; pl.cut_n = cut_n; pl.rest_swap = c.swap; pl.rest_pair = c.pair; pl.rest_bn = c.bn; pl.rest_splits = c.splits;
          }
        }
      }
    }
    if (best < 1e30) return pl;
  }
  const int rows = pl.swap ? N : M, cols = pl.swap ? M : N;
  pl.bn = bn_override > 0 ? bn_override : (elt == 4 && !(pair_ok && cols > 64) ? tf32_bn(cols) : pick_bn(cols));
  if (pair_ok && pl.bn == 256 && rows >= 256) {
    pl.kind = PLAIN_FLOW;
    pl.workers = pairs;
    return pl;
  }
  if (elt == 4 && pl.bn == 128) pl.bn = 256;
  const int tiles = ((rows + kBM - 1) / kBM) * ((cols + pl.bn - 1) / pl.bn);
  if (swap_ab < 0 && bn_override <= 0 && whole_chip && tiles <= d->num_sms) {
    // up to 64 rows of either operand: one wave with K splits
    const TileChoice c = best_tile(d, M, N, num_kb, elt, class_a, class_b, hbm_us, pair_ok, stats);
    if (c.splits > 0) {
      pl.kind = PLAIN_TILE; pl.swap = c.swap; pl.pair = c.pair; pl.bn = c.bn; pl.splits = c.splits;
      return pl;
    }
  }
  pl.kind = PLAIN_SINGLE;
  pl.workers = std::min(tiles, cap);
  return pl;
}

static thread_local PlanStats plan_stats;

// The plan of a problem, remembered per thread for the shapes a program repeats (a decode step calls the same few again and
// again). Working one out takes 3.8 us of host time on average over 3000 ragged problems of 65 rows and more, 10.3 at the 99th
// percentile, every candidate being bounded from below before its roots and powers are taken; without the bounds 10.0 and 29.3.
static PlainPlan known_plan(const DeviceState* d, int M, int N, int K, int elt, int swap_ab, int bn_override, int use_pair,
                            int max_ctas, long long lda, long long ldb) {
  const int class_a = row_class(lda, elt), class_b = row_class(ldb, elt);
  if (emu_recorder().active) return plain_plan(d, M, N, K, elt, swap_ab, bn_override, use_pair, max_ctas, class_a, class_b, &plan_stats);
  // 512 shapes (43 KB a thread): a server's prompts of many lengths times four projections. Eight to a set, replaced in turn: in a
  // direct-mapped table of 64, 8 of a block's 32 shapes (8 row counts x 4 projections) shared a place, 108 of 128 at 32 counts.
  constexpr int kSets = 64, kWays = 8;
  struct Set {
    int key[kWays][11];
    PlainPlan plan[kWays];
    int next;
  };
  static thread_local Set table[kSets];
  const int key[11] = {M, N, K, 1, d->device, elt, swap_ab, bn_override, use_pair, max_ctas, class_a * 3 + class_b};
  unsigned h = 2166136261u;
  for (int k : key) h = (h ^ (unsigned)k) * 16777619u;
  Set& set = table[(h ^ (h >> 15)) % kSets];
  for (int w = 0; w < kWays; ++w)
    if (memcmp(set.key[w], key, sizeof(key)) == 0) return set.plan[w];
  ++plan_stats.plans;
  const int w = set.next;
  set.next = (w + 1) % kWays;
  set.plan[w] = plain_plan(d, M, N, K, elt, swap_ab, bn_override, use_pair, max_ctas, class_a, class_b, &plan_stats);
  memcpy(set.key[w], key, sizeof(key));
  return set.plan[w];
}

template <int BN, int ELT>
static int launch_plain(const GemmParams& p, unsigned ctas, unsigned threads, cudaStream_t stream) {
  if (emu_recorder().active)
    return emu_record((const void*)gemm_plain_emu_kernel<BN, ELT>, &p, sizeof(p), ctas, threads, GemmCfg<BN>::SMEM);
  void* args[] = {(void*)&p};
  return launch_overlapped((const void*)gemm_plain_kernel<BN, ELT>, ctas, threads, args, GemmCfg<BN>::SMEM, stream);
}

}  // namespace kraken

using namespace kraken;

// What a call with these arguments would run. plan[0..5]: kernel (0 single CTAs, 1 one wave, 2 persistent pairs), weights as
// row operand, column tile, row blocks, K ranges, 1 when in two launches; plan[6..10] of the second launch: first row (column
// when plan[7] is 1) of the output, by column, weights as row operand, column tile, K ranges; plan[11], plan[12]: 1 when the
// one-wave kernel, as all of it or as the second launch, runs in CTA pairs.
KR_API int kr_gemm_plan(int M, int N, int K, long long lda, long long ldb, int in_fp32, int use_pair, int* plan) {
  DeviceState* d = device_state();
  if (!d) return KR_FAIL_CUDA;
  KR_REQUIRE(M >= 1 && N >= 1 && K >= 1, "GEMM needs positive sizes");
  const PlainPlan pl = known_plan(d, M, N, K, in_fp32 ? 4 : 2, -1, 0, use_pair, 0, lda, ldb);
  const int v[13] = {pl.kind, pl.swap, pl.bn, pl.rb, pl.splits, pl.cut > 0, pl.cut, pl.cut_n, pl.rest_swap, pl.rest_bn, pl.rest_splits,
                     pl.kind == PLAIN_TILE && pl.pair, pl.rest_pair};
  memcpy(plan, v, sizeof(v));
  return KR_SUCCESS;
}

// What planning cost the calling thread so far: plans worked out, and kernels whose time was worked out for them.
KR_API int kr_gemm_plan_stats(unsigned long long* plans, unsigned long long* timed) {
  *plans = plan_stats.plans;
  *timed = plan_stats.timed;
  return KR_SUCCESS;
}

// Counter words a call with these arguments needs (0: none).
KR_API int kr_gemm_scratch(int M, int N, int K, long long lda, long long ldb, int in_fp32, int swap_ab, int bn_override, int use_pair, int max_ctas,
                           unsigned long long* counter_words) {
  DeviceState* d = device_state();
  if (!d) return KR_FAIL_CUDA;
  KR_REQUIRE(M >= 1 && N >= 1 && K >= 1, "GEMM needs positive sizes");
  *counter_words = known_plan(d, M, N, K, in_fp32 ? 4 : 2, swap_ab, bn_override, use_pair, max_ctas, lda, ldb).kind == PLAIN_FLOW ? 2 : 0;
  return KR_SUCCESS;
}

// One launch of a call: all of it, or the part that a plan gives to it.
struct PlainCall {
  const void* a;
  long long lda;
  const void* bt;
  long long ldb;
  void* out;
  long long ldo;
  int M, N, K, out_fp32, act, in_fp32;
  uint32_t* counters;
  void* copy_dst;
  cudaStream_t stream;
  int copy_rows;                      // rows of `a` to copy when they are more than M
};
static int run_plain(const DeviceState* d, const PlainPlan& pl, const PlainCall& c, bool rest_follows, bool is_rest) {
  const int M = c.M, N = c.N, K = c.K, out_fp32 = c.out_fp32, act = c.act, in_fp32 = c.in_fp32, elt = in_fp32 ? 4 : 2;
  const long long lda = c.lda, ldb = c.ldb, ldo = c.ldo;
  const void *a = c.a, *bt = c.bt;
  void *out = c.out, *copy_dst = c.copy_dst;
  uint32_t* counters = c.counters;
  cudaStream_t stream = c.stream;
  const bool pair = pl.kind == PLAIN_FLOW || pl.pair;
  GemmParams p;
  memset(&p, 0, sizeof(p));
  int bn = 0;
  CUtensorMap tmap_last;
  const int cols = pl.swap ? M : N, last_cols = pl.bn > 0 ? ((cols - 1) % pl.bn + 16) / 16 * 16 : 0;
  const int narrow = pl.kind == PLAIN_FLOW && last_cols < pl.bn ? last_cols / 2 : 0;
  int rc = setup_problem(p, a, lda, bt, ldb, M, N, K, pl.swap, pl.bn, &bn, elt, pair ? pl.bn / 2 : pl.bn,
                         // Pairs on rows off the 128-byte lines: fetching past the line into L2 only gets in the way there
                         // (777 x 5120 x 13704 153 to 140 us); elsewhere it helps (16 x 8192 x 28672 78.6 to 76.0).
                         !pair || (lda * elt % 128 == 0 && ldb * elt % 128 == 0), narrow, &tmap_last);
  if (rc) return rc;
  p.mode = GEMM_PLAIN;
  p.out = out;
  p.ldo = ldo;
  p.out_rows = M;
  p.out_cols = N;
  p.out_fp32 = out_fp32;
  p.act = act;
  p.ws = 1;
  p.rest_follows = rest_follows;
  p.is_rest = is_rest;
  p.sync = sync_ctx(d);
  if (copy_dst != nullptr) {
    const int copy_rows = c.copy_rows > 0 ? c.copy_rows : M;
    KR_REQUIRE((lda == K || copy_rows == 1) && ((uintptr_t)copy_dst & 15) == 0 && ((unsigned long long)copy_rows * K * elt) % 16 == 0, "the copied operand must be contiguous and 16-byte aligned");
    p.cp_src = a;
    p.cp_dst = copy_dst;
    p.cp_bytes = (unsigned long long)copy_rows * K * elt;
  }
  if (pl.kind == PLAIN_FLOW) return launch_flow_gemm(p, bn, pl.rb, pl.workers, last_cols, tmap_last, counters, stream);
  if (pl.kind == PLAIN_TILE) {
    if (pl.pair) p.tiles_r = (p.rows_r + 255) / 256;
    return launch_tile_gemm(p, bn, pl.pair, pl.splits, stream);
  }
  const unsigned threads = copy_dst != nullptr ? kPlainThreads : kGemmThreads, ctas = (unsigned)pl.workers;
  if (!pl.swap && !out_fp32 && bn >= 64) p.use_tma_store = store_tmap(out, M, N, ldo, &p.tmap_out[0]) ? 1 : 0;
  p.num_mma_ctas = (int)ctas;
  if (in_fp32) {
    switch (bn) {
      case 256: return launch_plain<256, 4>(p, ctas, threads, stream);
      case 64: return launch_plain<64, 4>(p, ctas, threads, stream);
      case 16: return launch_plain<16, 4>(p, ctas, threads, stream);
      default: return fail(KR_FAIL_ARG, "tf32 GEMM supports column tiles of 16, 64 and 256");
    }
  }
  switch (bn) {
    case 256: return launch_plain<256, 2>(p, ctas, threads, stream);
    case 128: return launch_plain<128, 2>(p, ctas, threads, stream);
    case 64: return launch_plain<64, 2>(p, ctas, threads, stream);
    case 32: return launch_plain<32, 2>(p, ctas, threads, stream);
    default: return launch_plain<16, 2>(p, ctas, threads, stream);
  }
}

// out[M,N] (bf16 or fp32, row stride ldo) = act(a[M,K] (row stride lda) * bt[N,K]^T (row stride ldb)).
// act: 0 none, 1 GELU (tanh form), on the fp32 sums.
// swap_ab: -1 auto, 0/1 forced (1: the weights are the row operand).
// bn_override: 0 auto, 16 ... 256 a column tile, 1000 * b + n persistent pairs with b row blocks x n columns, 10000 * s +
// 1000 * p + n the one-wave kernel with s K ranges, single CTAs (p 0) or pairs (p 1) and n columns.
// use_pair: 0 forces the single-CTA kernels, anything else lets eligible shapes use CTA pairs.
// in_fp32: a and bt hold fp32 and are multiplied as tf32 (strides in elements).
// counters: as many zero words as kr_gemm_scratch says for the same arguments (zero again after the call;
// nothing else may use them while it runs), or nullptr: tiles are dealt in fixed shares.
// copy_dst: when not nullptr, receives a copy of a (which then has to be contiguous).
KR_API int kr_gemm(const void* a, long long lda, const void* bt, long long ldb, void* out, long long ldo, int M, int N, int K,
                   int out_fp32, int act, int swap_ab, int bn_override, int max_ctas, int use_pair, int in_fp32,
                   uint32_t* counters, void* copy_dst, cudaStream_t stream) {
  DeviceState* d = device_state();
  if (!d) return KR_FAIL_CUDA;
  KR_REQUIRE(M >= 1 && N >= 1, "GEMM needs positive sizes");
  const int elt = in_fp32 ? 4 : 2;
  PlainPlan pl = known_plan(d, M, N, K, elt, swap_ab, bn_override, use_pair, max_ctas, lda, ldb);
  // One tile whose K is too short to cut: bf16 rows that TMA stores leave the persistent kernel sooner (128 x 128 x 256 3.9 us,
  // the one-wave kernel 4.7); element stores take longer there (100 x 100 x 256 11.5 and 6.4), tiles of 64 columns as long.
  if (pl.kind == PLAIN_TILE && pl.splits == 1 && swap_ab < 0 && bn_override <= 0 && std::min(M, N) > 64 && std::max(M, N) <= 128 && elt == 2 &&
      !out_fp32 && ldo % 8 == 0 && ((uintptr_t)out & 15) == 0 && tma_store_enabled()) {
    pl.kind = PLAIN_SINGLE;
    pl.swap = pl.pair = false;
    pl.bn = 128;
    pl.workers = 1;
  }
  PlainCall c = {a, lda, bt, ldb, out, ldo, M, N, K, out_fp32, act, in_fp32, counters, copy_dst, stream};
  if (pl.cut == 0) return run_plain(d, pl, c, false, false);
  PlainCall rest = c;
  if (pl.cut_n) {
    c.N = pl.cut;
    rest.N -= pl.cut;
    rest.bt = (const char*)bt + (long long)pl.cut * ldb * elt;
    rest.out = (char*)out + (long long)pl.cut * (out_fp32 ? 4 : 2);
  } else {
    c.M = pl.cut;
    rest.M -= pl.cut;
    rest.a = (const char*)a + (long long)pl.cut * lda * elt;
    rest.out = (char*)out + (long long)pl.cut * ldo * (out_fp32 ? 4 : 2);
  }
  rest.counters = nullptr;
  rest.copy_dst = nullptr;
  if (copy_dst != nullptr) c.copy_rows = M;
  int rc = run_plain(d, pl, c, true, false);
  if (rc) return rc;
  pl.kind = PLAIN_TILE;
  pl.swap = pl.rest_swap;
  pl.pair = pl.rest_pair;
  pl.bn = pl.rest_bn;
  pl.splits = pl.rest_splits;
  return run_plain(d, pl, rest, false, true);
}

// The same without counters, activation or copy.
KR_API int kr_gemm_bf16(const void* a, long long lda, const void* bt, long long ldb, void* out, long long ldo, int M,
                        int N, int K, int out_fp32, int swap_ab, int bn_override, int max_ctas, int use_pair,
                        int in_fp32, cudaStream_t stream) {
  return kr_gemm(a, lda, bt, ldb, out, ldo, M, N, K, out_fp32, 0, swap_ab, bn_override, max_ctas, use_pair, in_fp32, nullptr, nullptr, stream);
}
