// The plain GEMM C[M,N] = act(A[M,K] * Bt[N,K]^T) on one GPU: what every fused op runs at world size 1
// and fused.matmul everywhere. bf16 operands, or fp32 operands multiplied as tf32; fp32 accumulation;
// bf16 or fp32 result. This file picks among three kernel families and launches:
//   tile    one wave, a tile or a K range of it per CTA or pair (gemm_tile.cu)
//   flow    persistent pairs that draw tiles in order (gemm_flow.cu)
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
};

// Where the rows of an operand start: 0 on 128-byte lines, 1 on 32-byte sectors, 2 in the middle of sectors
// (a row length of an odd number of 16-byte units): each 128 bytes then cost a fifth sector.
static int row_class(long long ld, int elt) { return ld * elt % 128 == 0 ? 0 : ld * elt % 32 == 0 ? 1 : 2; }

// Time model of the pair kernels, in microseconds, fitted to runs of every tile shape and split on 35 ragged and 4
// aligned problems on a B200 (it picks within 5 % of the best on average): per K block (64 bf16 or 32 fp32
// columns of K) 0.284 for the MMAs of 256 x 256 and a price per KB of operands that a CTA fetches, by the class
// of their rows (4096 x 4096 x 9512 against x 9472: 256 x 256 tiles 308 / 256 us, 512 x 256 266 / 249).
static double block_us(int bn, int rb, int class_r, int class_c) {
  static const double kPerKb[3] = {0.0035, 0.0051, 0.0105};
  // Two row blocks: fewer and larger stages in flight, which shows while the fetches are not what bounds the block
  // (2048 x 3584 x 8192: 512 x 224 tiles in one wave 90-100 us, 256 x 208 in two 86-92).
  const double two = rb == 2 && class_r < 2 && class_c < 2 ? 1.045 : 1.0;
  return (0.284 * rb * bn / 256 + kPerKb[class_r] * 16 * rb + kPerKb[class_c] * bn / 16.0) * two;
}

static double flow_us(int rows, int cols, int num_kb, int bn, int rb, int pairs, int class_r, int class_c, double hbm_us) {
  const int T = ((rows + 256 * rb - 1) / (256 * rb)) * ((cols + bn - 1) / bn);
  const int whole = T / pairs, rest = T % pairs;
  const double full = num_kb * block_us(bn, rb, class_r, class_c);
  double last = rest ? full * busy_factor((double)rest / pairs) : 0.0;
  if (rb == 2 && rest && 2 * rest <= pairs) last = num_kb * block_us(bn, 1, class_r, class_c) * busy_factor(2.0 * rest / pairs);
  // what is not hidden: start and last epilogue, and with one accumulator set the epilogue of every tile
  const double bubble = 2 * rb * bn <= 512 ? 0.0 : 3.2;
  return std::max(whole * (full + bubble) + last, hbm_us) + 6.3;
}

static PlainPlan plain_plan(const DeviceState* d, int M, int N, int K, int elt, int swap_ab, int bn_override, int use_pair,
                            int max_ctas, int class_a, int class_b) {
  PlainPlan pl;
  memset(&pl, 0, sizeof(pl));
  pl.rb = 1;
  const bool emu = emu_recorder().active;
  int cap = (int)grid_cap(d);
  if (max_ctas > 0 && max_ctas < cap) cap = max_ctas;
  const bool pair_ok = use_pair != 0 && pair_enabled() && !emu && cap >= 2;
  const int num_kb = (K + 128 / elt - 1) / (128 / elt), pairs = cap / 2;
  const double hbm_us = ((double)M + N) * K * elt / 5e6;         // with the rate that short kernels reach
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
    for (int swap = 0; swap < 2; ++swap) {
      const int rows = swap ? N : M, cols = swap ? M : N, cr = swap ? class_b : class_a, cc = swap ? class_a : class_b;
      if (rows <= 128) continue;
      if (whole_chip && cols <= 128) {
        // single CTAs of 128 x 128: up to eight K splits (100 x 4000 x 9000 21 us, with pairs 27)
        const int tiles = (rows + kBM - 1) / kBM;
        const double single_us = 1.06 * (0.142 + 2 * (block_us(128, 1, cr, cc) - 0.142) / 1.5);      // 32 KB a stage, not 24
        double us = 1e30;
        const int s = tiles <= d->num_sms ? tile_gemm_splits(d, tiles, num_kb, 128, false, elt, single_us, hbm_us, &us) : 0;
        if (s > 0 && us < best) {
          best = us;
          pl.kind = PLAIN_TILE; pl.swap = swap != 0; pl.pair = false; pl.bn = 128; pl.splits = s; pl.rb = 1;
        }
      }
      for (int bn = 64, step; bn <= 256; bn += step) {
        step = bn >= 128 && elt == 2 ? 16 : 32;
        if (bn > 64 && bn - step >= cols) continue;                  // wider than needed
        if (whole_chip && bn >= 128 && bn % 32 == 0) {
          const int tiles = ((rows + 255) / 256) * ((cols + bn - 1) / bn);
          double us = 1e30;
          const int s = tiles <= pairs ? tile_gemm_splits(d, tiles, num_kb, bn, true, elt, block_us(bn, 1, cr, cc), hbm_us, &us) : 0;
          if (s > 0 && us < best) {
            best = us;
            pl.kind = PLAIN_TILE; pl.swap = swap != 0; pl.pair = true; pl.bn = bn; pl.splits = s;
          }
        }
        for (int rb = 1; rb <= 2; ++rb) {
          if (rb == 2 && rows <= 256) continue;
          // a transposed store writes shorter runs: row-major unless the other way saves something
          const double us = flow_us(rows, cols, num_kb, bn, rb, pairs, cr, cc, hbm_us) * (swap ? 1.056 : 1.0);
          if (us < best) {
            best = us;
            pl.kind = PLAIN_FLOW; pl.swap = swap != 0; pl.pair = true; pl.bn = bn; pl.rb = rb; pl.splits = 0; pl.workers = pairs;
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
    pl.splits = tile_gemm_splits(d, tiles, num_kb, pl.bn, false, elt, 0.25, hbm_us, nullptr);
    if (pl.splits > 0) {
      pl.kind = PLAIN_TILE;
      return pl;
    }
  }
  pl.kind = PLAIN_SINGLE;
  pl.workers = std::min(tiles, cap);
  return pl;
}

// The plan of a problem, remembered per thread for the shapes a program repeats (a decode step calls the
// same few again and again; working a plan out takes microseconds).
static PlainPlan known_plan(const DeviceState* d, int M, int N, int K, int elt, int swap_ab, int bn_override, int use_pair,
                            int max_ctas, long long lda, long long ldb) {
  const int class_a = row_class(lda, elt), class_b = row_class(ldb, elt);
  struct Entry {
    int key[11];
    PlainPlan plan;
  };
  static thread_local Entry table[64];
  if (emu_recorder().active) return plain_plan(d, M, N, K, elt, swap_ab, bn_override, use_pair, max_ctas, class_a, class_b);
  const int key[11] = {1, d->device, M, N, K, elt, swap_ab, bn_override, use_pair, max_ctas, class_a * 3 + class_b};
  unsigned h = 2166136261u;
  for (int k : key) h = (h ^ (unsigned)k) * 16777619u;
  Entry& e = table[(h ^ (h >> 15)) % 64];
  if (memcmp(e.key, key, sizeof(key)) != 0) {
    e.plan = plain_plan(d, M, N, K, elt, swap_ab, bn_override, use_pair, max_ctas, class_a, class_b);
    memcpy(e.key, key, sizeof(key));
  }
  return e.plan;
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

// Counter words a call with these arguments needs (0: none).
KR_API int kr_gemm_scratch(int M, int N, int K, long long lda, long long ldb, int in_fp32, int swap_ab, int bn_override, int use_pair, int max_ctas,
                           unsigned long long* counter_words) {
  DeviceState* d = device_state();
  if (!d) return KR_FAIL_CUDA;
  KR_REQUIRE(M >= 1 && N >= 1 && K >= 1, "GEMM needs positive sizes");
  *counter_words = known_plan(d, M, N, K, in_fp32 ? 4 : 2, swap_ab, bn_override, use_pair, max_ctas, lda, ldb).kind == PLAIN_FLOW ? 2 : 0;
  return KR_SUCCESS;
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
  const PlainPlan pl = known_plan(d, M, N, K, elt, swap_ab, bn_override, use_pair, max_ctas, lda, ldb);
  const bool pair = pl.kind == PLAIN_FLOW || pl.pair;
  GemmParams p;
  memset(&p, 0, sizeof(p));
  int bn = 0;
  CUtensorMap tmap_last;
  const int cols = pl.swap ? M : N, last_cols = pl.bn > 0 ? ((cols - 1) % pl.bn + 16) / 16 * 16 : 0;
  const int narrow = pl.kind == PLAIN_FLOW && last_cols < pl.bn ? last_cols / 2 : 0;
  int rc = setup_problem(p, a, lda, bt, ldb, M, N, K, pl.swap, pl.bn, &bn, elt, pair ? pl.bn / 2 : pl.bn,
                         // Persistent pairs on rows off the 128-byte lines: fetching past the line into L2 only gets in the
                         // way there (777 x 5120 x 13704 153 to 140 us); elsewhere it helps (16 x 8192 x 28672 78.6 to 76.0).
                         pl.kind != PLAIN_FLOW || (lda * elt % 128 == 0 && ldb * elt % 128 == 0), narrow, &tmap_last);
  if (rc) return rc;
  p.mode = GEMM_PLAIN;
  p.out = out;
  p.ldo = ldo;
  p.out_rows = M;
  p.out_cols = N;
  p.out_fp32 = out_fp32;
  p.act = act;
  p.ws = 1;
  p.sync = sync_ctx(d);
  if (copy_dst != nullptr) {
    KR_REQUIRE(lda == K && ((uintptr_t)copy_dst & 15) == 0 && ((unsigned long long)M * K * elt) % 16 == 0, "the copied operand must be contiguous and 16-byte aligned");
    p.cp_src = a;
    p.cp_dst = copy_dst;
    p.cp_bytes = (unsigned long long)M * K * elt;
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

// The same without counters, activation or copy.
KR_API int kr_gemm_bf16(const void* a, long long lda, const void* bt, long long ldb, void* out, long long ldo, int M,
                        int N, int K, int out_fp32, int swap_ab, int bn_override, int max_ctas, int use_pair,
                        int in_fp32, cudaStream_t stream) {
  return kr_gemm(a, lda, bt, ldb, out, ldo, M, N, K, out_fp32, 0, swap_ab, bn_override, max_ctas, use_pair, in_fp32, nullptr, nullptr, stream);
}
