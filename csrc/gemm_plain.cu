// The plain GEMM C[M,N] = act(A[M,K] * Bt[N,K]^T) on one GPU: what every fused op runs at world size 1
// and fused.matmul everywhere. bf16 operands, or fp32 operands multiplied as tf32; fp32 accumulation;
// bf16 or fp32 result. Kernels: CTA pairs (256 x 256 and 256 x 128 tiles) and single CTAs (128 x 16 ...
// 128 x 256), all persistent, with the tiles of an uneven wave cut along K (stream-K, gemm_core.cuh).
// Optionally four more warps per CTA copy the row operand somewhere else while the tiles are computed
// (the all-gather GEMM at world size 1 returns its gathered operand).
#include <algorithm>
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
template <int BN, int ELT>
__global__ void __launch_bounds__(kPlainThreads, 1)
    gemm_plain_pair_kernel(const __grid_constant__ GemmParams p) {
  extern __shared__ unsigned char smem_raw[];
  PlainHooks h;
  h.bn = BN;
  gemm_mainloop_pair<PlainHooks, BN, ELT>(p, blockIdx.x / 2, gridDim.x / 2, h, smem_raw);
}

// ---- plan -------------------------------------------------------------------------------------
// Which kernel a problem runs on, and how its tiles are dealt. Times in microseconds, from runs of
// this kernel on a B200; only their ratios matter.
struct PlainPlan {
  bool swap;        // the weights (Bt) are the 128-row operand and the tile is stored transposed
  bool pair;
  int bn, tiles_r, tiles_c, num_kb;
  int workers;      // CTAs, or CTA pairs
  int sk_tiles;
  int splits;       // > 0: the one-wave kernel, every tile cut into this many parts along K
  size_t slot_bytes, counters;
};

static size_t sk_slot_bytes(const PlainPlan& pl) {
  return (size_t)2 * pl.workers * (pl.pair ? 2 : 1) * 4 * 32 * pl.bn * 4;
}

// Deals the tiles of `pl` to at most `max_workers` workers. With at least one whole wave, the tiles
// beyond the last whole wave (and one wave more when they are few, so that nobody gets slivers of
// many tiles) are cut along K; with less than a wave all tiles are. Cutting costs a meeting of the
// contributors, so a nearly full last wave stays whole.
static void deal_tiles(PlainPlan& pl, int max_workers, int sk_mode) {
  const int T = pl.tiles_r * pl.tiles_c;
  pl.workers = std::min(T, max_workers);
  pl.sk_tiles = 0;
  // one K block: the MMA (or what the shared-memory port feeds it), or the bytes of all workers from HBM
  const double mma = 0.375 * pl.bn / 256;
  const double load = (128.0 + (pl.pair ? pl.bn / 2 : pl.bn)) * 128 / 90e3;
  auto kb_us = [&](int w) {
    return std::max(std::max(mma, load), (double)w * (pl.pair ? 256 : 128) * 128 / 6.5e6);
  };
  // partial sums out, the count, and the last one's way through the slots
  auto meet_us = [&](double contributors) { return 1.5 + pl.bn / 128.0 * (0.8 + 0.8 * contributors); };
  const int waves = T / max_workers, rest = T % max_workers;
  double best = (double)((T + max_workers - 1) / max_workers) * pl.num_kb * kb_us(pl.workers);
  if (sk_mode == 0 || (rest == 0 && sk_mode < 0)) return;
  auto consider = [&](int tiles, int w) {
    const long long units = (long long)tiles * pl.num_kb;
    if (w > units || w < 2) return;
    const double per = (double)((units + w - 1) / w);
    if (per < 2) return;
    const double whole = (double)((T - tiles) / w) * pl.num_kb;
    const double n = (double)w / tiles + (w % tiles ? 1 : 0);
    double t = (whole + per) * kb_us(w) + meet_us(n);
    if (sk_mode > 0) t *= 1e-3;
    if (t < best) {
      best = t;
      pl.workers = w;
      pl.sk_tiles = tiles;
    }
  };
  if (waves == 0) {
    for (int i = 2; i <= 16 && i * T <= max_workers; ++i) consider(T, i * T);   // every tile in i equal parts
    consider(T, max_workers);
  } else {
    if (rest == 0) return;
    if (2 * rest >= max_workers || sk_mode == 1) consider(rest, max_workers);
    if (2 * rest < max_workers || sk_mode == 2) consider(rest + max_workers, max_workers);
  }
}

static PlainPlan plain_plan(const DeviceState* d, int M, int N, int K, int elt, int swap_ab, int bn_override, int use_pair,
                            int max_ctas, int sk_mode, bool have_scratch) {
  PlainPlan pl;
  memset(&pl, 0, sizeof(pl));
  const bool emu = emu_recorder().active;
  const bool pair_ok = use_pair != 0 && pair_enabled() && !emu;
  const bool free_choice = swap_ab < 0 && bn_override <= 0;
  pl.swap = swap_ab < 0 ? (M <= 64 && N >= 128) : swap_ab != 0;
  // Between one and two row tiles of 128 the tokens fit one 128-column tile of a pair: half the padding
  // of a 256-row tile.
  if (free_choice && pair_ok && M > 64 && M <= 128 && N >= 256) pl.swap = true;
  const int rows = pl.swap ? N : M, cols = pl.swap ? M : N;
  pl.bn = bn_override > 0 ? bn_override : (elt == 4 ? tf32_bn(cols) : pick_bn(cols));
  if (free_choice && pair_ok) {
    pl.pair = cols > 64 && rows > 128;
    if (pl.pair) pl.bn = cols <= 128 ? 128 : 256;
  } else {
    pl.pair = pair_ok && !pl.swap && pl.bn == 256 && rows >= 256;
  }
  const int unit = pl.pair ? 256 : kBM;
  pl.tiles_r = (rows + unit - 1) / unit;
  pl.tiles_c = (cols + pl.bn - 1) / pl.bn;
  pl.num_kb = (K + 128 / elt - 1) / (128 / elt);
  int cap = (int)grid_cap(d);
  if (max_ctas > 0 && max_ctas < cap) cap = max_ctas;
  if (pl.pair && cap < 2) {
    pl.pair = false;
    pl.tiles_r = (rows + kBM - 1) / kBM;
  }
  // An explicit layout is taken as given (its tests compare kernels bit by bit); parts of tiles are
  // summed in another order than whole ones.
  if (emu || (sk_mode < 0 && !free_choice)) sk_mode = 0;
  if ((sk_mode < 0 && max_ctas <= 0) || sk_mode >= 10) {
    pl.splits = tile_gemm_splits(d, pl.tiles_r * pl.tiles_c, pl.num_kb, pl.bn, pl.pair, elt);
    if (sk_mode > 10) pl.splits = std::min(pl.splits, sk_mode - 10);
    if (pl.splits > 0) {
      pl.workers = pl.tiles_r * pl.tiles_c;
      return pl;
    }
  }
  deal_tiles(pl, pl.pair ? cap / 2 : cap, have_scratch ? sk_mode : 0);
  if (pl.sk_tiles > 0) {
    pl.slot_bytes = sk_slot_bytes(pl);
    pl.counters = (size_t)pl.sk_tiles * (pl.pair ? 2 : 1) * 4;
  }
  return pl;
}

// The plan of a problem, remembered per thread for the shapes a program repeats (a decode step calls the
// same few again and again; working a plan out takes about a microsecond).
static const PlainPlan& known_plan(const DeviceState* d, int M, int N, int K, int elt, int swap_ab, int bn_override, int use_pair,
                                   int max_ctas, int sk_mode, bool have_scratch) {
  struct Entry {
    int key[11];
    PlainPlan plan;
  };
  static thread_local Entry table[64];
  const int key[11] = {1, d->device, M, N, K, elt, swap_ab, bn_override, use_pair, max_ctas, sk_mode * 2 + (have_scratch ? 1 : 0)};
  unsigned h = 2166136261u;
  for (int k : key) h = (h ^ (unsigned)k) * 16777619u;
  Entry& e = table[(h ^ (h >> 15)) % 64];
  if (emu_recorder().active || memcmp(e.key, key, sizeof(key)) != 0) {
    e.plan = plain_plan(d, M, N, K, elt, swap_ab, bn_override, use_pair, max_ctas, sk_mode, have_scratch);
    memcpy(e.key, key, sizeof(key));
    if (emu_recorder().active) e.key[0] = 0;       // an emulated launch is planned for fewer CTAs
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
template <int BN, int ELT>
static int launch_plain_pair(const GemmParams& p, unsigned ctas, unsigned threads, cudaStream_t stream) {
  void* args[] = {(void*)&p};
  return launch_overlapped((const void*)gemm_plain_pair_kernel<BN, ELT>, ctas, threads, args, PairCfgT<BN>::SMEM, stream, 2);
}

}  // namespace kraken

using namespace kraken;

// Scratch a call with these arguments needs: bytes of partial-sum slots (0: none) and counter words.
KR_API int kr_gemm_scratch(int M, int N, int K, int in_fp32, int swap_ab, int bn_override, int use_pair, int max_ctas,
                           int sk_mode, unsigned long long* slot_bytes, unsigned long long* counter_words) {
  DeviceState* d = device_state();
  if (!d) return KR_FAIL_CUDA;
  KR_REQUIRE(M >= 1 && N >= 1 && K >= 1, "GEMM needs positive sizes");
  const PlainPlan& pl = known_plan(d, M, N, K, in_fp32 ? 4 : 2, swap_ab, bn_override, use_pair, max_ctas, sk_mode, true);
  *slot_bytes = pl.slot_bytes;
  *counter_words = pl.counters;
  return KR_SUCCESS;
}

// out[M,N] (bf16 or fp32, row stride ldo) = act(a[M,K] (row stride lda) * bt[N,K]^T (row stride ldb)).
// act: 0 none, 1 GELU (tanh form), on the fp32 sums.
// swap_ab: -1 auto (weights on the 128-row side when M <= 64), 0/1 forced.
// use_pair: 0 forces the single-CTA kernel, anything else lets eligible shapes use CTA pairs.
// in_fp32: a and bt hold fp32 and are multiplied as tf32 (strides in elements).
// sk_mode: -1 auto, 0 whole tiles only, 1 / 2 forced. slots / counters: scratch as kr_gemm_scratch
// says for the same arguments (counters zero, zero again after the call; nothing else may use either
// while the call runs), or nullptr: whole tiles only.
// copy_dst: when not nullptr, receives a copy of a (which then has to be contiguous).
KR_API int kr_gemm(const void* a, long long lda, const void* bt, long long ldb, void* out, long long ldo, int M, int N, int K,
                   int out_fp32, int act, int swap_ab, int bn_override, int max_ctas, int use_pair, int in_fp32, int sk_mode,
                   void* slots, unsigned long long slot_bytes, uint32_t* counters, unsigned long long counter_words,
                   void* copy_dst, cudaStream_t stream) {
  DeviceState* d = device_state();
  if (!d) return KR_FAIL_CUDA;
  KR_REQUIRE(M >= 1 && N >= 1, "GEMM needs positive sizes");
  const int elt = in_fp32 ? 4 : 2;
  // a problem that needs no scratch has the same plan with and without
  PlainPlan pl = known_plan(d, M, N, K, elt, swap_ab, bn_override, use_pair, max_ctas, sk_mode, true);
  if (pl.sk_tiles > 0 && (slots == nullptr || counters == nullptr))
    pl = known_plan(d, M, N, K, elt, swap_ab, bn_override, use_pair, max_ctas, sk_mode, false);
  KR_REQUIRE(slot_bytes >= pl.slot_bytes && counter_words >= pl.counters, "GEMM scratch too small");
  GemmParams p;
  memset(&p, 0, sizeof(p));
  int bn = 0;
  int rc = setup_problem(p, a, lda, bt, ldb, M, N, K, pl.swap, pl.bn, &bn, elt, pl.pair ? pl.bn / 2 : pl.bn);
  if (rc) return rc;
  if (in_fp32) KR_REQUIRE(bn == 16 || bn == 64 || bn == 256 || pl.splits > 0 || (pl.pair && bn == 128), "tf32 GEMM supports column tiles of 16, 64 and 256");
  p.mode = GEMM_PLAIN;
  p.out = out;
  p.ldo = ldo;
  p.out_rows = M;
  p.out_cols = N;
  p.out_fp32 = out_fp32;
  p.act = act;
  p.ws = 1;
  p.sync = sync_ctx(d);
  p.sk_tiles = pl.sk_tiles;
  p.sk_slots = (float*)slots;
  p.sk_counters = counters;
  if (copy_dst != nullptr) {
    KR_REQUIRE(lda == K && ((uintptr_t)copy_dst & 15) == 0 && ((unsigned long long)M * K * elt) % 16 == 0, "the copied operand must be contiguous and 16-byte aligned");
    p.cp_src = a;
    p.cp_dst = copy_dst;
    p.cp_bytes = (unsigned long long)M * K * elt;
  }
  const unsigned threads = copy_dst != nullptr ? kPlainThreads : kGemmThreads;
  if (!pl.swap && !out_fp32 && bn >= 64) p.use_tma_store = store_tmap(out, M, N, ldo, &p.tmap_out[0]) ? 1 : 0;
  if (pl.splits > 0) {
    p.tiles_r = pl.tiles_r;
    return launch_tile_gemm(p, bn, pl.pair, pl.splits, stream);
  }
  const unsigned ctas = (unsigned)pl.workers * (pl.pair ? 2 : 1);
  p.num_mma_ctas = (int)ctas;
  if (pl.pair) {
    p.tiles_r = pl.tiles_r;
    p.group_r = std::max(1, p.group_r / 2);
    if (in_fp32) return bn == 128 ? launch_plain_pair<128, 4>(p, ctas, threads, stream) : launch_plain_pair<256, 4>(p, ctas, threads, stream);
    return bn == 128 ? launch_plain_pair<128, 2>(p, ctas, threads, stream) : launch_plain_pair<256, 2>(p, ctas, threads, stream);
  }
  if (in_fp32) {
    switch (bn) {
      case 256: return launch_plain<256, 4>(p, ctas, threads, stream);
      case 64: return launch_plain<64, 4>(p, ctas, threads, stream);
      default: return launch_plain<16, 4>(p, ctas, threads, stream);
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

// The same without scratch, activation or copy: whole tiles only.
KR_API int kr_gemm_bf16(const void* a, long long lda, const void* bt, long long ldb, void* out, long long ldo, int M,
                        int N, int K, int out_fp32, int swap_ab, int bn_override, int max_ctas, int use_pair,
                        int in_fp32, cudaStream_t stream) {
  return kr_gemm(a, lda, bt, ldb, out, ldo, M, N, K, out_fp32, 0, swap_ab, bn_override, max_ctas, use_pair, in_fp32, -1, nullptr, 0,
                 nullptr, 0, nullptr, stream);
}
