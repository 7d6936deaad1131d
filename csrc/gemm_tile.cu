// One-wave GEMM: every CTA (or CTA pair) computes ONE output tile, or one of `splits` equal K ranges of
// it, and the splits of a tile form a thread-block cluster that sums them through distributed shared
// memory. For the problems whose tiles do not fill the chip once — decode batches above all, where the
// time is the weights' way out of HBM and a tile per CTA leaves most SMs idle.
//
//   C[M,N] = act(A[M,K] * Bt[N,K]^T), bf16 operands or fp32 multiplied as tf32, fp32 sums in K order
//   (split by split), bf16 or fp32 result.
//
// Why clusters and not partial sums in global memory: a 256 x 256 tile split in two costs 15-18 us there
// (slots out to L2, an atomic, slots back in: measured with %globaltimer stamps) and about 1.5 us here.
//
// The sums are SENT: every CTA owns an equal share of the tile's rows, and the others store their partial sums of it
// straight from registers into its shared memory (st.async, counted on an mbarrier of the owner; the operand stages are
// free by then). The owner adds them in split order and stores its rows. One cluster barrier, whose latency the first
// read of the accumulator hides, says that the stages are free; nothing follows the stores. The other order was: own
// shared memory, cluster barrier, owners fetch, cluster barrier before anybody may leave, and the places of a thread's rows
// worked out here. With the plans of either, us a call in a graph of them, then and now: 8 x 4096 x 4096 9.3, 8.7;
// 35 x 4064 x 5416 13.7, 11.5; 102 x 1240 x 2816 8.5, 5.9; 100 x 4000 x 9000 21.4, 20.0. What bounds this part now is the
// way between SMs: 64 KB leave an SM in 2700 clocks (24 bytes each; bulk copies 3400, plain remote stores and a barrier
// 4200, fetches 3900), whatever the cluster size.
#include <algorithm>
#include <atomic>
#include <cmath>
#include "kraken/gemm_host.h"

namespace kraken {

constexpr int kTileThreads = 320;      // TMA warp, MMA warp, eight warps that empty the accumulator

struct alignas(64) TileParams {
  CUtensorMap tmap_r, tmap_c;
  int tiles_r, tiles_c, num_kb;
  int transposed, out_fp32, act, is_rest;
  int out_rows, out_cols;
  void* out;
  long long ldo;
  const void* cp_src;                  // optional copy of the row operand, as in gemm_plain.cu
  void* cp_dst;
  unsigned long long cp_bytes;
  SyncCtx sync;
};

template <int BN, bool PAIR>
struct TileCfg {
  static constexpr int A_BYTES = kBM * 128;
  static constexpr int B_BYTES = (PAIR ? BN / 2 : BN) * 128;
  static constexpr int B_BYTES_AL = (B_BYTES + 1023) / 1024 * 1024;
  static constexpr int STAGE = A_BYTES + B_BYTES_AL;
  static constexpr int RAW_STAGES = (kSmemLimit - 1024 - 512) / STAGE;
  static constexpr int STAGES = RAW_STAGES > 12 ? 12 : RAW_STAGES;
  static constexpr int TMEM_COLS = BN <= 32 ? 32 : BN <= 64 ? 64 : BN <= 128 ? 128 : 256;
  static constexpr int SMEM = 1024 + STAGES * STAGE + 512;
  // what arrives for the largest share: 48 rows of three pairs, 32 rows of seven CTAs, or 128 of one
  static_assert(BN / 4 * (PAIR ? 3 * 49 : 7 * 33) * 16 <= STAGES * STAGE && BN / 4 * 129 * 16 <= STAGES * STAGE, "the sums have to fit the stages");
};

__device__ __forceinline__ float4 ld_shared_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
// 16 bytes into the shared memory of a CTA of the cluster, counted on an mbarrier there.
__device__ __forceinline__ void push_cluster_u4(uint32_t addr, uint32_t bar, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1,%2,%3,%4}, [%5];"
               ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d), "r"(bar) : "memory");
}
// Relaxed: what it announces are this CTA's copies and MMAs, which mbarriers have shown to be over, and no store of the
// thread (with release semantics the arrival took 500 clocks).
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}

// Until all partial sums of this CTA's share are here. Longer than any other wait of the cluster can take, recorded
// error or not: who leaves early is written to after it has left.
__device__ __forceinline__ void wait_sums(uint32_t bar, const SyncCtx& c) {
  const uint64_t t0 = globaltimer_ns();
  while (!mbar_try_wait(bar, 0))
    if (globaltimer_ns() - t0 > 4 * c.timeout_ns + 50 * kMbarGraceNs) {
      set_status(c, make_status(KR_ERR_TIMEOUT_MBAR, 83, 0, blockIdx.x));
      return;
    }
}

// The rows of a CTA's 128 x BN part of the tile that split k sums and stores: groups of 16 rows (whole 32-byte
// sectors of a transposed bf16 store), as even as eight groups go.
__device__ __forceinline__ int share_begin(int k, int splits) { return (8 * k + splits - 1) / splits * 16; }

template <int BN, int ELT, bool PAIR>
__global__ void __launch_bounds__(kTileThreads, 1) gemm_tile_kernel(const __grid_constant__ TileParams p) {
  using Cfg = TileCfg<BN, PAIR>;
  constexpr int kStageK = 128 / ELT;
  constexpr uint32_t CTAS = PAIR ? 2 : 1;
  extern __shared__ unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank(), csize = cluster_size();
  const uint32_t half = PAIR ? (rank & 1u) : 0u;           // which CTA of the pair
  const bool leader = half == 0;
  const int split = (int)(rank / CTAS), splits = (int)(csize / CTAS);
  const int tile = (int)(blockIdx.x / csize);
  // consecutive tiles share the column operand of a column sweep
  const int tr2 = tile % p.tiles_r, tc = tile / p.tiles_r;
  const int tr = PAIR ? 2 * tr2 + (int)half : tr2;
  const int kb_lo = (int)((long long)p.num_kb * split / splits), kb_hi = (int)((long long)p.num_kb * (split + 1) / splits);

  const uint32_t stage0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t bars = stage0 + Cfg::STAGES * Cfg::STAGE;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (Cfg::STAGES + s); };
  const uint32_t done_bar = bars + 8u * (2 * Cfg::STAGES);
  const uint32_t sum_bar = done_bar + 8, tmem_slot = done_bar + 16;

  // Shares of this CTA's part of the tile. A split's partial sums arrive at the owner of a row as 16-byte units of
  // four columns, [split][unit][row]: what a warp sends is contiguous. Units past the output are not sent.
  const int valid_cols = (p.transposed ? p.out_rows : p.out_cols) - tc * BN;
  const int units = min(BN, valid_cols + 3) / 4;
  const int row_lo = share_begin(split, splits), rows = share_begin(split + 1, splits) - row_lo;
  const uint32_t unit_bytes = (uint32_t)rows * 16u + 16u;      // a row of padding against bank conflicts
  const int valid_rows = (p.transposed ? p.out_cols : p.out_rows) - tr * kBM;
  const int rows_left = min(max(valid_rows - row_lo, 0), rows);   // of the share; rows past the output are not sent either

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(done_bar, 1);
    mbar_init(sum_bar, 1 + kTileThreads / 32 - 2);
    mbar_fence_init();
    mbar_expect_tx(sum_bar, (uint32_t)((splits - 1) * units * rows_left) * 16u);
    tma_prefetch_desc(&p.tmap_r);
    tma_prefetch_desc(&p.tmap_c);
  }
  if (warp == 1) {
    if (PAIR) { tmem_alloc_pair(tmem_slot, Cfg::TMEM_COLS); tmem_relinquish_pair(); }
    else { tmem_alloc(tmem_slot, Cfg::TMEM_COLS); tmem_relinquish(); }
  }
  tc_fence_before();
  if (PAIR) cluster_sync_all();      // both CTAs' barriers exist before anyone signals across the pair
  else __syncthreads();
  tc_fence_after();
  uint32_t tmem_base;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));
  pdl_launch();
  if (p.is_rest == 0) pdl_wait();

  // Worked out now, while nothing waits for it (the divisions took 300 clocks of the tail): where this thread's row of the
  // accumulator goes, and which of the sums it stores first.
  constexpr int CH = BN < 32 ? BN : 32;                    // two warps per TMEM lane quarter take turns
  const int q = warp & 3, h = (warp - 2) >> 2, acc_row = q * 32 + lane;
  const int to = acc_row / 16 * splits / 8, to_lo = share_begin(to, splits);
  uint32_t to_bytes = (uint32_t)(share_begin(to + 1, splits) - to_lo) * 16u + 16u;
  const uint32_t to_rank = (uint32_t)to * CTAS + half;
  const uint32_t slot = (uint32_t)(split * units) * to_bytes + (uint32_t)(acc_row - to_lo) * 16u;
  uint32_t dst = to == split ? stage0 + slot : mapa_shared(stage0, to_rank) + slot, dst_bar = mapa_shared(sum_bar, to_rank);
  const int groups = (units + 1) / 2;                      // of eight columns
  const int items = p.transposed ? groups * rows : rows_left * groups, per = p.transposed ? rows : groups;
  int hi = (int)threadIdx.x / per, lo = (int)threadIdx.x - hi * per;
  asm volatile("" : "+r"(to_bytes), "+r"(dst), "+r"(dst_bar), "+r"(hi), "+r"(lo));

  if (warp == 0) {
    if (elect_one()) {
      int s = 0;
      uint32_t ph = 0;
      for (int kb = kb_lo; kb < kb_hi; ++kb) {
        if (!mbar_wait(empty_bar(s), ph ^ 1u, p.sync, 80)) break;
        const uint32_t sa = stage0 + s * Cfg::STAGE;
        if (PAIR) {
          const uint32_t lead_full = mapa_shared(full_bar(s), rank & ~1u);
          if (leader) mbar_expect_tx(full_bar(s), 2 * (Cfg::A_BYTES + Cfg::B_BYTES));
          tma_load_2d_pair(sa, &p.tmap_r, lead_full, kb * kStageK, tr * kBM);
          tma_load_2d_pair(sa + Cfg::A_BYTES, &p.tmap_c, lead_full, kb * kStageK, tc * BN + (int)half * (BN / 2));
        } else {
          mbar_expect_tx(full_bar(s), Cfg::A_BYTES + Cfg::B_BYTES);
          tma_load_2d(sa, &p.tmap_r, full_bar(s), kb * kStageK, tr * kBM);
          tma_load_2d(sa + Cfg::A_BYTES, &p.tmap_c, full_bar(s), kb * kStageK, tc * BN);
        }
        if (++s == Cfg::STAGES) { s = 0; ph ^= 1u; }
      }
    }
  } else if (warp == 1) {
    if (leader && elect_one()) {
      constexpr int UM = PAIR ? 256 : 128;
      constexpr uint32_t idesc = ELT == 2 ? make_idesc_bf16(UM, BN) : make_idesc_tf32(UM, BN);
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int kb = kb_lo; kb < kb_hi; ++kb) {
        ok = mbar_wait(full_bar(s), ph, p.sync, 81);
        if (!ok) break;
        tc_fence_after();
        const uint32_t sa = stage0 + s * Cfg::STAGE;
        const uint64_t adesc = make_smem_desc_sw128(sa), bdesc = make_smem_desc_sw128(sa + Cfg::A_BYTES);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t accumulate = (kb > kb_lo || k != 0) ? 1u : 0u;
          const uint64_t a = adesc + (uint64_t)(2 * k), b = bdesc + (uint64_t)(2 * k);
          if (PAIR) {
            if (ELT == 2) umma_bf16_pair(tmem_base, a, b, idesc, accumulate);
            else umma_tf32_pair(tmem_base, a, b, idesc, accumulate);
          } else {
            if (ELT == 2) umma_bf16(tmem_base, a, b, idesc, accumulate);
            else umma_tf32(tmem_base, a, b, idesc, accumulate);
          }
        }
        if (PAIR) {
          umma_commit_pair(empty_bar(s));
          umma_commit_pair(mapa_shared(empty_bar(s), rank | 1u));
        } else {
          umma_commit(empty_bar(s));
        }
        if (++s == Cfg::STAGES) { s = 0; ph ^= 1u; }
      }
      if (ok) {
        if (PAIR) {
          umma_commit_pair(done_bar);
          umma_commit_pair(mapa_shared(done_bar, rank | 1u));
        } else {
          umma_commit(done_bar);
        }
      }
    }
  } else {
    if (p.cp_bytes != 0) {
      // the copy of the row operand: this CTA's share, by the eight warps that have nothing to do yet
      const size_t nvec = p.cp_bytes / 16, lo = nvec * blockIdx.x / gridDim.x, hi = nvec * (blockIdx.x + 1) / gridDim.x;
      constexpr int T = kTileThreads - 64;
      size_t v = lo + threadIdx.x - 64;
      for (; v + 7 * T < hi; v += 8 * T) {
        U4 x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = ld16((const char*)p.cp_src + (v + (size_t)i * T) * 16);
#pragma unroll
        for (int i = 0; i < 8; ++i) st16((char*)p.cp_dst + (v + (size_t)i * T) * 16, x[i]);
      }
      for (; v < hi; v += T) st16((char*)p.cp_dst + v * 16, ld16((const char*)p.cp_src + v * 16));
    }
    mbar_wait(done_bar, 0, p.sync, 82);      // what a wait that ran out leaves is sent all the same: the others count on it
  }
  __syncwarp();
  tc_fence_after();
  // From here on this CTA's stages are free for what the others send. Nobody waits for more than that: the sums are
  // sent, not fetched, and whoever has them all stores and leaves.
  if (csize > 1) cluster_arrive();
  if (warp >= 2) {
    bool waited = csize == 1;
#pragma unroll 1
    for (int c0 = h * CH; c0 < units * 4; c0 += 2 * CH) {
      uint32_t r[32];
      const uint32_t t_addr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)c0;
      if (CH == 32) tmem_ld32(t_addr, r);
      else tmem_ld16(t_addr, r);
      tmem_ld_wait();
      if (!waited) cluster_wait();
      waited = true;
#pragma unroll
      for (int u = 0; u < CH / 4; ++u) {
        if (c0 / 4 + u >= units || acc_row >= valid_rows) continue;
        const uint32_t a = dst + (uint32_t)(c0 / 4 + u) * to_bytes;
        if (to == split) st_shared_u4(a, r[4 * u], r[4 * u + 1], r[4 * u + 2], r[4 * u + 3]);
        else push_cluster_u4(a, dst_bar, r[4 * u], r[4 * u + 1], r[4 * u + 2], r[4 * u + 3]);
      }
    }
    if (!waited) cluster_wait();
    __syncwarp();
    if (lane == 0) mbar_arrive(sum_bar);
  } else if (csize > 1) {
    cluster_wait();
  }
  __syncwarp();
  wait_sums(sum_bar, p.sync);

  // ---- sum over the splits, in order, and store
  const bool fp32 = p.out_fp32 != 0, act = p.act != 0, vec_ok = (p.ldo * (fp32 ? 4 : 2)) % 16 == 0 && ((uintptr_t)p.out & 15) == 0;
  const uint32_t split_bytes = (uint32_t)units * unit_bytes;
  auto unit_addr = [&](int unit, int row) { return stage0 + (uint32_t)unit * unit_bytes + (uint32_t)row * 16u; };
  // two units at a time: the loads of a split are in flight together
  auto sum_units = [&](uint32_t a, uint32_t b, float (&v)[8]) {
    float4 x = ld_shared_f4(a), y = ld_shared_f4(b);
#pragma unroll 1
    for (int k = 1; k < splits; ++k) {
      const float4 s = ld_shared_f4(a += split_bytes), t = ld_shared_f4(b += split_bytes);
      x = make_float4(x.x + s.x, x.y + s.y, x.z + s.z, x.w + s.w);
      y = make_float4(y.x + t.x, y.y + t.y, y.z + t.z, y.w + t.w);
    }
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
  };
#pragma unroll 1
  for (int e = (int)threadIdx.x; e < items;) {
    const int u = (p.transposed ? hi : lo) * 2, i = p.transposed ? lo : hi;
    float v[8];
    sum_units(unit_addr(u, i), unit_addr(min(u + 1, units - 1), i), v);
    if (act) {
#pragma unroll
      for (int c = 0; c < 8; ++c) v[c] = gelu_tanh(v[c]);
    }
    const int left = valid_cols - u * 4;                   // of the eight columns, those inside the output
    if (p.transposed) {
      // D(i, j) -> out[tc*BN + j][tr*128 + i]; lanes = consecutive i
      const long long o = (long long)(tc * BN + u * 4) * p.ldo + tr * kBM + row_lo + i;
      if (i < rows_left) {
        if (fp32) {
          float* out = (float*)p.out + o;
#pragma unroll
          for (int c = 0; c < 8; ++c, out += p.ldo)
            if (c < left) *out = v[c];
        } else {
          __nv_bfloat16* out = (__nv_bfloat16*)p.out + o;
#pragma unroll
          for (int c = 0; c < 8; ++c, out += p.ldo)
            if (c < left) *out = __float2bfloat16(v[c]);
        }
      }
    } else {
      // D(i, j) -> out[tr*128 + i][tc*BN + j]; lanes = consecutive groups of eight columns
      const long long o = (long long)(tr * kBM + row_lo + i) * p.ldo + tc * BN + u * 4;
      if (vec_ok && left >= 8) {
        if (fp32) {
          float* out = (float*)p.out + o;
          st16(out, U4{__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3])});
          st16(out + 4, U4{__float_as_uint(v[4]), __float_as_uint(v[5]), __float_as_uint(v[6]), __float_as_uint(v[7])});
        } else {
          st16((__nv_bfloat16*)p.out + o, pack8(v));
        }
      } else {
#pragma unroll
        for (int c = 0; c < 8; ++c)
          if (c < left) {
            if (fp32) ((float*)p.out)[o + c] = v[c];
            else ((__nv_bfloat16*)p.out)[o + c] = __float2bfloat16(v[c]);
          }
      }
    }
    if ((e += kTileThreads) < items) {
      hi = e / per;
      lo = e - hi * per;
    }
  }
  // Everything sent to this CTA has arrived, and who it sent to is still waiting for that: a single CTA may leave. The
  // CTAs of a pair give back their tensor memory together.
  tc_fence_before();
  if (PAIR) cluster_sync_all();
  else __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    if (PAIR) tmem_dealloc_pair(tmem_base, Cfg::TMEM_COLS);
    else tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
  // The rest of a problem starts when all blocks of the launch before it run and have seen their own predecessor
  // complete, reads what they read, writes other rows or columns, and is complete no sooner than they are.
  if (p.is_rest != 0) pdl_wait();
}

// ---- host ---------------------------------------------------------------------------------------
struct TileVariant {
  const void* fn;
  size_t smem;
};
template <int ELT>
static TileVariant tile_variant(int bn, bool pair) {
  if (pair) {
    switch (bn) {
      case 128: return {(const void*)gemm_tile_kernel<128, ELT, true>, TileCfg<128, true>::SMEM};
      case 160: return {(const void*)gemm_tile_kernel<160, ELT, true>, TileCfg<160, true>::SMEM};
      case 192: return {(const void*)gemm_tile_kernel<192, ELT, true>, TileCfg<192, true>::SMEM};
      case 224: return {(const void*)gemm_tile_kernel<224, ELT, true>, TileCfg<224, true>::SMEM};
      case 256: return {(const void*)gemm_tile_kernel<256, ELT, true>, TileCfg<256, true>::SMEM};
      default: return {nullptr, 0};
    }
  }
  switch (bn) {
    case 128: return {(const void*)gemm_tile_kernel<128, ELT, false>, TileCfg<128, false>::SMEM};
    case 16: return {(const void*)gemm_tile_kernel<16, ELT, false>, TileCfg<16, false>::SMEM};
    case 32: return {(const void*)gemm_tile_kernel<32, ELT, false>, TileCfg<32, false>::SMEM};
    case 64: return {(const void*)gemm_tile_kernel<64, ELT, false>, TileCfg<64, false>::SMEM};
    default: return {nullptr, 0};
  }
}

// How many clusters of `cluster` CTAs of this kernel the device holds at once (asked once; 0: none).
static int max_clusters(int device, const TileVariant& v, int elt, int bn, bool pair, unsigned cluster) {
  constexpr int kDevices = 16;
  static std::atomic<int> known[kDevices][2][2][17][9];        // answer + 1
  std::atomic<int>* slot = device < kDevices ? &known[device][elt == 4][pair][bn / 16][cluster] : nullptr;
  if (slot != nullptr)
    if (const int n = slot->load(std::memory_order_relaxed)) return n - 1;
  int n = 0;
  if (ensure_dynamic_smem(v.fn, v.smem) == KR_SUCCESS) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(cluster);
    cfg.blockDim = dim3(kTileThreads);
    cfg.dynamicSmemBytes = v.smem;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, v.fn, &cfg) != cudaSuccess) {
      (void)cudaGetLastError();
      n = 0;
    }
  }
  if (slot != nullptr) slot->store(n + 1, std::memory_order_relaxed);
  return n;
}

// The split count with which a one-wave problem takes less than *us, and its time there; 0 when there is none or its tiles do
// not fit the chip at once. kb_us: one K block with every SM busy (less when fewer are, the clock being what power leaves; not
// so for single CTAs of up to 64 columns). Near the operands' time out of HBM (hbm_us) the two slow each other down (norm of order 4). Then the partial
// sums' way between SMs (44 KB a us and SM); clusters of six CTAs and more start later.
int tile_gemm_splits(const DeviceState* d, int tiles, int num_kb, int bn, bool pair, int elt, double kb_us, double hbm_us,
                     double* us, PlanStats* stats) {
  const TileVariant v = elt == 4 ? tile_variant<4>(bn, pair) : tile_variant<2>(bn, pair);
  if (v.fn == nullptr) return 0;
  const int ctas = pair ? 2 : 1, most = 8 / ctas;
  const bool powered = pair || bn > 64;
  const double start_us = pair ? kTilePairUs : kTileSingleUs;
  // Most problems are asked for in vain, so whatever costs (roots and powers, 20 ns each) comes after a bound that does not.
  const int room = std::min(most, d->num_sms / (tiles * ctas));
  if (room < 1 || std::max((powered ? kBusyFloor : 1.0) * kb_us * num_kb / room, hbm_us) + start_us >= *us) return 0;
  int best = 0;
  for (int s = 1; s <= room && (s == 1 || num_kb >= 4 * s); ++s) {
    if (tiles > max_clusters(d->device, v, elt, bn, pair, (unsigned)(s * ctas))) continue;
    const double all_busy = (num_kb + s - 1) / s * kb_us, sent = (double)(s - 1) / s * kBM * bn * 4;
    const double ends = sent / 44500 + start_us + (pair && s >= 3 ? 0.5 : 0.0);
    if (std::max(powered ? kBusyFloor * all_busy : all_busy, hbm_us) + ends >= *us) continue;
    ++stats->timed;
    const double busy = (double)tiles * s * ctas / d->num_sms;
    const double blocks = all_busy * (powered ? busy_factor(busy) : 1.0), b2 = blocks * blocks, h2 = hbm_us * hbm_us;
    // (unsplit pairs: the persistent kernel stores bf16 rows faster, 636 x 4080 x 3152 29 us against 33; fp32 does not, 500 x
    // 4000 x 4000 34.6 against 29.4)
    const double t = std::sqrt(std::sqrt(b2 * b2 + h2 * h2)) * (pair && s == 1 && elt == 2 ? 1.05 : 1.0) + ends;
    if (t < *us) {
      *us = t;
      best = s;
    }
  }
  return best;
}

int launch_tile_gemm(const GemmParams& g, int bn, bool pair, int splits, cudaStream_t stream) {
  const TileVariant v = g.in_fp32 ? tile_variant<4>(bn, pair) : tile_variant<2>(bn, pair);
  const int num_kb = (g.K + (g.in_fp32 ? 32 : 64) - 1) / (g.in_fp32 ? 32 : 64);
  if (v.fn == nullptr || (pair && bn % 32 != 0)) return fail(KR_FAIL_ARG, "no one-wave kernel of this tile width");
  if (splits < 1 || splits * (pair ? 2 : 1) > 8 || splits > num_kb) return fail(KR_FAIL_ARG, "no such number of K ranges");
  TileParams p;
  p.tmap_r = g.tmap_r;
  p.tmap_c = g.tmap_c;
  p.tiles_r = g.tiles_r;
  p.tiles_c = g.tiles_c;
  p.num_kb = num_kb;
  p.transposed = g.transposed;
  p.out_fp32 = g.out_fp32;
  p.act = g.act;
  p.is_rest = g.is_rest;
  p.out_rows = g.out_rows;
  p.out_cols = g.out_cols;
  p.out = g.out;
  p.ldo = g.ldo;
  p.cp_src = g.cp_src;
  p.cp_dst = g.cp_dst;
  p.cp_bytes = g.cp_bytes;
  p.sync = g.sync;
  const unsigned cluster = (unsigned)splits * (pair ? 2 : 1);
  void* args[] = {(void*)&p};
  return launch_overlapped(v.fn, (unsigned)(g.tiles_r * g.tiles_c) * cluster, kTileThreads, args, v.smem, stream, cluster);
}

}  // namespace kraken
