// The plain GEMM for problems of a wave of tiles and more: persistent CTA pairs that draw their tiles from a
// counter, C[M,N] = act(A[M,K] * Bt[N,K]^T) with bf16 operands or fp32 multiplied as tf32.
//
// What bounds it: a B200 runs long GEMMs at its power limit (1.3-1.5 GHz), so besides feeding the tensor
// cores what counts is the data moved per operation. Two choices follow.
//  * Tiles are handed out in order, one atomic per tile. With a fixed share per pair the pairs drift apart (some
//    run 5 % slower), the tiles in flight stop sharing operands and HBM reads more than double: 8192 x 8192
//    x 14336 read 3.98 GB with fixed shares, 1.98 GB in order (ncu, dram__bytes_read.sum).
//  * RB = 2 row blocks: a pair computes 512 x 256, each operand stage feeds twice the MMAs (48 KB instead of 64
//    per CTA and 256 x 256 x 64 block pair). The accumulators then fill TMEM, so a tile's first MMAs wait for the
//    epilogue of the one before, row block by row block. RB = 1 keeps two accumulators in turn.
// Column tiles (BN) of 64 ... 256, in steps of 16 from 128 on, fit ragged sizes and waves; the launcher picks.
// The last column tile is as narrow as the output leaves it (16s), and a pair draws its next tile shortly before the end of
// the one in hand: drawn at its start, the last tiles of 777 x 5120 x 13704 (256 columns, three wide and one narrow tile per
// row of tiles) went to the pairs with the wide ones (172 us, now 141), those of 522 x 6156 x 4440 (tf32) as well (88, 73).
// (1000 x 4096 x 4096 in fp32: 240 columns 50.7 us, 256 columns 52.7; 404 x 5196 x 6084: 144 columns 69.1, 160 71.9.)
//
// Warps: 0 TMA producer (the leader's also draws the tiles), 1 MMA issuer (leader), 2-5 epilogue (one per TMEM
// lane quarter), 6-7 optional copy of the row operand. The common epilogues (MODE) are kernels of their own: with
// every store form in one kernel its unrolled code pushed the other roles' loops out of the instruction cache
// (8192 x 8192 x 3584 372 us against 366).
#include <algorithm>
#include "kraken/gemm_host.h"

namespace kraken {

constexpr int kFlowEpiWarps = 4;
constexpr int kFlowThreads = 64 + 32 * kFlowEpiWarps;
constexpr int kFlowCopyThreads = 64;
constexpr int kFlowSlots = 16;                            // more than the slowest role can be behind the producer, see next_item

struct alignas(64) FlowParams {
  CUtensorMap tmap_r, tmap_c, tmap_last, tmap_out, tmap_tail;      // tmap_tail: the last 16 columns of tiles with BN % 32 == 16
  int last_cols;                                          // columns of the last column tile, in 16s (tmap_last: boxes of half as many rows)
  int tiles_r, tiles_c, num_kb, group_r;                  // tiles of RB * 256 rows
  int items, split_from;                                  // tiles from split_from on are drawn as single row blocks
  int transposed, out_fp32, act, rest_follows;
  int out_rows, out_cols;
  uint32_t* sched;                                        // [0] items drawn beyond the first of each pair, [1] pairs done; or nullptr
  void* out;                                              // output without a tensor map (else nullptr) and its row stride
  long long ldo;
  const void* cp_src;
  void* cp_dst;
  unsigned long long cp_bytes;
  SyncCtx sync;
};

template <int BN, int RB>
struct FlowCfg {
  static constexpr int A_BYTES = kBM * 128;               // one row block of this CTA
  static constexpr int B_BYTES = BN / 2 * 128;
  static constexpr int STAGE = RB * A_BYTES + B_BYTES;
  static constexpr int EPI = kFlowEpiWarps * 8192;       // two panel slots per warp
  static constexpr int RAW_STAGES = (kSmemLimit - 1024 - EPI - 512) / STAGE;
  static constexpr int STAGES = RAW_STAGES > 8 ? 8 : RAW_STAGES;
  static constexpr int UNIT = (BN + 31) / 32 * 32;        // TMEM columns of an accumulator: read in chunks of 32
  static constexpr int BUFS = 2 * RB * UNIT <= 512 ? 2 : 1;
  static constexpr int UNITS = BUFS * RB;                 // accumulators
  static constexpr int TMEM_COLS = UNITS * UNIT <= 256 ? 256 : 512;
  static constexpr int SMEM = 1024 + STAGES * STAGE + EPI + 512;
  static_assert(BN % 16 == 0 && BN >= 64 && BN <= 256 && UNITS <= 4 && STAGES >= 3, "tile shape");
  static_assert(16 * STAGES + 16 * UNITS + 12 * kFlowSlots + 8 <= 512, "barrier area");
  static_assert(STAGES + BUFS + 2 < kFlowSlots, "a role could be lapped");
};

// One word into the shared memory of a CTA of the cluster, counted on an mbarrier there: whoever has waited for
// that phase sees the word. No fence at either end (a release / acquire pair at cluster scope per tile and
// role cost 0.8 us of every tile).
__device__ __forceinline__ void publish_cluster_u32(uint32_t addr, uint32_t bar, uint32_t v) {
  asm volatile("mbarrier.arrive.expect_tx.relaxed.cluster.shared::cluster.b64 _, [%0], 4;" ::"r"(bar) : "memory");
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.u32 [%0], %1, [%2];" ::"r"(addr), "r"(v), "r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t ld_shared_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}

struct FlowItem {
  int tr, tc, rb_lo, rb_hi;      // tile coordinates and the row blocks of it
};
template <int RB>
__device__ __forceinline__ FlowItem flow_item(const FlowParams& p, int t) {
  FlowItem it;
  int tile = t;
  it.rb_lo = 0;
  it.rb_hi = RB;
  if (RB == 2 && t >= p.split_from) {
    tile = p.split_from + ((t - p.split_from) >> 1);
    it.rb_lo = (t - p.split_from) & 1;
    it.rb_hi = it.rb_lo + 1;
  }
  const int per_group = p.group_r * p.tiles_c, g = tile / per_group, first = g * p.group_r;
  const int gsz = min(p.group_r, p.tiles_r - first), in = tile - g * per_group;
  it.tr = first + in % gsz;
  it.tc = in / gsz;
  return it;
}

enum FlowMode : int { FLOW_ROWS = 0, FLOW_ROWS_ACT = 1, FLOW_ANY = 2 };     // bf16 row-major through TMA; with GELU; anything

template <int BN, int RB, int ELT, int MODE>
__global__ void __launch_bounds__(kFlowThreads + kFlowCopyThreads, 1) gemm_flow_kernel(const __grid_constant__ FlowParams p) {
  using Cfg = FlowCfg<BN, RB>;
  constexpr int kStageK = 128 / ELT;
  extern __shared__ unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cta = cluster_ctarank();
  const bool leader = cta == 0;
  const int pair = (int)(blockIdx.x >> 1), pairs = (int)(gridDim.x >> 1);
  const uint32_t stage0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t epi0 = stage0 + Cfg::STAGES * Cfg::STAGE;
  const uint32_t bars = epi0 + Cfg::EPI;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (Cfg::STAGES + s); };
  auto tfull_bar = [&](int u) { return bars + 8u * (2 * Cfg::STAGES + u); };
  auto tempty_bar = [&](int u) { return bars + 8u * (2 * Cfg::STAGES + Cfg::UNITS + u); };
  const uint32_t sfull = bars + 8u * (2 * Cfg::STAGES + 2 * Cfg::UNITS), sdata = sfull + 8u * kFlowSlots;
  const uint32_t tmem_slot = sdata + 4u * kFlowSlots;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int u = 0; u < Cfg::UNITS; ++u) {
      mbar_init(tfull_bar(u), 1);
      mbar_init(tempty_bar(u), 2 * kFlowEpiWarps);
    }
    for (int k = 0; k < kFlowSlots; ++k) mbar_init(sfull + 8u * k, 1);
    mbar_fence_init();
    tma_prefetch_desc(&p.tmap_r);
    tma_prefetch_desc(&p.tmap_c);
    tma_prefetch_desc(&p.tmap_last);
    tma_prefetch_desc(&p.tmap_out);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();            // both CTAs' barriers exist before anyone signals across the pair
  tc_fence_after();
  const uint32_t tmem_base = ld_shared_u32(tmem_slot);
  // With a second launch for the rest of the problem, that one relies on the operands as this one does: it may only
  // start once they are there.
  if (p.rest_follows == 0) pdl_launch();
  pdl_wait();
  if (p.rest_follows != 0) pdl_launch();

  // A staged panel of `rows` x `cols` to an output that TMA cannot describe (rows not whole 16-byte
  // units) or may not store to (KRAKEN_TMA_STORE=0), element by element.
  auto store_plain = [&](uint32_t panel, int gx, int gy, int cols, int rows, bool fp32, int ln) {
    const int elt = fp32 ? 4 : 2, pitch = cols * elt;
    for (int r = 0; r < rows && gy + r < p.out_rows; ++r) {
      const int perm = pitch == 128 ? (r & 7) : pitch == 64 ? ((r >> 1) & 3) : 0;
      for (int c = ln; c < cols && gx + c < p.out_cols; c += 32) {
        const uint32_t a = panel + (uint32_t)(r * pitch + ((((c * elt) >> 4) ^ perm) << 4) + ((c * elt) & 15));
        const long long o = (long long)(gy + r) * p.ldo + gx + c;
        if (fp32) {
          ((uint32_t*)p.out)[o] = ld_shared_u32(a);
        } else {
          unsigned short v;
          asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
          ((unsigned short*)p.out)[o] = v;
        }
      }
    }
    __syncwarp();
  };

  // The item after item k of this pair, as the leader's producer published it. The slots need no "free" signal:
  // the producer is at most STAGES items ahead of the MMA issuer (one stage per item at least), which is at
  // most BUFS + 1 ahead of the epilogue.
  auto next_item = [&](int k, bool warp_wide, int& t) {
    const uint32_t slot = (uint32_t)(k % kFlowSlots);
    bool ok = mbar_wait(sfull + 8u * slot, (uint32_t)(k / kFlowSlots) & 1u, p.sync, 91);
    if (warp_wide) ok = __all_sync(0xffffffffu, ok);
    t = ok ? (int)ld_shared_u32(sdata + 4u * slot) : p.items;
    return ok;
  };

  if (warp == 0) {
    // ================= TMA producer (both CTAs) =================
    if (elect_one()) {
      // One thread has 130 ns a K block of 256 x 128 x 64: what does not change is kept out of the loop.
      const uint32_t lead_full0 = mapa_shared(full_bar(0), 0);
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      int t = pair;
      for (int k = 0; ok && t < p.items; ++k) {
        int drawn = 0;
        // Drawn shortly before the end of this tile, so that the pair that is done first takes it, and published a few
        // K blocks on, when the atomic has returned: the peer's producer goes on to the next tile without a gap.
        // Without a counter every pair takes its fixed share.
        const int draw_kb = max(0, p.num_kb - 10), publish_kb = max(min(3, p.num_kb - 1), p.num_kb - 4);
        const FlowItem it = flow_item<RB>(p, t);
        const int cols = it.tc + 1 == p.tiles_c ? p.last_cols : BN;
        const CUtensorMap* const map_c = it.tc + 1 == p.tiles_c ? &p.tmap_last : &p.tmap_c;
        const uint32_t bytes = 2u * (uint32_t)((it.rb_hi - it.rb_lo) * Cfg::A_BYTES + cols * 64);
        const int row0 = it.tr * (RB * 256) + (int)cta * kBM, col0 = it.tc * BN + (int)cta * (cols / 2);
        auto load_blocks = [&](int kb, int end) {
          for (; kb < end; ++kb) {
            ok = mbar_wait(empty_bar(s), ph ^ 1u, p.sync, 92);
            if (!ok) return;
            const uint32_t lead_full = lead_full0 + 8u * s, sa = stage0 + s * Cfg::STAGE;
            if (leader) mbar_expect_tx(full_bar(s), bytes);           // both CTAs' bytes complete on the leader's barrier
#pragma unroll
            for (int rb = 0; rb < RB; ++rb)
              if (RB == 1 || (rb >= it.rb_lo && rb < it.rb_hi))
                tma_load_2d_pair(sa + rb * Cfg::A_BYTES, &p.tmap_r, lead_full, kb * kStageK, row0 + rb * 256);
            tma_load_2d_pair(sa + RB * Cfg::A_BYTES, map_c, lead_full, kb * kStageK, col0);
            if (++s == Cfg::STAGES) { s = 0; ph ^= 1u; }
          }
        };
#pragma unroll 1
        for (int part = 0; ok && part < 3; ++part) {
          load_blocks(part == 0 ? 0 : part == 1 ? draw_kb : publish_kb + 1, part == 0 ? draw_kb : part == 1 ? publish_kb + 1 : p.num_kb);
          if (leader && part == 0) drawn = p.sched != nullptr ? (int)atomicAdd(p.sched, 1u) + pairs : t + pairs;
          if (leader && ok && part == 1) {
            // to both CTAs, even past the end (that is how the other roles learn of it)
            const uint32_t slot = (uint32_t)(k % kFlowSlots);
#pragma unroll
            for (uint32_t c = 0; c < 2; ++c)
              publish_cluster_u32(mapa_shared(sdata + 4u * slot, c), mapa_shared(sfull + 8u * slot, c), (uint32_t)drawn);
          }
        }
        if (leader) t = drawn;
        else ok = next_item(k, false, t) && ok;
      }
      if (leader && p.sched != nullptr) {
        // the last pair puts the counter back for the next launch on this stream (failed waits lead here as well)
        const uint32_t done = atom_add_acqrel_gpu(p.sched + 1, 1u);
        if (done == (uint32_t)pairs - 1u) {
          p.sched[0] = 0;
          p.sched[1] = 0;
        }
      }
    }
  } else if (warp == 1) {
    // ================= MMA issuer (leader CTA only) =================
    if (leader && elect_one()) {
      const uint32_t peer_empty0 = mapa_shared(empty_bar(0), 1);
      const uint64_t desc0 = make_smem_desc_sw128(stage0);
      int s = 0;
      uint32_t ph = 0, uph = 0;                            // uph: one phase bit per accumulator
      bool ok = true;
      int t = pair;
      for (int k = 0; ok && t < p.items; ++k) {
        const FlowItem it = flow_item<RB>(p, t);
        const int cols = it.tc + 1 == p.tiles_c ? p.last_cols : BN;
        const uint32_t idesc = ELT == 2 ? make_idesc_bf16(256, cols) : make_idesc_tf32(256, cols);
        const int u0 = Cfg::BUFS == 2 ? (k & 1) * RB : 0;
        for (int kb = 0; kb < p.num_kb; ++kb) {
          ok = mbar_wait(full_bar(s), ph, p.sync, 94);
          if (!ok) break;
          tc_fence_after();
          const uint64_t sdesc = desc0 + (uint64_t)(s * (Cfg::STAGE >> 4)), bdesc = sdesc + (uint64_t)(RB * Cfg::A_BYTES >> 4);
#pragma unroll
          for (int rb = 0; rb < RB; ++rb) {
            if (RB > 1 && (rb < it.rb_lo || rb >= it.rb_hi)) continue;
            const int u = u0 + rb;
            if (kb == 0) {
              ok = mbar_wait(tempty_bar(u), ((uph >> u) & 1u) ^ 1u, p.sync, 95) && ok;
              tc_fence_after();
            }
            const uint64_t adesc = sdesc + (uint64_t)(rb * Cfg::A_BYTES >> 4);
            const uint32_t d_tmem = tmem_base + (uint32_t)(u * Cfg::UNIT);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint32_t accumulate = (kb > 0 || i != 0) ? 1u : 0u;
              if (ELT == 2) umma_bf16_pair(d_tmem, adesc + (uint64_t)(2 * i), bdesc + (uint64_t)(2 * i), idesc, accumulate);
              else umma_tf32_pair(d_tmem, adesc + (uint64_t)(2 * i), bdesc + (uint64_t)(2 * i), idesc, accumulate);
            }
            if (kb == p.num_kb - 1) {
              umma_commit_pair(tfull_bar(u));
              umma_commit_pair(mapa_shared(tfull_bar(u), 1));
            }
          }
          if (!ok) break;
          umma_commit_pair(empty_bar(s));
          umma_commit_pair(peer_empty0 + 8u * s);
          if (++s == Cfg::STAGES) { s = 0; ph ^= 1u; }
        }
        for (int rb = it.rb_lo; rb < it.rb_hi; ++rb) uph ^= 1u << (u0 + rb);
        ok = next_item(k, false, t) && ok;
      }
    }
  } else if (warp < 2 + kFlowEpiWarps) {
    // ================= epilogue (both CTAs, own 128 rows of each block) =================
    const int q = warp & 3;                                // TMEM lane quarter
    const uint32_t slots = epi0 + (uint32_t)(warp - 2) * 8192u;
    constexpr int PW = BN % 64 == 0 ? 64 : 32;             // columns per panel of a bf16 row-major tile
    constexpr int CHUNKS = Cfg::UNIT / 32;
    constexpr bool TAIL = BN % 32 != 0;                    // the last chunk is 16 columns wide
    const bool fp32 = MODE == FLOW_ANY && p.out_fp32 != 0, transposed = MODE == FLOW_ANY && p.transposed != 0;
    const bool act = MODE == FLOW_ANY && p.act != 0;
    uint32_t uph = 0, sent = 0;
    bool ok = true;
    int t = pair;
    for (int k = 0; ok && t < p.items; ++k) {
      const FlowItem it = flow_item<RB>(p, t);
      const int u0 = Cfg::BUFS == 2 ? (k & 1) * RB : 0;
#pragma unroll 1
      for (int rb = it.rb_lo; rb < it.rb_hi && ok; ++rb) {
        const int u = u0 + rb;
        ok = mbar_wait(tfull_bar(u), (uph >> u) & 1u, p.sync, 96);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        uph ^= 1u << u;
        tc_fence_after();
        const uint32_t t_addr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(u * Cfg::UNIT);
        const int drow = it.tr * (RB * 256) + rb * 256 + (int)cta * kBM + q * 32;      // first row of D of this warp
        auto release = [&] {      // this warp has read its part of the accumulator
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(mapa_shared(tempty_bar(u), 0));
        };
        // The slot for the next panel, once the store that last read it (two panels ago) is done with it
        auto next_slot = [&] {
          if (lane == 0) bulk_wait_group_read<1>();
          __syncwarp();
          return slots + (sent++ & 1u) * 4096u;
        };
        // A panel in a slot goes out: rows gy ..., columns gx ... of the output
        auto send = [&](uint32_t slot, int gx, int gy, int cols, int rows, bool tail) {
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if ((MODE != FLOW_ANY || p.out == nullptr) && gx < p.out_cols && gy < p.out_rows) tma_store_2d(tail ? &p.tmap_tail : &p.tmap_out, slot, gx, gy);
            bulk_commit_group();
          }
          if (MODE == FLOW_ANY && p.out != nullptr) store_plain(slot, gx, gy, cols, rows, fp32, lane);
        };
        if (MODE == FLOW_ANY && (fp32 || transposed || act)) {
#pragma unroll 1
          for (int i = 0; i < CHUNKS; ++i) {
            const int col = i * 32;
            const bool tail = TAIL && i + 1 == CHUNKS;
            uint32_t r[32];
            tmem_ld32(t_addr + (uint32_t)col, r);
            tmem_ld_wait();
            if (i + 1 == CHUNKS) release();
            if (act) {
#pragma unroll
              for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(gelu_tanh(__uint_as_float(r[j])));
            }
            const uint32_t slot = next_slot();
            if (transposed) {
              // panel row j = column col + j of D; lanes = consecutive output columns
              if (fp32) {
#pragma unroll
                for (int j = 0; j < 32; ++j)
                  asm volatile("st.shared.u32 [%0], %1;" ::"r"(slot + j * 128u + (uint32_t)((((lane >> 2) ^ (j & 7)) << 4) + (lane & 3) * 4)), "r"(r[j]) : "memory");
              } else {
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                  const __nv_bfloat16 v = __float2bfloat16(__uint_as_float(r[j]));
                  asm volatile("st.shared.u16 [%0], %1;" ::"r"(slot + j * 64u + (uint32_t)((((lane >> 3) ^ ((j >> 1) & 3)) << 4) + (lane & 7) * 2)),
                               "h"(*reinterpret_cast<const unsigned short*>(&v)) : "memory");
                }
              }
              send(slot, drow, it.tc * BN + col, 32, tail ? 16 : 32, tail);
            } else if (!fp32) {
#pragma unroll
              for (int v = 0; v < 4; ++v) {
                if (tail && v >= 2) continue;
                uint32_t w[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) w[j] = pack_bf16x2(__uint_as_float(r[8 * v + 2 * j]), __uint_as_float(r[8 * v + 2 * j + 1]));
                const uint32_t a = tail ? slot + lane * 32u + v * 16u : slot + lane * 64u + (uint32_t)((v ^ ((lane >> 1) & 3)) << 4);
                st_shared_u4(a, w[0], w[1], w[2], w[3]);
              }
              send(slot, it.tc * BN + col, drow, tail ? 16 : 32, 32, tail);
            } else {
#pragma unroll
              for (int v = 0; v < 8; ++v) {
                if (tail && v >= 4) continue;
                const uint32_t a = tail ? slot + lane * 64u + (uint32_t)((v ^ ((lane >> 1) & 3)) << 4) : slot + lane * 128u + (uint32_t)((v ^ (lane & 7)) << 4);
                st_shared_u4(a, r[4 * v], r[4 * v + 1], r[4 * v + 2], r[4 * v + 3]);
              }
              send(slot, it.tc * BN + col, drow, tail ? 16 : 32, 32, tail);
            }
          }
        } else {
          // bf16 rows: everything is read, activated (on the fp32 sums) and rounded before anything is stored, so
          // that the next tile's MMAs do not wait for stores. With an activation 16 columns at a time: more raw
          // sums next to the rounded ones would spill. Releasing the accumulator before the activation would take
          // rounded sums (8192 x 28672 x 8192: 2868 us against 2895, two row blocks; with two accumulators no gain).
          uint32_t packed[CHUNKS][16];
          if (MODE == FLOW_ROWS_ACT) {
#pragma unroll
            for (int i = 0; i < BN / 16; ++i) {
              uint32_t raw[32];
              tmem_ld16(t_addr + (uint32_t)(i * 16), raw);
              tmem_ld_wait();
#pragma unroll
              for (int v = 0; v < 8; ++v)
                packed[i / 2][i % 2 * 8 + v] = pack_bf16x2(gelu_tanh(__uint_as_float(raw[2 * v])), gelu_tanh(__uint_as_float(raw[2 * v + 1])));
            }
          } else {
#pragma unroll
            for (int i = 0; i < CHUNKS; i += 2) {
              uint32_t r0[32], r1[32];
              tmem_ld32(t_addr + (uint32_t)(i * 32), r0);
              if (i + 1 < CHUNKS) tmem_ld32(t_addr + (uint32_t)(i * 32 + 32), r1);
              tmem_ld_wait();
#pragma unroll
              for (int v = 0; v < 16; ++v) {
                packed[i][v] = pack_bf16x2(__uint_as_float(r0[2 * v]), __uint_as_float(r0[2 * v + 1]));
                if (i + 1 < CHUNKS) packed[i + 1 < CHUNKS ? i + 1 : i][v] = pack_bf16x2(__uint_as_float(r1[2 * v]), __uint_as_float(r1[2 * v + 1]));
              }
            }
          }
          release();
          uint32_t slot = 0;
#pragma unroll
          for (int i = 0; i < CHUNKS; ++i) {
            if (PW == 32 || (i & 1) == 0) slot = next_slot();
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              const bool tail = TAIL && i + 1 == CHUNKS;
              if (tail && v >= 2) continue;
              const uint32_t a = tail ? slot + lane * 32u + v * 16u : PW == 64 ? slot + lane * 128u + (uint32_t)((((i & 1) * 4 + v) ^ (lane & 7)) << 4)
                                          : slot + lane * 64u + (uint32_t)((v ^ ((lane >> 1) & 3)) << 4);
              st_shared_u4(a, packed[i][4 * v], packed[i][4 * v + 1], packed[i][4 * v + 2], packed[i][4 * v + 3]);
            }
            if (TAIL && i + 1 == CHUNKS) send(slot, it.tc * BN + i * 32, drow, 16, 32, true);
            else if (PW == 32) send(slot, it.tc * BN + i * 32, drow, 32, 32, false);
            else if ((i & 1) == 1) send(slot, it.tc * BN + i * 32 - 32, drow, 64, 32, false);
          }
        }
      }
      if (ok) ok = next_item(k, true, t);
    }
    if (lane == 0) bulk_wait_group<0>();
  } else if (p.cp_bytes != 0) {
    // ================= copy of the row operand: this CTA's share =================
    const size_t nvec = p.cp_bytes / 16, lo = nvec * blockIdx.x / gridDim.x, hi = nvec * (blockIdx.x + 1) / gridDim.x;
    size_t v = lo + threadIdx.x - kFlowThreads;
    for (; v + 7 * kFlowCopyThreads < hi; v += 8 * kFlowCopyThreads) {
      U4 x[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = ld16((const char*)p.cp_src + (v + (size_t)i * kFlowCopyThreads) * 16);
#pragma unroll
      for (int i = 0; i < 8; ++i) st16((char*)p.cp_dst + (v + (size_t)i * kFlowCopyThreads) * 16, x[i]);
    }
    for (; v < hi; v += kFlowCopyThreads) st16((char*)p.cp_dst + v * 16, ld16((const char*)p.cp_src + v * 16));
  }
  __syncwarp();

  // ---- teardown: nobody leaves while the pair may still touch its shared memory or barriers
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, Cfg::TMEM_COLS);
  }
}

// ---- host ---------------------------------------------------------------------------------------
struct FlowVariant {
  const void* fn;
  size_t smem;
};
template <int ELT, int MODE>
static FlowVariant flow_variant(int bn, int rb) {
#define KR_FLOW(BN, RB) \
  if (bn == BN && rb == RB) return {(const void*)gemm_flow_kernel<BN, RB, ELT, MODE>, FlowCfg<BN, RB>::SMEM};
  KR_FLOW(256, 2)
  KR_FLOW(224, 2)
  KR_FLOW(192, 2)
  KR_FLOW(160, 2)
  KR_FLOW(128, 2)
  KR_FLOW(96, 2)
  KR_FLOW(64, 2)
  KR_FLOW(256, 1)
  KR_FLOW(224, 1)
  KR_FLOW(192, 1)
  KR_FLOW(160, 1)
  KR_FLOW(128, 1)
  KR_FLOW(96, 1)
  KR_FLOW(64, 1)
  KR_FLOW(240, 2)
  KR_FLOW(208, 2)
  KR_FLOW(176, 2)
  KR_FLOW(144, 2)
  KR_FLOW(240, 1)
  KR_FLOW(208, 1)
  KR_FLOW(176, 1)
  KR_FLOW(144, 1)
#undef KR_FLOW
  return {nullptr, 0};
}

int launch_flow_gemm(const GemmParams& g, int bn, int rb, int pairs, int last_cols, const CUtensorMap& tmap_last, uint32_t* sched,
                     cudaStream_t stream) {
  const bool tma_out = tma_store_enabled() && (g.ldo * (g.out_fp32 ? 4 : 2)) % 16 == 0 && ((uintptr_t)g.out & 15) == 0;
  const bool rows = tma_out && !g.out_fp32 && !g.transposed && !g.in_fp32;
  const FlowVariant v = g.in_fp32 ? flow_variant<4, FLOW_ANY>(bn, rb) : !rows ? flow_variant<2, FLOW_ANY>(bn, rb)
                        : g.act ? flow_variant<2, FLOW_ROWS_ACT>(bn, rb) : flow_variant<2, FLOW_ROWS>(bn, rb);
  if (v.fn == nullptr) return fail(KR_FAIL_ARG, "no persistent pair kernel of this tile shape");
  FlowParams p;
  memset(&p, 0, sizeof(p));
  p.tmap_r = g.tmap_r;
  p.tmap_c = g.tmap_c;
  const int out_elt = g.out_fp32 ? 4 : 2;
  // panels of 64 columns from the kernels that hold a tile's rounded rows, of 32 from those that go chunk by chunk
  const unsigned box_bytes = (out_elt == 4 || (!g.transposed && bn % 64 == 0 && (rows || !g.act))) ? 128u : 64u;
  if (tma_out) {
    int rc = get_tmap(g.out, g.out_rows, g.out_cols, g.ldo, 32, &p.tmap_out, out_elt, box_bytes);
    if (!rc && bn % 32 != 0)
      rc = g.transposed ? get_tmap(g.out, g.out_rows, g.out_cols, g.ldo, 16, &p.tmap_tail, out_elt, box_bytes)
                        : get_tmap(g.out, g.out_rows, g.out_cols, g.ldo, 32, &p.tmap_tail, out_elt, 16u * out_elt);
    if (rc) return rc;
  } else {
    p.tmap_out = g.tmap_r;          // prefetched, not used
    p.out = g.out;
    p.ldo = g.ldo;
  }
  p.tiles_r = (g.rows_r + 256 * rb - 1) / (256 * rb);
  p.tiles_c = (g.rows_c + bn - 1) / bn;
  p.num_kb = (g.K + (g.in_fp32 ? 32 : 64) - 1) / (g.in_fp32 ? 32 : 64);
  p.last_cols = last_cols;
  p.tmap_last = last_cols < bn ? tmap_last : p.tmap_c;
  p.group_r = std::max(1, g.group_r / (2 * rb));
  const int tiles = p.tiles_r * p.tiles_c;
  // A last wave that is at most half full is dealt as single row blocks
  p.split_from = tiles;
  if (rb == 2 && 2 * (tiles % pairs) <= pairs) p.split_from = tiles - tiles % pairs;
  p.items = p.split_from + (tiles - p.split_from) * rb;
  p.transposed = g.transposed;
  p.out_fp32 = g.out_fp32;
  p.act = g.act;
  p.rest_follows = g.rest_follows;
  p.out_rows = g.out_rows;
  p.out_cols = g.out_cols;
  p.sched = sched;
  p.cp_src = g.cp_src;
  p.cp_dst = g.cp_dst;
  p.cp_bytes = g.cp_bytes;
  p.sync = g.sync;
  pairs = std::min(pairs, p.items);
  if (pairs == p.items) p.sched = nullptr;        // one item each
  void* args[] = {(void*)&p};
  return launch_overlapped(v.fn, 2u * (unsigned)pairs, g.cp_bytes ? kFlowThreads + kFlowCopyThreads : kFlowThreads, args, v.smem, stream, 2);
}

}  // namespace kraken
