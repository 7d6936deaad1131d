"""Single-GPU numerics of the tcgen05 GEMM core and of the three fused GEMM + collective kernels
(emulated world sizes: all ranks in one cooperative launch). Goldens are plain PyTorch fp32
matmuls of the same bf16 inputs. Shapes include the reference's test shapes scaled to fit one GPU
(test/test_gemm_allreduce.py:57-117: 512x256x128, 256^3, rank-valued 32^3 with 1e-5 tolerance;
test/test_gemm_reduce_scatter.py:44-115; test/test_allgather_matmul.py:47-81)."""
import ctypes
import math

import pytest
import torch

from kraken_b200 import fused
from kraken_b200.ops import lib as klib
from kraken_b200.parallel import EmuWorld

pytestmark = pytest.mark.gpu


def _ab(M, N, K, seed=0, scale_b=0.05):
    g = torch.Generator().manual_seed(seed)
    a = torch.randn(M, K, generator=g).to(torch.bfloat16).cuda()
    bt = (scale_b * torch.randn(N, K, generator=g)).to(torch.bfloat16).cuda()
    return a, bt


def _close(c, ref, K):
    # bf16 inputs, fp32 accumulate: the only rounding is the bf16 output
    torch.testing.assert_close(c.float(), ref, atol=2e-2 * max(1.0, (K / 1024) ** 0.5), rtol=2e-2)


@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (128, 256, 128), (256, 512, 512), (1024, 1024, 1024),
                                   (4096, 2048, 1024), (384, 768, 4096), (8192, 256, 256)])
def test_gemm_basic(M, N, K):
    a, bt = _ab(M, N, K)
    c = fused.matmul(a, bt.t())
    _close(c, a.float() @ bt.float().t(), K)


@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (512, 512, 512), (4096, 2048, 1024), (1000, 520, 264), (8192, 4096, 512),
                                   (300, 1032, 136)])
def test_gemm_cta_pair_kernel_matches_single_cta_kernel(M, N, K):
    # 256 x 256 tiles on CTA pairs (tcgen05 cta_group::2) against the single-CTA kernel and fp32 PyTorch
    a, bt = _ab(M, N, K, seed=11)
    ref = a.float() @ bt.float().t()
    c_pair = fused.matmul(a, bt.t(), swap_ab=0, pair=1)
    c_single = fused.matmul(a, bt.t(), swap_ab=0, pair=0)
    _close(c_pair, ref, K)
    _close(c_single, ref, K)
    assert torch.equal(c_pair, c_single)      # same accumulation order per element


def test_gemm_cta_pair_many_tiles_per_pair():
    a, bt = _ab(2048, 2048, 256, seed=12)
    c = fused.matmul(a, bt.t(), max_ctas=6, pair=1)       # 64 pair tiles over 3 pairs
    _close(c, a.float() @ bt.float().t(), 256)
    c32 = fused.matmul(a, bt.t(), out_dtype=torch.float32, pair=1)
    torch.testing.assert_close(c32, a.float() @ bt.float().t(), atol=2e-3, rtol=2e-3)


@pytest.mark.parametrize("M,N,K", [(100, 200, 72), (129, 257, 136), (1000, 520, 264), (77, 1032, 8), (5, 8, 64)])
def test_gemm_ragged_shapes(M, N, K):
    a, bt = _ab(M, N, K, seed=1)
    c = fused.matmul(a, bt.t(), swap_ab=0)
    _close(c, a.float() @ bt.float().t(), K)


@pytest.mark.parametrize("bn", [16, 32, 64, 128, 256])
def test_gemm_every_column_tile_variant(bn):
    a, bt = _ab(256, 512, 512, seed=2)
    c = fused.matmul(a, bt.t(), swap_ab=0, bn=bn)
    _close(c, a.float() @ bt.float().t(), 512)


@pytest.mark.parametrize("M", [1, 16, 64, 256])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_gemm_decode_shapes_swap_ab(M, out_dtype):
    a, bt = _ab(M, 8192, 1024, seed=3, scale_b=0.02)
    ref = a.float() @ bt.float().t()
    for swap in (1, 0):
        c = fused.matmul(a, bt.t(), out_dtype=out_dtype, swap_ab=swap)
        assert c.dtype == out_dtype
        if out_dtype == torch.float32:
            torch.testing.assert_close(c, ref, atol=1e-3, rtol=1e-3)
        else:
            _close(c, ref, 1024)


def test_gemm_fp32_output_exact_on_integer_data():
    # values exactly representable in bf16 -> the fp32 result is exact
    a = torch.randint(-4, 5, (256, 256)).to(torch.bfloat16).cuda()
    bt = torch.randint(-4, 5, (384, 256)).to(torch.bfloat16).cuda()
    c = fused.matmul(a, bt.t(), out_dtype=torch.float32)
    assert torch.equal(c, a.float() @ bt.float().t())


def test_gemm_row_major_b_and_fp32_inputs():
    g = torch.Generator().manual_seed(4)
    a = torch.randn(512, 128, generator=g).cuda()                 # fp32, cast to bf16 inside
    b = (0.05 * torch.randn(128, 256, generator=g)).cuda()        # row-major [K, N]
    c = fused.matmul(a, b)
    ref = a.to(torch.bfloat16).float() @ b.to(torch.bfloat16).float()
    _close(c, ref, 128)
    c2 = fused.matmul(a, b)                                       # transposed weight comes from the cache
    assert torch.equal(c, c2)


@pytest.mark.parametrize("M,N,K", [(256, 512, 256), (1000, 520, 136), (16, 8192, 1024), (64, 1024, 512), (1, 2048, 64),
                                   (2048, 2048, 1024)])
def test_gemm_fp32_inputs_run_as_tf32(M, N, K):
    # fp32 x fp32 operands are multiplied as tf32 (10-bit mantissa), fp32 accumulation, fp32 output
    g = torch.Generator().manual_seed(21)
    a = torch.randn(M, K, generator=g).cuda()
    b = (0.05 * torch.randn(K, N, generator=g)).cuda()
    ref = a.double() @ b.double()
    c = fused.matmul(a, b, out_dtype=torch.float32)
    tol = 1e-2 * 0.05 * (K ** 0.5)                     # operands cut to 10 mantissa bits, random signs, max over the matrix
    assert float((c.double() - ref).abs().max()) < tol
    # and it is closer to the fp32 product than the bf16 path on the same data
    c16 = fused.matmul(a, b, out_dtype=torch.float32, tf32=False)
    assert float((c.double() - ref).abs().mean()) < float((c16.double() - ref).abs().mean())


def test_gemm_tf32_exact_on_small_integers():
    a = torch.randint(-8, 9, (384, 160)).float().cuda()
    b = torch.randint(-8, 9, (160, 272)).float().cuda()
    assert torch.equal(fused.matmul(a, b, out_dtype=torch.float32), a @ b)


def test_gemm_persistent_many_tiles_per_cta():
    a, bt = _ab(2048, 2048, 256, seed=5)
    c = fused.matmul(a, bt.t(), max_ctas=7)         # 128 tiles over 7 CTAs: both accumulators, many rounds
    _close(c, a.float() @ bt.float().t(), 256)


# ---- fused GEMM + collective, emulated ranks ---------------------------------------------------
@pytest.mark.parametrize("ws", [1, 2, 4, 8])
@pytest.mark.parametrize("splits", [1, 2, 4])
@pytest.mark.parametrize("backend", ["push", "sm"])
def test_all_gather_matmul(ws, splits, backend):
    world = EmuWorld(ws)
    shard_rows, K, N = 256, 512, 384
    g = torch.Generator().manual_seed(6)
    shards = [torch.randn(shard_rows, K, generator=g).to(torch.bfloat16).cuda() for _ in range(ws)]
    bt = (0.05 * torch.randn(N, K, generator=g)).to(torch.bfloat16).cuda()
    ts = world.symmetric((shard_rows, K), torch.bfloat16)
    for r in range(ws):
        ts[r].copy_(shards[r])
    a_full = torch.cat(shards, 0)
    ref = a_full.float() @ bt.float().t()
    for _ in range(3):          # three calls: both gathered-buffer halves / flag banks, then the first again
        progs = [torch.zeros(ws * splits, dtype=torch.uint32, device="cuda") for _ in range(ws)]
        outs = world.run(lambda r: fused.all_gather_matmul(ts[r], bt.t(), progress=progs[r], splits_per_rank=splits,
                                                           num_comm_sms=4, backend=backend))
        for r in range(ws):
            ag, c = outs[r]
            assert torch.equal(ag, a_full)
            _close(c, ref, K)
            assert bool((progs[r].to(torch.int64) != 0).all())


@pytest.mark.parametrize("symmetric_out", [True])
def test_all_gather_matmul_push_into_caller_buffers(symmetric_out):
    # a caller-owned symmetric a_out is written in place (entry barrier). (An ordinary a_out gets a
    # device copy after the kernel, which rank emulation cannot order after its deferred launch: that
    # form is covered by the multi-GPU test.)
    ws = 4
    world = EmuWorld(ws)
    shard_rows, K, N = 384, 256, 520
    g = torch.Generator().manual_seed(16)
    shards = [torch.randn(shard_rows, K, generator=g).to(torch.bfloat16).cuda() for _ in range(ws)]
    bt = (0.05 * torch.randn(N, K, generator=g)).to(torch.bfloat16).cuda()
    ts = world.symmetric((shard_rows, K), torch.bfloat16)
    for r in range(ws):
        ts[r].copy_(shards[r])
    outs_buf = world.symmetric((ws * shard_rows, K), torch.bfloat16) if symmetric_out else \
        [torch.empty(ws * shard_rows, K, dtype=torch.bfloat16, device="cuda") for _ in range(ws)]
    a_full = torch.cat(shards, 0)
    ref = a_full.float() @ bt.float().t()
    for _ in range(2):
        for o in outs_buf:
            o.zero_()
        outs = world.run(lambda r: fused.all_gather_matmul(ts[r], bt.t(), a_out=outs_buf[r], backend="push", num_comm_sms=2))
        for r in range(ws):
            ag, c = outs[r]
            assert ag.data_ptr() == outs_buf[r].data_ptr()
            assert torch.equal(ag, a_full)
            _close(c, ref, K)


@pytest.mark.parametrize("ws", [2, 4, 8])
@pytest.mark.parametrize("algo", ["pull", "scatter", "push"])
def test_gemm_reduce_scatter_fused(ws, algo):
    world = EmuWorld(ws)
    M, N, Kl = 128 * ws * 2, 512, 256
    g = torch.Generator().manual_seed(7)
    a_s = [torch.randn(M, Kl, generator=g).to(torch.bfloat16).cuda() for _ in range(ws)]
    bt_s = [(0.05 * torch.randn(N, Kl, generator=g)).to(torch.bfloat16).cuda() for _ in range(ws)]
    full = sum(a.float() @ bt.float().t() for a, bt in zip(a_s, bt_s))
    for _ in range(3):     # staging halves / counter banks alternate, then the first is reused
        outs = world.run(lambda r: fused.gemm_reduce_scatter(a_s[r], bt_s[r].t(), algo=algo))
        for r in range(ws):
            torch.testing.assert_close(outs[r].float(), full[r * (M // ws):(r + 1) * (M // ws)], atol=6e-2, rtol=3e-2)


@pytest.mark.parametrize("algo", ["pull", "scatter", "push"])
def test_gemm_reduce_scatter_fused_several_tiles_per_cta(algo):
    # 4 ranks x 37 CTAs, 16 x 5 tiles of 128 x 256 (last column tile ragged): every CTA walks two or
    # three tiles, owners interleaved (pull) or slab after slab (push)
    ws = 4
    world = EmuWorld(ws)
    M, N, Kl = 2048, 1160, 128
    g = torch.Generator().manual_seed(17)
    a_s = [torch.randn(M, Kl, generator=g).to(torch.bfloat16).cuda() for _ in range(ws)]
    bt_s = [(0.05 * torch.randn(N, Kl, generator=g)).to(torch.bfloat16).cuda() for _ in range(ws)]
    full = sum(a.float() @ bt.float().t() for a, bt in zip(a_s, bt_s))
    first = None
    for _ in range(2):
        outs = world.run(lambda r: fused.gemm_reduce_scatter(a_s[r], bt_s[r].t(), algo=algo))
        for r in range(ws):
            torch.testing.assert_close(outs[r].float(), full[r * (M // ws):(r + 1) * (M // ws)], atol=6e-2, rtol=3e-2)
        if first is None:
            first = [o.clone() for o in outs]
        else:
            assert all(torch.equal(x, y) for x, y in zip(first, outs))      # bit-reproducible


@pytest.mark.parametrize("algo", ["pull", "scatter", "push"])
@pytest.mark.parametrize("M,N,K", [(2048, 2048, 512), (4096, 1032, 256), (512, 256, 64)])
def test_gemm_reduce_scatter_kernel_at_world_size_one(algo, M, N, K):
    # the fused kernels (CTA pairs, reducer warps, counters, staging halves) on one real rank
    a, bt = _ab(M, N, K, seed=18)
    ref = a.float() @ bt.float().t()
    for _ in range(3):
        c = fused.gemm_reduce_scatter(a, bt.t(), algo=algo, _force_fused=True)
        _close(c, ref, K)


@pytest.mark.parametrize("ws", [2, 4])
def test_gemm_reduce_scatter_unaligned_slab_path(ws):
    world = EmuWorld(ws)
    M, N, Kl = 64 * ws, 256, 128            # slab of 64 rows: GEMM -> staging -> reduce-scatter kernel
    g = torch.Generator().manual_seed(8)
    a_s = [torch.randn(M, Kl, generator=g).to(torch.bfloat16).cuda() for _ in range(ws)]
    bt_s = [(0.05 * torch.randn(N, Kl, generator=g)).to(torch.bfloat16).cuda() for _ in range(ws)]
    full = sum(a.float() @ bt.float().t() for a, bt in zip(a_s, bt_s))
    # two kernels per rank cannot be recorded as one emulated launch: run each rank's GEMM into its
    # staging buffer eagerly, then the reduce-scatter kernel for all ranks at once
    from kraken_b200.parallel import symm_mem
    hdls = []
    for r in range(ws):
        with world.rank(r):
            hdl = symm_mem.get_symm_mem_workspace(None, M * N * 2)
            hdls.append(hdl)
            stage = hdl.get_buffer(r, (M, N), torch.bfloat16)
            stage.copy_(fused.matmul(a_s[r], bt_s[r].t()))
    from kraken_b200 import comm
    views = [hdls[r].get_buffer(r, (M, N), torch.bfloat16) for r in range(ws)]
    outs = world.run(lambda r: comm.reduce_scatter(views[r]))
    for r in range(ws):
        torch.testing.assert_close(outs[r].float(), full[r * (M // ws):(r + 1) * (M // ws)], atol=6e-2, rtol=3e-2)


@pytest.mark.parametrize("ws", [2, 4, 8])
@pytest.mark.parametrize("M", [1, 16, 64, 256])
@pytest.mark.parametrize("algo", ["one_shot", "two_shot"])
def test_gemm_one_shot_all_reduce(ws, M, algo):
    world = EmuWorld(ws)
    N, Kl = 1024, 256
    g = torch.Generator().manual_seed(9)
    a_s = [torch.randn(M, Kl, generator=g).to(torch.bfloat16).cuda() for _ in range(ws)]
    bt_s = [(0.02 * torch.randn(N, Kl, generator=g)).to(torch.bfloat16).cuda() for _ in range(ws)]
    full = sum(a.float() @ bt.float().t() for a, bt in zip(a_s, bt_s))
    for _ in range(3):       # three rounds: both staging halves / flag banks, then reuse of the first
        outs = world.run(lambda r: fused.gemm_one_shot_all_reduce_fused(a_s[r], bt_s[r].t(), algo=algo))
        for r in range(ws):
            assert outs[r].dtype == torch.float32
            torch.testing.assert_close(outs[r], full, atol=2e-3, rtol=2e-3)
        for r in range(1, ws):
            assert torch.equal(outs[0], outs[r])


@pytest.mark.parametrize("ws", [2, 4, 8])
@pytest.mark.parametrize("M", [1, 5, 16, 64])
@pytest.mark.parametrize("k_splits", [0, 2])
def test_gemm_all_reduce_tagged_two_shot(ws, M, k_splits):
    # partial tiles travel tagged to the tile's owner only; the owner publishes tagged results
    world = EmuWorld(ws)
    N, Kl = 1024, 256
    g = torch.Generator().manual_seed(41)
    for it in range(4):
        a_s = [torch.randn(M, Kl, generator=g).to(torch.bfloat16).cuda() for _ in range(ws)]
        bt_s = [(0.02 * torch.randn(N, Kl, generator=g)).to(torch.bfloat16).cuda() for _ in range(ws)]
        full = sum(a.float() @ bt.float().t() for a, bt in zip(a_s, bt_s))
        outs = world.run(lambda r: fused.gemm_one_shot_all_reduce_fused(a_s[r], bt_s[r].t(), algo="push_two_shot",
                                                                        k_splits=k_splits))
        for r in range(ws):
            torch.testing.assert_close(outs[r], full, atol=2e-3, rtol=2e-3)
            assert torch.equal(outs[0], outs[r])


@pytest.mark.parametrize("ws", [2, 4, 8])
@pytest.mark.parametrize("M", [1, 5, 16, 64])
@pytest.mark.parametrize("k_splits", [0, 1, 2])
def test_gemm_all_reduce_tagged_push(ws, M, k_splits):
    # decode exchange: {value, tag} pairs pushed into every rank's slots, summed as they land; with
    # k_splits = 2 two CTAs per tile each multiply half of K and the slots double
    world = EmuWorld(ws)
    N, Kl = 1024, 256
    g = torch.Generator().manual_seed(31)
    for it in range(4):      # both staging halves twice: a slot's previous tag must never satisfy a wait
        a_s = [torch.randn(M, Kl, generator=g).to(torch.bfloat16).cuda() for _ in range(ws)]
        bt_s = [(0.02 * torch.randn(N, Kl, generator=g)).to(torch.bfloat16).cuda() for _ in range(ws)]
        full = sum(a.float() @ bt.float().t() for a, bt in zip(a_s, bt_s))
        outs = world.run(lambda r: fused.gemm_one_shot_all_reduce_fused(a_s[r], bt_s[r].t(), algo="push", k_splits=k_splits))
        for r in range(ws):
            torch.testing.assert_close(outs[r], full, atol=2e-3, rtol=2e-3)
            assert torch.equal(outs[0], outs[r])


@pytest.mark.parametrize("ws,M", [(2, 16), (2, 64), (4, 64), (8, 16)])
def test_gemm_all_reduce_two_shot_split_k(ws, M):
    world = EmuWorld(ws)
    N, Kl = 1024, 512
    g = torch.Generator().manual_seed(32)
    a_s = [torch.randn(M, Kl, generator=g).to(torch.bfloat16).cuda() for _ in range(ws)]
    bt_s = [(0.02 * torch.randn(N, Kl, generator=g)).to(torch.bfloat16).cuda() for _ in range(ws)]
    full = sum(a.float() @ bt.float().t() for a, bt in zip(a_s, bt_s))
    for _ in range(3):
        outs = world.run(lambda r: fused.gemm_one_shot_all_reduce_fused(a_s[r], bt_s[r].t(), algo="two_shot", k_splits=2))
        for r in range(ws):
            torch.testing.assert_close(outs[r], full, atol=2e-3, rtol=2e-3)
            assert torch.equal(outs[0], outs[r])


def test_gemm_all_reduce_plan_prefers_push_for_decode_rows():
    import ctypes

    from kraken_b200.ops import lib as klib

    def plan(M, N, K, ws, S=32 << 20):
        out = (ctypes.c_int * 5)()
        klib.check(klib.lib().kr_gemm_ar_plan(M, N, K, ws, 0, -1, 0, S, 1, out))
        return list(out)

    algo, ks, bn, ctas, swap = plan(1, 8192, 1024, 8)
    assert algo == 2 and swap == 1 and ctas == 64 * ks
    algo, ks, *_ = plan(256, 8192, 1024, 8, 256 << 20)
    assert algo == 1                      # 8 MB of output: tile owners reduce
    algo, ks, *_ = plan(1, 8192, 4096, 2)
    assert algo == 2 and ks == 2          # long K per rank: two CTAs per tile stream the weights


def test_gemm_all_reduce_alternating_shapes_and_algorithms():
    # consecutive calls of different shapes and exchange algorithms share one staging buffer
    ws = 4
    world = EmuWorld(ws)
    g = torch.Generator().manual_seed(10)
    for M, N, algo in [(256, 1024, "two_shot"), (16, 512, "one_shot"), (64, 1024, "two_shot"), (1, 1024, "one_shot"),
                       (1, 1024, "push"), (16, 512, "push"), (16, 512, "push_two_shot"), (16, 512, "one_shot"), (3, 1024, "push"),
                       (3, 1024, "push_two_shot"), (64, 512, None), (64, 512, "push_two_shot"),
                       (200, 520, "two_shot"), (200, 520, "one_shot"), (8, 520, "push"), (8, 520, None)]:
        a_s = [torch.randn(M, 128, generator=g).to(torch.bfloat16).cuda() for _ in range(ws)]
        bt_s = [(0.02 * torch.randn(N, 128, generator=g)).to(torch.bfloat16).cuda() for _ in range(ws)]
        full = sum(a.float() @ bt.float().t() for a, bt in zip(a_s, bt_s))
        outs = world.run(lambda r: fused.gemm_one_shot_all_reduce_fused(a_s[r], bt_s[r].t(), algo=algo))
        for r in range(ws):
            torch.testing.assert_close(outs[r], full, atol=2e-3, rtol=2e-3)


@pytest.mark.parametrize("M", [1, 64, 256])
def test_gemm_all_reduce_fp32_operands(M):
    # the reference's GEMM + all-reduce tests feed fp32 operands (test/test_gemm_allreduce.py:57-58)
    ws = 4
    world = EmuWorld(ws)
    N, Kl = 512, 128
    g = torch.Generator().manual_seed(22)
    a_s = [torch.randn(M, Kl, generator=g).cuda() for _ in range(ws)]
    b_s = [(0.02 * torch.randn(Kl, N, generator=g)).cuda() for _ in range(ws)]
    full = sum(a.double() @ b.double() for a, b in zip(a_s, b_s)).float()
    for algo in ("one_shot", "two_shot"):
        outs = world.run(lambda r: fused.gemm_one_shot_all_reduce_fused(a_s[r], b_s[r], algo=algo))
        for r in range(ws):
            torch.testing.assert_close(outs[r], full, atol=2e-3, rtol=2e-3)
            assert torch.equal(outs[0], outs[r])


def test_gemm_all_reduce_rank_valued_exact():
    # the reference's exactness case: a = rank+1 everywhere, b = ones -> K * sum(rank+1), 1e-5
    ws, n = 4, 32
    world = EmuWorld(ws)
    a_s = [torch.full((n, n), float(r + 1), dtype=torch.bfloat16, device="cuda") for r in range(ws)]
    b = torch.ones(n, n, dtype=torch.bfloat16, device="cuda")
    outs = world.run(lambda r: fused.gemm_one_shot_all_reduce_fused(a_s[r], b))
    expect = torch.full((n, n), float(n * sum(range(1, ws + 1))), device="cuda")
    for r in range(ws):
        torch.testing.assert_close(outs[r], expect, atol=1e-5, rtol=1e-5)


def test_tensor_map_cache_is_hit_on_repeated_calls():
    import ctypes

    from kraken_b200.ops import lib as klib

    a, bt = _ab(512, 512, 256, seed=13)
    fused.matmul(a, bt.t())
    h0, m0 = ctypes.c_ulonglong(0), ctypes.c_ulonglong(0)
    klib.check(klib.lib().kr_tmap_cache_stats(ctypes.byref(h0), ctypes.byref(m0)))
    for _ in range(5):
        fused.matmul(a, bt.t())
    h1, m1 = ctypes.c_ulonglong(0), ctypes.c_ulonglong(0)
    klib.check(klib.lib().kr_tmap_cache_stats(ctypes.byref(h1), ctypes.byref(m1)))
    assert h1.value - h0.value >= 10           # both operand maps, five calls
    assert m1.value - m0.value <= 5            # at most the output map of a fresh output tensor


@pytest.mark.parametrize("M,N,K", [(1, 1024, 4096), (3, 8200, 264), (17, 520, 1032), (64, 1000, 8192), (65, 520, 2048),
                                   (128, 4096, 520), (129, 4096, 4104), (300, 1032, 136), (777, 5120, 1032), (2049, 1160, 264)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_gemm_split_tiles_match_fp32_reference(M, N, K, dtype):
    # the launcher's own choice: clusters that split a tile along K, tiles dealt in parts, swapped operands
    g = torch.Generator().manual_seed(31)
    a = torch.randn(M, K, generator=g).to(dtype).cuda()
    bt = (0.05 * torch.randn(N, K, generator=g)).to(dtype).cuda()
    ref = (a.double() @ bt.double().t()).float()
    for out_dtype in (torch.float32, torch.bfloat16):
        c = fused.matmul(a, bt.t(), out_dtype=out_dtype)
        rel = ((c.float() - ref).norm() / ref.norm()).item()
        assert rel < (3e-3 if out_dtype == torch.bfloat16 else (1e-5 if dtype == torch.bfloat16 else 1e-3)), rel
        assert torch.equal(c, fused.matmul(a, bt.t(), out_dtype=out_dtype))      # the parts are summed in K order


@pytest.mark.parametrize("M,N,K", [(1, 264, 64), (64, 1000, 136), (130, 520, 264), (777, 5120, 520), (2100, 2600, 264)])
def test_one_rank_all_gather_matmul_and_activation(M, N, K):
    from kraken_b200.fused.gemm_ops import all_gather_matmul_act
    from kraken_b200.parallel import symm_mem

    a, bt = _ab(M, N, K, seed=41, scale_b=0.1)
    x = symm_mem.empty(M, K, dtype=torch.bfloat16, device="cuda")
    x.copy_(a)
    ref = a.float() @ bt.float().t()
    prog = torch.zeros(1, dtype=torch.uint32, device="cuda")
    gathered, c = fused.all_gather_matmul(x, bt.t(), progress=prog)
    assert torch.equal(gathered, a) and gathered.data_ptr() != x.data_ptr() and int(prog[0]) == 1
    _close(c, ref, K)
    h = all_gather_matmul_act(x, bt.t(), "gelu_tanh")
    _close(h, torch.nn.functional.gelu(ref, approximate="tanh"), K)


@pytest.mark.parametrize("bn", [1064, 1096, 2064, 2096, 1144, 1176, 1208, 1240, 2144, 2176, 2208, 2240, 1128, 1160, 1192, 1224, 1256, 2128, 2160, 2192, 2224, 2256])
@pytest.mark.parametrize("swap", [0, 1])
def test_gemm_persistent_pairs_every_tile_shape(bn, swap):
    # row blocks x columns as 1000 * b + n; the last wave of two-block tiles is dealt as single blocks
    for M, N, K, dtype in [(300, 1032, 136, torch.bfloat16), (777, 2601, 72, torch.bfloat16), (2049, 520, 68, torch.float32)]:
        if dtype == torch.float32 and bn % 1000 % 32:
            dtype, K = torch.bfloat16, 72          # column tiles off the 32s: bf16 operands only
        g = torch.Generator().manual_seed(51)
        a = torch.randn(M, K, generator=g).to(dtype).cuda()
        bt = (0.05 * torch.randn(N, K, generator=g)).to(dtype).cuda()
        ref = (a.double() @ bt.double().t()).float()
        for out_dtype in (torch.bfloat16, torch.float32):
            for _ in range(2):                  # the tile counter is back at zero for the second call
                c = fused.matmul(a, bt.t(), out_dtype=out_dtype, bn=bn, swap_ab=swap)
                assert ((c.float() - ref).norm() / ref.norm()).item() < 3e-3
    c = fused.matmul(a, bt.t(), bn=bn, swap_ab=swap, max_ctas=6)        # many tiles per pair
    assert ((c.float() - ref).norm() / ref.norm()).item() < 3e-3


@pytest.mark.parametrize("splits", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("swap", [0, 1])
def test_gemm_one_wave_every_split_and_tile(splits, swap):
    # 10000 * splits + 1000 * pairs + columns: each split owns 16 ... 128 rows of a tile; rows and columns past the
    # output are neither sent nor waited for (last row block of 1 and of 0 rows in a pair, 1 ... 4 columns of a unit)
    for bn, dtype in [(16, 0), (32, 0), (64, 0), (128, 0), (16, 1), (128, 1), (1128, 0), (1160, 0), (1224, 1), (1256, 0)]:
        if bn >= 1000 and splits > 4:
            continue
        dtype = torch.float32 if dtype else torch.bfloat16
        for M, N, K in [(129, 264, 584), (1, 136, 1096), (300, 1032, 512)]:
            g = torch.Generator().manual_seed(71)
            a = torch.randn(M, K, generator=g).to(dtype).cuda()
            bt = (0.05 * torch.randn(N, K, generator=g)).to(dtype).cuda()
            ref = (a.double() @ bt.double().t()).float()
            for out_dtype, limit in ((torch.float32, 1e-5 if dtype == torch.bfloat16 else 1e-3), (torch.bfloat16, 3e-3)):
                c = fused.matmul(a, bt.t(), out_dtype=out_dtype, bn=10000 * splits + bn, swap_ab=swap)
                assert ((c.float() - ref).norm() / ref.norm()).item() < limit
                assert torch.equal(c, fused.matmul(a, bt.t(), out_dtype=out_dtype, bn=10000 * splits + bn, swap_ab=swap))


@pytest.mark.parametrize("bn", [1144, 1176, 1208, 1240, 2144, 2176, 2208, 2240])
@pytest.mark.parametrize("swap", [0, 1])
def test_gemm_persistent_pairs_fp32_steps_of_16(bn, swap):
    # fp32 stores of tiles whose last chunk is 16 columns; last column tiles of 16 columns and of less than a chunk
    for M, N, K in [(257, bn % 1000 * 2 + 1, 68), (600, bn % 1000 + 100, 132), (513, 520, 36)]:
        g = torch.Generator().manual_seed(52)
        a = torch.randn(M, K, generator=g).cuda()
        bt = (0.05 * torch.randn(N, K, generator=g)).cuda()
        ref = (a.double() @ bt.double().t()).float()
        for out_dtype in (torch.float32, torch.bfloat16):
            c = fused.matmul(a, bt.t(), out_dtype=out_dtype, bn=bn, swap_ab=swap)
            assert ((c.float() - ref).norm() / ref.norm()).item() < (1e-3 if out_dtype == torch.float32 else 3e-3)


def _plan(M, N, K, fp32, pair=1, lda=None):
    plan = (ctypes.c_int * 13)()
    klib.check(klib.lib().kr_gemm_plan(M, N, K, lda or K, K, int(fp32), pair, plan))
    return list(plan)


# Both dimensions up to 128: one tile, whose K is what can be shared out (router and gate projections of a decode step).
@pytest.mark.parametrize("M,N,K,fp32", [(64, 128, 8192, 0), (128, 128, 16384, 0), (1, 128, 7168, 0), (16, 64, 4096, 0), (128, 1, 520, 0),
                                        (33, 17, 5000, 0), (128, 128, 4096, 1), (8, 127, 260, 1)])
def test_one_tile_problems_are_cut_along_k(M, N, K, fp32):
    plan = _plan(M, N, K, fp32)
    assert plan[0] == 1 and plan[4] > 1, plan
    dtype = torch.float32 if fp32 else torch.bfloat16
    g = torch.Generator().manual_seed(97)
    a = torch.randn(M, K, generator=g).to(dtype).cuda()
    bt = (0.05 * torch.randn(N, K, generator=g)).to(dtype).cuda()
    ref = (a.double() @ bt.double().t()).float()
    # fp32 sums: one cut of the running sum (2**-23 of it) per MMA of 16 columns; tf32 operands: 10 bits; bf16 results: 2**-9
    for out_dtype, limit in ((torch.float32, 1e-3 if fp32 else 1e-6 + K / 16 * 2.0 ** -23), (torch.bfloat16, 3e-3)):
        c = fused.matmul(a, bt.t(), out_dtype=out_dtype)
        assert ((c.float() - ref).norm() / ref.norm()).item() < limit
        assert torch.equal(c, fused.matmul(a, bt.t(), out_dtype=out_dtype))


@pytest.mark.parametrize("M,N,K", [(128, 128, 256), (65, 72, 8), (72, 66, 448), (128, 128, 440)])
def test_one_tile_problems_too_short_to_cut(M, N, K):
    # the kernel depends on how the result can be stored: bf16 rows of whole 16 bytes, others, fp32
    assert _plan(M, N, K, 0)[4] == 1
    a, bt = _ab(M, N, K, seed=98)
    ref = (a.double() @ bt.double().t()).float()
    for out_dtype, limit in ((torch.float32, 1e-6 + K / 16 * 2.0 ** -23), (torch.bfloat16, 3e-3)):
        c = fused.matmul(a, bt.t(), out_dtype=out_dtype)
        assert ((c.float() - ref).norm() / ref.norm()).item() < limit


# The same in every form that these calls take, against the persistent kernel on one CTA (bn=64, weights as columns): padded rows on
# the left, weights as columns of a wider matrix, activation, a copy of the operand, results that TMA cannot store.
@pytest.mark.parametrize("M,N,K", [(128, 128, 256), (128, 72, 440), (65, 127, 1032), (1, 128, 2056), (128, 1, 2048), (17, 24, 8)])
@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("act", [None, "gelu_tanh"])
def test_forms_of_one_tile_problems(M, N, K, fp32, act):
    from kraken_b200.fused.gemm_ops import _gemm

    dtype = torch.float32 if fp32 else torch.bfloat16
    g = torch.Generator(device="cuda").manual_seed(100)
    a = torch.full((M, K + 24), float("nan"), device="cuda", dtype=dtype)[:, :K]
    a.copy_(torch.randn(M, K, generator=g, device="cuda"))
    bt = torch.full((N, K + 8), float("nan"), device="cuda", dtype=dtype)[:, :K]
    bt.copy_(torch.randn(N, K, generator=g, device="cuda") / K ** 0.5)
    # sums below 6, cut once per MMA of 32 bytes of K; the device's exp and divide: 1e-4; bf16 results: 2**-8 of the value, on
    # either side of what the sums differ by
    slack = 2 * 6 * (K * a.element_size() / 32) * 2.0 ** -23 + (6e-4 if act else 0)
    for out_fp32 in (True, False):
        want = _gemm(a, bt.t(), out_fp32, bool(fp32), 0, 64, act=act).double()
        c = _gemm(a, bt.t(), out_fp32, bool(fp32), act=act).double()
        assert (((c - want).abs() - (0 if out_fp32 else 2.0 ** -7) * want.abs()).max()).item() < slack
        whole = a.contiguous()
        copied = torch.zeros_like(whole)
        c = _gemm(whole, bt.t(), out_fp32, bool(fp32), act=act, copy_dst=copied).double()
        assert torch.equal(copied, whole) and (((c - want).abs() - (0 if out_fp32 else 2.0 ** -7) * want.abs()).max()).item() < slack


# Without pairs the one-wave kernel runs on single CTAs, also where pairs would be the faster choice.
@pytest.mark.parametrize("M,N,K,fp32,with_pairs", [(6120, 106, 8272, 0, 1), (100, 6152, 6200, 0, 1), (2, 9622, 8216, 0, 1), (4280, 122, 6472, 1, 1),
                                                   (16, 4096, 4096, 0, 0)])
def test_one_wave_without_pairs(M, N, K, fp32, with_pairs):
    assert _plan(M, N, K, fp32)[11] == with_pairs
    plan = _plan(M, N, K, fp32, pair=0)
    assert plan[0] == 1 and plan[11] == 0, plan
    dtype = torch.float32 if fp32 else torch.bfloat16
    g = torch.Generator(device="cuda").manual_seed(99)
    a = torch.randn(M, K, generator=g, device="cuda").to(dtype)
    bt = (0.05 * torch.randn(N, K, generator=g, device="cuda")).to(dtype)
    ref = a.double() @ bt.double().t()
    c = fused.matmul(a, bt.t(), out_dtype=torch.float32, pair=0)
    assert ((c - ref).norm() / ref.norm()).item() < (1e-3 if fp32 else 1e-6 + K / 16 * 2.0 ** -23)


def _plan_stats():
    plans, timed = ctypes.c_ulonglong(0), ctypes.c_ulonglong(0)
    klib.check(klib.lib().kr_gemm_plan_stats(ctypes.byref(plans), ctypes.byref(timed)))
    return plans.value, timed.value


def test_a_plan_is_worked_out_in_microseconds():
    # The time model's roots and powers are what a plan of a new shape costs on the host: 34 kernels of a problem are timed on
    # average and 93 at most, the others are out by a bound. Timing every kernel that fits is 350 and 960, and 10 to 40 us.
    import random

    r = random.Random(11)
    problems = {(r.randint(65, 4000), r.randint(128, 2000) * 8, r.randint(128, 2000) * 8) for _ in range(400)}
    timed = []
    for M, N, K in problems:
        plans, before = _plan_stats()
        _plan(M, N, K, 0)
        after = _plan_stats()
        assert after[0] == plans + 1
        timed.append(after[1] - before)
    assert sum(timed) / len(timed) < 70 and max(timed) < 200, (sum(timed) / len(timed), max(timed))


def test_plans_of_a_programs_shapes_are_all_remembered():
    # a block's four projections at 8 row counts, and at 32; a second pass over them works nothing out
    for row_counts in ([1, 7, 16, 64, 200, 777, 2048, 8192], list(range(100, 1700, 50))):
        shapes = [(m, n, k) for m in row_counts for n, k in ((10240, 8192), (8192, 8192), (28672, 8192), (8192, 28672))]
        want = [_plan(*s, 0) for s in shapes]
        before = _plan_stats()[0]
        assert [_plan(*s, 0) for s in shapes] == want
        assert _plan_stats()[0] == before, _plan_stats()[0] - before


def _two_launch_problem(index, fp32, same=lambda M, N, K: True, more_n=0, more_lda=0):
    """The index-th of a fixed series of ragged problems that the launcher gives to two launches."""
    import random

    r = random.Random(3)
    for _ in range(20000):
        M, N, K = r.randint(300, 3000), r.randint(60, 700) * 8 + more_n, r.randint(64, 400) * 8
        if _plan(M, N, K, fp32, lda=K + more_lda)[5] == 1 and same(M, N, K):
            if index == 0:
                return M, N, K
            index -= 1
    raise AssertionError("no such problem")


# whole waves on persistent pairs, the rest of the rows or columns by the one-wave kernel in a launch that overlaps it
@pytest.mark.parametrize("index,fp32", [(0, 0), (1, 0), (2, 0), (3, 0), (4, 0), (5, 0), (0, 1), (1, 1), (2, 1)])
def test_gemm_in_two_launches(index, fp32):
    from kraken_b200.fused.gemm_ops import _gemm
    from kraken_b200.parallel import symm_mem

    M, N, K = _two_launch_problem(index, fp32)
    dtype = torch.float32 if fp32 else torch.bfloat16
    g = torch.Generator(device="cuda").manual_seed(91)
    a = torch.randn(M, K, generator=g, device="cuda").to(dtype)
    bt = (0.05 * torch.randn(N, K, generator=g, device="cuda")).to(dtype)
    ref = (a.double() @ bt.double().t()).float()
    for out_dtype, limit in ((torch.float32, 1e-3 if fp32 else 1e-5), (torch.bfloat16, 3e-3)):
        c = fused.matmul(a, bt.t(), out_dtype=out_dtype)
        assert ((c.float() - ref).norm() / ref.norm()).item() < limit
        assert ((c.float() - ref).abs().amax(0) < 0.05 * ref.abs().amax()).all()              # no column or row left out
    h = _gemm(a, bt.t(), True, True, act="gelu_tanh")
    href = torch.nn.functional.gelu(ref, approximate="tanh")
    assert ((h - href).norm() / href.norm()).item() < 1e-3
    if not fp32:
        x = symm_mem.empty(M, K, dtype=dtype, device="cuda")
        x.copy_(a)
        gathered, c = fused.all_gather_matmul(x, bt.t())
        assert torch.equal(gathered, a) and ((c.float() - ref).norm() / ref.norm()).item() < 3e-3


# The forms of the first launch and what it shares with the second one: stores of whole rows, transposed, element by element
# (an output that TMA cannot describe), and a left operand with padded rows; cut by rows and by columns.
@pytest.mark.parametrize("by_col", [0, 1])
@pytest.mark.parametrize("swap,more_n,more_lda", [(0, 0, 0), (1, 0, 0), (0, 1, 0), (1, 1, 0), (0, 0, 72)])
@pytest.mark.parametrize("act", [None, "gelu_tanh"])
def test_forms_of_the_first_of_two_launches(by_col, swap, more_n, more_lda, act):
    from kraken_b200.fused.gemm_ops import _gemm

    def same(M, N, K):
        plan = _plan(M, N, K, 0, lda=K + more_lda)
        return plan[1] == swap and plan[7] == by_col

    M, N, K = _two_launch_problem(0, 0, same, more_n, more_lda)
    g = torch.Generator(device="cuda").manual_seed(93)
    a = torch.full((M, K + more_lda), float("nan"), device="cuda", dtype=torch.bfloat16)[:, :K]
    a.copy_(torch.randn(M, K, generator=g, device="cuda"))
    bt = (torch.randn(N, K, generator=g, device="cuda") / K ** 0.5).to(torch.bfloat16)
    ref = a.double() @ bt.double().t()
    if act is not None:
        ref = ref * torch.sigmoid(2 * (2 / math.pi) ** 0.5 * (ref + 0.044715 * ref ** 3))
    for out_fp32 in (False, True):
        c = _gemm(a, bt.t(), out_fp32, False, act=act)
        # One rounding of a bf16 result, 2**-8 of the value. The sums (rms 1, below 6) are cut once per MMA of 16 columns, at most
        # 200 * 2**-23 * 6; the device's exp and divide: 1e-4 of the value.
        assert (((c.double() - ref).abs() - (0 if out_fp32 else 2.0 ** -8) * ref.abs()).max()).item() < 1e-3
        assert torch.equal(c, _gemm(a, bt.t(), out_fp32, False, act=act))


def test_plans_can_be_launched():
    # every plan fits the chip and the kernels that exist, and the two launches of a problem share it out without a gap
    import random

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    r = random.Random(12)

    def one_wave(M, N, kb, swap, pair, bn, splits):
        rows, cols = (N, M) if swap else (M, N)
        tiles = -(-rows // (256 if pair else 128)) * -(-cols // bn)
        assert bn in ((128, 160, 192, 224, 256) if pair else (16, 32, 64, 128))
        assert 1 <= splits <= kb and splits * (1 + pair) <= 8 and tiles * splits * (1 + pair) <= sms

    kinds = set()
    for _ in range(4000):
        M, N = (int(2 ** r.uniform(0, 13)) for _ in range(2))
        fp32, pair = r.randint(0, 1), int(r.random() < 0.8)
        K = int(2 ** r.uniform(0, 12)) * (4 if fp32 else 8)
        kb = -(-K // (32 if fp32 else 64))
        kind, swap, bn, rb, splits, two, cut, cut_n, rest_swap, rest_bn, rest_splits, pairs, rest_pairs = _plan(M, N, K, fp32, pair)
        kinds.add((kind, two))
        assert pair or (kind != 2 and not pairs)
        if kind == 1:
            one_wave(M, N, kb, swap, pairs, bn, splits)
        elif kind == 2:
            assert bn in (64, 96, 128, 144, 160, 176, 192, 208, 224, 240, 256) and rb in (1, 2)
            if two:
                assert 0 < cut < (N if cut_n else M) and cut % (bn if cut_n != swap else 256 * rb) == 0
                one_wave(*((M, N - cut) if cut_n else (M - cut, N)), kb, rest_swap, rest_pairs, rest_bn, rest_splits)
        assert two in (0, int(kind == 2))
    assert kinds == {(0, 0), (1, 0), (2, 0), (2, 1)}


def test_gemms_in_two_launches_chained_and_captured():
    # The second launch does not wait for the first one, but nothing after them may start before both are complete, and it
    # must not start before what the first one waits for: every call reads the result of the one before, whose memory the
    # one after next writes.
    M, N, K = _two_launch_problem(0, 0, lambda M, N, K: 2000 < K < N)
    g = torch.Generator(device="cuda").manual_seed(92)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w1 = (torch.randn(N, K, generator=g, device="cuda") / K ** 0.5).to(torch.bfloat16)
    w2 = (torch.randn(K, N, generator=g, device="cuda") / N ** 0.5).to(torch.bfloat16)

    def chain(n, sync):
        y = x
        for _ in range(n):
            y = fused.matmul(y, w1.t())
            if sync:
                torch.cuda.synchronize()
            y = fused.matmul(y, w2.t())
            if sync:
                torch.cuda.synchronize()
        return y

    want = chain(6, True)
    for _ in range(5):
        assert torch.equal(chain(6, False), want)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        chain(1, False)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            y = chain(6, False)
    torch.cuda.current_stream().wait_stream(s)
    for _ in range(3):
        y.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want)


@pytest.mark.parametrize("M,N,bn,swap", [(520, 1024, 1256, 0), (1500, 2080, 2256, 0), (520, 1024, 2144, 0), (777, 1160, 1096, 0), (520, 1024, 1192, 1),
                                         (520, 1001, 1144, 0), (520, 1001, 2128, 1), (16, 1024, 0, -1), (200, 520, 0, -1), (64, 136, 64, 0), (77, 520, 256, 0)])
@pytest.mark.parametrize("out_fp32", [False, True])
def test_activation_is_applied_to_the_fp32_sums_in_every_kernel(M, N, bn, swap, out_fp32):
    # Operands are multiples of 1/32, so the sums are exact in fp32 and mostly not in bf16. What remains is one
    # rounding of the result (8 significant bits: 2**-8 of the value) and the error of the device's exp and divide (below 1e-4).
    from kraken_b200.fused.gemm_ops import _gemm

    K = 72
    g = torch.Generator().manual_seed(61)
    a = (torch.randint(-32, 33, (M, K), generator=g) / 32).to(torch.bfloat16).cuda()
    bt = (torch.randint(-32, 33, (N, K), generator=g) / 32).to(torch.bfloat16).cuda()
    s = a.double() @ bt.double().t()
    ref = s * torch.sigmoid(2 * (2 / math.pi) ** 0.5 * (s + 0.044715 * s ** 3))      # the tanh form, without its cancellation
    h = _gemm(a, bt.t(), out_fp32, False, swap, bn, act="gelu_tanh").double()
    worst = float(((h - ref).abs() / (ref.abs() + 1e-30)).max())
    assert worst <= (0 if out_fp32 else 2.0 ** -8) + 1e-4, worst


def test_one_rank_all_gather_matmul_fills_a_out_like_a_copy():
    # what a_out.copy_(a_shared) accepts is filled, what it refuses is refused
    from kraken_b200.parallel import symm_mem

    M, N, K = 96, 136, 64
    a, bt = _ab(M, N, K, seed=42)
    x = symm_mem.empty(M, K, dtype=torch.bfloat16, device="cuda")
    x.copy_(a)
    ref = fused.matmul(a, bt.t())
    for out in (torch.zeros_like(a), torch.zeros(1, M, K, dtype=torch.bfloat16, device="cuda"), torch.zeros(M, K, device="cuda"),
                torch.zeros(M, 2 * K, dtype=torch.bfloat16, device="cuda")[:, :K]):
        gathered, c = fused.all_gather_matmul(x, bt.t(), a_out=out)
        assert gathered is out and torch.equal(out.reshape(M, K).to(torch.bfloat16), a)
        _close(c, ref.float(), K)
    for out in (torch.zeros(K, M, dtype=torch.bfloat16, device="cuda"), torch.zeros(M * K, dtype=torch.bfloat16, device="cuda"),
                torch.zeros(M, K, dtype=torch.bfloat16, device="cuda", requires_grad=True)):
        with pytest.raises(RuntimeError):
            fused.all_gather_matmul(x, bt.t(), a_out=out)


def test_one_rank_all_gather_matmul_of_one_row_of_a_wider_buffer():
    # one row is contiguous whatever its stride
    from kraken_b200.parallel import symm_mem

    wide = symm_mem.empty(1, 520, dtype=torch.bfloat16, device="cuda")
    a, bt = _ab(1, 136, 264, seed=43)
    x = wide[:, :264]
    x.copy_(a)
    gathered, c = fused.all_gather_matmul(x, bt.t())
    assert torch.equal(gathered, a)
    _close(c, a.float() @ bt.float().t(), 264)


_TMA_STORE_PROBE = """
import ctypes, torch
from kraken_b200 import fused
from kraken_b200.ops import lib as klib
g = torch.Generator().manual_seed(71)
a = torch.randn(520, 264, generator=g).to(torch.bfloat16).cuda()
bt = (0.05 * torch.randn(1032, 264, generator=g)).to(torch.bfloat16).cuda()
ref = a.float() @ bt.float().t()
hits, before, after = ctypes.c_ulonglong(0), ctypes.c_ulonglong(0), ctypes.c_ulonglong(0)
keep = []
for bn in ({bn}):
    for out_dtype in (torch.bfloat16, torch.float32):
        klib.check(klib.lib().kr_tmap_cache_stats(ctypes.byref(hits), ctypes.byref(before)))
        c = fused.matmul(a, bt.t(), out_dtype=out_dtype, bn=bn, swap_ab=0)
        assert ((c.float() - ref).norm() / ref.norm()).item() < 3e-3
        klib.check(klib.lib().kr_tmap_cache_stats(ctypes.byref(hits), ctypes.byref(after)))
        print("maps", after.value - before.value)
        keep.append((a, bt, c))          # fresh addresses for the next call
        a, bt = a.clone(), bt.clone()
"""


@pytest.mark.parametrize("setting,maps", [("1", 3), ("0", 2)])
def test_tma_store_setting_reaches_the_persistent_pairs(setting, maps):
    # read once per process; without TMA stores a call describes its two operands and no output
    import os
    import subprocess
    import sys

    r = subprocess.run([sys.executable, "-c", _TMA_STORE_PROBE.format(bn="1256, 2192")], env={**os.environ, "KRAKEN_TMA_STORE": setting},
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))), capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
    assert [int(line.split()[1]) for line in r.stdout.splitlines() if line.startswith("maps")] == [maps] * 4, r.stdout


@pytest.mark.parametrize("M,hidden,ffn", [(65, 264, 1096), (300, 512, 1032), (777, 520, 2024), (2100, 1160, 4104), (300, 512, 1088)])
def test_prefill_at_one_rank_with_ragged_ffn(M, hidden, ffn):
    # the up projection's rows are padded to whole 128-byte lines when ffn is not a multiple of 64; what the padding
    # holds (NaN here) must not reach the down projection
    from kraken_b200.fused.gemm_ops import all_gather_matmul_act
    from kraken_b200.models import TPMLP

    mlp = TPMLP(hidden, ffn, device="cuda", seed=5)
    x = (0.5 * torch.randn(M, hidden, generator=torch.Generator().manual_seed(92))).to(torch.bfloat16).cuda()
    xs = mlp.stage_input(x)
    padded = -(-ffn // 64) * 64
    h = all_gather_matmul_act(xs, mlp.w_up_t.t(), "gelu_tanh")
    assert h.shape == (M, ffn) and h.stride(0) == padded
    if padded != ffn:
        torch.as_strided(h, (M, padded - ffn), (padded, 1), ffn).fill_(float("nan"))
    s = x.double() @ mlp.w_up_t.double().t()
    gelu = s * torch.sigmoid(2 * (2 / math.pi) ** 0.5 * (s + 0.044715 * s ** 3))
    # one bf16 rounding per element: at most 2**-8, half of that root mean square or less
    assert ((h.double() - gelu).norm() / gelu.norm()).item() < 2.0 ** -9 + 1e-4
    ref = gelu.to(torch.bfloat16).double() @ mlp.w_down_t.double().t()
    y = fused.gemm_reduce_scatter(h, mlp.w_down_t.t())
    assert y.shape == (M, hidden) and ((y.double() - ref).norm() / ref.norm()).item() < 3e-3
    assert torch.equal(mlp.prefill(xs), y)


def test_tile_counters_of_many_streams_and_threads():
    # Every stream has counter words of its own, more streams than the pool keeps among them, used by two threads
    # at a time. Whole tiles would be missing or stale if two launches drew from the same words.
    import threading

    a, bt = _ab(2048, 2600, 264, seed=93)
    want = fused.matmul(a, bt.t())
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(priority=p) for p in (0, -1) for _ in range(24)]
    outs, errors = {}, []

    def work(mine):
        try:
            for i in mine:
                with torch.cuda.stream(streams[i]):
                    outs[i] = [fused.matmul(a, bt.t()) for _ in range(4)]
        except Exception as e:
            errors.append(e)

    for _ in range(2):
        threads = [threading.Thread(target=work, args=(range(k, len(streams), 2),)) for k in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        torch.cuda.synchronize()
        assert not errors, errors
        for i in range(len(streams)):
            assert all(torch.equal(c, want) for c in outs[i]), i
        outs.clear()


def test_tile_counters_stay_out_of_dispatch_modes():
    # the counter words of a new stream are made under a lock: a mode that sees their allocation could replace them
    # or wait in Python while it is held
    from torch.utils._python_dispatch import TorchDispatchMode

    class Recorder(TorchDispatchMode):
        def __init__(self):
            super().__init__()
            self.seen = []

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.seen.append(str(func))
            return func(*args, **(kwargs or {}))

    a, bt = _ab(2048, 2600, 264, seed=96)
    b = bt.t()
    want = fused.matmul(a, b)
    for _ in range(2):                      # the first call on a stream, and on one whose words are there
        for stream in [torch.cuda.Stream() for _ in range(40)]:
            with torch.cuda.stream(stream), Recorder() as mode:
                stream.wait_stream(torch.cuda.default_stream())
                c = fused.matmul(a, b)
            assert mode.seen == []
            stream.synchronize()
            assert torch.equal(c, want)
