"""Single-GPU numerics of the memory-bound collectives and the fused bias / RMSNorm epilogues,
at world size 1 and at emulated world sizes 2/4/8 (all ranks of a kernel run as ONE cooperative
launch on one GPU). Every result is compared with a plain PyTorch fp32 computation of the same op.
Shapes follow the reference's tests: [1024, 1024] bf16 for all-reduce (test/test_allreduce.py:52),
x/bias [b, 5120] for the bias ops (test/test_allreduce_bias.py:57-71)."""
import pytest
import torch

from kraken_b200 import comm, fused
from kraken_b200.parallel import EmuWorld, symm_mem

pytestmark = pytest.mark.gpu


def _inputs(ws, shape, seed=0):
    return [torch.randn(*shape, generator=torch.Generator().manual_seed(seed + 42 + r)).to(torch.bfloat16).cuda()
            for r in range(ws)]


def _poison(t):
    t.view(torch.int16).fill_(-1)     # NaN pattern: unwritten outputs are detected


@pytest.mark.parametrize("ws", [1, 2, 4, 8])
@pytest.mark.parametrize("shape", [(1024, 1024), (3, 40), (7, 1000)])
def test_one_shot_all_reduce(ws, shape):
    world = EmuWorld(ws)
    xs = _inputs(ws, shape)
    ts = world.symmetric(shape, torch.bfloat16)
    for r in range(ws):
        ts[r].copy_(xs[r])
    expect = sum(x.float() for x in xs)
    outs = world.run(lambda r: comm.one_shot_all_reduce(ts[r]))
    for r in range(ws):
        torch.testing.assert_close(outs[r].float(), expect, atol=1e-1, rtol=1e-1)
    # bitwise-identical across ranks? (rotated peer order -> not required); but repeatable:
    outs2 = world.run(lambda r: comm.one_shot_all_reduce(ts[r]))
    for r in range(ws):
        assert torch.equal(outs[r], outs2[r])


@pytest.mark.parametrize("ws", [1, 2, 4, 8])
@pytest.mark.parametrize("numel", [1024 * 1024, 8 * 4096 + 64, 40])
def test_two_shot_all_reduce(ws, numel):
    world = EmuWorld(ws)
    xs = _inputs(ws, (numel,))
    expect = sum(x.float() for x in xs)
    for _ in range(2):        # second round: staging workspace reused, pads must have reset
        outs = world.run(lambda r: comm.two_shot_all_reduce(xs[r]))
        for r in range(ws):
            torch.testing.assert_close(outs[r].float(), expect, atol=1e-1, rtol=1e-1)
        for r in range(1, ws):
            assert torch.equal(outs[0], outs[r])      # every rank receives the same bits


@pytest.mark.parametrize("ws", [1, 2, 4])
def test_multimem_all_reduce_falls_back_in_place(ws):
    world = EmuWorld(ws)          # emulated ranks have no multicast mapping: P2P form, same contract
    xs = _inputs(ws, (64, 1024))
    ts = world.symmetric((64, 1024), torch.bfloat16)
    for r in range(ws):
        ts[r].copy_(xs[r])
    expect = sum(x.float() for x in xs)
    outs = world.run(lambda r: comm.multimem_all_reduce(ts[r]))
    for r in range(ws):
        assert outs[r].data_ptr() == ts[r].data_ptr()
        torch.testing.assert_close(ts[r].float(), expect, atol=1e-1, rtol=1e-1)


@pytest.mark.parametrize("ws", [1, 2, 4, 8])
@pytest.mark.parametrize("symmetric_input", [True, False])
def test_reduce_scatter(ws, symmetric_input):
    world = EmuWorld(ws)
    shape = (ws * 96, 256)
    xs = _inputs(ws, shape)
    expect = sum(x.float() for x in xs)
    if symmetric_input:
        ts = world.symmetric(shape, torch.bfloat16)
        for r in range(ws):
            ts[r].copy_(xs[r])
        src = ts
    else:
        src = xs
    outs = world.run(lambda r: comm.reduce_scatter(src[r]))
    for r in range(ws):
        torch.testing.assert_close(outs[r].float(), expect[r * 96:(r + 1) * 96], atol=1e-1, rtol=1e-1)


@pytest.mark.parametrize("ws", [1, 2, 4, 8])
@pytest.mark.parametrize("splits", [1, 2, 4])
def test_all_gather_w_progress_sm(ws, splits):
    world = EmuWorld(ws)
    shape = (256, 1024)
    xs = _inputs(ws, shape)
    ts = world.symmetric(shape, torch.bfloat16)
    for r in range(ws):
        ts[r].copy_(xs[r])
    progs = [torch.zeros(ws * splits, dtype=torch.uint32, device="cuda") for _ in range(ws)]
    outs = world.run(lambda r: comm.all_gather_w_progress(ts[r], progress=progs[r], splits_per_rank=splits,
                                                          backend="sm"))
    expect = torch.cat(xs, 0)
    for r in range(ws):
        assert torch.equal(outs[r], expect)
        assert bool((progs[r].to(torch.int64) != 0).all())


@pytest.mark.parametrize("ws", [1, 2, 4, 8])
@pytest.mark.parametrize("b", [1, 2, 16, 64])
@pytest.mark.parametrize("full_bias", [True, False])
def test_all_reduce_bias(ws, b, full_bias):
    world = EmuWorld(ws)
    D = 5120
    xs = _inputs(ws, (b, D))
    bias = torch.randn(b, D).to(torch.bfloat16).cuda() if full_bias else torch.randn(D).to(torch.bfloat16).cuda()
    pads = world.symmetric((1024, 1024), torch.bfloat16)
    expect = sum(x.float() for x in xs) + bias.float()
    for fn in (fused.one_shot_all_reduce_bias, fused.two_shot_all_reduce_bias):
        outs = [torch.empty_like(xs[0]) for _ in range(ws)]
        for o in outs:
            _poison(o)
        world.run(lambda r: fn(pads[r], xs[r], bias, outs[r]))
        for r in range(ws):
            torch.testing.assert_close(outs[r].float(), expect, atol=5e-2, rtol=5e-2)
    # no bias
    outs = [torch.empty_like(xs[0]) for _ in range(ws)]
    world.run(lambda r: fused.one_shot_all_reduce_bias(pads[r], xs[r], None, outs[r]))
    torch.testing.assert_close(outs[0].float(), sum(x.float() for x in xs), atol=5e-2, rtol=5e-2)


def _rms_ref(x, w, eps):
    xf = x.float()
    return xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + eps) * w.float()


@pytest.mark.parametrize("rows,D", [(1, 5120), (64, 5120), (300, 8192), (5, 64), (2, 40000)])
def test_rms_norm(rows, D):
    x = torch.randn(rows, D).to(torch.bfloat16).cuda()
    w = (1 + 0.1 * torch.randn(D)).to(torch.bfloat16).cuda()
    y = fused.rms_norm(x, w, 1e-5)
    torch.testing.assert_close(y.float(), _rms_ref(x, w, 1e-5), atol=4e-2, rtol=4e-2)


@pytest.mark.parametrize("ws", [1, 2, 4, 8])
@pytest.mark.parametrize("b", [1, 4, 32, 200])
@pytest.mark.parametrize("D", [5120, 8192])
def test_all_reduce_bias_rms_norm(ws, b, D):
    world = EmuWorld(ws)
    xs = _inputs(ws, (b, D))
    bias = torch.randn(D).to(torch.bfloat16).cuda()
    fullbias = torch.randn(b, D).to(torch.bfloat16).cuda()
    w = (1 + 0.1 * torch.randn(D)).to(torch.bfloat16).cuda()
    pads = world.symmetric((b * D + 64,), torch.bfloat16)
    for bb in (bias, fullbias):
        total = sum(x.float() for x in xs) + bb.float()
        expect = _rms_ref(total, w, 1e-5)
        for fn in (fused.one_shot_all_reduce_bias_rms_norm, fused.two_shot_all_reduce_bias_rms_norm):
            ys = [torch.empty_like(xs[0]) for _ in range(ws)]
            for y in ys:
                _poison(y)
            world.run(lambda r: fn(pads[r], xs[r], bb, w, ys[r], 1e-5))
            for r in range(ws):
                torch.testing.assert_close(ys[r].float(), expect, atol=4e-2, rtol=4e-2)


# ---- push-style one-shot kernels (small messages) ------------------------------------------------
@pytest.mark.parametrize("ws", [1, 2, 4, 8])
@pytest.mark.parametrize("numel", [8, 2048, 5120 * 3, 64 * 1024])
@pytest.mark.parametrize("with_bias", [False, True])
def test_push_and_pull_one_shot_agree(ws, numel, with_bias):
    world = EmuWorld(ws)
    xs = _inputs(ws, (numel,), seed=31)
    bias = torch.randn(numel, generator=torch.Generator().manual_seed(5)).to(torch.bfloat16).cuda() if with_bias else None
    expect = sum(x.float() for x in xs) + (bias.float() if with_bias else 0.0)
    pads = world.symmetric((numel,), torch.bfloat16)
    res = {}
    for algo in ("push", "pull"):
        for _ in range(3):          # three calls: both workspace halves, then the first again
            outs = [torch.empty_like(xs[r]) for r in range(ws)]
            for o in outs:
                _poison(o)
            world.run(lambda r: fused.one_shot_all_reduce_bias(pads[r], xs[r], bias, outs[r], algo=algo))
            for r in range(ws):
                torch.testing.assert_close(outs[r].float(), expect, atol=5e-2, rtol=5e-2)
        res[algo] = outs
    for r in range(ws):
        assert torch.equal(res["push"][0], res["push"][r])      # rank-order sums: same bits on every rank


@pytest.mark.parametrize("ws", [1, 2, 4, 8])
@pytest.mark.parametrize("b,D", [(1, 5120), (3, 5120), (16, 1024), (40, 8192), (2, 64), (2, 8192), (4, 4096)])
def test_push_all_reduce_bias_rms_norm(ws, b, D):
    world = EmuWorld(ws)
    xs = _inputs(ws, (b, D), seed=33)
    g = torch.Generator().manual_seed(6)
    bias = torch.randn(D, generator=g).to(torch.bfloat16).cuda()
    w = (1 + 0.1 * torch.randn(D, generator=g)).to(torch.bfloat16).cuda()
    s = sum(x.float() for x in xs) + bias.float()
    expect = s * torch.rsqrt(s.pow(2).mean(-1, keepdim=True) + 1e-5) * w.float()
    pads = world.symmetric((b, D), torch.bfloat16)
    for algo in ("push", "pull"):
        for _ in range(2):
            ys = [torch.empty_like(xs[r]) for r in range(ws)]
            for y in ys:
                _poison(y)
            world.run(lambda r: fused.one_shot_all_reduce_bias_rms_norm(pads[r], xs[r], bias, w, ys[r], 1e-5, algo=algo))
            for r in range(ws):
                torch.testing.assert_close(ys[r].float(), expect, atol=4e-2, rtol=4e-2)


def test_push_tagged_and_flag_forms_share_a_workspace(monkeypatch):
    # small messages travel tagged (no barrier), larger ones behind one barrier; both forms alternate
    # workspace halves by the same call counter and must never read each other's leftovers
    ws, numel = 4, 4096
    world = EmuWorld(ws)
    pads = world.symmetric((numel,), torch.bfloat16)
    for i, kb in enumerate([64, 0, 64, 64, 0, 0, 64, 0, 64]):
        monkeypatch.setenv("KRAKEN_PUSH_TAGGED_KB", str(kb))
        xs = _inputs(ws, (numel,), seed=100 + i)
        expect = sum(x.float() for x in xs)
        outs = [torch.empty_like(xs[r]) for r in range(ws)]
        for o in outs:
            _poison(o)
        world.run(lambda r: fused.one_shot_all_reduce_bias(pads[r], xs[r], None, outs[r], algo="push"))
        for r in range(ws):
            torch.testing.assert_close(outs[r].float(), expect, atol=5e-2, rtol=5e-2)
            assert torch.equal(outs[0], outs[r])


@pytest.mark.parametrize("rows,D", [(1, 8), (2, 1032), (1, 8200), (3, 16392), (2, 32768), (297, 1024), (300, 1032),
                                    (297, 8192), (300, 8200), (300, 16392)])
@pytest.mark.parametrize("bias", ["none", "row", "full"])
def test_one_rank_forms(rows, D, bias):
    # world size 1 outside any emulation: no exchange, one pass (few rows: a thread per vector; many: 128-thread blocks)
    x = symm_mem.empty(rows, D, dtype=torch.bfloat16, device="cuda")
    x.copy_(_inputs(1, (rows, D))[0])
    w = (1 + 0.1 * torch.randn(D)).to(torch.bfloat16).cuda()
    b = {"none": None, "row": torch.randn(D).to(torch.bfloat16).cuda(), "full": torch.randn(rows, D).to(torch.bfloat16).cuda()}[bias]
    s = x.float() + (b.float() if b is not None else 0)
    for fn in (fused.one_shot_all_reduce_bias_rms_norm, fused.two_shot_all_reduce_bias_rms_norm):
        y = torch.empty_like(x)
        _poison(y)
        fn(x, x, b, w, y)
        torch.testing.assert_close(y.float(), _rms_ref(s, w, 1e-5), atol=4e-2, rtol=2e-2)
    for fn in (fused.one_shot_all_reduce_bias, fused.two_shot_all_reduce_bias):
        out = torch.empty_like(x)
        _poison(out)
        fn(x, x, b, out)
        assert torch.equal(out, s.to(torch.bfloat16))
    assert torch.equal(comm.all_reduce(x), x) and torch.equal(comm.reduce_scatter(x), x)
    torch.testing.assert_close(fused.rms_norm(x, w).float(), _rms_ref(x, w, 1e-5), atol=4e-2, rtol=2e-2)


@pytest.mark.parametrize("rows,D", [(1, 8), (5, 1000), (16, 8192), (300, 5120)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_rounded_bias_rms_norm_rounds_like_separate_ops(rows, D, dtype):
    from kraken_b200.ops import host

    p = torch.randn(rows, D, device="cuda", dtype=dtype)
    bias = torch.randn(D, device="cuda").to(torch.bfloat16)
    w = (1 + 0.1 * torch.randn(D, device="cuda")).to(torch.bfloat16)
    x = (p.to(torch.bfloat16).float() + bias.float()).to(torch.bfloat16)
    y = host.rounded_bias_rms_norm(p, bias, w, 1e-5)
    torch.testing.assert_close(y.float(), _rms_ref(x, w, 1e-5), atol=1e-2, rtol=1e-2)
    assert torch.equal(y, fused.rms_norm(x, w))


@pytest.mark.parametrize("rows,D", [(3552, 8), (3552, 2552), (3600, 2560), (4000, 1000), (3552, 32768), (3552, 32776)])
def test_rms_norm_of_thousands_of_rows(rows, D):
    x = torch.randn(rows, D, device="cuda").to(torch.bfloat16)
    w = (1 + 0.1 * torch.randn(D, device="cuda")).to(torch.bfloat16)
    torch.testing.assert_close(fused.rms_norm(x, w).float(), _rms_ref(x, w, 1e-5), atol=4e-2, rtol=2e-2)


@pytest.mark.parametrize("ws", [1, 2, 4])
@pytest.mark.parametrize("form", ["one_shot", "two_shot"])
@pytest.mark.parametrize("rows,D", [(3, 1024), (300, 5120)])
def test_where_bias_rms_norm_rounds_its_sums(ws, form, rows, D):
    # Inputs are multiples of 1/64 below 4, so the sums are exact in fp32. What is normalised: the bf16 sums where they are
    # published (two-shot, several ranks), else the fp32 sums. Left over: one bf16 rounding of the result (2**-8) and
    # a few fp32 roundings (below 1e-5); the other choice of sums is off by about 2**-8 more for many elements.
    g = torch.Generator().manual_seed(91)
    grid = lambda *shape: (torch.randint(-255, 256, shape, generator=g) / 64).to(torch.bfloat16).cuda()
    xs, bias = [grid(rows, D) for _ in range(ws)], grid(D)
    w = (1 + 0.1 * torch.randn(D, generator=g)).to(torch.bfloat16).cuda()
    op = fused.one_shot_all_reduce_bias_rms_norm if form == "one_shot" else fused.two_shot_all_reduce_bias_rms_norm
    ys = [torch.empty_like(x) for x in xs]
    if ws == 1:
        scratch = symm_mem.empty(rows, D, dtype=torch.bfloat16, device="cuda")
        op(scratch, xs[0], bias, w, ys[0])
    else:
        world = EmuWorld(ws)
        scratch = world.symmetric((rows, D), torch.bfloat16)
        world.run(lambda r: op(scratch[r], xs[r], bias, w, ys[r]))
    s = sum(x.double() for x in xs) + bias.double()
    published = form == "two_shot" and ws > 1

    def worst(sums):
        ref = sums * torch.rsqrt(sums.pow(2).mean(-1, keepdim=True) + 1e-5) * w.double()
        return max(float(((y.double() - ref).abs() / (ref.abs() + 1e-30)).max()) for y in ys)

    rounded = s.to(torch.bfloat16).double()
    assert worst(rounded if published else s) <= 2.0 ** -8 + 1e-5
    assert worst(s if published else rounded) > 2.0 ** -8 + 1e-5


@pytest.mark.parametrize("rows,D,K", [(128, 40960, 2048), (3600, 4096, 1024), (16, 8192, 4096), (600, 5120, 2048), (40, 16392, 2048)])
def test_chain_of_overlapped_launches(rows, D, K):
    # Each kernel starts while the one before it still runs and must wait for it before it reads; the norms here are
    # the long-row, the streaming and the row-per-block kernels. Same bits as with a synchronisation after every step.
    g = torch.Generator().manual_seed(95)
    bt = (0.05 * torch.randn(D, K, generator=g)).to(torch.bfloat16).cuda()
    w = (1 + 0.1 * torch.randn(D, generator=g)).to(torch.bfloat16).cuda()
    scratch = symm_mem.empty(rows, D, dtype=torch.bfloat16, device="cuda")
    bias = torch.randn(D, generator=g).to(torch.bfloat16).cuda()
    bufs = [torch.empty(rows, D, dtype=torch.bfloat16, device="cuda") for _ in range(2)]

    def chain(a, after):
        x = fused.matmul(a, bt.t())
        after()
        x = fused.rms_norm(x, w)
        after()
        fused.one_shot_all_reduce_bias(scratch, x, bias, bufs[0])
        after()
        x = fused.rms_norm(bufs[0], w)
        after()
        fused.two_shot_all_reduce_bias(scratch, x, bias, bufs[1])
        after()
        return fused.rms_norm(bufs[1], w)

    for _ in range(4):
        a = torch.randn(rows, K, generator=g).to(torch.bfloat16).cuda()
        want = chain(a, torch.cuda.synchronize)
        torch.cuda.synchronize()
        for b in bufs:
            _poison(b)
        torch.cuda.synchronize()
        assert torch.equal(chain(a, lambda: None), want)
