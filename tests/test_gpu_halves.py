"""GPU: products of fp16 halves on the tensor-core kernel: what holds for operands of any magnitude, in every family that runs on it
and under capture."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def halves(ctx, monkeypatch):
    monkeypatch.setenv("PETB200_TC_MATH", "f16x3")
    monkeypatch.setattr(ctx, "_plans", {})  # none that another test made with another arithmetic


def _weights(shape, small, filter_dim, seed):
    """Gaussian weights in which the filters `small` are too small for a half."""
    w = torch.randn(shape, generator=torch.Generator().manual_seed(seed))
    w.movedim(filter_dim, 0)[small] *= 1e-6
    return w.cuda()


def _captured(call):
    """`call` captured into a CUDA graph, and what it returned there."""
    call()  # (lazily made plans)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = call()
    return graph, out


def _replay(graph, out):
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    return out.clone()


# A captured launch is replayed after its plan's operand has been packed again: with the same weights, with others whose small
# filters are elsewhere, and with none small
@pytest.mark.parametrize("kind", ["conv2d", "convtrans_phases", "convtrans", "matmul"])
def test_captured_launch_after_a_new_packing(ctx, monkeypatch, kind):
    if kind == "conv2d":
        x, shape, fdim = torch.randn(2, 32, 12, 12, device="cuda"), (40, 32, 3, 3), 0
        plan = ctx.conv2d_plan(x.shape, shape, 1, 1)
        set_weights, run = lambda w: ctx.conv2d_set_weights(plan, w), lambda: ctx.conv2d_run(plan, x)
    elif kind == "matmul":
        x, shape, fdim = torch.randn(1, 70, 96, device="cuda"), (1, 96, 65), 2
        plan = ctx.matmul_plan(x.shape, shape)
        set_weights, run = lambda w: ctx.matmul_set_weights(plan, w), lambda: ctx.matmul_run(plan, x, None)
    else:
        monkeypatch.setenv("PETB200_CONVTRANS_PHASES", "1" if kind == "convtrans_phases" else "0")
        x, shape, fdim = torch.randn(2, 8, 8, 32, device="cuda"), (4, 4, 32, 24), 3
        plan = ctx.convtrans_plan(x.shape, shape, 1, 1, 2, 2)
        set_weights, run = lambda w: ctx.convtrans_run(plan, x, w), lambda: ctx.convtrans_run(plan, x)
    assert plan.kernel == "tc_3xtf32_f16_ts"
    first = _weights(shape, [3, 7], fdim, 1)
    set_weights(first)
    graph, out = _captured(run)
    for w in (first, _weights(shape, [5], fdim, 2), _weights(shape, [], fdim, 3), first):
        set_weights(w)
        assert torch.equal(run(), _replay(graph, out))
    ctx.sync_check()


# A declared weight packed again because another B came in between
def test_captured_matmul_after_another_operand(ctx):
    a, w, other = torch.randn(1, 70, 96, device="cuda"), _weights((1, 96, 65), [3, 7], 2, 1), _weights((1, 96, 65), [], 2, 2)
    plan = ctx.matmul_plan(a.shape, w.shape)
    ctx.matmul_set_weights(plan, w)
    graph, out = _captured(lambda: ctx.matmul_run(plan, a, None))
    want = ctx.matmul_run(plan, a, None)
    ctx.matmul_run(plan, a, other)
    assert torch.equal(ctx.matmul_run(plan, a, None), want) and torch.equal(_replay(graph, out), want)
    ctx.sync_check()


# The packing itself captured with the product, and other operands packed between two replays
@pytest.mark.parametrize("kind", ["conv2d", "conv3d", "matmul", "matmul_trans_b"])
def test_captured_packing_after_another(ctx, kind):
    if kind.startswith("matmul"):
        x, shape, fdim = torch.randn(3, 70, 96, device="cuda"), (3, 65, 96) if kind == "matmul_trans_b" else (3, 96, 65), 1 if kind == "matmul_trans_b" else 2
        call = lambda w: ctx.matmul(x, w, False, kind == "matmul_trans_b")
    elif kind == "conv2d":
        x, shape, fdim = torch.randn(2, 32, 12, 12, device="cuda"), (40, 32, 3, 3), 0
        call = lambda w: ctx.conv2d(x, w, 1, 1)
    else:
        x, shape, fdim = torch.randn(1, 16, 4, 8, 8, device="cuda"), (33, 16, 3, 3, 3), 0
        call = lambda w: ctx.conv3d(x, w, (1, 1, 1))
    w = _weights(shape, [3, 7], fdim, 1)
    graph, out = _captured(lambda: call(w))
    for i, new in enumerate((w, _weights(shape, [5], fdim, 2), _weights(shape, [], fdim, 3))):
        w.copy_(new)  # what the captured packing reads
        between = _weights(shape, [1] if i != 1 else [], fdim, 4 + i)
        want = call(w)
        call(between)
        assert torch.equal(_replay(graph, out), want)
    ctx.sync_check()


# Operator by operator (the profiled run) and as one captured graph in turn: the same sums of a filter that is too small for a half
def test_graph_runs_around_a_profiled_run(ctx):
    from pet_b200 import configs
    from pet_b200.graph import Graph
    graph = Graph(ctx)
    b = configs.GraphBuilder(graph)
    x, w = np.random.default_rng(0).standard_normal((2, 32, 12, 12), np.float32), _weights((40, 32, 3, 3), [3, 7], 0, 1).cpu().numpy()
    out = b.conv(b.input(x), b.const(w), 1, 1)
    graph.setOutputs([out])
    graph.compile()
    b.load()
    assert [k for _, k in graph.steps()] == ["tc_3xtf32_f16_ts"]
    graph.run()
    before = graph.get_data(out).copy()
    graph.run_profiled(0, 1)
    assert np.array_equal(graph.get_data(out), before)
    graph.run()
    assert np.array_equal(graph.get_data(out), before)
    ctx.sync_check()


# Row and filter both so large (or small) that the product of their factors is no float, while the results are: zero sums of huge values that
# meet zeros, sums of tiny values near the smallest normal number, huge rows with tiny filters and the other way round.  One tile per CTA,
# several (narrow, wide), K split.
@pytest.mark.parametrize("m,n,k", [(130, 40, 64), (5000, 60, 130), (5000, 200, 900), (64, 64, 2048)])
@pytest.mark.parametrize("row,filt", [(2.0 ** 100, 2.0 ** 100), (2.0 ** -62, 2.0 ** -61), (2.0 ** 90, 2.0 ** -100), (2.0 ** -110, 2.0 ** 96)])
def test_factors_of_row_and_filter_beyond_a_float(ctx, m, n, k, row, filt):
    gen = torch.Generator().manual_seed(m + n)
    a, w = torch.randn(m, k, generator=gen), torch.randn(k, n, generator=gen)
    if row * filt > 2.0 ** 128:  # nothing huge meets anything but zero
        a[:, k // 2:], w[:k // 2] = 0, 0
    a, w = a * row, w * filt
    plan = ctx.matmul_plan((1, m, k), (1, k, n))
    assert plan.kernel == "tc_3xtf32_f16_ts"
    ctx.matmul_set_weights(plan, w.cuda()[None])
    got = ctx.matmul_run(plan, a.cuda()[None], None)[0].cpu().double()
    ctx.sync_check()
    a, w = a.double(), w.double()
    # (3 * 2^-22 of each product dropped, K / 16 MMAs that each truncate a sum twice: see the tests over all magnitudes)
    bound = 2.0 ** -22 * ((4 + k / 8) * (a.abs() @ w.abs()) + a.abs().amax(1, keepdim=True) * w.abs().sum(0, keepdim=True) * (row * filt <= 2.0 ** 128))
    assert bool(((got - a @ w).abs() <= bound + 2.0 ** -149).all())


# Values of very different size in one row or filter, the largest of which meet zeros: what is left of the small ones decides.  No less
# precise than three products of TF32.
@pytest.mark.parametrize("top,rest", [(1.0, 1.0), (1.0, 1e-6), (1.0, 1e-7), (1e-4, 1e-7), (200.0, 1e-6), (900.0, 1e-4), (0.02, 1e-6), (3e-3, 1e-7), (1e-9, 1e-15), (1e9, 1e3)])
@pytest.mark.parametrize("where", ["rows", "filters"])
@pytest.mark.parametrize("kind", ["matmul", "matmul_trans_b", "matmul_weight", "conv2d"])
def test_mixed_magnitudes_no_less_precise_than_tf32(ctx, monkeypatch, kind, where, top, rest):
    gen = torch.Generator().manual_seed(7)
    m, n, k = 288, 64, 512
    big, other = torch.randn(m if where == "rows" else n, k, generator=gen) * rest, torch.randn(n if where == "rows" else m, k, generator=gen)
    big[:, 5], other[:, 5] = top, 0.0
    x, w = ((big, other) if where == "rows" else (other, big))
    want = x.double() @ w.double().t()

    def product(math):
        monkeypatch.setenv("PETB200_TC_MATH", math)
        if kind == "conv2d":
            xd, wd = x.t().reshape(1, k, 12, 24).contiguous().cuda(), w.reshape(n, k, 1, 1).cuda()
            plan = ctx.conv2d_plan(xd.shape, wd.shape, 0, 0)
            ctx.conv2d_set_weights(plan, wd)
            got = ctx.conv2d_run(plan, xd).reshape(n, m).t()
        else:
            wd = (w if kind == "matmul_trans_b" else w.t().contiguous()).cuda()[None]
            plan = ctx.matmul_plan((1, m, k), wd.shape, False, kind == "matmul_trans_b")
            if kind == "matmul_weight":
                ctx.matmul_set_weights(plan, wd)
            got = ctx.matmul_run(plan, x.cuda()[None], None if kind == "matmul_weight" else wd)[0]
        assert plan.kernel == ("tc_3xtf32_f16_ts" if math == "f16x3" else "tc_3xtf32_ts")
        return float((got.cpu().double() - want).norm() / want.norm())

    halves, tf32 = product("f16x3"), product("3xtf32")
    ctx.sync_check()
    assert halves <= tf32, (halves, tf32)


# Many tiles per CTA: with one row out of range a CTA repeats all of its tiles, those of more than eight twice in a row; narrow tiles, wide ones
# with a flush, tiles of a single K stage (which one transform set sees alone)
@pytest.mark.parametrize("m,n,k", [(148 * 128 * 8, 60, 130), (148 * 128 * 11 + 5, 60, 130), (148 * 128 * 9, 40, 50), (148 * 128 * 3, 40, 50), (20000, 1280, 800), (9000, 1280, 800)])
@pytest.mark.parametrize("rows", ["some", "all"])
def test_second_pass_of_many_tiles(ctx, m, n, k, rows):
    gen = torch.Generator(device="cuda").manual_seed(m + k)
    a, w = torch.randn(m, k, device="cuda", generator=gen), torch.randn(k, n, device="cuda", generator=gen)
    a[:: 997 if rows == "some" else 1] *= 1e-9
    a[5::1999] *= 1e7
    w[:, 3] *= 1e-7
    plan = ctx.matmul_plan((1, m, k), (1, k, n))
    assert plan.kernel == "tc_3xtf32_f16_ts"
    ctx.matmul_set_weights(plan, w[None])
    got = ctx.matmul_run(plan, a[None], None)[0].double()
    ctx.sync_check()
    a, w = a.double(), w.double()
    # (as in the tests over all magnitudes; the values of a row or filter are of one magnitude here)
    bound = 2.0 ** -22 * ((4 + k / 8) * (a.abs() @ w.abs()) + a.abs().amax(1, keepdim=True) * w.abs().sum(0, keepdim=True))
    assert bool(((got - a @ w).abs() <= bound).all())


# What a context asks of the device once (cluster sizes, shared-memory limits) is kept per context: contexts of several threads plan the same
def test_contexts_of_two_threads(ctx):
    import threading
    from pet_b200.ops import Context
    x, w = torch.randn(2, 64, 16, 16, device="cuda"), torch.randn(48, 64, 3, 3, device="cuda")
    a, b = torch.randn(1, 16, 2048, device="cuda"), torch.randn(1, 2048, 96, device="cuda")
    want, got = (ctx.conv2d(x, w, 1, 1), ctx.matmul(a, b)), {}
    torch.cuda.synchronize()

    def work(i):
        own = Context(0)
        got[i] = (own.conv2d(x, w, 1, 1), own.matmul(a, b))
        own.sync_check()
        own.close()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i in range(2):
        assert all(torch.equal(p, q) for p, q in zip(got[i], want))


# What a product of halves, or three of TF32, may be off by: what the products leave out (2^-21 and 3 * 2^-20 of each), and the sum that the
# tensor core truncates after each of K / 8 or fewer MMAs, twice 2^-23 of it at most for each of the two accumulators.
def _within_bound(got, x2, w2):
    """x2 [rows, K], w2 [K, cols], float64, the values of a row or filter of one magnitude."""
    bound = 2.0 ** -22 * ((12 + x2.shape[1] / 4) * (x2.abs() @ w2.abs()) + x2.abs().amax(1, keepdim=True) * w2.abs().sum(0, keepdim=True))
    return bool(((got.double() - x2 @ w2).abs() <= bound).all())


def _some_rows(shape, channel_dim, gen):
    """Values of which some pixels are too small and some too large for halves."""
    x = torch.randn(shape, generator=gen).movedim(channel_dim, -1)
    scale = torch.tensor([1.0, 1.0, 1e-9, 1e7])[torch.randint(0, 4, x.shape[:-1], generator=gen)]
    return (x * scale.unsqueeze(-1)).movedim(-1, channel_dim).contiguous()


# A group's rows are scaled by the group's own values: the last channels that are fetched with 48 or 40 of a group are its neighbour's
@pytest.mark.parametrize("cpg,fg,groups,h,w,k", [(48, 64, 2, 12, 12, 3), (40, 48, 3, 10, 16, 3), (36, 33, 2, 9, 11, 3), (36, 33, 2, 90, 110, 1), (64, 64, 2, 12, 12, 3), (16, 40, 4, 8, 20, 3), (96, 130, 2, 30, 64, 1)])
@pytest.mark.parametrize("scale", [1e-13, 1e-9, 1.0, 1e9])
def test_groups_of_different_magnitude(ctx, cpg, fg, groups, h, w, k, scale):
    gen = torch.Generator().manual_seed(cpg + fg)
    x, wt = torch.randn(2, groups * cpg, h, w, generator=gen), torch.randn(groups * fg, cpg, k, k, generator=gen)
    x[:, :cpg] *= scale
    wt[fg + 3] *= 1e-7  # a filter of the second group has a factor
    plan = ctx.conv2d_plan(x.shape, wt.shape, k // 2, k // 2)
    ctx.conv2d_set_weights(plan, wt.cuda())
    got = ctx.conv2d_run(plan, x.cuda()).cpu()
    ctx.sync_check()
    for g in range(groups):
        cols = torch.nn.functional.unfold(x[:, g * cpg:(g + 1) * cpg].double(), k, padding=k // 2).transpose(1, 2).reshape(-1, cpg * k * k)
        mine = got[:, g * fg:(g + 1) * fg].permute(0, 2, 3, 1).reshape(-1, fg)
        assert _within_bound(mine, cols, wt[g * fg:(g + 1) * fg].reshape(fg, -1).double().t())
    # (36 channels in planes of odd width are fetched whole, in chunks that divide the group)
    assert plan.kernel == ("tc_3xtf32_ts" if cpg in (48, 40) else "tc_3xtf32_f16_ts")


# A correction window borrows its plan's packed filters and their factors; rows out of range are scaled as in the whole result
@pytest.mark.parametrize("n,c,h,w,f,k,win", [(1, 64, 20, 20, 64, 3, (3, 5, 0, 20)), (3, 32, 16, 24, 130, 3, (0, 2, 7, 9)), (2, 96, 11, 13, 48, 3, (4, 7, 2, 11)), (40, 64, 28, 28, 128, 3, (26, 2, 0, 28)),
                                             (1, 512, 14, 14, 64, 3, (1, 1, 1, 1)), (2, 3, 30, 150, 33, 5, (10, 9, 100, 50))])
def test_windows_with_factors_bit_identical(ctx, n, c, h, w, f, k, win):
    gen = torch.Generator().manual_seed(c + f)
    x, wt = _some_rows((n, c, h, w), 1, gen).cuda(), _weights((f, c, k, k), [1, f - 1], 0, 5)
    plan = ctx.conv2d_plan(x.shape, wt.shape, k // 2, k // 2)
    assert plan.kernel == "tc_3xtf32_f16_ts"
    ctx.conv2d_set_weights(plan, wt)
    whole, part = ctx.conv2d_run(plan, x), torch.full(plan.out_shape, 7.0, device="cuda")
    r0, rn, c0, cn = win
    ctx.conv2d_correct(plan, x, part, r0, rn, c0, cn)
    ctx.sync_check()
    inside = (slice(None), slice(None), slice(r0, r0 + rn), slice(c0, c0 + cn))
    assert torch.equal(part[inside], whole[inside])
    part[inside] = 7.0
    assert bool((part == 7.0).all())


# Neighbouring pixels of different magnitude in one row of operands would leave the bound above no meaning: here a whole image is of one
# magnitude.  One tile per CTA, several, K split.
@pytest.mark.parametrize("n,c,d,hw,f", [(3, 16, 4, 8, 33), (3, 64, 4, 14, 64), (6, 64, 8, 28, 64), (3, 256, 2, 4, 128)])
def test_conv3d_second_pass(ctx, n, c, d, hw, f):
    gen = torch.Generator().manual_seed(c + f)
    x, wt = torch.randn(n, c, d, hw, hw, generator=gen), _weights((f, c, 3, 3, 3), [2, f - 1], 0, 6)
    x *= torch.tensor([1.0, 1e-9, 1e7])[torch.arange(n) % 3].reshape(-1, 1, 1, 1, 1)
    plan = ctx.conv3d_plan(x.shape, wt.shape, (1, 1, 1))
    assert plan.kernel == "tc_3xtf32_f16_ts"
    got = ctx.conv3d(x.cuda(), wt, (1, 1, 1)).cpu()
    ctx.sync_check()
    pad = torch.nn.functional.pad(x, (1,) * 6)
    cols = pad.unfold(2, 3, 1).unfold(3, 3, 1).unfold(4, 3, 1).permute(0, 2, 3, 4, 1, 5, 6, 7).reshape(-1, c * 27)
    rows = torch.randperm(cols.shape[0], generator=gen)[:3000]
    assert _within_bound(got.permute(0, 2, 3, 4, 1).reshape(-1, f)[rows], cols[rows].double(), wt.cpu().reshape(f, -1).double().t())


# The phases of a transposed convolution are a chain of launches that fill every second row and column (channels last); with rows out of
# range each makes its second pass
@pytest.mark.parametrize("phases", ["1", "0"])
@pytest.mark.parametrize("n,hw,f,c,k,act", [(3, 8, 32, 24, 4, "none"), (3, 16, 128, 64, 4, "none"), (3, 9, 40, 33, 4, "relu"), (12, 32, 64, 66, 4, "none"), (3, 4, 512, 64, 4, "none")])
def test_convtrans_second_pass(ctx, monkeypatch, phases, n, hw, f, c, k, act):
    monkeypatch.setenv("PETB200_CONVTRANS_PHASES", phases)
    gen = torch.Generator().manual_seed(f + c)
    x, wt, bias = torch.randn(n, hw, hw, f, generator=gen), _weights((k, k, f, c), [0, c - 1], 3, 8), torch.randn(c, generator=gen)
    scale = torch.tensor([1.0, 1e-9, 1e7])[torch.arange(n) % 3].reshape(-1, 1, 1, 1)
    x *= scale
    plan = ctx.convtrans_plan(x.shape, wt.shape, 1, 1, 2, 2, bias=True, act=act)
    assert plan.kernel == "tc_3xtf32_f16_ts"
    got = ctx.convtrans_run(plan, x.cuda(), wt, bias.cuda()).cpu().double()
    ctx.sync_check()
    w4 = wt.cpu().permute(2, 3, 0, 1).double()  # [f, c, k, k]
    exact = lambda a, b: torch.nn.functional.conv_transpose2d(a.double().permute(0, 3, 1, 2), b, stride=2, padding=1).permute(0, 2, 3, 1)
    want = exact(x, w4) + bias.double()
    want = want.clamp_min(0) if act == "relu" else want
    bound = 2.0 ** -22 * (12 + f * k) * exact(x.abs(), w4.abs()) + 2.0 ** -22 * (want.abs() + bias.abs().double())
    bound += 2.0 ** -22 * x.abs().amax((1, 2, 3)).double().reshape(-1, 1, 1, 1) * w4.abs().sum((0, 2, 3))
    assert bool(((got - want).abs() <= bound).all())


# Operands that are strided views, heads of [sequence, heads, width]: the same bits as on dense copies
@pytest.mark.parametrize("seq,heads,d", [(128, 12, 64), (77, 3, 68), (384, 8, 128)])
def test_strided_operands_second_pass(ctx, seq, heads, d):
    gen = torch.Generator().manual_seed(seq)
    q, v = _some_rows((seq, heads, d), 2, gen).cuda(), _some_rows((seq, heads, d), 2, gen).cuda()
    plan = ctx.matmul_plan((heads, seq, d), (heads, seq, d), transB=True, strides=(d, heads * d, d, heads * d, seq * seq, seq))
    assert plan.kernel == "tc_3xtf32_f16_ts"
    out = torch.empty(heads, seq, seq, device="cuda")
    ctx.matmul_run(plan, q, v, out=out)
    qh, vh = q.permute(1, 0, 2).contiguous(), v.permute(1, 0, 2).contiguous()
    assert torch.equal(out, ctx.matmul(qh, vh, transB=True))
    ctx.sync_check()
    for i in range(heads):
        assert _within_bound(out[i].cpu(), qh[i].cpu().double(), vh[i].cpu().double().t())


# Factors are taken out before bias, residual and activation.  (The activations agree with torch's to a few units in the last place, on
# sums that are the same: 2^-20 of the value, or of 1 where the result is the small rest of larger terms.)
@pytest.mark.parametrize("act", ["none", "relu", "sigmoid", "tanh", "gelu"])
@pytest.mark.parametrize("n,c,hw,f", [(1, 64, 12, 40), (30, 64, 28, 72), (20, 128, 28, 128), (1, 512, 8, 64)])
def test_epilogue_after_factors(ctx, act, n, c, hw, f):
    gen = torch.Generator().manual_seed(c + f)
    x, wt = _some_rows((n, c, hw, hw), 1, gen).cuda() * 0.05, _weights((f, c, 3, 3), [0, f - 1], 0, 9)
    bias, res = torch.randn(f, generator=gen).cuda(), torch.randn(n, f, hw, hw, generator=gen).cuda()
    plain, plan = ctx.conv2d_plan(x.shape, wt.shape, 1, 1), ctx.conv2d_plan(x.shape, wt.shape, 1, 1, bias=True, act=act)
    assert plain.kernel == plan.kernel == "tc_3xtf32_f16_ts"
    for p in (plain, plan):
        ctx.conv2d_set_weights(p, wt)
    sums = ctx.conv2d_run(plain, x) + bias.reshape(1, -1, 1, 1) + res
    got = ctx.conv2d_run(plan, x, bias, residual=res)
    ctx.sync_check()
    want = {"none": lambda t: t, "relu": torch.relu, "sigmoid": torch.sigmoid, "tanh": torch.tanh, "gelu": torch.nn.functional.gelu}[act](sums)
    assert bool(((got - want).abs() <= 2.0 ** -20 * torch.maximum(want.abs(), torch.ones_like(want))).all())


# Packing B: columns in strips of 32 or of 8 (few columns), rows of B by one warp or several; more units of K than have room in shared memory
# or registers; one unit, remainders of a unit
@pytest.mark.parametrize("b,n,k", [(1, 40, 20000), (1, 1300, 5000), (3, 9, 200), (2, 33, 64), (5, 8, 1000), (1, 1, 4100), (2, 2000, 70), (1, 600, 12300)])
@pytest.mark.parametrize("trans_b", [False, True])
def test_packing_of_halves(ctx, b, n, k, trans_b):
    gen = torch.Generator().manual_seed(n + k)
    a, w = torch.randn(b, 24, k, generator=gen), torch.randn(b, n, k, generator=gen)
    w *= torch.tensor([1.0, 1.0, 1e-9, 1e9])[torch.randint(0, 4, (b, n, 1), generator=gen)]
    wd = (w if trans_b else w.transpose(1, 2).contiguous()).cuda()
    plan = ctx.matmul_plan(a.shape, wd.shape, False, trans_b)
    assert plan.kernel == "tc_3xtf32_f16_ts"
    got = ctx.matmul_run(plan, a.cuda(), wd).cpu()
    ctx.sync_check()
    for i in range(b):
        assert _within_bound(got[i], a[i].double(), w[i].double().t())


# Left to itself a plan takes halves only where their stages are well filled and there is work enough: chunks of 1, 4 and 8 channels (planes
# of odd width), K of 89; batched products of few stages, whose B is packed in every call
@pytest.mark.parametrize("x,w,takes", [((2, 119, 66, 66), (23, 119, 1, 1), False), ((9, 144, 75, 75), (33, 144, 3, 3), False), ((3, 480, 43, 43), (64, 480, 3, 3), False),
                                       ((1, 512, 64, 64), (512, 512, 3, 3), True), ((18, 120, 1088), (18, 1088, 232), False), ((1, 2000, 89), (1, 89, 2000), False),
                                        ((1, 384, 768), (1, 768, 3072), True), ((4, 1000, 1024), (4, 1024, 1000), True)])
def test_which_plans_take_halves(ctx, monkeypatch, x, w, takes):
    monkeypatch.delenv("PETB200_TC_MATH")
    plan = ctx.matmul_plan(x, w) if len(x) == 3 else ctx.conv2d_plan(x, w, w[2] // 2, w[2] // 2)
    assert plan.kernel == ("tc_3xtf32_f16_ts" if takes else "tc_3xtf32_ts")
