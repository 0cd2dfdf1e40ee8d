"""GPU: variants of kernels that a dispatch rule picks by size or alignment, at the sizes where each can go wrong (edges of
tiles, remainders, the smallest and largest of its range), against the CPU oracle."""
import numpy as np
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu
TOL = 1e-3


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


# n around a block of 128 (B as [k][n]) or 32 (B as [n][k]) columns; k below one warp pass, at a split over a whole cluster of eight
# and, with that split, at slices of one shared-memory tile of A (512 values for m > 4, else 1024) and of one value more; rows of B
# on and off the 16-byte grid
@pytest.mark.parametrize("n,k", [(1, 1), (31, 69), (128, 8), (129, 511), (260, 1025), (33, 2052), (100, 9001), (4100, 640),
                                 (100, 4096), (100, 4097), (100, 8192), (100, 8193)])
@pytest.mark.parametrize("m,trans_a,trans_b", [(1, False, False), (1, False, True), (2, True, False), (3, False, True), (8, True, True), (8, False, False)])
def test_matrix_vector_products_exact(ctx, m, trans_a, trans_b, n, k):
    rng = np.random.default_rng(n + k + m)
    b = 2
    a = rng.integers(-4, 5, (b, k, m) if trans_a else (b, m, k)).astype(np.float32)
    w = rng.integers(-4, 5, (b, n, k) if trans_b else (b, k, n)).astype(np.float32)
    bias, res = rng.integers(-4, 5, n).astype(np.float32), rng.integers(-4, 5, (b, m, n)).astype(np.float32)
    want = np.maximum((a.transpose(0, 2, 1) if trans_a else a) @ (w.transpose(0, 2, 1) if trans_b else w) + bias + res, 0)
    got = ctx.matmul(dev(a), dev(w), trans_a, trans_b, bias=dev(bias), act="relu", residual=dev(res))
    ctx.sync_check()
    assert np.array_equal(got.cpu().numpy(), want)


# Tensor-core matmul: k off the 16-byte grid (A re-pitched), n off it (rows stored one by one), one tile per CTA and several,
# narrow tiles and wide ones with an accumulator flush (k > 768), tiles that end inside the last rows and columns
@pytest.mark.parametrize("b,m,n,k", [(1, 33, 9, 31), (2, 129, 65, 70), (80, 130, 70, 33), (160, 128, 64, 34), (3, 1025, 129, 801), (4, 1921, 330, 773), (1, 257, 2047, 998)])
@pytest.mark.parametrize("trans_a,trans_b", [(False, False), (False, True), (True, False)])
def test_matmul_off_the_16_byte_grid(ctx, b, m, n, k, trans_a, trans_b):
    rng = np.random.default_rng(m + n + k)
    a = rng.integers(-2, 3, (b, k, m) if trans_a else (b, m, k)).astype(np.float32)
    w = rng.integers(-2, 3, (b, n, k) if trans_b else (b, k, n)).astype(np.float32)
    bias, res = rng.integers(-4, 5, n).astype(np.float32), rng.integers(-4, 5, (b, m, n)).astype(np.float32)
    lin = torch.matmul(dev(a).double().transpose(1, 2) if trans_a else dev(a).double(), dev(w).double().transpose(1, 2) if trans_b else dev(w).double()) + dev(bias).double()
    got = ctx.matmul(dev(a), dev(w), trans_a, trans_b, bias=dev(bias), act="relu", residual=dev(res))
    assert np.array_equal(got.cpu().numpy(), torch.relu(lin + dev(res)).float().cpu().numpy())
    got = ctx.matmul(dev(a), dev(w), trans_a, trans_b, bias=dev(bias), act="tanh")
    ctx.sync_check()
    assert rel_err(got.cpu().numpy(), torch.tanh(lin).cpu().numpy()) <= TOL


# Several tiles per CTA: 16-byte runs of pixels that end inside a warp's 32 (10 x 14, 10 x 10), pixels off the 16-byte grid, two images in a
# tile, filters that end inside a block; with and without a flush (c*9 > 768); each way of storing with and without a residual
@pytest.mark.parametrize("n,c,h,w,f,act", [(300, 8, 13, 13, 70, "relu"), (170, 8, 16, 16, 64, "none"), (310, 5, 10, 10, 33, "relu"), (160, 90, 10, 14, 72, "relu"),
                                           (320, 96, 7, 7, 130, "none"), (160, 6, 12, 18, 31, "sigmoid")])
def test_conv_persistent_tiles_stores(ctx, n, c, h, w, f, act):
    rng = np.random.default_rng(n + c)
    x, wt = dev(rng.integers(-2, 3, (n, c, h, w)).astype(np.float32)), dev(rng.integers(-2, 3, (f, c, 3, 3)).astype(np.float32))
    bias, res = dev(rng.integers(-4, 5, f).astype(np.float32)), dev(rng.integers(-4, 5, (n, f, h, w)).astype(np.float32))
    lin = torch.nn.functional.conv2d(x.double().cpu(), wt.double().cpu(), bias.double().cpu(), padding=1)
    fn = {"relu": torch.relu, "none": lambda v: v, "sigmoid": torch.sigmoid}[act]
    for r in (None, res):
        plan = ctx.conv2d_plan(x.shape, wt.shape, 1, 1, bias=True, act=act)
        ctx.conv2d_set_weights(plan, wt)
        got = ctx.conv2d_run(plan, x, bias, residual=r)
        ctx.sync_check()
        want = fn(lin if r is None else lin + r.double().cpu())
        assert torch.equal(got.cpu(), want.float()) if act != "sigmoid" else rel_err(got.cpu().numpy(), want.numpy()) <= TOL


# last register-resident rows of a warp (enough of them for a warp each: 1300), of a block, and the first row past them; fewer rows
# than a wave of blocks, and more than there are blocks (a block then takes several)
@pytest.mark.parametrize("rows,cols", [(r, c) for c in (255, 256, 1024, 1025, 1279, 2048, 2049, 4095, 4096, 4097) for r in (1, 3, 700, 1300)] +
                         [(9600, 1025), (9600, 4097)])
def test_softmax_rows_by_length(ctx, oracle, rows, cols):
    x = np.random.default_rng(cols).standard_normal((rows, cols)).astype(np.float32) * 4
    x[0, cols - 1] = 40.0
    got = ctx.softmax(dev(x))
    ctx.sync_check()
    assert rel_err(got.cpu().numpy(), oracle.softmax(x)) <= 1e-5


# 2w+1 around a 16-byte piece, a K stage and more than a tile of keys; rows that end inside a tile; the first and last rows'
# windows reach past the keys
@pytest.mark.parametrize("b,n,m,w", [(1, 130, 64, 1), (2, 257, 32, 3), (3, 300, 64, 16), (1, 1000, 96, 130), (5, 129, 16, 200), (2, 2051, 64, 67)])
def test_banded_products_by_width(ctx, oracle, b, n, m, w):
    rng = np.random.default_rng(n + w)
    q, k = (rng.integers(-2, 3, (b, n, m)).astype(np.float32) for _ in range(2))
    p = rng.integers(-2, 3, (b, n, 2 * w + 1)).astype(np.float32)
    scores, out = ctx.g2bmm(dev(q), dev(k), w), ctx.gbmml(dev(p), dev(k))
    ctx.sync_check()
    assert np.array_equal(scores.cpu().numpy(), oracle.g2bmm(q, k, w))
    assert np.array_equal(out.cpu().numpy(), oracle.gbmml(p, k))


# Phases side by side: with and without a K split, one launch per phase or persistent tiles (many images), calls back to back (the next
# call's layout pass must wait for every phase), phases of different size
@pytest.mark.parametrize("n,hw,f,c,k,s,pad", [(3, 9, 40, 33, 3, 2, 1), (16, 4, 512, 64, 4, 2, 1), (200, 16, 8, 64, 4, 2, 1), (2, 12, 96, 48, 5, 3, 1)])
def test_convtrans_phases_back_to_back(ctx, oracle, monkeypatch, n, hw, f, c, k, s, pad):
    monkeypatch.setenv("PETB200_CONVTRANS_PHASES", "1")
    rng = np.random.default_rng(n + hw)
    w = rng.integers(-2, 3, (k, k, f, c)).astype(np.float32)
    xs = [rng.integers(-2, 3, (n, hw, hw, f)).astype(np.float32) for _ in range(3)]
    plan = ctx.convtrans_plan((n, hw, hw, f), (k, k, f, c), pad, pad, s, s)
    got = [ctx.convtrans_run(plan, x, dev(w) if i == 0 else None) for i, x in enumerate([dev(x) for x in xs])]
    ctx.sync_check()
    for g, x in zip(got, xs):
        ref = torch.nn.functional.conv_transpose2d(dev(x).double().cpu().permute(0, 3, 1, 2), torch.from_numpy(w).double().permute(2, 3, 0, 1), stride=s, padding=pad)
        assert np.array_equal(g.cpu().numpy(), ref.permute(0, 2, 3, 1).float().numpy())


# Operands that are views: each is copied, and the copies have sizes that the allocator could give the same memory
def test_operands_that_are_views(ctx):
    rng = np.random.default_rng(3)
    ints = lambda *s: dev(rng.integers(-3, 4, s).astype(np.float32))
    a, b, bias, res = ints(2, 64, 96).transpose(1, 2), ints(2, 96, 64).transpose(1, 2), ints(192)[::2], ints(2, 96, 96).transpose(1, 2)
    assert torch.equal(ctx.matmul(a, b, bias=bias, residual=res).double(), a.double() @ b.double() + bias.double() + res.double())
    x, r, w = ints(1, 8, 8, 8, 16).transpose(3, 4), ints(1, 8, 8, 8, 16).transpose(3, 4), ints(8, 8, 1, 1, 1)
    want = torch.nn.functional.conv3d(x.double().cpu(), w.double().cpu(), bias[:8].double().cpu()) + r.double().cpu()
    assert torch.equal(ctx.conv3d(x, w, (0, 0, 0), bias=bias[:8], residual=r).double().cpu(), want)
    x, r, w = ints(1, 8, 8, 16).transpose(2, 3), ints(1, 8, 8, 16).transpose(2, 3), ints(8, 8, 1, 1)
    want = torch.nn.functional.conv2d(x.double().cpu(), w.double().cpu(), bias[:8].double().cpu()) + r.double().cpu()
    assert torch.equal(ctx.conv2d(x, w, 0, 0, bias=bias[:8], residual=r).double().cpu(), want)
    ctx.sync_check()


# A plan with a declared weight that is given another B in between: the weight's packed operand has been overwritten and is made again
@pytest.mark.parametrize("m,k", [(32, 64), (33, 70), (4, 64)])
def test_matmul_weight_after_another_operand(ctx, m, k):
    rng = np.random.default_rng(m + k)
    a, w, other = (dev(rng.integers(-3, 4, s).astype(np.float32)) for s in ((1, m, k), (1, k, 40), (1, k, 40)))
    plan = ctx.matmul_plan(a.shape, w.shape)
    ctx.matmul_set_weights(plan, w)
    for b in (None, other, None, w, other, w):
        assert torch.equal(ctx.matmul_run(plan, a, b).double(), a.double() @ (w if b is None else b).double())
    ctx.sync_check()


# Timing a plan or a graph leaves its weights as they are
@pytest.mark.parametrize("algo", ["auto", "simt_fp32"])
def test_timing_keeps_the_weights(ctx, algo, monkeypatch):
    from pet_b200 import configs
    from pet_b200.graph import Graph
    x, w = torch.randn(2, 16, 12, 12, device="cuda"), torch.randn(24, 16, 3, 3, device="cuda")
    plan = ctx.conv2d_plan(x.shape, w.shape, 1, 1, algo=algo)
    ctx.conv2d_set_weights(plan, w)
    before = ctx.conv2d_run(plan, x)
    plan.time(rounds=2, warmup=1)
    assert torch.equal(ctx.conv2d_run(plan, x), before)
    for phases in ("0", "1"):
        monkeypatch.setenv("PETB200_CONVTRANS_PHASES", phases)
        wt = torch.randn(4, 4, 16, 8, device="cuda")
        plan = ctx.convtrans_plan((2, 12, 12, 16), wt.shape, 1, 1, 2, 2, algo=algo)
        xt = torch.randn(2, 12, 12, 16, device="cuda")
        before = ctx.convtrans_run(plan, xt, wt)
        plan.time(rounds=2, warmup=1)
        assert torch.equal(ctx.convtrans_run(plan, xt), before)
    graph = Graph(ctx)
    b = configs.GraphBuilder(graph)
    out = b.matmul(b.reshape(b.conv(b.input(x.cpu().numpy()), b.const(w.cpu().numpy()), 1, 1), [1, 2 * 24, 144]), b.const(np.ones((1, 144, 16), np.float32)))
    graph.setOutputs([out])
    graph.compile()
    b.load()
    graph.run()
    before = graph.get_data(out).copy()
    graph.perf(rounds=2, warmup=1)
    graph.run()
    assert np.array_equal(graph.get_data(out), before)
    ctx.sync_check()


# fp16 halves: hi and lo carry 22 bits of each operand (what is dropped is below 3 * 2^-22 of a product, and below 2^-22 of the
# row's largest value for values that a half cannot hold as normal numbers); the tensor core truncates its sum after each of K / 16
# MMAs, twice 2^-23 of it at most.  So |error| <= 2^-22 * ((4 + K / 8) * sum |x||w| + max |x| * sum |w|), elementwise.
def _check_halves(got, x2, w2):
    """x2 [rows, K], w2 [K, cols], float64; rows and filters of any magnitude."""
    k = x2.shape[1]
    fin = torch.isfinite(x2).all(1)
    bound = 2.0 ** -22 * ((4 + k / 8) * (x2.abs() @ w2.abs()) + x2.abs().amax(1, keepdim=True) * w2.abs().sum(0, keepdim=True))
    err = (got.double() - x2 @ w2).abs()
    assert bool((err[fin] <= bound[fin] + 1e-37).all()), float((err[fin] / (bound[fin] + 1e-37)).max())
    assert not bool(torch.isfinite(got[~fin]).any())


def _outlandish(x2d, kind, gen):
    """Rows (or filters) of magnitudes that a half cannot hold, beside ordinary ones."""
    rows = x2d.shape[0]
    pick = torch.randperm(rows, generator=gen)[: max(1, rows // 3)]
    scale = {"ordinary": 1.0, "tiny": 1e-9, "huge": 1e7, "mixed": 10.0 ** torch.randint(-12, 13, (len(pick), 1), generator=gen).double()}[kind]
    x2d[pick] = (x2d[pick].double() * scale).float()
    if kind == "mixed":
        x2d[pick[0]] = 0
    return x2d


# one stage and several, K remainders around a stage of 64 and a flush (K > 768), rows around a tile, one tile per CTA, several, K splits
@pytest.mark.parametrize("b,m,n,k", [(1, 16, 32, 64), (1, 129, 65, 63), (2, 300, 130, 65), (1, 128, 96, 768), (1, 257, 129, 833), (3, 1000, 200, 260), (1, 64, 64, 4096),
                                     (1, 5000, 300, 900)])
@pytest.mark.parametrize("kind", ["ordinary", "tiny", "huge", "mixed"])
@pytest.mark.parametrize("trans_b", [False, True])
def test_matmul_of_halves_over_all_magnitudes(ctx, monkeypatch, b, m, n, k, kind, trans_b):
    monkeypatch.setenv("PETB200_TC_MATH", "f16x3")
    gen = torch.Generator().manual_seed(m + n + k)
    a = _outlandish(torch.randn(b * m, k, generator=gen), kind, gen).reshape(b, m, k)
    w = torch.stack([_outlandish(torch.randn(n, k, generator=gen), kind, gen) for _ in range(b)])
    if kind == "ordinary":
        a[0, m // 2, 0], a[0, 0, k - 1] = float("inf"), float("nan")
    wd = (w if trans_b else w.transpose(1, 2).contiguous()).cuda()
    plan = ctx.matmul_plan(tuple(a.shape), tuple(wd.shape), False, trans_b)
    assert plan.kernel == "tc_3xtf32_f16_ts"
    c = torch.empty(b, m, n, device="cuda")
    for weights in (True, False):
        if weights:
            ctx.matmul_set_weights(plan, wd)
        got = ctx.matmul_run(plan, a.cuda(), None if weights else wd.clone())
        ctx.sync_check()
        for i in range(b):
            _check_halves(got[i].cpu(), a[i].double(), w[i].double().t())


# the ways of gathering: chunks of 32 channels, of 8, the offset table, whole unpadded planes (odd widths); one tile per CTA, several (narrow
# and, with a flush, wide), K split; a residual that is also the result's buffer must be added once
@pytest.mark.parametrize("n,c,h,w,f,k,stride", [(1, 64, 20, 20, 64, 3, 1), (2, 24, 9, 12, 40, 3, 1), (3, 3, 20, 24, 33, 5, 2), (4, 10, 7, 7, 20, 3, 1), (1, 256, 14, 14, 64, 3, 1),
                                                (40, 32, 32, 32, 64, 3, 1), (40, 96, 24, 24, 128, 3, 1), (30, 64, 28, 28, 130, 1, 2), (1, 7, 30, 150, 16, 3, 1)])
@pytest.mark.parametrize("kind", ["ordinary", "tiny", "huge", "mixed"])
def test_conv_of_halves_over_all_magnitudes(ctx, monkeypatch, n, c, h, w, f, k, stride, kind):
    monkeypatch.setenv("PETB200_TC_MATH", "f16x3")
    gen = torch.Generator().manual_seed(n + c + f)
    x = _outlandish(torch.randn(n * h * w, c, generator=gen), kind, gen).reshape(n, h, w, c).permute(0, 3, 1, 2).contiguous()
    wt = _outlandish(torch.randn(f, c * k * k, generator=gen), kind, gen).reshape(f, c, k, k)
    if kind == "ordinary":
        x[0, 0, h // 2, w // 2], x[-1, c - 1, 0, 0] = float("nan"), float("inf")
    pad = k // 2
    plan = ctx.conv2d_plan(tuple(x.shape), tuple(wt.shape), pad, pad, stride, stride)
    assert plan.kernel == "tc_3xtf32_f16_ts"
    ctx.conv2d_set_weights(plan, wt.cuda())
    got = ctx.conv2d_run(plan, x.cuda())
    ctx.sync_check()
    oh, ow = plan.out_shape[2:]
    cols = torch.nn.functional.unfold(x.double(), k, padding=pad, stride=stride)  # [n, c*k*k, L]
    full = [(d + 2 * pad - k) // stride + 1 for d in (h, w)]
    cols = cols.reshape(n, c * k * k, *full)[:, :, :oh, :ow].permute(0, 2, 3, 1).reshape(n * oh * ow, -1)
    _check_halves(got.permute(0, 2, 3, 1).reshape(n * oh * ow, f).cpu(), cols, wt.reshape(f, -1).double().t())
    if kind != "ordinary":
        res = torch.ones_like(got)
        y = ctx.conv2d_run(plan, x.cuda(), out=res, residual=res)
        ctx.sync_check()
        scale = got.abs().amax()
        assert bool((y - (got + 1) <= 1e-6 * (scale + 1)).all()) and bool(((got + 1) - y <= 1e-6 * (scale + 1)).all())


# Tiled permutations whose input run is an innermost pair and a second digit (the interleave of the space-to-batch rewrites): runs of 4, of
# 6 and 10 (off the 16-byte grid), around a tile's 64 words and beyond, channels around a tile; inputs off the 16-byte grid
@pytest.mark.parametrize("shape", [(1, 3, 4, 4), (2, 5, 8, 8), (1, 33, 6, 10), (3, 7, 12, 64), (2, 40, 8, 68), (1, 64, 64, 132), (4, 512, 4, 16)])
@pytest.mark.parametrize("shift", [0, 1, 4])
def test_tiled_permutation_of_pairs(ctx, oracle, shape, shift):
    from pet_b200.configs import SPACE_TO_BATCH
    x = np.random.default_rng(shape[3]).standard_normal(shape).astype(np.float32)
    buf = torch.empty(x.size + shift, device="cuda")
    xd = buf[shift:].view(shape)
    xd.copy_(torch.from_numpy(x))
    want = x
    for op in SPACE_TO_BATCH:
        want = oracle.transpose(want, *op)
    got = ctx.transpose_chain(xd, SPACE_TO_BATCH)
    ctx.sync_check()
    assert np.array_equal(got.cpu().numpy(), want)
