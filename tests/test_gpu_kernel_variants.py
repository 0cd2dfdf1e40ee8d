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


# n around a block of 128 (B as [k][n]) or 32 (B as [n][k]) columns; k below one warp pass, around a shared-memory tile of A
# (512 / 1024 values) and past a split over a whole cluster; rows of B on and off the 16-byte grid
@pytest.mark.parametrize("n,k", [(1, 1), (31, 69), (128, 8), (129, 511), (260, 1025), (33, 2052), (100, 9001), (4100, 640)])
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
