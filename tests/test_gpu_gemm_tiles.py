"""Grouped FP64 GEMM at its tile edges: units are cut into equal tiles of at
most 32 x 32, whose outputs are dealt to 128 threads, and K slabs of 32 rows
are filled from consecutive items.  Renormalisations (one item per unit,
transposed A) and density matrices (one item per root and sector, transposed
B or A) of one-sector blocks at sizes around 32, 64 and 128, against numpy.

Every output is a sum of k products rounded at most k + 1 times, so the error
of an element is at most (k + 2) eps times the product of the absolute
matrices; the tolerance is twice that (numpy's own sum included)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def one_sector(ctx, n, keys):
    h, size = ctx.block_define([0], "c1", np.array([[1, 1, 0]]), np.array([n]), np.array(keys, np.int32).reshape(-1, 4))
    return h, size


@pytest.mark.parametrize("n,m", [(1, 1), (2, 1), (31, 5), (32, 32), (33, 31), (64, 33), (65, 64), (101, 97), (130, 129)])
def test_renormalise_tiles(gpu_ctx, n, m):
    rng = np.random.default_rng(n * 1000 + m)
    gpu_ctx.set_precision("fp64")
    h, size = one_sector(gpu_ctx, n, [(0, -1, -1, 0)])
    assert size == n * n
    o, u = rng.standard_normal((n, n)), rng.standard_normal((n, m))
    gpu_ctx.block_upload(h, o)
    small, out, _ = gpu_ctx.renormalise(h, [m], [(0, -1, -1, 0)], rotations=u)
    got = gpu_ctx.block_download(small, out).reshape(m, m)
    bound = 2 * (2 * n + 4) * EPS * (np.abs(u).T @ np.abs(o) @ np.abs(u))
    assert np.all(np.abs(got - u.T @ o @ u) <= bound)


@pytest.mark.parametrize("roots", [1, 3, 20])
@pytest.mark.parametrize("rows,cols", [(1, 1), (7, 40), (33, 3), (65, 31), (101, 1), (130, 65)])
def test_density_tiles(gpu_ctx, rows, cols, roots):
    rng = np.random.default_rng(rows * 1000 + cols)
    none = np.zeros((0, 4), np.int32)
    hl, _ = one_sector(gpu_ctx, rows, none)
    hr, _ = one_sector(gpu_ctx, cols, none)
    sb, n = gpu_ctx.superblock_define(hl, hr, [2, 0, 0], np.zeros(0), none)
    assert n == rows * cols
    psi = rng.standard_normal((roots, n))
    w = rng.random(roots)
    gpu_ctx.set_wavefunctions(sb, psi)
    for left, size in ((True, rows), (False, cols)):
        gpu_ctx.density_eig(sb, left, size, w)
        rho, _ = gpu_ctx.density_download(size * size)
        p = psi.reshape(roots, rows, cols) if left else psi.reshape(roots, rows, cols).transpose(0, 2, 1)
        ref = np.einsum("r,rik,rjk->ij", w, p, p)
        k = roots * p.shape[2]
        bound = 2 * (k + 4) * EPS * np.einsum("r,rik,rjk->ij", w, np.abs(p), np.abs(p))
        assert np.all(np.abs(rho.reshape(size, size) - ref) <= bound)
