"""Tensor-core products at the edges of their tiles and stages: one-sector
superblocks with 1 to 270 rows and columns (tiles of 128 rows and 64 or 128
columns, 64 columns per epilogue warp, stages cut to the largest piece), a
stage-1 product, both identity terms and repeated terms (accumulation groups
and single items with their own factors), against numpy.

Tolerances, of the 2-norm: 2e-5 for two 16-bit slices (the split products'
bound of the other tests), 1e-11 for the exact slices."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def superblock(ctx, rows, cols, rng, nterms, sa=1.0, sb_=1.0):
    keys = np.array([[0, -1, -1, 0], [2, 0, 0, 0]], np.int32)  # HAM, CD(0,0;0): both rank 0
    hl, n = ctx.block_define([0], "c1", [[1, 1, 0]], [rows], keys)
    hr, m = ctx.block_define([0], "c1", [[1, 1, 0]], [cols], keys)
    A, B = rng.standard_normal((2, rows, rows)), rng.standard_normal((2, cols, cols))
    A[1] *= sa
    B[1] *= sb_
    ctx.block_upload(hl, A.reshape(-1))
    ctx.block_upload(hr, B.reshape(-1))
    ops = [(0, 0, -1, 0), (-1, 0, 0, 1)] + [(1, t % 2, 1, t // 2 % 2) for t in range(nterms)]
    coef = np.concatenate([[1.0, -0.5], rng.uniform(0.5, 1.5, nterms)])
    sb, size = ctx.superblock_define(hl, hr, [2, 0, 0], coef, np.array(ops, np.int32), 0.25)
    assert size == rows * cols

    def sigma(psi):
        out = 0.25 * psi + coef[0] * A[0] @ psi + coef[1] * psi @ B[0]
        for c, (_, lt, _, rt) in zip(coef[2:], ops[2:]):
            out += c * (A[1].T if lt else A[1]) @ psi @ (B[1] if rt else B[1].T)
        return out

    return sb, sigma


@pytest.mark.parametrize("width", [64, 128])
@pytest.mark.parametrize("rows,cols", [(1, 1), (8, 9), (17, 63), (64, 65), (65, 120), (127, 128), (129, 136), (270, 200), (128, 270)])
def test_split_edges(gpu_ctx, rows, cols, width):
    rng = np.random.default_rng(1000 * rows + cols)
    try:
        gpu_ctx.set_tc_tile_width(width)
        for nterms in (0, 1, 5, 40):
            sb, sigma = superblock(gpu_ctx, rows, cols, rng, nterms)
            for prec in ("bf16x3tc", "fp16x2tc"):
                gpu_ctx.set_precision(prec)
                psi = rng.standard_normal((rows, cols))
                ref = sigma(psi)
                got = gpu_ctx.sigma(sb, psi.reshape(-1)).reshape(rows, cols)
                assert np.linalg.norm(got - ref) <= 2e-5 * np.linalg.norm(ref), (nterms, prec)
    finally:
        gpu_ctx.set_tc_tile_width(0)
        gpu_ctx.set_precision("fp64")


@pytest.mark.parametrize("rows,cols", [(1, 1), (8, 9), (17, 63), (65, 120), (129, 136), (270, 200)])
def test_exact_edges(gpu_ctx, rows, cols):
    rng = np.random.default_rng(1000 * rows + cols)
    try:
        gpu_ctx.set_precision("exacttc")
        for nterms in (0, 1, 5, 40):
            sb, sigma = superblock(gpu_ctx, rows, cols, rng, nterms)
            psi = rng.standard_normal((rows, cols))
            ref = sigma(psi)
            got = gpu_ctx.sigma(sb, psi.reshape(-1)).reshape(rows, cols)
            assert np.linalg.norm(got - ref) <= 1e-11 * np.linalg.norm(ref), nterms
    finally:
        gpu_ctx.set_precision("fp64")


# tiles of 1 to 4 lane quarters and 16 or 32 columns, K of 128 and 144 (two
# ways to read the accumulators), of 512, 528 and 1040 (read-outs of 512)
@pytest.mark.parametrize("rows,cols", [(32, 33), (33, 16), (96, 31), (97, 128), (129, 144), (40, 512), (520, 24), (1030, 530)])
def test_exact_tiles_and_blocks(gpu_ctx, rows, cols):
    rng = np.random.default_rng(1000 * rows + cols)
    try:
        gpu_ctx.set_precision("exacttc")
        for nterms in (1, 7):
            sb, sigma = superblock(gpu_ctx, rows, cols, rng, nterms)
            psi = rng.standard_normal((rows, cols))
            ref = sigma(psi)
            for _ in range(2):
                got = gpu_ctx.sigma(sb, psi.reshape(-1)).reshape(rows, cols)
                assert np.linalg.norm(got - ref) <= 1e-11 * np.linalg.norm(ref), nterms
    finally:
        gpu_ctx.set_precision("fp64")


# scales of the products out of the range of one power of two
@pytest.mark.parametrize("ea,eb,ep", [(500, -500, 0), (510, -500, 505), (-480, 490, -470), (300, 200, 460)])
def test_exact_far_scales(gpu_ctx, ea, eb, ep):
    rng = np.random.default_rng(7)
    try:
        gpu_ctx.set_precision("exacttc")
        sb, sigma = superblock(gpu_ctx, 21, 19, rng, 4, 2.0**ea, 2.0**eb)
        psi = 2.0**ep * rng.standard_normal((21, 19))
        ref = sigma(psi)
        got = gpu_ctx.sigma(sb, psi.reshape(-1)).reshape(21, 19)
        assert np.isfinite(ref).all()
        big = np.abs(ref).max()
        assert np.linalg.norm((got - ref) / big) <= 1e-11 * np.linalg.norm(ref / big)
    finally:
        gpu_ctx.set_precision("fp64")


def test_split_knob_sets_the_pieces(gpu_ctx, monkeypatch):
    """The split knob cuts the phase-2 tiles into more pieces, for the same
    product (a sector of 12 x 12 or more tiles, each above a piece's least)."""
    rng = np.random.default_rng(12)
    tasks = []
    try:
        gpu_ctx.set_precision("bf16x3tc")
        sb, sigma = superblock(gpu_ctx, 1500, 1500, rng, 40)
        psi = rng.standard_normal((1500, 1500))
        ref = sigma(psi)
        for split in ("1", "3", "6"):
            monkeypatch.setenv("BGPU_TC_SPLIT", split)
            gpu_ctx.set_tc_stacking(64 if split == "3" else 56)  # (another limit: the plan is made again)
            got = gpu_ctx.sigma(sb, psi.reshape(-1)).reshape(1500, 1500)
            assert np.linalg.norm(got - ref) <= 2e-5 * np.linalg.norm(ref)
            info = gpu_ctx.superblock_info(sb)
            assert info["tc_split"] == float(split)
            tasks.append(info["tc_phase2_tasks"])
    finally:
        gpu_ctx.set_tc_stacking(64)
        gpu_ctx.set_precision("fp64")
    assert tasks[0] < tasks[1] < tasks[2], tasks
