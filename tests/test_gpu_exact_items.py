"""Exact-slice products whose blocks mix items of K from 17 to 600 and tiles
of one to four lane quarters: several sectors with scalar operators, against
numpy (1e-11 of the 2-norm, the exact slices' bound of the other tests), and
the same bits from every repetition."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# rows and columns of the sectors: K on both sides of 512 in every phase
SHAPES = [
    [(20, 600), (600, 24), (40, 530), (64, 17)],
    [(33, 513), (530, 20), (100, 100), (17, 600), (600, 33), (5, 512)],
]


@pytest.mark.parametrize("shapes", SHAPES)
@pytest.mark.parametrize("nterms", [3, 24])
def test_mixed_items(gpu_ctx, shapes, nterms):
    rng = np.random.default_rng(100 * len(shapes) + nterms)
    ns = len(shapes)
    keys = np.array([[0, -1, -1, 0], [2, 0, 0, 0]], np.int32)  # HAM, CD(0,0;0): both rank 0
    # one sector for each left quantum: 2 q + 1 electrons, spin 1/2
    ql = [[2 * q + 1, 1, 0] for q in range(ns)]
    rows, cols = [s[0] for s in shapes], [s[1] for s in shapes]
    hl, _ = gpu_ctx.block_define([0], "c1", ql, rows, keys)
    hr, _ = gpu_ctx.block_define([0], "c1", ql, cols[::-1], keys)
    A = [[rng.standard_normal((r, r)) for r in rows] for _ in keys]
    B = [[rng.standard_normal((c, c)) for c in cols[::-1]] for _ in keys]
    gpu_ctx.block_upload(hl, np.concatenate([m.reshape(-1) for op in A for m in op]))
    gpu_ctx.block_upload(hr, np.concatenate([m.reshape(-1) for op in B for m in op]))
    ops = [(0, 0, -1, 0), (-1, 0, 0, 1)] + [(1, t % 2, 1, t // 2 % 2) for t in range(nterms)]
    coef = np.concatenate([[1.0, -0.5], rng.uniform(0.5, 1.5, nterms)])
    sb, size = gpu_ctx.superblock_define(hl, hr, [2 * ns, 0, 0], coef, np.array(ops, np.int32), 0.25)
    assert size == sum(r * c for r, c in shapes)
    psi = [rng.standard_normal(s) for s in shapes]
    ref = []
    for q, p in enumerate(psi):
        a, b = [op[q] for op in A], [op[ns - 1 - q] for op in B]
        out = 0.25 * p + coef[0] * a[0] @ p + coef[1] * p @ b[0]
        for c, (_, lt, _, rt) in zip(coef[2:], ops[2:]):
            out += c * (a[1].T if lt else a[1]) @ p @ (b[1] if rt else b[1].T)
        ref.append(out.reshape(-1))
    ref, psi = np.concatenate(ref), np.concatenate([p.reshape(-1) for p in psi])
    try:
        gpu_ctx.set_precision("exacttc")
        first = gpu_ctx.sigma(sb, psi).copy()
        assert np.linalg.norm(first - ref) <= 1e-11 * np.linalg.norm(ref)
        for _ in range(20):
            assert np.array_equal(gpu_ctx.sigma(sb, psi), first)
    finally:
        gpu_ctx.set_precision("fp64")
