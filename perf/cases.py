"""Performance cases of the sweep hot path: what a DMRG program has this library do.

A case is a dict of plain values with a "kind":

  sigma    H psi on a superblock, device vectors (the Davidson functor) or host
           vectors (a caller that keeps its own vectors), in every precision
  renorm   U^T O U of a block's whole catalogue, the new block copied to the
           host (a program that stores its blocks)
  step     enlarged block built from a system block and a site, renormalised
           with given rotations and copied to the host
  density  density matrix of a wavefunction and its eigenvalues per sector
  eig      eigenpairs of a batch of dense symmetric matrices
  dmrg     whole sweeps from a dmrg.conf

The superblocks have the sector structure of a two-site step in the middle of
the chain: each side is a block of M kept states (multiplets spread over
particle number, spin and irrep around half filling) enlarged by one site, with
the operator catalogue and pair list of the Hamiltonian in normal and
complementary operators.  Operator values are random with the scale of
normalised operators: the cost of a product depends on the sectors alone.
"""
import math
import os
import tempfile

import numpy as np
import torch

import block_gb300

HAM, CRE, CD, CC, CDCOMP, DDCOMP, CCD, OVERLAP = 0, 1, 2, 3, 4, 5, 6, 7


def listed():
    def sigma(name, norb, m, prec, s2=0, group="c1", host=False):
        return {"name": name, "kind": "sigma", "norb": norb, "m": m, "prec": prec, "s2": s2, "group": group, "host": host}

    return [
        # the first sweeps of a small active space, vectors held by the caller: latency
        sigma("sigma_fp64_m50_host", 12, 50, "fp64", host=True),
        # the plain FP64 path at an ordinary size
        sigma("sigma_fp64_m150", 16, 150, "fp64"),
        # split precision, small and odd: a triplet state in 13 orbitals
        sigma("sigma_split_m101_triplet", 13, 101, "bf16x3tc", s2=2),
        # split precision at the 24-orbital size of the benchmark's second configuration
        sigma("sigma_split_m500", 24, 500, "bf16x3tc"),
        # the largest: sectors of several hundred states
        sigma("sigma_split_m1000", 18, 1000, "bf16x3tc"),
        # many uneven sectors: D2h irreps round-robin over the orbitals
        sigma("sigma_split_d2h_m500", 20, 500, "bf16x3tc", group="d2h"),
        # the FP64-level products that verify a split-precision solve
        sigma("sigma_exact_m300", 20, 300, "exacttc"),
        # a block step of a program that keeps its own sweep: build, renormalise, store
        {"name": "step_m60", "kind": "step", "norb": 14, "m": 60, "prec": "fp64"},
        # renormalisation of a split-precision run
        {"name": "renorm_m250", "kind": "renorm", "norb": 16, "m": 250, "prec": "bf16x3tc"},
        # truncation of a step: density matrix and its spectrum
        {"name": "density_m500", "kind": "density", "norb": 24, "m": 500, "nroots": 2},
        # the eigensolver on a batch of uneven sectors
        {"name": "eig_to_400", "kind": "eig", "largest": 400, "count": 12},
        # whole sweeps of a small system, Hamiltonian generated from a seed
        {"name": "dmrg_10_m40", "kind": "dmrg", "norb": 10, "m": 40, "prec": "fp64"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sigma"] * 7 + ["step", "renorm", "density", "eig", "dmrg"])
    if kind == "sigma":
        prec = rng.choice(["bf16x3tc"] * 4 + ["fp16x2tc", "fp64", "exacttc"])
        group = rng.choice(["c1", "c1", "c2v", "d2h"])
        norb = rng.randint(8, 20)
        most = {"fp64": 160, "exacttc": 300}.get(prec, 700)
        m = _log(rng, 30, most)
        s2 = rng.choice([0, 0, 0, 2, 4])
        return {"kind": kind, "norb": norb, "m": m, "prec": prec, "s2": s2, "group": group, "host": rng.random() < 0.2}
    if kind == "step":
        return {"kind": kind, "norb": rng.randint(10, 16), "m": _log(rng, 20, 70), "prec": rng.choice(["fp64", "bf16x3tc"])}
    if kind == "renorm":
        return {"kind": kind, "norb": rng.randint(10, 16), "m": _log(rng, 40, 250), "prec": rng.choice(["fp64", "bf16x3tc"])}
    if kind == "density":
        return {"kind": kind, "norb": rng.randint(12, 30), "m": _log(rng, 40, 700), "nroots": rng.randint(1, 3)}
    if kind == "eig":
        return {"kind": kind, "largest": _log(rng, 20, 450), "count": rng.randint(1, 12)}
    return {"kind": kind, "norb": rng.randint(8, 10), "m": _log(rng, 20, 50), "prec": rng.choice(["fp64", "bf16x3tc"])}


# ---- state spaces and catalogues


def _nirrep(group):
    return {"c1": 1, "c2v": 4, "d2h": 8}[group]


def _orbsym(norb, group):
    return [i % _nirrep(group) for i in range(norb)]


def _multiplets(nsites, n, s2):
    """Multiplets of n electrons with spin s2 / 2 in nsites orbitals (Weyl)."""
    a, b = (n - s2) // 2, (n + s2) // 2 + 1
    if (n + s2) % 2 or n < s2 or b > nsites + 1:
        return 0
    return (s2 + 1) * math.comb(nsites + 1, a) * math.comb(nsites + 1, b) // (nsites + 1)


def _kept(nsites, m, group, share):
    """{(n, 2S, irrep): kept states}: m states around half filling, low spins favoured."""
    ni = _nirrep(group)
    w = {}
    for n in range(2 * nsites + 1):
        for s2 in range(n % 2, min(n, 2 * nsites - n) + 1, 2):
            for g in range(ni):
                full = _multiplets(nsites, n, s2) / ni
                if full < 0.5:
                    continue
                uneven = 1.0 + 0.6 * math.cos(1.7 * g + 0.9 * n + 0.5 * s2)  # sectors of one n differ in size
                w[(n, s2, g)] = (math.exp(-((n - nsites) ** 2) / (2 * 1.3**2)) * math.exp(-0.6 * abs(s2 - share)) * uneven, full)
    lo, hi = 0.0, 1e9
    for _ in range(80):  # the scale at which m states are kept, no sector holding more than it has
        scale = (lo + hi) / 2
        total = {q: min(int(round(scale * x)), int(full)) for q, (x, full) in w.items()}
        lo, hi = (lo, scale) if sum(total.values()) > m else (scale, hi)
    total = {q: min(int(round(lo * x)), int(full)) for q, (x, full) in w.items()}
    return {q: k for q, k in total.items() if k > 0}


def _enlarge(kept, sym):
    out = {}
    for (n, s2, g), k in kept.items():
        for dn, ds, dg in ((0, 0, 0), (1, 1, sym), (2, 0, 0)):
            for t in range(abs(s2 - ds), s2 + ds + 1, 2):
                q = (n + dn, t, g ^ dg)
                out[q] = out.get(q, 0) + k
    return out


def _sides(norb, m, group, s2):
    """Sorted (quanta, states) of the two enlarged blocks, quanta that meet no partner dropped."""
    nl = norb // 2
    sym = _orbsym(norb, group)
    share = s2 / 2.0
    left = _enlarge(_kept(nl - 1, m, group, share), sym[nl - 1])
    right = _enlarge(_kept(norb - nl - 1, m, group, share), sym[nl])
    nelec = norb - norb % 2

    def meets(a, b):
        return a[0] + b[0] == nelec and a[2] == b[2] and abs(a[1] - b[1]) <= s2 <= a[1] + b[1] and (a[1] + b[1] + s2) % 2 == 0

    left2 = {q: k for q, k in left.items() if any(meets(q, r) for r in right)}
    right2 = {q: k for q, k in right.items() if any(meets(q, r) for r in left2)}
    return sorted(left2.items()), sorted(right2.items()), (nelec, s2, 0)


def _pairs(sites):
    return [(a, b) for a in sites for b in sites if a >= b]


def _normal(sites):
    k = []
    for a, b in _pairs(sites):
        k += [(CD, a, b, 0), (CD, a, b, 2), (CC, a, b, 0)] + ([(CC, a, b, 2)] if a != b else [])
    return k


def _complementary(sites):
    k = []
    for a, b in _pairs(sites):
        k += [(CDCOMP, a, b, 0), (CDCOMP, a, b, 2), (DDCOMP, a, b, 0)] + ([(DDCOMP, a, b, 2)] if a != b else [])
    return k


def _catalogue(own, other, extra):
    return [(HAM, -1, -1, 0)] + [(CRE, i, -1, 1) for i in own] + extra + [(CCD, i, -1, 1) for i in other]


def _terms(lk, rk, left, right, loop_left):
    """(coef, left op, transposed, right op, transposed) of H = sum of operator pairs."""
    li, ri = {k: i for i, k in enumerate(lk)}, {k: i for i, k in enumerate(rk)}
    out = [(1.0, li[lk[0]], 0, -1, 0), (1.0, -1, 0, ri[rk[0]], 0)]
    for i in right:
        out += [(1.0, li[(CCD, i, -1, 1)], t, ri[(CRE, i, -1, 1)], 1 - t) for t in (0, 1)]
    for i in left:
        out += [(1.0, li[(CRE, i, -1, 1)], t, ri[(CCD, i, -1, 1)], 1 - t) for t in (1, 0)]
    for a, b in _pairs(left if loop_left else right):
        for k2 in (0, 2):
            x, y = (CD, a, b, k2), (CDCOMP, a, b, k2)
            x, y = (x, y) if loop_left else (y, x)
            out += [(1.0, li[x], t, ri[y], t) for t in ((0, 1) if a != b else (0,))]
        for k2 in (0, 2) if a != b else (0,):
            x, y = (CC, a, b, k2), (DDCOMP, a, b, k2)
            x, y = (x, y) if loop_left else (y, x)
            out += [(2.0 if a != b else 1.0, li[x], t, ri[y], t) for t in (0, 1)]
    return out


def _dq(key, sym):
    t, i, j, k2 = key
    n = {HAM: 0, OVERLAP: 0, CRE: 1, CCD: 1, CD: 0, CDCOMP: 0, CC: 2, DDCOMP: -2}[t]
    return n, k2, (sym[i] if i >= 0 else 0) ^ (sym[j] if j >= 0 else 0)


def _op_blocks(space, dq):
    """(bra, ket, offset) of an operator's reduced blocks and its size."""
    out, off = [], 0
    for b, (qb, nb) in enumerate(space):
        for k, (qk, nk) in enumerate(space):
            if qb[0] == qk[0] + dq[0] and qb[2] == qk[2] ^ dq[2] and abs(qk[1] - dq[1]) <= qb[1] <= qk[1] + dq[1] and (qb[1] + qk[1] + dq[1]) % 2 == 0:
                out.append((b, k, off))
                off += nb * nk
    return out, off


class _Block:
    """Layout of a block's arena: operators back to back in the order of their sorted keys."""

    def __init__(self, space, keys, sym):
        self.space, self.keys, layouts = space, keys, {}
        self.ops, self.size = {}, 0
        for k in sorted(keys):
            dq = _dq(k, sym)
            if dq not in layouts:
                layouts[dq] = _op_blocks(space, dq)
            blocks, n = layouts[dq]
            self.ops[k] = (self.size, blocks)
            self.size += n

    def quanta(self):
        return np.array([q for q, _ in self.space], np.int32)

    def states(self):
        return np.array([k for _, k in self.space], np.int32)

    def values(self, seed):
        """Random operators whose norm is about one."""
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        x = torch.randn(self.size, dtype=torch.float64, device="cuda", generator=g)
        x *= 1.0 / math.sqrt(max(1.0, sum(k * k for _, k in self.space) / sum(k for _, k in self.space)))
        return x.cpu().numpy()


_shapes = {}


def _superblock(case):
    """Blocks, pair list and sectors of a case (host bookkeeping, no values)."""
    key = (case["norb"], case["m"], case.get("group", "c1"), case.get("s2", 0))
    if key not in _shapes:
        norb, m, group, s2 = key
        sym = _orbsym(norb, group)
        ls, rs, target = _sides(norb, m, group, s2)
        left, right = list(range(norb // 2)), list(range(norb // 2, norb))
        loop_left = len(left) <= len(right)
        loop = left if loop_left else right
        lk = _catalogue(left, right, _normal(loop) if loop_left else _complementary(loop))
        rk = _catalogue(right, left, _complementary(loop) if loop_left else _normal(loop))
        L, R = _Block(ls, lk, sym), _Block(rs, rk, sym)
        sectors, n = [], 0
        for a, (qa, na) in enumerate(ls):
            for b, (qb, nb) in enumerate(rs):
                if qa[0] + qb[0] == target[0] and qa[2] ^ qb[2] == target[2] and abs(qa[1] - qb[1]) <= s2 <= qa[1] + qb[1] and (qa[1] + qb[1] + s2) % 2 == 0:
                    sectors.append((a, b, n))
                    n += na * nb
        while len(_shapes) > 40:
            _shapes.pop(next(iter(_shapes)))
        _shapes[key] = (sym, group, L, R, _terms(lk, rk, left, right, loop_left), target, sectors, n)
    return _shapes[key]


def _define(ctx, block, sym, group, values=None, sites=None, is_dot=False):
    h, n = ctx.block_define(sym, group, block.quanta(), block.states(), np.array(block.keys, np.int32).reshape(-1, 4), is_dot)
    assert n == block.size
    if values is not None:
        ctx.block_upload(h, values)
    if sites is not None:
        ctx.block_set_sites(h, sites)
    return h


def _psi(n, seed, count=1):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = torch.randn(count, n, dtype=torch.float64, device="cuda", generator=g)
    return x / x.norm(dim=1, keepdim=True)


# ---- what a program has in hand before the call


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return globals()["_run_" + state["kind"]](state)


def _prepare_sigma(case, seed):
    sym, group, L, R, terms, target, _, n = _superblock(case)
    ctx = block_gb300.Context(0)
    ctx.set_precision(case["prec"])
    hl = _define(ctx, L, sym, group, L.values(3 * seed + 1))
    hr = _define(ctx, R, sym, group, R.values(3 * seed + 2))
    coef = np.array([t[0] for t in terms])
    ops = np.array([t[1:] for t in terms], np.int32)
    sb, size = ctx.superblock_define(hl, hr, target, coef, ops, -1.25)
    assert size == n
    psi = _psi(n, 3 * seed)[0]
    s = {"kind": "sigma", "host": case["host"], "ctx": ctx, "sb": sb}
    if case["host"]:
        s["psi"] = psi.cpu().numpy()
    else:
        s["psi"], s["out"] = psi, torch.zeros_like(psi)
    torch.cuda.synchronize()
    return s


def _run_sigma(s):
    if s["host"]:
        return s["ctx"].sigma(s["sb"], s["psi"])
    s["ctx"].sigma_device(s["sb"], s["psi"].data_ptr(), s["out"].data_ptr())
    return s["out"]


def _renorm_shape(norb, m):
    """An enlarged block in the middle of the chain and the m states kept of it."""
    sym, nl = _orbsym(norb, "c1"), norb // 2
    own, other = list(range(nl)), list(range(nl, norb))
    space = sorted(_enlarge(_kept(nl - 1, m, "c1", 0.0), 0).items())
    keys = [(OVERLAP, -1, -1, 0)] + _catalogue(own, other, _normal(own) + _complementary(other))
    full = sum(k for _, k in space)
    kept = np.array([min(k, max(1, k * m // full)) if k * m >= full // 2 else 0 for _, k in space], np.int32)
    return sym, own, other, _Block(space, keys, sym), kept


def _rotations(space, kept, seed):
    """Orthonormal columns, states x kept per quantum."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    u = [torch.linalg.qr(torch.randn(k, int(m), dtype=torch.float64, device="cuda", generator=g))[0] for (_, k), m in zip(space, kept) if m]
    return torch.cat([x.reshape(-1) for x in u]).cpu().numpy()


def _prepare_renorm(case, seed):
    sym, own, other, big, kept = _renorm_shape(case["norb"], case["m"])
    ctx = block_gb300.Context(0)
    ctx.set_precision(case["prec"])
    h = _define(ctx, big, sym, "c1", big.values(2 * seed), sites=own)
    return {"kind": "renorm", "ctx": ctx, "big": h, "kept": kept, "keys": np.array(big.keys, np.int32), "rot": _rotations(big.space, kept, 2 * seed + 1)}


def _stored(ctx, h, n):
    """The block on the host; its device storage is released."""
    out = ctx.block_download(h, n)
    _free(ctx, h)
    return out


def _free(ctx, h):
    if ctx.lib.bgpu_block_free(ctx.h, h) != 0:
        raise block_gb300.BgpuError("bgpu_block_free")


def _run_renorm(s):
    h, n, _ = s["ctx"].renormalise(s["big"], s["kept"], s["keys"], rotations=s["rot"])
    return _stored(s["ctx"], h, n)


def _prepare_step(case, seed):
    norb, nl = case["norb"], case["norb"] // 2
    sym, own, other, big, kept = _renorm_shape(norb, case["m"])
    sys_sites, dot = own[:-1], own[-1]
    system = _Block(sorted(_kept(nl - 1, case["m"], "c1", 0.0).items()), [(OVERLAP, -1, -1, 0)] + _catalogue(sys_sites, [dot] + other, _normal(sys_sites) + _complementary([dot] + other)), sym)
    rest = [i for i in range(norb) if i != dot]
    site = _Block([((0, 0, 0), 1), ((1, 1, 0), 1), ((2, 0, 0), 1)], [(OVERLAP, -1, -1, 0)] + _catalogue([dot], rest, _normal([dot]) + _complementary(rest)), sym)
    rng = np.random.default_rng(seed)
    h1 = rng.standard_normal((norb, norb)) * 0.05
    chol = rng.standard_normal((2 * norb, norb, norb)) * 0.1
    chol = chol + chol.transpose(0, 2, 1)
    ctx = block_gb300.Context(0)
    ctx.set_precision(case["prec"])
    ints = ctx.integrals_define(sym, h1 + h1.T + np.diag(np.linspace(-3, 1, norb)), np.einsum("kpq,krs->pqrs", chol, chol))
    hs = _define(ctx, system, sym, "c1", system.values(2 * seed), sites=sys_sites)
    hd = _define(ctx, site, sym, "c1", rng.standard_normal(site.size), sites=[dot], is_dot=True)
    return {"kind": "step", "ctx": ctx, "ints": ints, "sys": hs, "dot": hd, "keys": np.array(big.keys, np.int32), "kept": kept, "rot": _rotations(big.space, kept, 2 * seed + 1)}


def _run_step(s):
    ctx = s["ctx"]
    big, _, _ = ctx.build_enlarged_ops(s["ints"], s["sys"], s["dot"], s["keys"])
    small, n, _ = ctx.renormalise(big, s["kept"], s["keys"], rotations=s["rot"])
    _free(ctx, big)
    return _stored(ctx, small, n)


def _prepare_density(case, seed):
    sym, group, L, R, _, target, _, n = _superblock(case)
    ctx = block_gb300.Context(0)
    none = np.zeros((0, 4), np.int32)
    hl, _ = ctx.block_define(sym, group, L.quanta(), L.states(), none)
    hr, _ = ctx.block_define(sym, group, R.quanta(), R.states(), none)
    sb, _ = ctx.superblock_define(hl, hr, target, np.zeros(0), none, 0.0)
    psi = _density_psi(case, seed)
    states = L.states()
    return {"kind": "density", "ctx": ctx, "sb": sb, "psi": psi.cpu().numpy(), "states": int(states.sum()), "elems": int((states.astype(np.int64) ** 2).sum()),
            "weights": np.full(case["nroots"], 1.0 / case["nroots"])}


def _density_psi(case, seed):
    """Wavefunctions whose singular values fall over some decades in every sector, as a truncated state's do."""
    _, _, L, R, _, _, sectors, n = _superblock(case)
    x = _psi(n, seed, case["nroots"])
    for a, b, off in sectors:
        na, nb = L.space[a][1], R.space[b][1]
        x[:, off:off + na * nb] *= torch.exp(-6.0 * torch.arange(nb, device="cuda", dtype=torch.float64) / nb).repeat(na)
    return x / x.norm(dim=1, keepdim=True)


def _run_density(s):
    # the eigenvectors stay on the device for the renormalisation (those of equal eigenvalues are a choice)
    s["ctx"].set_wavefunctions(s["sb"], s["psi"])
    eig = s["ctx"].density_eig(s["sb"], True, s["states"], s["weights"])
    rho, _ = s["ctx"].density_download(s["elems"])
    return {"eig": eig, "rho": rho}


def _eig_dims(case):
    top, count = case["largest"], case["count"]
    return [max(1, round(top * (j + 1) ** 1.4 / count**1.4)) for j in range(count)]


def _eig_matrices(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    out = []
    for n in _eig_dims(case):
        x = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g)
        out.append((x + x.T) / math.sqrt(2 * n))
    return out


def _prepare_eig(case, seed):
    return {"kind": "eig", "ctx": block_gb300.Context(0), "a": [x.cpu().numpy() for x in _eig_matrices(case, seed)]}


def _run_eig(s):
    got = s["ctx"].diagonalise(s["a"])
    return {"w": np.concatenate([w for w, _ in got]), "v": np.concatenate([v.reshape(-1) for _, v in got])}


def _prepare_dmrg(case, seed):
    where = tempfile.TemporaryDirectory()
    conf = os.path.join(where.name, "dmrg.conf")
    n = case["norb"]
    with open(conf, "w") as f:
        f.write("nelec %d\nspin 0\nschedule\n0 %d 1e-12 0\nend\nmaxiter 2\nsweep_tol 1e-12\nnoreorder\norbitals synthetic:%d:%d:%d:%d:0\n" % (n - n % 2, case["m"], n, n - n % 2, 2 * n, 1000 + seed % 100000))
    ctx = block_gb300.Context(0)
    ctx.set_precision(case["prec"])
    return {"kind": "dmrg", "ctx": ctx, "where": where, "conf": conf}


def _run_dmrg(s):
    e, stats = s["ctx"].run_dmrg(s["conf"])
    return {"energies": e, "sweeps": stats["sweep_energies"]}


# ---- 64-bit values in plain torch and numpy


def _fact(n):
    return math.factorial(n)


def _sixj(a, b, c, d, e, f):
    """Wigner 6j of doubled spins (Racah)."""
    def tri(x, y, z):
        if (x + y + z) % 2 or z < abs(x - y) or z > x + y:
            return None
        return _fact((x + y - z) // 2) * _fact((x - y + z) // 2) * _fact((y + z - x) // 2) / _fact((x + y + z) // 2 + 1)

    t = [tri(a, b, c), tri(a, e, f), tri(d, b, f), tri(d, e, c)]
    if any(x is None for x in t):
        return 0.0
    lo = max(a + b + c, a + e + f, d + b + f, d + e + c) // 2
    hi = min(a + b + d + e, b + c + e + f, a + c + d + f) // 2
    s = 0.0
    for k in range(lo, hi + 1):
        den = _fact(k - (a + b + c) // 2) * _fact(k - (a + e + f) // 2) * _fact(k - (d + b + f) // 2) * _fact(k - (d + e + c) // 2)
        den *= _fact((a + b + d + e) // 2 - k) * _fact((b + c + e + f) // 2 - k) * _fact((a + c + d + f) // 2 - k)
        s += (-1) ** k * _fact(k + 1) / den
    return math.sqrt(t[0] * t[1] * t[2] * t[3]) * s


def _coupling(lp, rp, j, k, l, r):
    """Normalised 9j {lp rp j; k k 0; l r j}."""
    sign = (rp + j + k + l) // 2 + (lp + rp + l + r) // 2 + j + k
    x = _sixj(lp, rp, j, r, l, k) * (-1) ** sign / math.sqrt((j + 1) * (k + 1))
    return math.sqrt((l + 1) * (r + 1) * (j + 1)) * x


def _adjoint(bra, ket, k):
    """Scale of the adjoint tensor's block (bra, ket) against the operator's (ket, bra)."""
    return (-1) ** ((bra + k - ket) // 2) * math.sqrt((ket + 1) / (bra + 1))


def _exact_sigma(case, seed):
    sym, group, L, R, terms, target, sectors, n = _superblock(case)
    J, work = target[1], _sigma_work(case)
    if group == "d2h" and work[3] > 400000 or work[0] > 6e12:
        return None
    on = "cuda" if case["m"] > 60 and group != "d2h" else "cpu"
    xl = torch.from_numpy(L.values(3 * seed + 1)).to(on)
    xr = torch.from_numpy(R.values(3 * seed + 2)).to(on)
    psi = _psi(n, 3 * seed)[0].to(on)
    out = -1.25 * psi
    view = {(a, b): psi[o:o + L.space[a][1] * R.space[b][1]].view(L.space[a][1], R.space[b][1]) for a, b, o in sectors}
    res = {(a, b): out[o:o + L.space[a][1] * R.space[b][1]].view(L.space[a][1], R.space[b][1]) for a, b, o in sectors}
    by_left = {}
    for a, b, _ in sectors:
        by_left.setdefault(a, []).append(b)

    def side(B, x, index, trans):
        """[(bra, ket, matrix, scale)] of an operand."""
        if index < 0:
            return [(q, q, None, 1.0) for q in range(len(B.space))]
        base, blocks = B.ops[B.keys[index]]
        k = B.keys[index][3]
        got = []
        for b, c, off in blocks:
            nb, nc = B.space[b][1], B.space[c][1]
            m = x[base + off:base + off + nb * nc].view(nb, nc)
            got.append((c, b, m.T, _adjoint(B.space[c][0][1], B.space[b][0][1], k)) if trans else (b, c, m, 1.0))
        return got

    factor = {}
    for coef, lo, lt, ro, rt in terms:
        k = L.keys[lo][3] if lo >= 0 else R.keys[ro][3] if ro >= 0 else 0
        odd = ro >= 0 and R.keys[ro][0] in (CRE, CCD)
        right = {}
        for rq, rp, m, s in side(R, xr, ro, rt):
            right.setdefault(rp, []).append((rq, m, s))
        for lq, lp, A, sa in side(L, xl, lo, lt):
            for rp in by_left.get(lp, ()):
                into = [(rq, B, sb) for rq, B, sb in right.get(rp, ()) if (lq, rq) in res]
                if not into:
                    continue
                t = view[(lp, rp)] if A is None else A @ view[(lp, rp)]
                for rq, B, sb in into:
                    key = (L.space[lp][0][1], R.space[rp][0][1], k, L.space[lq][0][1], R.space[rq][0][1])
                    if key not in factor:
                        factor[key] = _coupling(key[0], key[1], J, k, key[3], key[4])
                    f = coef * sa * sb * factor[key] * (-1.0 if odd and L.space[lp][0][0] % 2 else 1.0)
                    if f:
                        res[(lq, rq)].add_(t if B is None else t @ B.T, alpha=f)
    return out.cpu().numpy() if case["host"] else out


def _exact_renorm(case, seed):
    sym, own, other, big, kept = _renorm_shape(case["norb"], case["m"])
    x = torch.from_numpy(big.values(2 * seed)).cuda()
    rot, u, o = torch.from_numpy(_rotations(big.space, kept, 2 * seed + 1)).cuda(), [], 0
    for (_, k), m in zip(big.space, kept):
        u.append(rot[o:o + k * int(m)].view(k, int(m)) if m else None)
        o += k * int(m)
    out = []
    for key in sorted(big.keys):
        base, blocks = big.ops[key]
        for b, c, off in blocks:
            if u[b] is not None and u[c] is not None:
                nb, nc = big.space[b][1], big.space[c][1]
                out.append((u[b].T @ x[base + off:base + off + nb * nc].view(nb, nc) @ u[c]).reshape(-1))
    return torch.cat(out).cpu().numpy()


def _exact_density(case, seed):
    _, _, L, R, _, _, sectors, _ = _superblock(case)
    x = _density_psi(case, seed)
    rho = [torch.zeros(k, k, dtype=torch.float64, device="cuda") for _, k in L.space]
    for a, b, off in sectors:
        na, nb = L.space[a][1], R.space[b][1]
        for r in range(case["nroots"]):
            p = x[r, off:off + na * nb].view(na, nb)
            rho[a] += p @ p.T / case["nroots"]
    eig = torch.cat([torch.linalg.eigvalsh(m) for m in rho])
    return {"eig": eig.cpu().numpy(), "rho": torch.cat([m.reshape(-1) for m in rho]).cpu().numpy()}


def _exact_eig(case, seed):
    # the signs of eigenvectors are a choice: no value for them
    return {"w": np.concatenate([torch.linalg.eigvalsh(a).cpu().numpy() for a in _eig_matrices(case, seed)]), "v": None}


def exact(case, seed):
    f = globals().get("_exact_" + case["kind"])
    return f(case, seed) if f else None


# ---- what a pass cannot do without


def _sigma_work(case):
    """(flops of the products, operator elements, wavefunction elements, products)."""
    _, _, L, R, terms, target, sectors, n = _superblock(case)
    have, by_left, flops, count = {(a, b) for a, b, _ in sectors}, {}, 0.0, 0
    for a, b, _ in sectors:
        by_left.setdefault(a, []).append(b)
    used, cache = set(), {}
    for _, lo, lt, ro, rt in terms:
        lb = [(q, q) for q in range(len(L.space))] if lo < 0 else [(c, b) if lt else (b, c) for b, c, _ in L.ops[L.keys[lo]][1]]
        rb = [(q, q) for q in range(len(R.space))] if ro < 0 else [(c, b) if rt else (b, c) for b, c, _ in R.ops[R.keys[ro]][1]]
        used |= {(0, lo), (1, ro)}
        key = (lo < 0, ro < 0, tuple(lb), tuple(rb))
        if key not in cache:
            f, items, right = 0.0, 0, {}
            for rq, rp in rb:
                right.setdefault(rp, []).append(rq)
            for lq, lp in lb:
                for rp in by_left.get(lp, ()):
                    into = [rq for rq in right.get(rp, ()) if (lq, rq) in have]
                    if not into:
                        continue
                    ml, kl, kr = L.space[lq][1], L.space[lp][1], R.space[rp][1]
                    if lo >= 0:
                        f += 2.0 * ml * kl * kr
                        items += 1
                    if ro >= 0:
                        f += sum(2.0 * ml * kr * R.space[rq][1] for rq in into)
                        items += len(into)
            cache[key] = (f, items)
        flops += cache[key][0]
        count += cache[key][1]
    elems = 0
    for side, index in used:
        if index >= 0:
            B = R if side else L
            elems += sum(B.space[b][1] * B.space[c][1] for b, c, _ in B.ops[B.keys[index]][1])
    return flops, elems, n, count


def work(case):
    kind = case["kind"]
    if kind == "sigma":
        flops, elems, n, _ = _sigma_work(case)
        # 16-bit products per logical product and bytes per stored operator element (two 16-bit slices, six digits, FP64)
        products, per = {"fp64": (1, 8), "exacttc": (21, 12)}.get(case["prec"], (3, 4))
        return {"bytes": per * elems + 16.0 * n, "flops": products * flops}
    if kind in ("renorm", "step"):
        _, _, _, big, kept = _renorm_shape(case["norb"], case["m"])
        flops, read, wrote = 0.0, 0, 0
        for _, blocks in big.ops.values():
            for b, c, _ in blocks:
                nb, nc, mb, mc = big.space[b][1], big.space[c][1], int(kept[b]), int(kept[c])
                if mb and mc:
                    flops += 2.0 * nb * nc * mc + 2.0 * mb * nb * mc
                    read += nb * nc
                    wrote += mb * mc
        products = 21 if case["prec"] != "fp64" else 1
        # a step reads the system block, the new site's half-sized source, instead of the enlarged one
        return {"bytes": 8.0 * ((read if kind == "renorm" else read / 9.0) + wrote), "flops": products * flops}
    if kind == "density":
        _, _, L, R, _, _, sectors, n = _superblock(case)
        rho = sum(k * k for _, k in L.space)
        flops = sum(2.0 * L.space[a][1] ** 2 * R.space[b][1] * case["nroots"] for a, b, _ in sectors) + sum(9.0 * k**3 for _, k in L.space)
        return {"bytes": 8.0 * (n * case["nroots"] + rho), "flops": flops}
    if kind == "eig":
        d = _eig_dims(case)
        return {"bytes": 8.0 * sum(2 * n * n + n for n in d), "flops": sum(9.0 * n**3 for n in d)}
    # sweeps: the products of about ten Davidson iterations in each of 2 (norb - 3) steps of two sweeps
    flops, elems, n, _ = _sigma_work({"norb": case["norb"], "m": case["m"]})
    steps = 2 * 2 * (case["norb"] - 3)
    products = 3 if case["prec"] != "fp64" else 1
    return {"bytes": steps * 10 * (8.0 * elems + 16.0 * n), "flops": products * steps * 10 * flops}
