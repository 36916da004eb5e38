"""Performance cases: what a user of the library has it do, with an independent 64-bit answer for each.

A case names a workload by its sizes; `prepare` makes its inputs from a seed (displaced or turned atoms,
a strained cell, jittered k points), `run` makes one call of a public entry point with host buffers, and `exact` says
what that call computes, from the formulas of the NRL tight-binding model in plain numpy and torch.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tight-binding_gb300"))
from nrltb import Context, KMesh, Opts, abi, synth  # noqa: E402
from nrltb.api import Structure  # noqa: E402

LATTICES = {"fcc": (synth.FCC_BASIS, 6.82), "bcc": (synth.BCC_BASIS, 5.42), "sc": (synth.SC_BASIS, 4.6),
            "b2": (synth.BCC_BASIS, 5.5)}
PRECISION = {"fp64": abi.PREC_FP64, "mixed": abi.PREC_MIXED}
DNN = 16.5   # pair cut-off of the synthetic parameter sets, bohr


def listed():
    """The library's own range: one-atom cells on dense meshes to 216-atom cells on sparse ones, both
    precision forms, every kind of result (energies, pressures, bands, charges), and the stages a program
    calls by themselves."""
    return [
        # neighbour list of a molecular-dynamics frame (128 atoms), the stage before everything else
        dict(name="pairs_128", call="pairs", lattice="fcc", nx=4, ny=4, nz=2),
        # E_F of one structure's bands for a scan over fillings and temperatures: the smallest call
        dict(name="fermi_27x1152", call="fermi", nv=1152, nk=27),
        # equation of state / elastic constants of an elemental metal: a strained one-atom cell, dense mesh
        dict(name="cell_fp64", call="bande", lattice="fcc", nx=0, ny=0, nz=0, basis="spd", mesh=12, mode=4,
             precision="fp64"),
        # an sp3 cell with the T -> 0 extrapolation (mode 2), small matrices in the fast form
        dict(name="sp3_8_mixed", call="bande", lattice="sc", nx=2, ny=2, nz=2, basis="sp3", mesh=5, mode=2,
             precision="mixed"),
        # band structure along a path: eigenvalues only (mode 9)
        dict(name="bands_12_fp64", call="bande", lattice="fcc", nx=3, ny=1, nz=1, basis="spd", path=121, mode=9,
             precision="fp64"),
        # orbital charges of every state (mode 6)
        dict(name="charges_16_fp64", call="bande", lattice="bcc", nx=2, ny=2, nz=2, basis="spd", mesh=3, mode=6,
             precision="fp64"),
        # the 32-atom bcc supercell on its 4^3 mesh, both forms
        dict(name="bcc32_fp64", call="bande", lattice="bcc", nx=2, ny=2, nz=4, basis="spd", mesh=4, mode=4,
             precision="fp64"),
        dict(name="bcc32_mixed", call="bande", lattice="bcc", nx=2, ny=2, nz=4, basis="spd", mesh=4, mode=4,
             precision="mixed"),
        # many structures of uneven size in one call (fitting sets)
        dict(name="batch_24_mixed", call="batch", count=24, precision="mixed"),
        # the 128-atom supercell: a few k points in plain FP64, its whole mesh in the fast form
        dict(name="fcc128_4k_fp64", call="bande", lattice="fcc", nx=4, ny=4, nz=2, basis="spd", nk=4, mode=4,
             precision="fp64"),
        dict(name="fcc128_mixed", call="bande", lattice="fcc", nx=4, ny=4, nz=2, basis="spd", mesh=3, mode=4,
             precision="mixed"),
        # the largest: a two-species 216-atom alloy cell, 8 k points
        dict(name="b2_216_mixed", call="bande", lattice="b2", nx=6, ny=6, nz=3, basis="spd", mesh=2, mode=4,
             precision="mixed"),
    ]


def draw(rng):
    """One more case of the same ranges: sizes over their logarithm, odd ones included."""
    call = rng.choice(["bande"] * 7 + ["pairs", "fermi", "batch"])
    if call == "fermi":
        nv = int(round(math.exp(rng.uniform(math.log(9), math.log(1500)))))
        return dict(call="fermi", nv=nv, nk=max(1, min(2000, int(rng.uniform(2e3, 6e4) / nv))))
    if call == "pairs":
        nx, ny, nz = (rng.randint(1, 4) for _ in range(3))
        return dict(call="pairs", lattice=rng.choice(["fcc", "bcc", "sc"]), nx=nx, ny=ny, nz=nz)
    precision = rng.choice(["fp64", "mixed"])
    if call == "batch":
        return dict(call="batch", count=rng.randint(6, 24 if precision == "mixed" else 10), precision=precision)
    flops = 1.6e11 if precision == "fp64" else 9e11   # 24 N^3 a k point: what the largest listed ones take
    while True:
        lattice = rng.choice(["fcc", "bcc", "sc", "b2"])
        nx, ny, nz = (rng.randint(1, 5) for _ in range(3))
        if rng.random() < 0.15 and lattice in ("fcc", "bcc"):
            nx = ny = nz = 0
        case = dict(call="bande", lattice=lattice, nx=nx, ny=ny, nz=nz,
                    basis=rng.choice(["spd", "spd", "sp3"]), mode=rng.choice([4, 4, 4, 2, 3, 9, 6]), precision=precision)
        n = order(case)
        if case["mode"] == 6 and n > 400:
            continue
        most = int(min(2000, flops / (24.0 * n ** 3), 6e7 / n ** 2 if case["mode"] == 6 else 1e9))
        # no draws so small that a listed cell of the same kind covers them
        if most < 1 or n > 1404 or n < 9:
            continue
        nk = max(1, int(most ** rng.uniform(0.3, 1.0)))
        if case["mode"] == 9:
            return dict(case, path=nk)
        mesh = int(nk ** (1 / 3) + 1e-9)
        return dict(case, mesh=min(mesh, 12)) if mesh >= 2 else dict(case, nk=min(nk, 7))


# ---- inputs -------------------------------------------------------------------------------------------------
def parameters(lattice, basis):
    if lattice == "b2":
        return synth.make_params([9, 4], [10.0, 4.0], synth.PARAM_SEED)
    if basis == "sp3":
        return synth.make_params([4], [4.0], synth.BATCH_SP3_SEED)
    return synth.make_params([9], [11.0 if lattice == "fcc" else 8.0], synth.PARAM_SEED)


def order(case):
    """Orbitals of the structure."""
    nb = len(LATTICES[case["lattice"]][0])
    cells = case["nx"] * case["ny"] * case["nz"]
    if case["lattice"] == "b2":
        return cells * 13
    return max(1, cells * nb) * (9 if case["basis"] == "spd" else 4)


def structure(lattice, nx, ny, nz, rng):
    """A supercell with displaced atoms; with no repeats, the strained primitive cell."""
    basis, a = LATTICES[lattice]
    if nx:
        return synth.supercell(basis, a, (nx, ny, nz), (lambda b: 1 + b) if lattice == "b2" else (lambda b: 1),
                               0.1, rng, dnn=DNN)
    plv = a / 2 * (np.array([[0., 1, 1], [1, 0, 1], [1, 1, 0]]) if lattice == "fcc" else
                   np.array([[-1., 1, 1], [1, -1, 1], [1, 1, -1]]))
    plv = plv @ (np.eye(3) + rng.normal(0.0, 0.01, (3, 3)))
    return Structure(np.array([1], np.int32), np.zeros((1, 3)), plv, synth.search_box(plv, DNN),
                     abs(np.linalg.det(plv)), 0.0)


def k_points(case, rng):
    if "path" in case:   # a line from one general point to another
        a, b = rng.uniform(-0.5, 0.5, (2, 3))
        t = np.linspace(0.0, 1.0, case["path"])[:, None]
        return KMesh(a + t * (b - a), np.full(case["path"], 1.0 / case["path"]))
    if "nk" in case:
        return KMesh(rng.uniform(-0.5, 0.5, (case["nk"], 3)), np.full(case["nk"], 1.0 / case["nk"]))
    km = synth.mp_mesh(case["mesh"])
    return KMesh(km.k + rng.uniform(-0.02, 0.02, 3), km.w)


def bande_inputs(case, rng):
    par = parameters(case["lattice"], case["basis"])
    st = structure(case["lattice"], case["nx"], case["ny"], case["nz"], rng)
    opts = Opts(mode=case["mode"], precision=PRECISION[case["precision"]], tkb=0.005, eigcut=1e3, fermi_tol=1e-11)
    return st, par, k_points(case, rng), opts


def batch_inputs(case, rng):
    """Uneven structures of 4 to 64 atoms, spd and sp3 in turn, as a fitting set has them."""
    out = []
    for i in range(case["count"]):
        while True:
            lattice = ("fcc", "bcc", "sc")[rng.integers(3)]
            nx, ny, nz = (int(x) for x in rng.integers(1, 5, 3))
            if 4 <= len(LATTICES[lattice][0]) * nx * ny * nz <= 64:
                break
        out.append(bande_inputs(dict(lattice=lattice, nx=nx, ny=ny, nz=nz, basis="spd" if i % 2 == 0 else "sp3",
                                     mesh=int(rng.integers(2, 4)), mode=4, precision=case["precision"]), rng))
    return out


def fermi_inputs(case, rng):
    eig = np.sort(rng.normal(0.0, 0.5, (case["nk"], case["nv"])), axis=1)
    w = rng.uniform(0.5, 1.5, case["nk"])
    return eig, w / w.sum(), rng.uniform(0.003, 0.02), case["nv"] * rng.uniform(0.5, 1.5)


def inputs(case, seed):
    # the sizes of a batch are its own, not the seed's: every seed is the same amount of work
    rng = np.random.default_rng([7, seed])
    call = case["call"]
    if call == "pairs":
        # the same displaced crystal in another frame: as many pairs for every seed
        st = structure(case["lattice"], case["nx"], case["ny"], case["nz"], np.random.default_rng(case["nx"]))
        turn = np.linalg.qr(rng.normal(size=(3, 3)))[0]
        return (Structure(st.kkind, st.posn @ turn, st.plv @ turn, st.nd, st.volume),
                parameters(case["lattice"], "spd"))
    if call == "fermi":
        return fermi_inputs(case, rng)
    if call == "batch":
        sized = batch_inputs(case, np.random.default_rng(case["count"]))
        return [(Structure(st.kkind, st.posn + rng.normal(0.0, 0.02, st.posn.shape), st.plv, st.nd, st.volume),
                 par, km, op) for st, par, km, op in sized]
    return bande_inputs(case, rng)


_context = []


def context():
    """The one context that a program keeps for all its structures."""
    if not _context:
        _context.append(Context(0))
    return _context[0]


def prepare(case, seed):
    ctx, inp = context(), inputs(case, seed)
    if case["call"] != "batch":
        return case, ctx, inp
    n = len(inp)
    rows = [km.nk * par.nv(st) for st, par, km, _ in inp]
    flat = {k: np.zeros(sum(rows)) for k in ("eig", "deig")}
    res = (abi.Result_ * n)()
    at = 0
    for r, m in zip(res, rows):
        for k, a in flat.items():
            setattr(r, k, a[at:].ctypes.data_as(C.POINTER(C.c_double)))
        at += m
    args = [(t * n)(*[x[i].to_c() for x in inp])
            for i, t in enumerate((abi.Structure_, abi.Params_, abi.KMesh_, abi.Opts_))]
    return case, ctx, (n, args, res, flat, inp)


def run(state):
    case, ctx, inp = state
    call = case["call"]
    if call == "pairs":
        pairs, kneigh, dismin = ctx.search2(*inp)
        return dict(pairs, kneigh=kneigh, dismin=dismin)
    if call == "fermi":
        eig, w, tkb, zfill = inp
        return ctx.fermi(eig, w, tkb, zfill, tol=1e-11)
    if call == "batch":
        n, args, res, flat, _ = inp
        if ctx.lib.nrltb_bande_batch(ctx.h, n, *args, res):
            raise RuntimeError(ctx.lib.nrltb_last_error().decode())
        return dict({k: a.copy() for k, a in flat.items()},
                    **{k: np.array([getattr(r, k) for r in res]) for k in ("efermi", "e_total", "pressure", "npairs")})
    r = ctx.bande(*inp)
    out = dict(efermi=r.efermi, e_total=r.e_total, fermi_shift=r.fermi_shift, dismin=r.dismin, earg1=r.earg1,
               npairs=r.npairs, kneigh=r.kneigh_out, eig=r.eig, k_status=r.k_status, ncut=r.ncut)
    if case["mode"] in (2, 4):
        out.update(pressure=r.pressure, deig=r.deig)
    if case["mode"] in (1, 2):
        out.update(entropy=r.entropy, entropy_shift=r.entropy_shift, earg2=r.earg2)
    if case["mode"] == 6:
        out.update(orbocc=r.orbocc)
    return out


# ---- what one pass cannot do without ----------------------------------------------------------------------------
def solve_work(n, nk, mode):
    """24 N^3 flops of a generalized eigensolve with vectors (20 N^3 / 3 without), 16 N^3 for the two
    Hellmann-Feynman products (modes 2, 4) and 16 N^3 + 24 N^3 for S^1/2 and the charges (mode 6); the k list
    in, eigenvalues and per-state results out."""
    f = 24.0 if mode in (2, 4, 6) else 20.0 / 3.0
    f += 16.0 if mode in (2, 4) else 40.0 if mode == 6 else 0.0
    b = 8.0 * n * (2 if mode in (2, 4) else 1) + (8.0 * n * n if mode == 6 else 0.0) + 40.0
    return nk * b, nk * f * float(n) ** 3


def k_count(case):
    return case.get("path") or case.get("nk") or case["mesh"] ** 3


def work(case):
    call = case["call"]
    if call == "fermi":
        return dict(bytes=8.0 * case["nv"] * case["nk"], flops=20.0 * 30 * case["nk"])
    if call == "pairs":
        nat = case["nx"] * case["ny"] * case["nz"] * len(LATTICES[case["lattice"]][0])
        a = LATTICES[case["lattice"]][1]
        near = 4.19 * DNN ** 3 / (a ** 3 / len(LATTICES[case["lattice"]][0]))
        return dict(bytes=nat * near / 2 * 76.0, flops=nat * near / 2 * 40.0)
    if call == "batch":
        parts = [solve_work(par.nv(st), km.nk, op.mode)
                 for st, par, km, op in batch_inputs(case, np.random.default_rng(case["count"]))]
    else:
        parts = [solve_work(order(case), k_count(case), case["mode"])]
    return dict(bytes=sum(p[0] for p in parts), flops=sum(p[1] for p in parts))


# ---- the same results in 64 bits ----------------------------------------------------------------------------------
def neighbour_pairs(st):
    """Every ordered pair within the cut-off (iat <= jat) in the order atom, atom, image."""
    nd = st.nd
    im = np.stack(np.meshgrid(*[np.arange(-m, m + 1) for m in nd], indexing="ij"), -1).reshape(-1, 3)
    shift = im @ st.plv
    found = []
    for i in range(st.natoms):
        t = st.posn[i:, None, :] + shift[None] - st.posn[i]
        d2 = (t ** 2).sum(-1) - 1e-3
        j, m = np.nonzero((d2 < DNN ** 2) & (d2 > 1e-3))
        found.append((np.full(len(j), i), j + i, im[m], t[j, m]))
    i, j, m, t = (np.concatenate(x) for x in zip(*found))
    return i, j, m, t, np.sqrt((t ** 2).sum(-1))


def screening(dist, screenl):
    x = np.exp((dist - (DNN - 5.0 * screenl)) / screenl)
    return 1.0 / (1.0 + x), -x / (1.0 + x) / screenl   # the factor and its logarithmic derivative


def bond_blocks(u, v):
    """Two-centre 9 x 9 blocks of unit vectors u from the 14 integrals v, by projecting the orbitals on the
    bond: p as vectors, d as traceless symmetric matrices Q (yz, zx, xy, x2-y2, 3z2-r2)."""
    p = len(u)
    q = np.zeros((5, 3, 3))
    for n, (a, b) in enumerate([(1, 2), (2, 0), (0, 1)]):
        q[n, a, b] = q[n, b, a] = math.sqrt(0.5)
    q[3] = np.diag([1, -1, 0]) / math.sqrt(2)
    q[4] = np.diag([-1, -1, 2]) / math.sqrt(6)
    qu = np.einsum("aij,pj->pai", q, u)
    ds = math.sqrt(1.5) * np.einsum("pai,pi->pa", qu, u)
    dp = math.sqrt(2.0) * (qu - np.einsum("pai,pi->pa", qu, u)[..., None] * u[:, None, :])
    v = [v[:, n][:, None, None] for n in range(14)]
    e = np.zeros((p, 9, 9))
    uu, pp = u[:, :, None] * u[:, None, :], np.eye(3)[None] - u[:, :, None] * u[:, None, :]
    e[:, 0:1, 0:1] = v[0]
    e[:, 0:1, 1:4] = v[1] * u[:, None, :]
    e[:, 1:4, 0:1] = v[10] * u[:, :, None]
    e[:, 1:4, 1:4] = v[2] * uu + v[3] * pp
    e[:, 0:1, 4:9] = v[4] * ds[:, None, :]
    e[:, 4:9, 0:1] = v[11] * ds[:, :, None]
    pd = np.einsum("pi,pa->pia", u, ds)
    e[:, 1:4, 4:9] = v[5] * pd + v[6] * dp.transpose(0, 2, 1)
    e[:, 4:9, 1:4] = v[12] * pd.transpose(0, 2, 1) + v[13] * dp
    sig, pi = ds[:, :, None] * ds[:, None, :], np.einsum("pai,pbi->pab", dp, dp)
    e[:, 4:9, 4:9] = v[7] * sig + v[8] * pi + v[9] * (np.eye(5)[None] - sig - pi)
    return e


def model(st, par):
    """(first orbital of each atom, atom pairs, images, [H, S, dH/dV, dS/dV] blocks, on-site terms and their
    volume derivatives) of a structure."""
    kinds, P = par.kinds, par.param
    i, j, m, t, dist = neighbour_pairs(st)
    k1, k2 = st.kkind[i] - 1, st.kkind[j] - 1
    scr, dscr = screening(dist, par.screenl[0])
    vd = dist / (3.0 * st.volume)   # dR/dV
    den, dden = np.zeros((2, st.natoms, kinds))
    for a, b, kb in ((i, j, k2), (j, i, k1)):
        own = (a != b) | (a is i)   # an atom's own images come both ways in the list
        beta = P[17 * kb] ** 2      # density parameter by the neighbour's kind
        d = np.exp(-beta * dist) * scr
        np.add.at(den, (a[own], kb[own]), d[own])
        np.add.at(dden, (a[own], kb[own]), ((dscr - beta) * d * vd)[own])
    on, don = np.zeros((2, st.natoms, 4))
    for a in range(st.natoms):
        k = st.kkind[a] - 1
        x = den[a, k] ** (2 / 3)
        dx = 2 / 3 * den[a, k] ** (-1 / 3) * dden[a, k]
        c = P[17 * k + 1:17 * k + 17].reshape(4, 4)
        on[a] = c @ x ** np.arange(4)
        don[a] = c[:, 1:] @ (np.arange(1, 4) * x ** np.arange(3)) * dx
        for b in range(kinds):
            if b != k and den[a, b] != 0:
                hi, lo = max(k, b), min(k, b)
                at = kinds * 17 + 24 * (hi * (hi - 1) // 2 + lo) + (12 if b < hi else 0)
                x, c = den[a, b] ** (2 / 3), P[at:at + 12].reshape(4, 3)
                dx = 2 / 3 * den[a, b] ** (-1 / 3) * dden[a, b]
                on[a] += c @ x ** np.arange(1, 4)
                don[a] += c @ (np.arange(1, 4) * x ** np.arange(3)) * dx
    base, unlike = kinds * (1 + 4 * (3 * kinds + 1)), kinds * (kinds - 1) // 2
    lo, hi = np.minimum(k1, k2), np.maximum(k1, k2)
    blocks = []
    for s in range(2):
        at = base + s * (40 * kinds + 56 * unlike) + np.where(lo == hi, 40 * lo, 40 * kinds + 56 * (hi * (hi - 1) // 2 + lo))
        c = P[np.minimum(at[:, None] + np.arange(56), len(P) - 1)].reshape(-1, 14, 4)
        c = np.where(((lo == hi)[:, None] & (np.arange(14) >= 10)[None])[..., None], 0.0, c)
        r = dist[:, None]
        poly, dpoly, g = c[..., 0] + r * (c[..., 1] + r * c[..., 2]), c[..., 1] + 2 * r * c[..., 2], -c[..., 3] ** 2
        ex = np.exp(g * r) * scr[:, None]
        blocks += [poly * ex, vd[:, None] * ((dpoly + g * poly) * ex + dscr[:, None] * poly * ex)]
    full = []
    for b in (blocks[0], blocks[2], blocks[1], blocks[3]):
        # (second orbital, first orbital) integrals: their own for unlike kinds, else by the bond's parity
        v = b.copy()
        flip = [(10, 1, -1), (11, 4, 1), (12, 5, -1), (13, 6, -1)]
        for x, y, sg in flip:
            v[:, x] = np.where(k1 == k2, sg * b[:, y], np.where(k1 > k2, sg * b[:, y], b[:, x]))
            v[:, y] = np.where(k1 > k2, sg * b[:, x], b[:, y])
        full.append(bond_blocks(t / dist[:, None], v))
    first = np.concatenate([[0], np.cumsum(par.kbas[st.kkind - 1])])
    return first, (i, j), m, full, (on, don)


def dense(st, par, mod, k, which):
    """H or S (or dH/dV, dS/dV) of k points k as torch complex128 on the GPU."""
    first, (i, j), m, full, on = mod
    n, nk = int(first[-1]), len(k)
    kb = par.kbas[st.kkind - 1]
    ph = np.exp(2j * np.pi * (k @ m.T.astype(float)))
    a, b = np.meshgrid(np.arange(9), np.arange(9), indexing="ij")
    keep = (a[None] < kb[i][:, None, None]) & (b[None] < kb[j][:, None, None])
    row, col = (first[i][:, None, None] + a)[keep], (first[j][:, None, None] + b)[keep]
    pair = np.broadcast_to(np.arange(len(i))[:, None, None], keep.shape)[keep]
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    val = torch.from_numpy(np.ascontiguousarray(full[which][keep])).to(dev)
    at, pr = torch.from_numpy(row * n + col).to(dev), torch.from_numpy(pair.copy()).to(dev)
    out = torch.zeros((nk, n * n), dtype=torch.complex128, device=dev)
    pht = torch.from_numpy(ph).to(dev)
    for q in range(nk):
        out[q].index_add_(0, at, val * pht[q][pr])
    out = out.reshape(nk, n, n)
    # only iat <= jat is listed: the blocks below are the conjugates of those above
    below = torch.from_numpy(np.repeat(np.arange(st.natoms), kb)).to(dev)
    below = below[:, None] > below[None, :]
    out = torch.where(below, out.mH, out)
    cls = np.array([0, 1, 1, 1, 2, 2, 2, 3, 3])
    diag = np.concatenate([on[which // 2][a][cls[:kb[a]]] for a in range(st.natoms)]) if which % 2 == 0 else \
        np.full(n, 1.0 if which == 1 else 0.0)
    out += torch.diag(torch.from_numpy(diag).to(dev)).to(torch.complex128)
    return 0.5 * (out + out.mH)


def occupation(e, mu, tkb):
    """Fermi factors, exactly 1 and 0 beyond 20 kT."""
    x = np.clip((e - mu) / tkb, -40.0, 40.0)
    return np.where(e < mu - 20 * tkb, 1.0, np.where(e < mu + 20 * tkb, 1.0 / (1.0 + np.exp(x)), 0.0))


def fermi_level(e, w, tkb, zfill, tol=1e-11):
    fill = int(zfill / 2 + 1e-5)
    if abs(zfill / 2 - fill) < tol and 1 <= fill < e.shape[1]:
        below, above = e[:, fill - 1].max(), e[:, fill].min()
        if above - below > 20 * tkb:
            return 0.5 * (below + above)
    lo, hi = e.min(), e.max()
    while True:
        mu = 0.5 * (lo + hi)
        if mu in (lo, hi):
            return mu
        if 2.0 * math.fsum((w[:, None] * occupation(e, mu, tkb)).ravel()) < zfill:
            lo = mu
        else:
            hi = mu


def exact_bande(case_mode, st, par, km, op):
    mod = model(st, par)
    n, eig, deig, orb = int(mod[0][-1]), [], [], []
    step = max(1, int(2e8 / (16 * n * n)))
    for a in range(0, km.nk, step):
        k = km.k[a:a + step]
        h, s = (dense(st, par, mod, k, q) for q in (0, 1))
        low = torch.linalg.cholesky(s)
        x = torch.linalg.solve_triangular(low, h, upper=False)
        x = torch.linalg.solve_triangular(low, x.mH, upper=False)
        e, z = torch.linalg.eigh(0.5 * (x + x.mH))
        z = torch.linalg.solve_triangular(low.mH, z, upper=True)
        eig.append(e.cpu().numpy())
        if case_mode in (2, 4):
            dh, ds = ((z.conj() * (dense(st, par, mod, k, q) @ z)).sum(-2).real for q in (2, 3))
            deig.append((dh - e * ds).cpu().numpy())
        if case_mode == 6:
            o, v = torch.linalg.eigh(s)
            uz = v @ (o.sqrt()[..., None] * (v.mH @ z))
            orb.append((uz.abs() ** 2).mT.cpu().numpy())
    eig, tkb = np.concatenate(eig), op.tkb
    mu = fermi_level(eig, km.w, tkb, par.zfill(st))
    f, w = occupation(eig, mu, tkb), 2.0 * km.w[:, None]
    out = dict(efermi=mu, e_total=float((w * f * eig).sum()), eig=eig, earg1=float((w * f * eig).sum()))
    win = (eig >= mu - 20 * tkb) & (eig < mu + 20 * tkb)
    df = np.where(win, -f * (1.0 - f) / tkb, 0.0)
    if case_mode in (2, 4):
        deig = np.concatenate(deig)
        shift = float((w * df * deig).sum() / (w * df).sum()) if abs((w * df).sum()) > 1e-10 else 0.0
        press = -float((w * f * deig).sum() + (w * df * eig * deig).sum() - shift * (w * df * eig).sum())
        out.update(deig=deig, fermi_shift=shift, pressure=press)
    if case_mode in (1, 2):
        g = np.where(win, f, 0.5)
        ent = -float(np.where(win, w * (g * np.log(g) + (1 - g) * np.log(1 - g)), 0.0).sum())
        out.update(entropy=ent, earg1=out["e_total"] - 0.5 * tkb * ent)
    if case_mode == 6:
        out.update(orbocc=np.concatenate(orb))
    return out


def exact(case, seed):
    inp = inputs(case, seed)
    call = case["call"]
    if call == "pairs":
        st, par = inp
        _, _, _, t, dist = neighbour_pairs(st)
        scr, dscr = screening(dist, par.screenl[0])
        return dict(tt=t / dist[:, None], dist=dist, screen=scr, dscrn=dscr, dismin=float(dist.min()))
    if call == "fermi":
        return float(fermi_level(*inp))
    if call == "batch":
        got = [exact_bande(op.mode, st, par, km, op) for st, par, km, op in inp]
        return dict({k: np.concatenate([g[k].ravel() for g in got]) for k in ("eig", "deig")},
                    **{k: np.array([g[k] for g in got]) for k in ("efermi", "e_total", "pressure")})
    n, nk = order(case), k_count(case)
    if 24.0 * n ** 3 * nk > 2.5e11:   # a minute and more of dense eigensolves
        return None
    return exact_bande(case["mode"], *inp)
