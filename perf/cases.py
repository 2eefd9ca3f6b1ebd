"""Performance cases: what a user of the recursion library runs, from the smallest call to the largest.

Every case is one call of a public entry point on an operator (or supercell) that the caller's program built before:

* ``green``   -- ``chains_run``: the batched chains of an SCF contour or of a real-axis DOS (edc route), and the real
                 chains of the plain route;
* ``blk``     -- ``edc_green_blk``: one group of energies, the reference's own block call;
* ``proj``    -- ``chains_proj``: the projected chains of the Bloch spectral function;
* ``adjoint`` -- ``chains_adjoint`` / ``chains_adjoint_ext``: the reverse sweep behind ``torch.autograd``;
* ``kpm``     -- ``Supercell.kpm_moments``: Chebyshev moments of an explicit supercell.

The operators are those of the benchmark, the shipped examples and the tests; bond blocks, species parameters and
energies are drawn from the seed.  ``exact`` gives the same results in 64 bits from plain torch and numpy: the chains on
the unreduced augmented space (no group, no orbits), the moments by dense block products, the gradients by autograd.
"""
import numpy as np
import torch

import asr_b200 as A
from asr_b200 import kpm as K
from asr_b200 import lattices as lat
from asr_b200 import spectral as SP
from asr_b200 import synthetic as S

# name: lattice, conventional cells per edge, species fractions, closure levels (rank 1), group, start orbitals that are
# one dimensional under the group, nodes and group order (for the work counts), share of the neighbour slots that hold a
# link inside the node set
OPERATORS = {
    "bcc_binary_levels2": dict(lattice="bcc", cells=3, conc=(0.5, 0.5), levels=2, group="d2h", orbs=9, nodes=395, order=8, links=0.90),
    "bcc_binary": dict(lattice="bcc", cells=4, conc=(0.5, 0.5), levels=4, group="d2h", orbs=9, nodes=2536, order=8, links=1.0),
    "fcc_ternary_levels2": dict(lattice="fcc", cells=4, conc=(0.66, 0.14, 0.20), levels=2, group="d2h", orbs=9, nodes=3256, order=8, links=0.70),
    "fcc_quinary_levels2": dict(lattice="fcc", cells=3, conc=(0.2,) * 5, levels=2, group="d2h", orbs=9, nodes=3900, order=8, links=0.81),
    "fcc_ternary": dict(lattice="fcc", cells=5, conc=(0.66, 0.14, 0.20), levels=3, group="d2h", orbs=9, nodes=20969, order=8, links=0.81),
    "cuzn_alloy": dict(lattice="cuzn", cells=8, conc=(0.5, 0.5), levels=4, group="class", orbs=4, nodes=17515, order=16, links=0.85),
    "l21": dict(lattice="l21", cells=4, conc=(0.6, 0.4), levels=3, group="d2", orbs=9, nodes=994, order=4, links=0.96),
}
CUZN_ORBS = (1, 3, 5, 7)   # s, p_z, d_xy, d_3z2-r2: one dimensional under the class group


def listed():
    return [
        # one contour block of one orbital: the smallest call of a program that schedules its own chains; latency counts
        dict(name="blk_small", kind="blk", op="bcc_binary_levels2", groups=1, energies=32, depth=16, tail="hull",
             precision="fp64", depth_tol=0.0, o=0.0, axis="contour"),
        # the plain route: nine real chains, Beer-Pettifor tail, DOS at 2000 energies
        dict(name="plain_bcc_bp", kind="green", mode="plain", op="bcc_binary", groups=9, energies=2000, depth=12, tail="bp",
             precision="fp64", depth_tol=0.0, o=0.0, axis="real"),
        # a slice of the real-axis DOS, all species, orbitals and spins, with the batch shape of an earlier autotune
        dict(name="dos_fcc", kind="green", mode="edc", op="fcc_ternary", groups=54, energies=96, depth=22, tail="hull",
             precision="fp64", depth_tol=0.0, o=0.0, axis="real", tuned=True),
        # an SCF iteration's contour in the mixed form (FP32 vectors and matvec, FP64 coefficients and fractions), one spin
        # channel; 48 points: the last tile of a group is half full
        dict(name="contour_fcc_fp32", kind="green", mode="edc", op="fcc_ternary", groups=27, energies=48, depth=22, tail="hull",
             precision="fp32", depth_tol=0.0, o=0.0, axis="contour"),
        # the shipped bcc example: class group, adaptive depth, one contour of 77 points
        dict(name="cuzn_depth_test", kind="green", mode="edc", op="cuzn_alloy", groups=8, energies=77, depth=24, tail="hull",
             precision="fp64", depth_tol=1e-5, o=0.0, axis="contour"),
        # the whole operator form H = E + h - h o h + X(z): every self-consistent potential has o != 0
        dict(name="general_fcc", kind="green", mode="edc", op="fcc_ternary", groups=9, energies=64, depth=20, tail="hull",
             precision="fp64", depth_tol=0.0, o=0.15, axis="contour"),
        # the same on the small ordered cell with one disordered sublattice, Beer-Pettifor tails
        dict(name="general_l21_bp", kind="green", mode="edc", op="l21", groups=18, energies=32, depth=20, tail="bp",
             precision="fp64", depth_tol=0.0, o=0.15, axis="contour"),
        # gradients of the contour charges for the mixing step
        dict(name="adjoint_fcc", kind="adjoint", op="fcc_ternary", groups=9, energies=48, depth=20, tail="hull",
             precision="fp64", depth_tol=0.0, o=0.0, axis="contour"),
        # the Jacobian's gradient on the whole operator form
        dict(name="adjoint_l21", kind="adjoint", op="l21", groups=9, energies=32, depth=20, tail="hull", precision="fp64",
             depth_tol=0.0, o=0.15, axis="contour"),
        # one spectral window: projections on 55 target sites
        dict(name="proj_fcc", kind="proj", op="fcc_ternary", groups=9, energies=64, depth=24, tail="hull", precision="fp64",
             depth_tol=0.0, o=0.0, axis="real"),
        # moments of the large supercell in the mixed form
        dict(name="kpm_40_fp32", kind="kpm", cells=40, moments=128, vectors=64, precision="fp32", order=True, doubling=True),
        # and of a smaller, odd-sized one in FP64
        dict(name="kpm_23_fp64", kind="kpm", cells=23, moments=200, vectors=50, precision="fp64", order=True, doubling=True),
    ]


def draw(rng):
    kind = rng.choice(["blk", "green", "green", "green", "plain", "proj", "adjoint", "kpm", "kpm"])

    def log(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    if kind == "kpm":
        return dict(kind="kpm", cells=log(5, 28), moments=2 * log(12, 64) + rng.randint(0, 1), vectors=log(8, 80),
                    precision=rng.choice(["fp32", "fp64"]), order=rng.random() < 0.5, doubling=rng.random() < 0.8)
    names = {"blk": ["bcc_binary_levels2", "bcc_binary", "fcc_ternary_levels2", "fcc_quinary_levels2", "l21"],
             "plain": ["bcc_binary", "fcc_ternary_levels2", "fcc_quinary_levels2", "fcc_ternary"],
             "proj": ["bcc_binary", "fcc_ternary_levels2"],
             "adjoint": ["bcc_binary", "fcc_ternary_levels2", "fcc_quinary_levels2", "l21"],
             "green": [n for n in OPERATORS if n != "bcc_binary_levels2"]}[kind]
    name = rng.choice(names)
    op = OPERATORS[name]
    most = 2 * len(op["conc"]) * op["orbs"]
    case = dict(kind=kind, op=name, groups=log(1, min(most, 27)), energies=log(5, 96), depth=rng.randint(9, 28),
                tail=rng.choice(["hull", "hull", "bp", "avg2", "none"]), precision=rng.choice(["fp64", "fp64", "fp32"]),
                depth_tol=0.0, o=0.0, axis=rng.choice(["contour", "real"]))
    if kind == "blk":
        case.update(groups=1)
    elif kind == "plain":
        case.update(kind="green", mode="plain", groups=log(1, 9), energies=log(100, 2000), axis="real", precision="fp64")
    elif kind == "green":
        case.update(mode="edc", depth_tol=rng.choice([0.0, 0.0, 1e-5]), o=rng.choice([0.0, 0.0, 0.15]))
        if op["nodes"] > 10000:
            case.update(groups=min(case["groups"], 9))
    elif kind == "proj":
        case.update(groups=min(case["groups"], 9), precision="fp64")
    else:
        case.update(groups=min(case["groups"], 9), precision="fp64", tail=rng.choice(["hull", "avg2", "none"]),
                    o=0.15 if name == "l21" else 0.0)
    return case


# ---------------------------------------------------------------------------------------------------------- inputs
def _operator_inputs(op, seed):
    """Graph, group and model of an operator; the bond blocks come from the seed."""
    if op["lattice"] == "cuzn":
        c = S.example_case("cuzn_alloy", 1, seed=seed, l=op["cells"])
    elif op["lattice"] == "l21":
        c = S.heusler_case(op["cells"], seed, 4, op["levels"], 1)
    else:
        c = S.cubic_case(op["lattice"], op["cells"], len(op["conc"]), list(op["conc"]), seed=seed, group=op["group"])
        fl = np.ones(c["graph"].n, np.int32)
        fl[0] = 0
        c["flippable"] = fl
    return c


def _chain_inputs(case, seed):
    """Everything a chain call is given: operator inputs, chain specs, energies, seeds of the adjoint, targets."""
    op = OPERATORS[case["op"]]
    c = _operator_inputs(op, seed)
    mdl = c["model"]
    rng = np.random.default_rng([seed, 7])
    kap = int(c["cls"][0]) - 1
    centres = [int(x) for x in mdl.spc[: mdl.nsc[kap], kap]]
    orbs = CUZN_ORBS if op["lattice"] == "cuzn" else tuple(range(1, 10))
    deep = case["depth"]
    specs, eds = [], []
    for spin in range(2):
        sp = S.draw_species(mdl.nsp, seed + 100003 * spin)
        ol = S.draw_o(mdl.nsp, seed + 100003 * spin, case["o"]) if case["o"] else None
        for cen in centres:
            ed = S.edc_params(sp, cen) if ol is None else S.edc_params_o(sp, ol, cen)
            plain = S.plain_params(sp)
            for l0 in orbs:
                nlev = int(deep + (rng.integers(-6, 7) if case["kind"] == "green" and case.get("mode") == "edc" and deep > 15 else 0))
                if case.get("mode") == "plain":
                    specs.append(A.ChainSpec(c=plain[0], d=plain[1], o=plain[2], e=plain[3], start_orb=l0, nlev=nlev))
                else:
                    specs.append(A.ChainSpec(c=ed["c"], d=ed["d"], o=ed["o"], e=ed["e"], pa=ed["pa"], pb=ed["pb"],
                                             frozen_sp=0 if case["kind"] == "blk" else cen, start_orb=l0, nlev=nlev))
                eds.append((cen, ed))
    specs, eds = specs[: case["groups"]], eds[: case["groups"]]
    ne, shift = case["energies"], 0.1 * rng.random()
    if case["axis"] == "contour":
        x, _ = np.polynomial.legendre.leggauss(ne)
        ebot, ef = -1.2 - shift, 0.3 - shift
        z = 0.5 * (ebot + ef) + 0.5 * (ef - ebot) * np.exp(0.5j * np.pi * (1.0 - x))
    else:
        z = np.linspace(-1.5 + shift, 1.0 + shift, ne) + 0.005j
    out = dict(c, specs=specs, eds=eds, z=z, orbs=orbs, levels=op["levels"])
    if case["kind"] == "adjoint":
        out["w"] = rng.standard_normal((ne, len(specs))) + 1j * rng.standard_normal((ne, len(specs)))
    if case["kind"] == "proj":   # the sites within 1.5 lattice constants of the origin (minimum image)
        m = 2 * op["cells"]
        h = (c["coord"] + m // 2) % m - m // 2
        out["tsite"] = (np.nonzero(np.sum(h * h, axis=0) <= 9)[0] + 1).astype(np.int32)
        t0 = int(np.nonzero(out["tsite"] == 1)[0][0])
        nsm = int(np.max(mdl.nsc))
        tw = np.zeros((9, nsm, len(out["tsite"]), len(specs)), order="F")
        for q, (cen, ed) in enumerate(eds):
            free = SP.spectral_dressing(ed["dc"], ed["dl"], [1 + s for s in range(mdl.nsp)], list(op["conc"]), False, nsm)
            tw[:, :, :, q] = free[:, :, None]
            tw[:, :, t0, q] = SP.spectral_dressing(ed["dc"], ed["dl"], [1 + s for s in range(mdl.nsp)], list(op["conc"]), True, nsm)
        out["tw"] = tw
    return out


def _kpm_inputs(case, seed):
    conc = [0.66, 0.14, 0.20]
    if case["order"]:
        nbr, spc, bvec, _ = K.fcc_supercell(case["cells"], conc, -0.10, seed, sweeps=4)
    else:
        g, _, bvec = lat.periodic_graph_shells("fcc", case["cells"], 4)
        nbr = np.asfortranarray(g.nbr.reshape(g.n, bvec.shape[1]).T)
        spc = np.random.default_rng([seed, 3]).choice(3, size=g.n, p=conc).astype(np.int32) + 1
    block, block0 = S.sk_blocks(bvec, seed)
    c, d, o, e = S.plain_params(S.draw_species(3, seed))
    # spectral bound: |H| <= max |c| + max d^2 (sum over the slots of |B|_inf)
    rows = np.sum([np.abs(block[:, :, k]).sum(1).max() for k in range(block.shape[2])]) + np.abs(block0).sum(1).max()
    sc = 1.05 * (np.max(np.abs(c)) + np.max(d) ** 2 * rows)
    return dict(nbr=nbr, spc=spc, block=block, block0=block0, c=c, d=d, o=o, e=e, cen=0.0, sc=float(sc), seed=seed)


def prepare(case, seed):
    if case["kind"] == "kpm":
        i = _kpm_inputs(case, seed)
        return dict(case=case, sc=K.Supercell(i["nbr"], i["spc"], i["c"], i["d"], i["o"], i["e"], i["block"], i["block0"]), inp=i)
    i = _chain_inputs(case, seed)
    args = (i["graph"], i["model"], i["cls"], i["perm"], i["dmat"], 1, i["levels"])
    if case["kind"] == "proj":
        op, tnode, tgop = A.build_augcls_operator(*args, maxrank=1, flippable=i["flippable"], tsite=i["tsite"])
        return dict(case=case, op=op, inp=i, tnode=tnode, tgop=tgop)
    op = A.build_augcls_operator(*args, maxrank=1, flippable=i["flippable"])
    if case.get("tuned"):
        A.set_tuning(op, case["precision"], 16, 4, "fixed-offset")
    if case["kind"] == "blk":
        s, (cen, _) = i["specs"][0], i["eds"][0]
        op.set_params(s.c, s.d, s.o, s.e)
        op.freeze_site(1, cen)
        op.set_start(s.start_orb)
    return dict(case=case, op=op, inp=i)


def run(state):
    case, i = state["case"], state["inp"]
    if case["kind"] == "kpm":
        return state["sc"].kpm_moments(i["cen"], i["sc"], case["moments"], case["vectors"], seed=i["seed"],
                                       precision=case["precision"], doubling=case["doubling"])
    op, specs, z = state["op"], i["specs"], i["z"]
    if case["kind"] == "blk":
        g, m, a, b = A.edc_green_blk(op, i["eds"][0][1], z, specs[0].start_orb, specs[0].nlev, case["depth_tol"], case["tail"],
                                     case["precision"])
        return dict(g=g, m=m, a=a, b=b)
    if case["kind"] == "proj":
        return A.chains_proj(op, specs, z, state["tnode"], state["tgop"], i["tw"], case["tail"], case["precision"])
    if case["kind"] == "adjoint":
        if case["o"]:
            g, m, grad = A.chains_adjoint_ext(op, specs, z, i["w"], case["depth_tol"], case["tail"], case["precision"])
            return dict(g=g, m=m, grad=grad)
        g, grad = A.chains_adjoint(op, specs, z, i["w"], case["tail"], case["precision"])
        return dict(g=g, grad=grad)
    return A.chains_run(op, specs, z, case["mode"], case["depth_tol"], case["tail"], case["precision"])


def work(case):
    """A chain step: one S application (162 real-complex products per block) per chain, reading the vector and its
    predecessor and writing the next one; the general form applies S twice; the reverse sweep applies the operator once
    more and reads what it differentiates.  A Chebyshev step: one block product per slot, two vectors read, one written."""
    if case["kind"] == "kpm":
        n, b = 4 * case["cells"] ** 3, 4 if case["precision"] == "fp32" else 8
        steps = (case["moments"] + 1) // 2 if case["doubling"] else case["moments"] - 1
        return {"bytes": float(3 * b * 9 * n * case["vectors"] * steps), "flops": float(2 * 81 * 19 * n * case["vectors"] * steps)}
    op = OPERATORS[case["op"]]
    slots = 18 if op["lattice"] == "fcc" else 14
    real = 1 if case.get("mode") == "plain" else 2
    chains = case["groups"] * (1 if real == 1 else case["energies"])
    b = 4 if case["precision"] == "fp32" else 8
    applies = (2 if case["o"] else 1) * (2 if case["kind"] == "adjoint" else 1)
    steps = chains * case["depth"]
    vec = 9 * op["nodes"] * real
    return {"bytes": float(3 * b * vec * steps * applies), "flops": float(2 * 9 * (op["links"] * slots + 1) * vec * steps * applies)}


# ---------------------------------------------------------------------------------------------------------- exact
DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


def exact(case, seed):
    if case["kind"] == "kpm":
        return _exact_kpm(case, _kpm_inputs(case, seed))
    op = OPERATORS[case["op"]]
    lanes = case["groups"] * (1 if case.get("mode") == "plain" else case["energies"])
    size = lanes * case["depth"] * op["nodes"] * op["order"] * (2 if case["o"] else 1) * (6 if case["kind"] == "adjoint" else 1)
    if size > 6e9:   # the unreduced chains would take too long
        return None
    return _exact_chains(case, _chain_inputs(case, seed))


class _Space:
    """The unreduced augmented space at rank 1: a node is (site, the one site not in its reference state and its state)."""

    def __init__(self, i):
        g, mdl = i["graph"], i["model"]
        self.nbr = torch.as_tensor(g.nbr.reshape(g.n, -1).astype(np.int64) - 1, device=DEVICE)
        nsm = int(np.max(mdl.nsc))
        cls = torch.as_tensor(np.asarray(i["cls"], np.int64) - 1, device=DEVICE)
        nsc = torch.as_tensor(np.asarray(mdl.nsc, np.int64), device=DEVICE)
        can = torch.as_tensor(np.asarray(i["flippable"]) != 0, device=DEVICE)
        nst = torch.where(can, nsc[cls], torch.ones_like(cls))
        M = 1 + g.n * nsm
        two = torch.cat([torch.arange(g.n, device=DEVICE)[:, None], self.nbr], 1)
        known = front = torch.zeros(1, dtype=torch.int64, device=DEVICE)
        for _ in range(i["levels"]):
            r, code = front // M, front % M
            j = torch.where(code > 0, (code - 1) // nsm, torch.full_like(code, -1))
            new = []
            for k1 in range(two.shape[1]):
                r1 = two[r, k1]
                for k2 in range(two.shape[1]):
                    r2 = two[r1, k2]
                    inside = (code == 0) | (j == r) | (j == r1) | (j == r2)
                    new.append(r2[~inside] * M + code[~inside])
                    new.append(r2[inside] * M)
                    for s in (r[inside], r1[inside], r2[inside]):
                        for k in range(1, nsm):
                            ok = k < nst[s]
                            new.append(r2[inside][ok] * M + 1 + s[ok] * nsm + k)
                new = [torch.unique(torch.cat(new))]
            front = new[0][~torch.isin(new[0], known)]
            known = torch.unique(torch.cat([known, front]))
        self.key, self.n, self.M, self.nsm = known, known.numel(), M, nsm
        self.site = r = known // M
        code = known % M
        j = torch.where(code > 0, (code - 1) // nsm, torch.full_like(code, -1))
        self.own = own = torch.where(j == r, (code - 1) % nsm, torch.zeros_like(code))
        self.cls = cls[r]
        self.hop = [self.find(self.nbr[r, k] * M + code) for k in range(self.nbr.shape[1])]   # n where absent
        self.flips = []   # (state k, nodes, target nodes)
        for k in range(nsm):
            free = (code == 0) | (j == r)
            to = torch.where(free, r * M + (1 + r * nsm + k if k else 0), torch.full_like(r, -1))
            t = self.find(to)
            at = torch.nonzero((t < self.n) & (k != own) & (k < nsc[self.cls]) & (can[r] | (k == 0))).flatten()
            if at.numel():
                self.flips.append((k, at, t[at]))
        self.start = self.find(torch.zeros(1, dtype=torch.int64, device=DEVICE))
        self.phi = np.zeros((len(mdl.nsc), nsm, nsm, mdl.nsp))   # x_s phi_own(s) phi_flip(s) per class
        for kap in range(len(mdl.nsc)):
            n = int(mdl.nsc[kap])
            x = np.asarray(mdl.conc[:n, kap], float)
            v = np.concatenate([np.ones((n, 1)), np.eye(n)[:, : n - 1]], 1)
            for c in range(n):
                for _ in range(2):
                    for b in range(c):
                        v[:, c] -= np.sum(x * v[:, b] * v[:, c]) * v[:, b]
                v[:, c] /= np.sqrt(np.sum(x * v[:, c] ** 2))
            for s in range(n):
                self.phi[kap, :n, :n, mdl.spc[s, kap] - 1] += x[s] * np.outer(v[s], v[s])
        self.phi = torch.as_tensor(self.phi, device=DEVICE)
        block = torch.as_tensor(np.ascontiguousarray(mdl.block[..., 0]), device=DEVICE)
        self.blocks = [torch.as_tensor(np.ascontiguousarray(mdl.block0[..., 0]), device=DEVICE)] + [block[:, :, k] for k in range(block.shape[2])]

    def find(self, key):
        at = torch.searchsorted(self.key, key).clamp(max=self.n - 1)
        return torch.where(self.key[at] == key, at, torch.full_like(at, self.n))

    def weights(self, par, frozen):
        """Diagonal weights (n, 9) of one species parameter (9, nsp), and (nodes, targets, weights) of its flips."""
        fz = (self.site == 0) & (frozen > 0)
        W = torch.einsum("aijs,ls->aijl", self.phi, par)
        diag = torch.where(fz[:, None], par[:, max(frozen, 1) - 1][None, :], W[self.cls, self.own, self.own])
        off = []
        for k, at, to in self.flips:
            keep = ~fz[at]
            off.append((at[keep], to[keep], W[self.cls[at[keep]], self.own[at[keep]], k]))
        return diag, off

    def rand(self, wt, x):   # x (9, n, lanes)
        diag, off = wt
        y = diag.T[:, :, None] * x
        for at, to, w in off:
            y = y.index_add(1, at, w.T[:, :, None] * x[:, to])
        return y

    def smul(self, x):
        xr = torch.view_as_real(x).flatten(2)                       # (9, n, 2 lanes)
        pad = torch.cat([xr, torch.zeros_like(xr[:, :1])], 1)
        acc = (self.blocks[0] @ xr.flatten(1)).view_as(xr)
        for B, hop in zip(self.blocks[1:], self.hop):
            acc = acc + (B @ pad[:, hop].flatten(1)).view_as(xr)
        return torch.view_as_complex(acc.view(9, self.n, -1, 2))


def _recursion(sp, par, frozen, l0, nlev, z, plain, targets=None):
    """Coefficients a, b (lists of (lanes,)) of the chain from orbital l0 of the start node, and the projections of every
    vector on the targets."""
    wt = {k: sp.weights(v, frozen) for k, v in par.items() if v is not None}
    general = bool((par["o"] != 0).any())

    def h(x):
        return sp.rand(wt["d"], sp.smul(sp.rand(wt["d"], x))) + sp.rand(wt["c"], x)

    def apply(x):
        y = h(x)
        if general:
            y = y - h(sp.rand(wt["o"], y))
        y = y + sp.rand(wt["e"], x)
        if "pa" in wt:
            y = y + z[None, None, :] * sp.rand(wt["pa"], x) + sp.rand(wt["pb"], x)
        return y

    u = torch.zeros(9, sp.n, z.numel(), dtype=torch.complex128, device=DEVICE)
    u[l0 - 1, sp.start] = 1.0
    up, bp, a, b, proj = torch.zeros_like(u), torch.zeros_like(z), [], [], []
    for k in range(nlev):
        if targets is not None:
            proj.append(targets(u))
        y = apply(u)
        a.append((u * y).sum((0, 1)))
        w = y - a[-1] * u - bp * up
        b2 = (w * w).sum((0, 1))
        bp = torch.sqrt(b2.real.clamp(min=0)).to(b2.dtype) if plain else torch.sqrt(b2)
        b.append(bp)
        up, u = u, w / bp
    return a, b, proj


def _tail_limits(a, b, tail, plain):
    """(aa, bb) of the square-root tail for chains a (lanes, m), b (lanes, >= m - 1)."""
    m = a.shape[1]
    if tail == "none":
        return None
    if tail == "avg2" and m >= 3 or plain and tail == "avg2" and m >= 2:
        last = (b[:, m - 1], b[:, m - 2]) if plain else (b[:, m - 2], b[:, m - 3])
        return 0.5 * (a[:, m - 1] + a[:, m - 2]), torch.sqrt(0.5 * (last[0] ** 2 + last[1] ** 2))

    def edges(shift):
        T = torch.diag_embed(a.clone()) + torch.diag_embed(b[:, : m - 1], 1) + torch.diag_embed(b[:, : m - 1], -1)
        if shift is not None:
            e = torch.zeros(m, m, dtype=T.dtype, device=T.device)
            e[m - 1, m - 1] = 1.0
            T = T + shift[:, None, None] * e
        lam = torch.linalg.eigvals(T.cpu()).to(a.device)
        at = lam.real.detach()
        return (lam.gather(1, at.argmin(1, keepdim=True))[:, 0], lam.gather(1, at.argmax(1, keepdim=True))[:, 0])

    lo, hi = edges(None)
    aa, bb = 0.5 * (lo + hi), 0.25 * (hi - lo)
    if tail == "bp":
        if plain:
            aa = 0.5 * (a[:, m - 1] + a[:, m - 2])
            bb = torch.sqrt(0.5 * (b[:, m - 1] ** 2 + b[:, m - 2] ** 2))
        done = torch.zeros(aa.shape, dtype=torch.bool, device=aa.device)
        first = (aa, bb)
        for _ in range(500 if plain else 200):
            an_hi, an_lo = edges(bb)[1], edges(-bb)[0]
            an, bn = 0.5 * (an_hi + an_lo), 0.25 * (an_hi - an_lo)
            close = (an - aa).abs() + (bn - bb).abs() < (1e-13 if plain else 1e-12 * (1.0 + bn.abs()))
            aa, bb = torch.where(done, aa, an), torch.where(done, bb, bn)
            done = done | close
            if bool(done.all()):
                break
        if not plain:   # a fixed point that was not reached: the hull's
            aa, bb = torch.where(done, aa, first[0]), torch.where(done, bb, first[1])
    return aa, bb


def _fraction(a, b, z, tail, plain=False):
    """Terminated fraction of a (lanes, m), b at z (lanes, ...); returns G and the factors gt of every level."""
    m = a.shape[1]
    more = (slice(None),) + (None,) * (z.dim() - 1)
    tl = 0.0
    lim = _tail_limits(a, b, tail, plain)
    if lim is not None:
        aa, bb = lim[0][more], lim[1][more]
        d = z - aa
        s = torch.sqrt(d * d - 4 * bb * bb)
        t1, t2 = 0.5 * (d - s), 0.5 * (d + s)
        tl = torch.where(t1.abs() <= t2.abs(), t1, t2)
    gt = [1.0 / (z - a[:, m - 1][more] - tl)]
    for j in range(m - 2, -1, -1):
        gt.insert(0, 1.0 / (z - a[:, j][more] - (b[:, j] ** 2)[more] * gt[0]))
    return gt[0], gt


def _exact_chains(case, i):
    sp = _Space(i)
    specs, ne, ng = i["specs"], case["energies"], len(i["specs"])
    z = torch.as_tensor(i["z"], device=DEVICE)
    plain, nmax = case.get("mode") == "plain", max(s.nlev for s in specs)
    grads = case["kind"] == "adjoint"
    chunk = 1 if plain else max(1, int((2.5e7 if grads else 1e9) / (sp.n * 9 * 16)))
    g = np.zeros((ne, ng), np.complex128)
    mm = np.zeros((ne, ng), np.int32)
    A_, B_ = np.zeros((2, nmax, ne), np.complex128)
    gp, gp4 = None, None
    kinds = ("c", "d", "pa", "o", "e") if case["o"] else ("c", "d", "pa")
    grad = np.zeros((ng, len(kinds), i["model"].nsp, 9), np.complex128)
    for q, s in enumerate(specs):
        par = {k: None if getattr(s, k) is None else torch.as_tensor(np.ascontiguousarray(getattr(s, k)), device=DEVICE)
               for k in ("c", "d", "o", "e", "pa", "pb")}
        frozen = i["eds"][q][0] if case["kind"] == "blk" else s.frozen_sp
        targets = None
        if case["kind"] == "proj":
            r = torch.as_tensor(i["tsite"].astype(np.int64) - 1, device=DEVICE)
            tw = torch.as_tensor(np.ascontiguousarray(i["tw"][..., q]), device=DEVICE)
            nodes = [sp.find(r * sp.M + (1 + r * sp.nsm + k if k else 0)) for k in range(sp.nsm)]
            nodes = [torch.where((r == 0) & (k > 0), torch.full_like(n, sp.n), n) for k, n in enumerate(nodes)]

            def targets(u):
                pad = torch.cat([u, torch.zeros_like(u[:, :1])], 1)
                return sum(tw[:, k, :, None] * pad[:, n] for k, n in enumerate(nodes))
            if gp is None:
                gp, gp4 = np.zeros((2, 9, len(r), ne, ng), np.complex128)
        for at in range(0, 1 if plain else ne, chunk):
            zz = torch.zeros(1, dtype=torch.complex128, device=DEVICE) if plain else z[at: at + chunk]
            if grads:
                for k in kinds:
                    par[k] = par[k].detach().requires_grad_(True)
            with torch.set_grad_enabled(grads):
                a, b, proj = _recursion(sp, par, frozen, s.start_orb, s.nlev, zz, plain, targets)
                a, b = torch.stack(a, 1), torch.stack(b, 1)
                zs = z[None, :] if plain else zz
                m = torch.full(zz.shape, s.nlev, dtype=torch.int32, device=DEVICE)
                if case["depth_tol"] > 0 and not plain:
                    prev, live = None, torch.ones(zz.shape, dtype=torch.bool, device=DEVICE)
                    for k in range(8, s.nlev, 4):
                        gk = _fraction(a[:, :k], b, zz, case["tail"])[0]
                        if prev is not None:
                            stop = live & ((gk - prev).abs() <= case["depth_tol"] * gk.abs())
                            m[stop] = k
                            live = live & ~stop
                        prev = gk
                G = torch.zeros(zs.shape, dtype=torch.complex128, device=DEVICE)
                for k in torch.unique(m).tolist():
                    sel = m == k
                    v, gt = _fraction(a[sel][:, :k], b[sel], zs if plain else zs[sel], case["tail"], plain)
                    G = v if bool(sel.all()) else G.index_put((sel,), v)
            if grads:
                w = torch.as_tensor(i["w"][at: at + chunk, q], device=DEVICE)
                for f in (1.0, -1j):
                    d = torch.autograd.grad((f * w * G).sum().real, [par[k] for k in kinds], retain_graph=True, allow_unused=True)
                    for n, v in enumerate(d):
                        grad[q, n] += (1.0 if f == 1.0 else 1j) * v.T.cpu().numpy()
            if targets is not None:
                for out, k in ((gp, s.nlev), (gp4, max(1, s.nlev - 4))):
                    pv = _fraction(a[:, :k], b, zz, case["tail"])[1]
                    acc, prod = 0.0, pv[0]
                    for n in range(k):
                        acc = acc + proj[n] * prod
                        prod = prod * b[:, n] * pv[n + 1] if n + 1 < k else prod
                    out[:, :, at: at + chunk, q] = acc.cpu().numpy()
            to = slice(0, ne) if plain else slice(at, at + chunk)
            g[to, q] = (G[0] if plain else G).detach().cpu().numpy()
            mm[to, q] = s.nlev if plain else m.cpu().numpy()
            if case["kind"] == "blk":
                A_[: s.nlev, to], B_[: s.nlev, to] = a.T.cpu().numpy(), b.T.cpu().numpy()
            del a, b, proj, G
    if case["kind"] == "blk":
        B_[specs[0].nlev - 1] = 0.0   # the edc chain ends before its last b
        return dict(g=g[:, 0], m=mm[:, 0], a=A_, b=B_)
    if case["kind"] == "proj":
        return dict(g=g, m=mm, gp=gp, gp4=gp4)
    if grads:
        return dict(g=g, m=mm, grad=grad) if case["o"] else dict(g=g, grad=grad)
    return dict(g=g, m=mm)


def _exact_kpm(case, i):
    n, ns, nmom = i["nbr"].shape[1], i["nbr"].shape[0], case["moments"]

    def dev(x, dt=torch.float64):
        return torch.as_tensor(np.ascontiguousarray(x), dtype=dt, device=DEVICE)

    nbr, spc = dev(i["nbr"].astype(np.int64) - 1, torch.int64), dev(i["spc"].astype(np.int64) - 1, torch.int64)
    block, block0 = dev(i["block"]), dev(i["block0"])
    c, d = dev(i["c"])[:, spc][:, :, None], dev(i["d"])[:, spc][:, :, None]
    mu = np.zeros(nmom)
    for v0 in range(0, case["vectors"], 16):
        v = np.arange(v0, min(case["vectors"], v0 + 16), dtype=np.uint64)
        with np.errstate(over="ignore"):   # splitmix64 of the documented counter
            q = np.arange(9 * n, dtype=np.uint64)[:, None]
            x = np.uint64(i["seed"]) * np.uint64(0x9E3779B97F4A7C15) + (v << np.uint64(40))[None, :] + q + np.uint64(0x9E3779B97F4A7C15)
            x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
            x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
            x = x ^ (x >> np.uint64(31))
        r = dev(np.where(x >> np.uint64(63), -1.0, 1.0)).view(n, 9, -1).permute(1, 0, 2).contiguous()

        def h(t):
            u = d * t
            acc = (block0 @ u.flatten(1)).view_as(u)
            for k in range(ns):
                acc += (block[:, :, k] @ u[:, nbr[k]].flatten(1)).view_as(u)
            return (c * t + d * acc - i["cen"] * t) / i["sc"]

        t0, t1 = r, h(r)
        dim = 9.0 * n
        m0, m1 = r.shape[2] * 1.0, float((r * t1).sum()) / dim
        mu[0] += m0
        if nmom > 1:
            mu[1] += m1
        k = 1
        while (2 * k if case["doubling"] else k + 1) < nmom:
            if case["doubling"]:
                mu[2 * k] += 2.0 * float((t1 * t1).sum()) / dim - m0
            if not case["doubling"] or 2 * k + 1 < nmom:
                t0, t1 = t1, 2.0 * h(t1) - t0
                mu[2 * k + 1 if case["doubling"] else k + 1] += 2.0 * float((t1 * t0).sum()) / dim - m1 if case["doubling"] else float((r * t1).sum()) / dim
            k += 1
    return mu / case["vectors"]
