"""The work that programs on this framework have it do, as cases that can be timed.

Each case is one call sequence that a user's program makes through the public
entry points of ``tenes_b200``, on inputs made from a seed:

* ``environment``: new site tensors go to the GPU, the CTM environment is
  computed from scratch (``Environment.calc_ctm_environment``, the reference's
  ``Calc_CTM_Environment``), and the observables are read off: <Sz> of every
  site and the reduced density matrix of every bond.  The options are those of
  an input file: full-SVD or randomised projectors, built from the left
  corners or from all four, FP64 or mixed precision, ground state (iTPS) or
  density operator (iTPO);
* ``simple_update``: imaginary-time steps over every bond of the cell;
* ``observables``: multi-site windows and long correlation strips in a given
  environment;
* ``gradient``: the energy and its gradient through the environment, forward
  and backward.

Environment tensors are defined up to a unitary on each of their legs and site
tensors after a simple update up to the sign (phase) of each bond index, so a
case returns what does not depend on these: density matrices, norms, weights,
and the magnitudes of the updated site tensors.
"""

import numpy as np
import torch

from tenes_b200.env import CTMParams, Environment
from tenes_b200.grad import j1j2_terms
from tenes_b200.std_ops import evolution_twosite, heisenberg_bond, real_if_close

SZ = np.diag([0.5, -0.5])


# ------------------------------------------------------------------ the cases
def environment(LX, LY, D, chi, sweeps, solver="full", corner=True, is_complex=False, mixed=False, density=False,
                brick=False):
    return {"kind": "environment", "LX": LX, "LY": LY, "D": D, "chi": chi, "sweeps": sweeps, "solver": solver,
            "corner": corner, "complex": is_complex, "mixed": mixed, "density": density, "brick": brick}


def listed():
    return [
        # an input file's first try: the transverse-field Ising size of the tutorials, latency and launches alone
        dict(environment(2, 2, 2, 10, 6), name="env 2x2 D2 chi10"),
        # an odd, small complex cell with projectors from all four corners and the randomised SVD
        dict(environment(2, 1, 3, 15, 4, solver="rsvd", corner=False, is_complex=True),
             name="env 2x1 D3 chi15 complex updown rsvd"),
        # an ordinary ground-state run, the default projectors
        dict(environment(2, 2, 4, 32, 4), name="env 2x2 D4 chi32"),
        # the same kind of run with odd sizes and complex tensors
        dict(environment(2, 2, 3, 27, 4, is_complex=True), name="env 2x2 D3 chi27 complex"),
        # production accuracy, randomised projectors: the headline benchmark's sizes
        dict(environment(2, 2, 6, 72, 4, solver="rsvd"), name="env 2x2 D6 chi72 rsvd"),
        # the same in mixed precision
        dict(environment(2, 2, 6, 72, 4, solver="rsvd", mixed=True), name="env 2x2 D6 chi72 rsvd mixed"),
        # the same with the reference's default projectors
        dict(environment(2, 2, 6, 72, 3), name="env 2x2 D6 chi72"),
        # a frustrated magnet on a brick wall: 16 sites, uneven bonds, complex
        dict(environment(4, 4, 4, 48, 3, solver="rsvd", is_complex=True, brick=True),
             name="env 4x4 brick chi48 complex rsvd"),
        # finite temperature: the single-layer environment of a density operator
        dict(environment(2, 2, 8, 64, 4, density=True), name="env 2x2 D8 chi64 density"),
        # imaginary-time evolution between two environments
        {"name": "simple update 2x2 D4", "kind": "simple_update", "LX": 2, "LY": 2, "D": 4, "steps": 20,
         "complex": False},
        # the measurements after a run: plaquettes, and correlations up to ten sites away
        {"name": "observables 2x2 D4 chi40", "kind": "observables", "LX": 2, "LY": 2, "D": 4, "chi": 40, "r_max": 10,
         "complex": False},
        # one evaluation of a variational optimisation
        {"name": "gradient 2x2 D3 chi18", "kind": "gradient", "D": 3, "chi": 18, "sweeps": 2},
    ]


def draw(rng):
    """One more case of the ranges above: the kinds of environment for the most part."""
    kind = rng.choice(["environment"] * 8 + ["simple_update", "observables"])
    log_int = lambda a, b: int(round(a * (b / a) ** rng.random()))  # noqa: E731
    if kind == "simple_update":
        return {"kind": kind, "LX": rng.randint(1, 3) * 2, "LY": 2, "D": rng.randint(2, 6), "steps": log_int(5, 40),
                "complex": rng.random() < 0.4}
    if kind == "observables":
        return {"kind": kind, "LX": 2, "LY": 2, "D": rng.randint(2, 4), "chi": log_int(10, 48),
                "r_max": rng.randint(4, 12), "complex": rng.random() < 0.4}
    density, is_complex = rng.random() < 0.15, rng.random() < 0.4
    if density:
        D = rng.randint(3, 8)
        return environment(2, 2, D, log_int(max(12, D), 64), rng.randint(2, 4), "full", True, is_complex, False, True)
    solver, corner = rng.choice(["full", "rsvd"]), rng.random() < 0.8
    mixed = not is_complex and rng.random() < 0.2
    # the randomised projectors are for environments that are wider than the sketch from the start
    D = rng.randint(3 if solver == "rsvd" else 2, 4 if is_complex or not corner else 6)
    chi = log_int(8, 40 if is_complex or not corner else 72)
    LX, LY = rng.choice([(2, 2), (2, 2), (2, 1), (1, 2), (3, 2), (2, 3)])
    sweeps = rng.randint(1, 2) if D * D * chi * LX * LY > 3000 else rng.randint(2, 4)
    return environment(LX, LY, D, chi, sweeps, solver, corner, is_complex, mixed)


# ----------------------------------------------------------------- the inputs
def bond_dims(case):
    """(left, up, right, down) bond dimensions of every site."""
    LX, LY = case.get("LX", 2), case.get("LY", 2)
    if not case.get("brick"):
        return [[case["D"]] * 4 for _ in range(LX * LY)]
    # brick wall (honeycomb): every other vertical bond is absent, the others around D
    dims = [[0] * 4 for _ in range(LX * LY)]
    for x in range(LX):
        for y in range(LY):
            i, right, top = x + y * LX, (x + 1) % LX + y * LX, x + (y + 1) % LY * LX
            dims[i][2] = dims[right][0] = case["D"] + (x + 2 * y) % 3 - 1
            dims[i][1] = dims[top][3] = case["D"] + (2 * x + y) % 3 - 1 if (x + y) % 2 else 1
    return dims


def site_tensors(case, seed):
    """Site tensors as an imaginary-time evolution leaves them: random
    entries, with weights that fall off along every bond."""
    rng = np.random.default_rng(seed)
    out = []
    for dims in bond_dims(case):
        phys = (2, 2) if case.get("density") else (2,)
        shape = tuple(dims) + phys
        t = rng.normal(size=shape) + (1j * rng.normal(size=shape) if case.get("complex") else 0.0)
        if case.get("density"):  # around the identity of infinite temperature
            t = 0.3 * t
            t[0, 0, 0, 0] += np.eye(2)
        for leg, d in enumerate(dims):
            w = np.exp(-0.5 * np.arange(d)) * (1.0 + 0.1 * rng.random(d))
            t = t * w.reshape([-1 if a == leg else 1 for a in range(t.ndim)])
        out.append(np.ascontiguousarray(t / np.abs(t).max()))
    return out


def params(case):
    p = CTMParams(chi=case.get("chi", 2), max_ctm_iteration=case.get("sweeps", 4), ctm_convergence_epsilon=1e-10)
    p.projector_corner = case.get("corner", True)
    p.mixed = case.get("mixed", False)
    p.density = case.get("density", False)
    if case.get("solver") == "rsvd":
        p.use_rsvd, p.rsvd_oversample_abs = True, 10
    return p


def bonds(case):
    """(site, dx, dy) of every bond to the right and up that is present."""
    return [(i, 1 - v, v) for i, d in enumerate(bond_dims(case)) for v in (0, 1) if d[2 - v] > 1]


def prepare(case, seed):
    dims, tensors = bond_dims(case), site_tensors(case, seed)
    env = Environment(case.get("LX", 2), case.get("LY", 2), [2] * len(dims), dims, params(case),
                      case.get("complex", False))
    state = {"case": case, "env": env, "tensors": tensors, "sz": SZ.astype(env.dtype), "id": np.eye(2, dtype=env.dtype)}
    for i, t in enumerate(tensors):
        env.set_site_tensor(i, t)
    if case["kind"] == "simple_update":
        gate = real_if_close(evolution_twosite(heisenberg_bond(1.0), 0.01))
        state["steps"] = [(i, leg, gate) for leg in (2, 1) for i in range(len(dims))] * case["steps"]
    if case["kind"] == "observables":
        env.calc_ctm_environment(True)
    if case["kind"] == "gradient":
        state["terms"] = j1j2_terms(len(dims), 1.0, 0.5)
    return state


# ------------------------------------------------------------------ one pass
def values(env, v):
    """Measured values as numbers of the site tensors' type (their imaginary part is zero for real ones)."""
    return np.array(v) if env.is_complex else np.array(v).real


def run(state):
    case, env = state["case"], state["env"]
    if case["kind"] == "environment":
        for i, t in enumerate(state["tensors"]):
            env.set_site_tensor(i, t)
        env.calc_ctm_environment(True)
        return {"sz": values(env, [env.contract_one_site(i, state["sz"]) for i in range(env.N)]),
                "rdm": np.stack([env.contract_bond_rdm(*b) for b in bonds(case)])}
    if case["kind"] == "simple_update":
        for i, t in enumerate(state["tensors"]):
            env.set_site_tensor(i, t)
            for leg in range(4):
                env.set_lambda(i, leg, np.ones(t.shape[leg]))
        env.simple_update_many(state["steps"])
        return {"tensors": [np.abs(env.get_site_tensor(i)) for i in range(env.N)],
                "lambda": np.array([[env.get_lambda(i, leg) for leg in range(4)] for i in range(env.N)])}
    if case["kind"] == "observables":
        corners = {(0, 0): state["sz"], (0, 1): state["sz"], (1, 0): state["sz"], (1, 1): state["sz"]}
        plaquettes = [env.contract_window(i, 2, 2, 1, 0, ops) for i in range(env.N) for ops in (corners, None)]
        strips = [env.correlation_strip(i, vertical, case["r_max"], state["sz"], lambda site: [state["sz"]])
                  for i in range(env.N) for vertical in (False, True)]
        return {"plaquettes": values(env, plaquettes), "strips": values(env, strips)}
    for i, t in enumerate(state["tensors"]):
        env.set_site_tensor(i, t)
    energy, grads = env.energy_grad(state["terms"], case["sweeps"], checkpoint_every=case["sweeps"])
    return {"energy": energy, "gradient": grads}


def work(case):
    """Floating-point operations of the contractions that one pass cannot do
    without, and the bytes of its inputs and outputs."""
    size = 16 if case.get("complex") else 8
    mul = 8 if case.get("complex") else 2  # a multiply-add
    dims = bond_dims(case)
    D = float(np.mean([max(d) for d in dims]))
    n, chi, sites = D ** 4 * 2 * (2 if case.get("density") else 1), case.get("chi", 0), len(dims)
    b = 1 if case.get("density") else D  # the conjugated layer's bond dimension
    p = 1 if case.get("density") else 2
    if case["kind"] == "simple_update":
        m = 2 * D  # Theta is m x m; two QRs of (D^3, m), Theta, its SVD, two products back
        step = 2 * 2 * D ** 3 * m * m + 2 * m ** 3 + 20 * m ** 3 + 2 * 2 * D ** 3 * m * D
        return {"bytes": 2 * size * n * sites, "flops": mul / 2 * step * 2 * sites * case["steps"]}
    absorb = mul * (chi ** 3 * D * b + chi ** 2 * D * D * b * b * 2 * p)  # one site's tensors onto one corner
    if case["kind"] == "observables":
        return {"bytes": size * sites * (n + 4 * chi * chi * (1 + D * b)),
                "flops": sites * absorb * (2 * 4 + 2 * 2 * case["r_max"])}
    # a move at one site: two corner blocks, their product with chi columns
    # for the projectors, the new corners and the new edge
    big = chi * D * b
    move = 2 * absorb + mul * 2 * big * big * chi + mul * 2 * chi ** 3 * D * b + 2 * absorb
    flops = 4 * sites * move * case["sweeps"]
    if case["kind"] == "gradient":
        flops *= 3  # forward, and two products for each in the backward
    return {"bytes": size * sites * n * (2 if case["kind"] == "gradient" else 1) + size * 2 * sites * 16, "flops": flops}


# ------------------------------------------------- the same in plain 64 bits
def exact(case, seed):
    """The environment with full-SVD projectors from the left corners, and the
    simple update, in plain torch FP64; the randomised projectors are defined
    by their random test matrix, and the others follow from these."""
    tensors = [torch.from_numpy(t) for t in site_tensors(case, seed)]
    if case["kind"] == "simple_update":
        return exact_simple_update(case, tensors)
    if case["kind"] != "environment" or case["solver"] != "full" or not case["corner"] or case["mixed"]:
        return None
    wide = case["chi"] * case["D"] ** (1 if case["density"] else 2)
    if case["sweeps"] * case["LX"] * case["LY"] * wide ** 3 > 2.2e9:
        return None  # dense SVDs that would take minutes
    return exact_environment(case, tensors)


def exact_simple_update(case, tensors):
    gate = torch.from_numpy(real_if_close(evolution_twosite(heisenberg_bond(1.0), 0.01))).to(tensors[0].dtype)
    nn = neighbours(case["LX"], case["LY"])
    lam = [[torch.ones(d, dtype=torch.float64) for d in t.shape[:4]] for t in tensors]

    def weighted(t, weights, power, skip):
        for leg in range(4):
            if leg != skip:
                shape = [-1 if a == leg else 1 for a in range(5)]
                t = t * (weights[leg] ** power).reshape(shape)
        return t

    for _ in range(case["steps"]):
        for leg in (2, 1):
            back = (leg + 2) % 4
            for i in range(len(tensors)):
                j = nn[i][leg]
                halves = []
                for s, l in ((i, leg), (j, back)):
                    t = weighted(tensors[s], lam[s], 1.0, l).movedim(l, 3)  # outer legs, the bond, the spin
                    q, r = torch.linalg.qr(t.reshape(-1, t.shape[3] * 2))
                    halves.append((t.shape[:3], q, r.reshape(-1, t.shape[3], 2)))
                (so, q1, r1), (to, q2, r2) = halves
                theta = torch.einsum("acp,bcq,pqxy->axby", r1, r2, gate)
                d = r1.shape[1]
                u, s, vh = torch.linalg.svd(theta.reshape(theta.shape[0] * 2, -1), full_matrices=False)
                w = torch.sqrt(s[:d] / torch.linalg.norm(s[:d]))
                lam[i][leg] = lam[j][back] = w
                a = torch.einsum("na,apc->ncp", q1, u[:, :d].reshape(-1, 2, d) * w).reshape(*so, d, 2)
                b = torch.einsum("nb,cbp->ncp", q2, (w[:, None] * vh[:d]).reshape(d, -1, 2)).reshape(*to, d, 2)
                tensors[i] = weighted(a.movedim(3, leg), lam[i], -1.0, leg)
                tensors[j] = weighted(b.movedim(3, back), lam[j], -1.0, back)
    return {"tensors": [t.abs().numpy() for t in tensors],
            "lambda": np.array([[w.numpy() for w in x] for x in lam])}


def neighbours(LX, LY):
    """(left, up, right, down) of every site."""
    at = lambda x, y: x % LX + y % LY * LX  # noqa: E731
    return [(at(x - 1, y), at(x, y + 1), at(x + 1, y), at(x, y - 1)) for y in range(LY) for x in range(LX)]


def contract(spec, *tensors):
    """An einsum, pair by pair from the left."""
    inputs, out = spec.split("->")
    names = inputs.split(",")
    a, ta = names[0], tensors[0]
    for q in range(1, len(names)):
        rest = set("".join(names[q + 1:])) | set(out)
        keep = "".join(c for c in dict.fromkeys(a + names[q]) if c in rest)
        ta = torch.einsum("%s,%s->%s" % (a, names[q], keep), ta, tensors[q])
        a = keep
    return torch.einsum("%s->%s" % (a, out), ta)


def exact_environment(case, tensors):
    LX, LY, chi = case["LX"], case["LY"], case["chi"]
    nn, N = neighbours(LX, LY), LX * LY

    def padded(x, legs):
        if case["density"]:
            x = x[..., None][:chi, :chi] if legs == 4 else x[:chi, :chi]
        else:
            x = x.reshape(x.shape[0] ** 2, x.shape[2] ** 2, *x.shape[4:])[:chi, :chi]
        y = torch.zeros(chi, chi, *x.shape[2:], dtype=x.dtype)
        y[:x.shape[0], :x.shape[1]] = x
        return y

    # corners C[0..3] (top left, top right, bottom right, bottom left) and edges
    # E[0..3] (top, right, bottom, left) of every site, legs clockwise, from the
    # double layers of the neighbours
    C, E = [[None] * N for _ in range(4)], [[None] * N for _ in range(4)]
    if case["density"]:
        # one layer: the density tensors with their spin legs traced, boundary
        # bonds summed over, and a unit tensor in the place of the other layer
        tn, tensors = tensors, [torch.einsum("lurbpp->lurb", t)[..., None] for t in tensors]
        bra = lambda t: torch.ones(1, 1, 1, 1, t.shape[4], dtype=t.dtype)  # noqa: E731
        corners = ["lurbp->br", "lurbp->lb", "lurbp->ul", "lurbp->ru"]
        edges = ["lurbp->lrb", "lurbp->ubl", "lurbp->rlu", "lurbp->bur"]
        double = lambda spec, t: torch.einsum(spec, t)  # noqa: E731
    else:
        tn, bra = tensors, torch.conj
        corners = ["lurbp,luRBp->bBrR", "lurbp,LurBp->lLbB", "lurbp,LUrbp->uUlL", "lurbp,lURbp->rRuU"]
        edges = ["lurbp,LuRBp->lLrRbB", "lurbp,LUrBp->uUbBlL", "lurbp,LURbp->rRlLuU", "lurbp,lURBp->bBuUrR"]
        double = lambda spec, t: torch.einsum(spec, t, t.conj())  # noqa: E731
    for i in range(N):
        for k, (v, h) in enumerate(((1, 0), (1, 2), (3, 2), (3, 0))):
            C[k][i] = padded(double(corners[k], tensors[nn[nn[i][h]][v]]), 2)
        for k, way in enumerate((1, 2, 3, 0)):
            E[k][i] = padded(double(edges[k], tensors[nn[i][way]]), 4)

    def move(r, line):
        """The left move in the lattice turned r times by a quarter: corner k
        stands in for k + r, the direction w for w + r."""
        c, e = (lambda k, i: C[(k + r) % 4][i]), (lambda k, i: E[(k + r) % 4][i])
        go = lambda i, way: nn[i][(way + r) % 4]  # noqa: E731
        site = lambda i: tensors[i].permute(*[(w + r) % 4 for w in range(4)], 4)  # noqa: E731
        P = {}
        for i in line:
            down = go(i, 3)
            t, u = site(i), site(down)
            lt = contract("xa,aekm,yxln->ekmyln", c(0, i), e(0, i), e(3, i))
            lt = contract("ekmyln,nmRBp,lkrbp->reRbyB", lt, bra(t), t)
            lb = contract("xa,ayln,exkm->ylnekm", c(3, down), e(3, down), e(2, down))
            lb = contract("ylnekm,nURmp,lurkp->uyUreR", lb, bra(u), u)
            rows, mid, cols = lt.shape[:3].numel(), lt.shape[3:].numel(), lb.shape[3:].numel()
            mt, mb = lt.reshape(rows, mid), lb.reshape(mid, cols)
            U, s, Vh = torch.linalg.svd(mt @ mb, full_matrices=False)
            s = s[:chi]
            s = s[s > 1e-12 * s[0]]
            scale = torch.zeros(min(chi, U.shape[1]), dtype=s.dtype)
            scale[:len(s)] = 1.0 / torch.sqrt(s)
            w = len(scale)
            shape = (lt.shape[3], lt.shape[4], lt.shape[5], w)
            P[i] = [(mb @ Vh[:w].mH * scale).reshape(shape).permute(1, 0, 2, 3),
                    (mt.T @ U[:, :w].conj() * scale).reshape(shape).permute(1, 0, 2, 3)]
            P[i] = [torch.nn.functional.pad(x, (0, chi - w)) for x in P[i]]
        new = []
        for i in line:
            down = go(i, 3)
            up = P[go(i, 1)]
            c1 = contract("xa,aekm,xkmw->we", c(0, i), e(0, i), up[0])
            c4 = contract("exkm,xa,akmw->ew", e(2, down), c(3, down), P[down][1])
            t = site(i)
            x = contract("yxln,xkmw,nmRBp,lkrbp->yrbRBw", e(3, i), up[1], bra(t), t)
            x = contract("yrbRBw,ybBv->vwrR", x, P[i][0])
            new.append((go(i, 2), go(down, 2), [y / y.abs().max() for y in (c1, c4, x)]))
        for j, k, (c1, c4, x) in new:
            C[r][j], C[(3 + r) % 4][k], E[(3 + r) % 4][j] = c1, c4, x

    column = lambda x: [x + y * LX for y in range(LY)]  # noqa: E731
    row = lambda y: [x + y * LX for x in range(LX)]  # noqa: E731
    for _ in range(case["sweeps"]):
        for x in range(LX):
            move(0, column(x))
        # the turned moves' lines are given by their "top left" site
        for x in range(LX):
            move(2, column((1 - x) % LX))
        for y in range(LY):
            move(1, row((1 - y) % LY))
        for y in range(LY):
            move(3, row(y))

    def half(r, i):
        """The site i with the left half of its environment (turned r times):
        legs (upper edge, lower edge, r, r*, p, p*)."""
        c, e = (lambda k: C[(k + r) % 4][i]), (lambda k: E[(k + r) % 4][i])
        t = tn[i].permute(*[(w + r) % 4 for w in range(4)], *range(4, tn[i].dim())).flatten(4)
        x = contract("xa,aekm,yxln,zy,fzgh->ekmlnfgh", c(0), e(0), e(3), c(3), e(2))
        if case["density"]:  # the pair of spin legs is the site's own
            return contract("ekmlnfgh,lkrgp->efrp", x, t).unflatten(3, (2, 2))[:, :, :, None]
        return contract("ekmlnfgh,nmRhq,lkrgp->efrRpq", x, t.conj(), t)

    rdm, sz = [], []
    for i, dx, dy in bonds(case):
        if dx:
            rdm.append(torch.einsum("efrRpq,ferRst->psqt", half(0, i), half(2, nn[i][2])))
        else:
            rdm.append(torch.einsum("efrRpq,ferRst->sptq", half(1, nn[i][1]), half(3, i)))
    for i in range(N):
        a = contract("efrRpq,pq->efrR", half(0, i), torch.from_numpy(SZ).to(tensors[0].dtype))
        sz.append(contract("efrR,eg,ghrR,hf->", a, C[1][i], E[1][i], C[2][i]))
    return {"sz": torch.stack(sz).numpy(), "rdm": torch.stack(rdm).numpy()}
