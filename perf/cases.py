"""The work a user has this library do, as cases that can be timed and checked.

A case is a dict of plain values:

  kind        "mdot"      U(, W) = Mdot(F(, T)) at positions set before, as in an
                          iterative solver that applies M many times per time step
              "step"      a deterministic time step: setPositions, Mdot
              "sqrt"      a Brownian displacement: setPositions, sqrtMdotW
              "brownian"  a fluctuating time step: setPositions, Mdot, sqrtMdotW
              "learned"   "sqrt" with the learned preconditioner, whose blocks are built
                          for the new positions as part of the pass
              "ensemble"  many independent systems of uneven size, open and wall mixed:
                          Mdot and sqrtMdotW of all of them
  wall        single bottom wall or open space
  torques     forces and torques with angular velocities, or forces alone
  precision   "float" or "double"
  n           particles of one batch (ensembles: the largest system)
  batches     equal batches (ensembles: systems)
  tolerance   of the Lanczos iteration

Units are the configurations' own: radius 1, viscosity 1 / (6 pi), so the translational
self mobility is 1.  Noise is given, not drawn inside, so a pass can be repeated.
"""
import math

import torch

from libmobility_gb300 import NBody
from libmobility_gb300.ensemble import Ensemble

VISCOSITY = 1.0 / (6.0 * math.pi)
# rotational and coupling prefactors over the translational one, 1 / (8 pi eta) = 3/4
ROT = 0.75

# Flops (FMA = 2) of one unordered pair, both particles' velocities from it: differences,
# squared distances, reciprocal square roots, the scalar coefficients of the blocks, and
# the blocks applied to either particle's force and torque.  The mobility is symmetric, so
# coefficients are needed once per pair.
PAIR_FLOPS = {(False, False): 53, (False, True): 153, (True, False): 130, (True, True): 270}


def _case(name, kind, n, wall=False, torques=False, precision="float", batches=1,
          tolerance=1e-5):
    c = {"kind": kind, "wall": wall, "torques": torques, "precision": precision, "n": n,
         "batches": batches, "tolerance": tolerance}
    return dict(name=name, **c) if name else c


def listed():
    return [
        # the smallest call in use: a few hundred particles, a time step at a time
        _case("open_small_step", "step", 200),
        # translational product of a 4096-particle suspension at volume fraction 0.05, in
        # both precisions
        _case("open_4096", "mdot", 4096),
        _case("open_4096_double", "mdot", 4096, precision="double"),
        # many small replicas in one handle (Nbatch, NperBatch), odd size
        _case("open_batches", "mdot", 333, batches=64),
        # rotating particles (bacteria, rods of beads) in open space, ragged size
        _case("open_torques", "mdot", 6001, torques=True),
        # the largest: a colloidal monolayer-like suspension above a wall, forces only
        _case("wall_forces_large", "mdot", 100003, wall=True),
        # the 16 384-particle single-wall product with torques
        _case("wall_torques_16384", "mdot", 16384, wall=True, torques=True),
        # the same physics in double precision, ragged size
        _case("wall_torques_double", "mdot", 3001, wall=True, torques=True,
              precision="double"),
        # Brownian displacements of the 4096-particle suspension to 1e-6
        _case("open_sqrt_4096", "sqrt", 4096, tolerance=1e-6),
        # a whole fluctuating step above a wall with torques, to 1e-5
        _case("wall_brownian_step", "brownian", 2048, wall=True, torques=True),
        # displacements of a dense suspension (volume fraction 0.2) with the learned
        # preconditioner
        _case("open_learned_16384", "learned", 16384, tolerance=1e-6),
        # parameter sweeps: 48 small systems of uneven size, half above a wall
        _case("ensemble_48", "ensemble", 2000, batches=48),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above (sizes over their logarithm, mostly odd ones)."""
    kind = rng.choice(["mdot"] * 5 + ["step", "sqrt", "brownian", "learned", "ensemble"])
    wall, torques = rng.random() < 0.5, rng.random() < 0.5
    if kind == "mdot":
        if rng.random() < 0.3:  # double
            return _case(None, kind, _log_int(rng, 100, 4000), wall, torques, "double")
        if rng.random() < 0.25:  # batches
            return _case(None, kind, _log_int(rng, 20, 1000), wall, torques,
                         batches=rng.randint(2, 100))
        return _case(None, kind, _log_int(rng, 100, 30000), wall, torques)
    if kind == "step":
        return _case(None, kind, _log_int(rng, 100, 5000), wall, torques)
    tol = 1e-5 if wall else rng.choice([1e-5, 1e-6])
    if kind in ("sqrt", "brownian"):
        precision = "double" if rng.random() < 0.2 else "float"
        return _case(None, kind, _log_int(rng, 100, 1000 if precision == "double" else 3000),
                     wall, torques, precision, tolerance=tol)
    if kind == "learned":
        return _case(None, kind, _log_int(rng, 1000, 16000), tolerance=rng.choice([1e-5, 1e-6]))
    return _case(None, kind, _log_int(rng, 300, 2000), batches=rng.randint(4, 48))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _dtype(case):
    return torch.float64 if case["precision"] == "double" else torch.float32


def _positions(gen, n, batches, wall, lattice):
    """(batches * n, 3) in 64 bits: uniform in a cube at volume fraction 0.05, uniform in
    a slab 1.5..20 radii above a wall with one particle per unit area, or (lattice) a
    jittered cubic lattice without overlaps at volume fraction 0.2, in random order."""
    dev = gen.device
    if lattice:
        m = math.ceil(n ** (1.0 / 3.0) - 1e-9)
        cell = (4.0 * math.pi / 3.0 / 0.2) ** (1.0 / 3.0)
        k = torch.randperm(m ** 3, generator=gen, device=dev)[:n]
        p = torch.stack([k // (m * m), (k // m) % m, k % m], 1).double()
        jitter = torch.rand((n, 3), generator=gen, device=dev, dtype=torch.float64) - 0.5
        return (p + 0.5) * cell + jitter * (cell - 2.0)
    u = torch.rand((batches * n, 3), generator=gen, device=dev, dtype=torch.float64)
    if wall:
        side = math.sqrt(n)
        return torch.stack([side * u[:, 0], side * u[:, 1], 1.5 + 18.5 * u[:, 2]], 1)
    return u * (4.0 * math.pi / 3.0 * n / 0.05) ** (1.0 / 3.0)


def _systems(case):
    """Sizes and geometries of an ensemble: sizes uniform between a tenth of the largest
    and the largest, every other system above a wall."""
    g = torch.Generator().manual_seed(1 + case["n"])
    k, big = case["batches"], case["n"]
    lo = max(16, big // 10)
    sizes = torch.randint(lo, big + 1, (k,), generator=g).tolist()
    sizes[0] = big
    return sizes, ["single_wall" if s % 2 else "open" for s in range(k)]


def _inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dt = _dtype(case)
    if case["kind"] == "ensemble":
        sizes, geometry = _systems(case)
        pos = torch.cat([_positions(gen, n, 1, g == "single_wall", False)
                         for n, g in zip(sizes, geometry)])
    else:
        pos = _positions(gen, case["n"], case["batches"], case["wall"],
                         case["kind"] == "learned")
    total = pos.shape[0]
    normal = [torch.randn((total, 3), generator=gen, device="cuda", dtype=torch.float64).to(dt)
              for _ in range(4)]
    pos = pos.to(dt).contiguous()
    F, T = normal[0], normal[1] if case["torques"] else None
    dW = torch.cat([normal[2].reshape(-1), normal[3].reshape(-1)]) if case["torques"] \
        else normal[2].reshape(-1)
    return pos, F, T, dW


def prepare(case, seed):
    pos, F, T, dW = _inputs(case, seed)
    if case["kind"] == "ensemble":
        sizes, geometry = _systems(case)
        h = Ensemble(precision=case["precision"])
        h.setSystems(sizes, geometry, [0.0] * len(sizes))
        h.initialize(VISCOSITY, 1.0, tolerance=case["tolerance"], seed=1)
    else:
        h = NBody("open", "open", "single_wall" if case["wall"] else "open",
                  precision=case["precision"])
        batches = {"Nbatch": case["batches"], "NperBatch": case["n"]} if case["batches"] > 1 else {}
        h.setParameters(wallHeight=0.0 if case["wall"] else None, **batches)
        h.initialize(VISCOSITY, 1.0, includeAngular=case["torques"],
                     tolerance=case["tolerance"], seed=1)
        if case["kind"] == "learned":
            h.setPreconditioner("mlp")
    if case["kind"] in ("mdot", "ensemble"):
        h.setPositions(pos)
    return {"kind": case["kind"], "h": h, "pos": pos, "F": F, "T": T, "dW": dW}


def run(state):
    h, kind = state["h"], state["kind"]
    if kind == "ensemble":
        return h.Mdot(state["F"]), h.sqrtMdotW(state["dW"])[0]
    out = []
    if kind != "mdot":
        h.setPositions(state["pos"])
    if kind in ("mdot", "step", "brownian"):
        out += h.Mdot(state["F"], state["T"])
    if kind in ("sqrt", "brownian", "learned"):
        out += h.sqrtMdotW_noise(state["dW"])[:2]
    return [x for x in out if x is not None]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _iterations(case):
    """Products of a Lanczos solve, typical of these inputs (they depend on the matrix)."""
    per_digit = 5 if case["kind"] == "learned" else 12
    return round(per_digit * -math.log10(case["tolerance"]))


def work(case):
    size = 8 if case["precision"] == "double" else 4
    blocks = 2 if case["torques"] else 1
    if case["kind"] == "ensemble":
        # sizes uniform between n / 10 and n, half of the systems open
        n1, n2 = 0.55 * case["n"], 0.37 * case["n"] ** 2
        flops = 0.5 * n2 * case["batches"] * (PAIR_FLOPS[False, False] +
                                              PAIR_FLOPS[True, False]) / 2
        vec = 3.0 * n1 * case["batches"] * size
    else:
        flops = 0.5 * case["n"] ** 2 * case["batches"] * PAIR_FLOPS[case["wall"], case["torques"]]
        vec = 3.0 * blocks * case["n"] * case["batches"] * size
    pos = vec / blocks
    products = {"mdot": 1, "step": 1}.get(case["kind"], 0)
    total = pos + products * 2 * vec
    if not products:
        its = _iterations(case)
        products = its + (case["kind"] in ("brownian", "ensemble"))
        # each basis vector written once and read once for the result
        total += 2 * its * vec + (products - its) * 2 * vec
    return {"bytes": total, "flops": products * flops}


# ---------------------------------------------------------------------------
# the same in 64 bits, entry by entry
# ---------------------------------------------------------------------------
def _outer(x, y):
    return x[..., :, None] * y[..., None, :]


def _cross_matrix(v):
    """C with C w = v x w."""
    x, y, z = v.unbind(-1)
    o = torch.zeros_like(x)
    return torch.stack([torch.stack([o, -z, y], -1), torch.stack([z, o, -x], -1),
                        torch.stack([-y, x, o], -1)], -2)


def _blocks(pi, pj, wall, torques):
    """3x3 blocks (n, m, 3, 3) between targets pi (n, 3) and sources pj (m, 3): U from F,
    and with torques also W from T and W from F.  Rotne-Prager-Yamakawa, and above a wall
    the corrections of Swan and Brady (2007)."""
    eye = torch.eye(3, dtype=pi.dtype, device=pi.device)
    z = eye[2]

    def iso(s):
        return s[..., None, None] * eye

    def by(s, t):
        return s[..., None, None] * t

    d = pi[:, None] - pj[None]
    r = d.norm(dim=-1)
    same = r == 0
    far = r >= 2
    i = 1 / torch.where(same, torch.ones_like(r), r)
    dd = _outer(d, d)
    tt = iso(torch.where(far, 0.75 * i + 0.5 * i ** 3, 1 - 9 / 32 * r)) + by(
        torch.where(far, (0.75 - 1.5 * i ** 2) * i ** 3, 3 / 32 * i), dd)
    rr = rt = None
    if torques:
        rr = iso(torch.where(far, -0.5 * i ** 3, 1 - 27 / 32 * r + 5 / 64 * r ** 3)) + by(
            torch.where(far, 1.5 * i ** 5, 9 / 32 * i - 3 / 64 * r), dd)
        # W = c (F x d)
        rt = by(torch.where(far, i ** 3, 0.5 - 3 / 16 * r), -_cross_matrix(d))
    if wall:
        hi, hj = pi[:, None, 2], pj[None, :, 2]
        R = torch.stack([d[..., 0], d[..., 1], hi + hj], -1)
        n1 = 1 / R.norm(dim=-1)
        n3, n5 = n1 ** 3, n1 ** 5
        e = R * n1[..., None]
        ez = e[..., 2]
        q = ez * ez
        h = hj / R[..., 2]
        k = h * (1 - h)
        A = -0.25 * (3 * (1 + 2 * k * q) * n1 + 2 * (1 - 3 * q) * n3 - 2 * (1 - 5 * q) * n5)
        B = -0.25 * (3 * (1 - 6 * k * q) * n1 - 6 * (1 - 5 * q) * n3 + 10 * (1 - 7 * q) * n5)
        C = 0.5 * ez * (3 * h * (1 - 6 * (1 - h) * q) * n1 - 6 * (1 - 5 * q) * n3
                        + 10 * (2 - 7 * q) * n5)
        D = 0.5 * ez * (3 * h * n1 - 10 * n5)
        E = -(3 * h * h * q * n1 + 3 * q * n3 + (2 - 15 * q) * n5)
        ee, zv = _outer(e, e), z.expand_as(e)
        image = iso(A) + by(B, ee) + by(C, _outer(e, zv)) + by(D, _outer(zv, e)) + by(
            E, _outer(zv, zv))
        ih = (1 / hi).expand_as(r)
        own = torch.diag_embed(torch.stack(
            [-(9 * ih - 2 * ih ** 3 + ih ** 5) / 16, -(9 * ih - 2 * ih ** 3 + ih ** 5) / 16,
             -(9 * ih - 4 * ih ** 3 + ih ** 5) / 8], -1))
        tt = tt + torch.where(same[..., None, None], own, image)
        if torques:
            p = torch.stack([-e[..., 1], e[..., 0], torch.zeros_like(ez)], -1)  # z x e
            image = iso(0.5 * (1 - 6 * q) * n3) + by(-1.5 * n3, ee) + by(
                3 * n3 * ez, _outer(zv, e)) + by(3 * n3, _outer(p, p))
            own = torch.diag_embed(torch.stack([-5 / 16 * ih ** 3, -5 / 16 * ih ** 3,
                                                -ih ** 3 / 8], -1))
            rr = rr + torch.where(same[..., None, None], own, image)
            n2, n4 = n1 ** 2, n1 ** 4
            f2 = 2 * (6 * h * q * n2 + (1 - 10 * q) * n4)
            f3 = -2 * ez * (3 * h * n2 - 5 * n4)
            f4 = -2 * ez * (h * n2 - n4)
            image = by(n2, _cross_matrix(e)) + by(f3, _outer(-p, e)) + by(
                f2, _outer(-p, zv)) + by(f4, _cross_matrix(zv))
            own = by(ih ** 4 / 8, _cross_matrix(zv))
            rt = rt + torch.where(same[..., None, None], own, image)
    if torques:
        rr, rt = ROT * rr, ROT * rt
    return tt, rr, rt


def _rows(pi, pj, wall, torques):
    """The rows of the mobility matrix of targets pi: blocks tt, and with torques also
    tr (U from T), rt and rr.  U from T of (i, j) is the transpose of W from F of (j, i)."""
    tt, rr, rt = _blocks(pi, pj, wall, torques)
    if not torques:
        return tt, None, None, None
    tr = _blocks(pj, pi, wall, True)[2].transpose(0, 1).transpose(-1, -2)
    return tt, tr, rt, rr


def _exact_mdot(pos, F, T, wall):
    U, W = torch.empty_like(F), torch.empty_like(F) if T is not None else None
    n = pos.shape[0]
    chunk = max(1, (1 << 21) // n)

    def dot(block, v):
        return torch.einsum("nmij,mj->ni", block, v)

    for b in range(0, n, chunk):
        s = slice(b, min(n, b + chunk))
        tt, tr, rt, rr = _rows(pos[s], pos, wall, T is not None)
        U[s] = dot(tt, F)
        if T is not None:
            U[s] += dot(tr, T)
            W[s] = dot(rt, F) + dot(rr, T)
    return U, W


def _dense(pos, wall, torques):
    n = pos.shape[0]
    M = torch.empty((3 * n * (2 if torques else 1),) * 2, dtype=pos.dtype, device=pos.device)
    chunk = max(1, (1 << 21) // n)

    def flat(block):
        return block.permute(0, 2, 1, 3).reshape(3 * block.shape[0], 3 * n)

    for b in range(0, n, chunk):
        e = min(n, b + chunk)
        tt, tr, rt, rr = _rows(pos[b:e], pos, wall, torques)
        M[3 * b:3 * e, :3 * n] = flat(tt)
        if torques:
            M[3 * b:3 * e, 3 * n:] = flat(tr)
            M[3 * (n + b):3 * (n + e), :3 * n] = flat(rt)
            M[3 * (n + b):3 * (n + e), 3 * n:] = flat(rr)
    return M


def _exact_sqrt(pos, dW, wall, torques):
    """M^{1/2} dW by a Lanczos iteration in 64 bits with full reorthogonalisation, far past
    any tolerance asked for."""
    M = _dense(pos, wall, torques)
    size = M.shape[0]
    limit = min(size, 240)
    V = torch.zeros((limit, size), dtype=M.dtype, device=M.device)
    norm = dW.norm()
    V[0] = dW / norm
    alpha, beta, last = [], [], None
    for k in range(limit):
        w = M @ V[k]
        alpha.append(float(w @ V[k]))
        for _ in range(2):
            w = w - V[:k + 1].T @ (V[:k + 1] @ w)
        beta.append(float(w.norm()))
        end = k + 1 == limit or beta[-1] < 1e-12 * alpha[0]
        if end or k % 20 == 19:
            t = torch.diag(torch.tensor(alpha, dtype=torch.float64))
            if k:
                off = torch.tensor(beta[:-1], dtype=torch.float64)
                t = t + torch.diag(off, 1) + torch.diag(off, -1)
            lam, P = torch.linalg.eigh(t)
            c = (P * lam.clamp(min=0).sqrt()) @ P[0]
            y = norm * (V[:k + 1].T @ c.to(M.device))
            if end or (last is not None and float((y - last).norm() / y.norm()) < 1e-12):
                return y
            last = y
        V[k + 1] = w / beta[-1]
    return y


def exact(case, seed):
    if case["kind"] == "learned":
        # P^{-1} (P M P^T)^{1/2} dW depends on the network's P: no value of its own
        return None
    pos, F, T, dW = (x.double() if x is not None else None for x in _inputs(case, seed))
    if case["kind"] == "ensemble":
        U, y, b = torch.empty_like(F), torch.empty_like(dW), 0
        for n, g in zip(*_systems(case)):
            p = pos[b:b + n]
            U[b:b + n] = _exact_mdot(p, F[b:b + n], None, g != "open")[0]
            y[3 * b:3 * (b + n)] = _exact_sqrt(p, dW[3 * b:3 * (b + n)], g != "open", False)
            b += n
        return U, y
    out = []
    n, wall, torques = case["n"], case["wall"], case["torques"]
    if case["kind"] in ("mdot", "step", "brownian"):
        parts = [_exact_mdot(pos[b * n:(b + 1) * n], F[b * n:(b + 1) * n],
                             T[b * n:(b + 1) * n] if torques else None, wall)
                 for b in range(case["batches"])]
        out += [torch.cat([p[k] for p in parts]) for k in range(2 if torques else 1)]
    if case["kind"] in ("sqrt", "brownian"):
        y = _exact_sqrt(pos, dW, wall, torques)
        out += [y[:3 * n].reshape(n, 3), y[3 * n:].reshape(n, 3)] if torques \
            else [y.reshape(n, 3)]
    return out
