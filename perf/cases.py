"""The work that a user of this framework has it do, case by case, through its public entry points.

Kinds of case:

- ``step``   one eager ``System.iterate_step`` (latency of a small mesh)
- ``run``    ``System.run``: steps replayed from a captured graph, then the state is read back (a run's output cadence)
- ``stages`` one step through the reference's own call sequence, one member function after another
- ``host``   a host code that rebuilds its mesh: ``set_mesh``, ``set_positions``, ``step_host`` on pinned host state
- ``train``, ``grad``, ``eval``  the network of the learned face flux on host arrays
- ``flux``   a batch of face states through the exact Riemann solver on host arrays

Meshes: ``tile``^3 jittered generators in Peano-Hilbert order, the Voronoi mesh of which is repeated rx x ry x rz times
(the repeated mesh is the periodic Voronoi mesh of the repeated generators), or the generators of the Keplerian disk.
Generators that move with the flow on a mesh that is not rebuilt degenerate after thousands of steps (in the reference as
well), so such runs start from one saved state each time; the others go on.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import fvmhd3d_b200 as F
from fvmhd3d_b200 import learned

DISK = dict(gamma=1.0, courant=0.4, dtmax=1.0 / 16, eos=1, iso_GM=1.0, iso_cfac=0.05, static_mesh=True)
NPARAM = learned.MLP_NPARAM
NOISE = 1e-4  # of the initial states: no field is flat to round-off, where the limiter's value would be round-off's
LINKS = 7.96  # faces per cell of the jittered lattices (links are twice that)


def mesh_case(kind, name, problem, tile, reps, precision, steps, **more):
    return dict(kind=kind, name=name, problem=problem, tile=tile, rx=reps[0], ry=reps[1], rz=reps[2],
                precision=precision, steps=steps, **{**dict(shared=True, static=True, learned=False, fused=0), **more})


def listed():
    return [
        # the smallest call: a unit-test sized mesh stepped by hand, bound by launches and the host
        mesh_case("step", "step_6cubed", "blast", 6, (1, 1, 1), "fp64", 1),
        # configuration 1 of the benchmark: 32^3 Alfven wave, moving generators, ten global steps
        mesh_case("run", "alfven_32cubed", "alfven", 32, (1, 1, 1), "fp64", 10, static=False),
        # configuration 2: the 64^3 blast in the FP32 bulk form
        mesh_case("run", "blast_64cubed_fp32", "blast", 32, (2, 2, 2), "fp32", 30),
        # the headline: 2.1 million cells, plain FP64, global timestep
        mesh_case("run", "blast_128cubed", "blast", 32, (4, 4, 4), "fp64", 12),
        # a drop-in that keeps the reference's call sequence, on a ragged box of odd side
        mesh_case("stages", "stages_vortex_23", "orszag_tang", 23, (3, 1, 2), "fp64", 1),
        # individual timesteps (configuration 3, smaller): small rung steps beside full ones
        dict(kind="run", name="disk_rungs_fp32", problem="disk", cells=100000, precision="fp32", steps=32, shared=False,
             static=True, learned=False, fused=16384),
        # individual timesteps of a blast in FP64, with the stage kernels (the defaults)
        mesh_case("run", "blast_rungs_29", "blast", 29, (1, 1, 1), "fp64", 32, shared=False),
        # a host code that rebuilds its mesh every step and keeps the state in its own (pinned) arrays
        mesh_case("host", "remesh_40cubed", "alfven", 20, (2, 2, 2), "fp64", 1, static=False),
        # the learned face flux (the shipped network) with the FP32 bulk form
        mesh_case("run", "learned_48cubed", "blast", 24, (2, 2, 2), "fp32", 10, learned=True),
        # training of that network: the minibatch of the shipped pipeline
        dict(kind="train", name="train_8192", rows=120000, batch=8192, steps=20),
        # the network alone on a harvested set's worth of rows
        dict(kind="eval", name="eval_200k", rows=200000),
        # a host integrator's batch of boundary or sub-grid faces
        dict(kind="flux", name="flux_3000", rows=3000),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "rungs", "step", "stages", "host", "learned", "train", "grad", "eval", "flux"])
    if kind == "train":
        return dict(kind="train", rows=int(_log(rng, 20000, 300000)), batch=int(_log(rng, 256, 16384)), steps=rng.randint(5, 25))
    if kind in ("grad", "eval"):
        return dict(kind=kind, rows=int(_log(rng, 100, 20000 if kind == "grad" else 1000000)))
    if kind == "flux":
        return dict(kind="flux", rows=int(_log(rng, 1, 200000)))
    if kind == "rungs" and rng.random() < 0.5:
        return dict(kind="run", problem="disk", cells=int(_log(rng, 3000, 120000)), precision=rng.choice(["fp64", "fp32"]),
                    steps=rng.randint(8, 40), shared=False, static=True, learned=False, fused=rng.choice([0, 16384]))
    most = {"run": 2000000, "rungs": 60000, "step": 30000, "stages": 300000, "host": 100000, "learned": 200000}[kind]
    cells = _log(rng, 216, most)
    # a side of at most 32 generators, repeated along each axis by about the same number
    rep = max(1, math.ceil((cells / 32768.0) ** (1.0 / 3.0)))
    reps = [max(1, rep + rng.choice([-1, 0, 0, 1])) if rep > 1 else 1 for _ in range(3)]
    tile = min(32, max(6, round((cells / (reps[0] * reps[1] * reps[2])) ** (1.0 / 3.0))))
    steps = {"run": max(1, min(30, int(2.5e7 / (tile ** 3 * reps[0] * reps[1] * reps[2])))), "rungs": rng.randint(8, 40),
             "learned": rng.randint(2, 10)}.get(kind, 1)
    c = mesh_case({"rungs": "run", "learned": "run"}.get(kind, kind), "", rng.choice(["alfven", "blast", "orszag_tang"]), tile, reps,
                  "fp32" if kind == "learned" else rng.choice(["fp64", "fp64", "fp32"]), steps, shared=kind != "rungs",
                  learned=kind == "learned", fused=rng.choice([0, 16384]) if kind == "rungs" else 0)
    del c["name"]
    return c


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


# ---- meshes and initial states ----------------------------------------------------------------------------------

def tiled_mesh(tile, reps, seed):
    """The Voronoi mesh of tile^3 jittered generators (Peano-Hilbert order) repeated reps times, the longest side of the
    box 1; cells tile after tile, faces by their lower cell, a cell's faces by number."""
    pos = F.jittered_lattice(tile, 0.1, seed=seed)
    pos = np.ascontiguousarray(pos[F.sort_local_data(pos, 1.0)])
    m = F.build_periodic(pos, 1.0)
    if tuple(reps) == (1, 1, 1):
        return m
    dev, nt, nf = _dev(), m.ncell, m.nface
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    r = torch.tensor(reps, device=dev)
    s = 1.0 / max(reps)
    p, a, b = t(m.pos), t(m.s1).long(), t(m.s2).long()
    shift = -torch.round(p[b] - p[a]).long()  # tiles from a's to b's
    grid = torch.cartesian_prod(*[torch.arange(k, device=dev) for k in reps[::-1]]).reshape(-1, 3).flip(1)  # x fastest
    K = grid.shape[0]
    other = torch.remainder(grid[:, None] + shift[None], r)  # K x nf x 3
    number = (other[..., 2] * r[1] + other[..., 1]) * r[0] + other[..., 0]
    A = (torch.arange(K, device=dev)[:, None] * nt + a[None]).reshape(-1)
    B = (number * nt + b[None]).reshape(-1)
    n = t(m.n).repeat(K, 1) * s * s
    c = (t(m.centroid)[None] + grid[:, None]).reshape(-1, 3)
    back = (other - (grid[:, None] + shift[None])).reshape(-1, 3).double()  # from a's frame to b's
    swap = A > B
    n[swap] = -n[swap]
    c[swap] += back[swap]
    s1, s2 = torch.where(swap, B, A), torch.where(swap, A, B)
    order = torch.sort(s1, stable=True)[1]
    s1, s2, n, c = s1[order], s2[order], n[order].contiguous(), (c[order] * s).contiguous()
    total, nft = K * nt, K * nf
    ids = torch.arange(nft, device=dev)
    key = torch.cat([s1 * nft + ids, s2 * nft + ids]).sort()[0]
    count = torch.bincount(torch.cat([s1, s2]), minlength=total)
    off = torch.zeros(total + 1, dtype=torch.long, device=dev)
    off[1:] = count.cumsum(0)
    h = lambda x, ty: x.cpu().numpy().astype(ty, copy=False)  # noqa: E731
    place = lambda x: ((x[None] + grid[:, None]) * s).reshape(-1, 3)  # noqa: E731
    return F.Mesh(np.asarray(reps, np.float64) * s, h(place(p), np.float64), h(s1, np.int32), h(s2, np.int32),
                  h(n, np.float64), h(c, np.float64), h(t(m.volume).repeat(K) * s ** 3, np.float64),
                  h(place(t(m.cell_centroid)), np.float64), h(off, np.int64), h(key % nft, np.int32))


def inputs(case, seed):
    """(mesh, W, bnd, arguments of System) of a case on a mesh."""
    if case["problem"] == "disk":
        pos, box = F.problems.disk_generators(case["cells"], seed=seed + 3)
        pos = pos[F.sort_local_data(pos, box)]
        m = F.build_periodic(pos, box)
        W, bnd = F.problems.disk(pos, box, seed=seed + 4)
        return m, F.problems.perturbed(W, NOISE, seed), bnd, dict(DISK, box=tuple(box))
    m = tiled_mesh(case["tile"], (case["rx"], case["ry"], case["rz"]), seed + 1)
    W = getattr(F.problems, case["problem"])(m.pos / m.box)
    return m, F.problems.perturbed(W, NOISE, seed), None, dict(box=tuple(m.box), static_mesh=case["static"])


STATE = (("vel", 3), ("tlast", 1), ("tend", 1), ("rung", 1), ("U", 10), ("dU", 14), ("wrec", 50))


def pinned(shape, dtype=torch.float64):
    return torch.zeros(shape, dtype=dtype, pin_memory=torch.cuda.is_available())


class State:
    pass


def prepare(case, seed):
    st = State()
    st.case, st.kind = case, case["kind"]
    if st.kind in ("train", "grad", "eval"):
        st.sys = F.System()
        X, T = rows(case, seed)
        st.X, st.T = X, T
        st.sys.mlp_set_weights(weights(case, seed))
        return st
    if st.kind == "flux":
        st.sys = F.System()
        st.args = faces(case, seed)
        return st
    m, W, bnd, args = inputs(case, seed)
    st.single = case["precision"] == "fp32"
    st.sys = F.System(precision=F.FVM_PREC_FP32 if st.single else F.FVM_PREC_FP64, **args)
    st.sys.set_mesh(m)
    st.sys.init_problem(W, bnd=bnd)
    if case["fused"]:
        st.sys.set_fused(case["fused"])
    if case["learned"]:
        learned.apply(st.sys, learned.load_model())
        st.sys.set_flux_mode(1, **learned.GATE)
    st.out = {k: pinned((m.ncell, w) if w > 1 else m.ncell, torch.int32 if k == "rung" else torch.float64) for k, w in STATE}
    if st.single:  # a single-precision run's analysis keeps the bulk data on the GPU in single precision
        st.bulk = {k: (torch.empty(v.shape, dtype=torch.float64, device=_dev()), torch.empty(v.shape, dtype=torch.float32, device=_dev()))
                   for k, v in st.out.items() if k in ("vel", "U", "dU", "wrec")}
    # where a step's work depends on the state (rungs, gated faces, moving generators), each pass is a run from one saved
    # state
    st.start = None
    if not (case["shared"] and case["static"]) or case["learned"]:
        read_state(st)
        st.start = {k: v.clone().pin_memory().numpy() for k, v in st.out.items()}
    if st.kind == "host":  # the mesh and the state in the host code's own pinned arrays
        st.host = {k: v.numpy() for k, v in st.out.items()}
        read_state(st)
        keep = lambda a, ty: torch.from_numpy(np.ascontiguousarray(a, ty)).pin_memory().numpy()  # noqa: E731
        f, i = np.float64, np.int32
        st.mesh = F.Mesh(m.box, keep(m.pos, f), keep(m.s1, i), keep(m.s2, i), keep(m.n, f), keep(m.centroid, f), keep(m.volume, f),
                         keep(m.cell_centroid, f), keep(m.cell_face_off, np.int64), keep(m.cell_face_ids, i))
    return st


def read_state(st):
    """The whole state into the program's own pinned arrays (fvm_get_state)."""
    s = st.sys
    p = [st.out[k].data_ptr() for k, _ in STATE]
    s._check(s.L.fvm_get_state(s.h, None, *p), "fvm_get_state")


def run(st):
    s, c = st.sys, st.case
    if st.kind == "train":
        loss = s.mlp_train(st.X, st.T, learned.OUTPUT_WEIGHTS, batch=c["batch"], steps=c["steps"], lr=1e-3, seed=5)
        return {"loss": loss, "params": s.mlp_get_weights()}
    if st.kind == "grad":
        loss, g = s.mlp_grad(st.X, st.T, learned.OUTPUT_WEIGHTS)
        return {"loss": np.float32(loss), "grad": g}
    if st.kind == "eval":
        return {"Y": s.mlp_eval(st.X)}
    if st.kind == "flux":
        psi, Bn, flux = s.compute_flux(*st.args)
        return {"psi": psi, "Bn": Bn, "flux": flux}
    faces_done = 0
    if st.kind == "run":
        if st.start:  # restart from the saved state
            s.set_state(**st.start, tsys_ticks=0)
        cells, faces_done = s.run(c["steps"], shared=c["shared"])
        read_state(st)
    elif st.kind == "step":
        cells = s.iterate_step(shared=c["shared"])
        read_state(st)
    elif st.kind == "stages":
        cells = s.begin_step()
        s.fluid_update(True, shared=c["shared"])
        s.collect_results()
        s.fluid_update(False)
        s.end_step(c["shared"])
        read_state(st)
    else:
        s.set_mesh(st.mesh)
        s.set_positions(st.mesh.pos)
        cells = s.step_host(st.host, shared=c["shared"])
    out = dict(st.out, cells=cells, faces=faces_done)
    if st.single:
        out.update((k, single.copy_(double.copy_(st.out[k], non_blocking=True))) for k, (double, single) in st.bulk.items())
    return out


def work(case):
    k = case["kind"]
    per_row = 2 * (16 * 128 + 2 * 128 * 128 + 128 * 8)
    if k == "eval":
        return {"bytes": case["rows"] * 24 * 4, "flops": case["rows"] * per_row}
    if k == "grad":
        return {"bytes": case["rows"] * 24 * 4 + 8 * NPARAM, "flops": 3 * case["rows"] * per_row}
    if k == "train":
        return {"bytes": case["steps"] * (case["batch"] * 24 * 4 + 24 * NPARAM), "flops": 3 * case["steps"] * case["batch"] * per_row}
    if k == "flux":
        return {"bytes": case["rows"] * (38 * 8 + 4), "flops": case["rows"] * 650}
    n = case["cells"] if case["problem"] == "disk" else case["tile"] ** 3 * case["rx"] * case["ry"] * case["rz"]
    w = 4 if case["precision"] == "fp32" else 8
    state = 31 * 8 + 4 + 50 * 8  # what a read of the whole state gives, per cell
    # a step reads each face's geometry and cells, and reads and writes each cell's state and reconstruction once
    step = n * (LINKS * 56 + 2 * (31 * 8 + 4 + 50 * w) + 80)
    share = 1.0 if case["shared"] else 0.3  # of the cells are active in a mean step of the individual timesteps
    flops = n * LINKS * 2500 * case["steps"] * share
    if case["learned"]:
        flops += n * LINKS * 2 * per_row * case["steps"]
    mesh = n * (LINKS * (8 + 48 + 8) + 8 + 24 + 8 + 24) if k == "host" else 0
    return {"bytes": step * case["steps"] * share + n * state * (3 if k == "host" else 1) + mesh, "flops": flops}


# ---- the network's and the solver's inputs -----------------------------------------------------------------------

def weights(case, seed):
    return learned.load_model()["params"] if case["kind"] == "eval" else learned.init_params(seed + 1)


def rows(case, seed):
    """Standardised features and, for training, targets a smooth function of them."""
    rng = np.random.default_rng(seed + 10)
    X = rng.standard_normal((case["rows"], 16), dtype=np.float32)
    if case["kind"] == "eval":
        return X, None
    M = rng.standard_normal((16, 8)).astype(np.float32) / 4
    return X, np.tanh(X @ M) + 0.3 * np.sin(X[:, :8])


def faces(case, seed):
    """Face states of a magnetised gas: (wij, Wi, Wj, jbnd, normal), a few faces at a boundary."""
    rng = np.random.default_rng(seed + 20)
    n = case["rows"]
    Wi = np.empty((n, 10))
    Wi[:, 0] = np.exp(rng.normal(0, 0.5, n))
    Wi[:, 1:4] = rng.normal(0, 0.7, (n, 3))
    Wi[:, 4] = np.exp(rng.normal(0, 0.7, n))
    Wi[:, 5:8] = rng.normal(0, 0.5, (n, 3))
    Wi[:, 8] = rng.normal(0, 0.05, n)
    Wi[:, 9] = np.exp(rng.normal(0, 0.3, n))
    Wj = Wi * np.exp(rng.normal(0, 0.2, (n, 10))) + 0.05 * np.array([0, 1, 1, 1, 0, 1, 1, 1, 0.2, 0]) * rng.normal(0, 1, (n, 10))
    normal = rng.normal(0, 1, (n, 3))
    normal /= np.linalg.norm(normal, axis=1)[:, None]
    wij = 0.5 * (Wi[:, 1:4] + Wj[:, 1:4]) + rng.normal(0, 0.1, (n, 3))
    jbnd = np.where(rng.random(n) < 0.02, rng.integers(1, 4, n), 0).astype(np.int32)
    return wij, Wi, Wj, jbnd, normal


# ---- what the outputs are in 64 bits, in plain torch -------------------------------------------------------------

GAMMA, COURANT, DTMAX, HUGE = 5.0 / 3.0, 0.4, 1.0 / 64, float(np.float32(3.40282347e+38))
D, VX, VY, VZ, E, BX, BY, BZ, PSI, ENTR = range(10)


def _prim(U, V):
    W = torch.empty_like(U)
    W[:, 0] = U[:, 0] / V
    for a in (1, 2, 3, 8, 9):
        W[:, a] = U[:, a] / U[:, 0]
    for a in (5, 6, 7):
        W[:, a] = U[:, a] / V
    W[:, E] = U[:, E] / V - 0.5 * (W[:, 5:8] ** 2).sum(1) - 0.5 * (W[:, 1:4] ** 2).sum(1) * W[:, 0]
    return W


def _cons(W, V):
    M = W[:, 0] * V
    U = W * M[:, None]
    U[:, 0] = M
    U[:, 5:8] = W[:, 5:8] * V[:, None]
    U[:, E] = W[:, E] * V + 0.5 * (W[:, 5:8] ** 2).sum(1) * V + 0.5 * (W[:, 1:4] ** 2).sum(1) * M
    return U


def _flux(wij, Wi, Wj, jbnd, nrm):
    """Rotated-frame HLLD flux at a moving face: (psi, Bn, flux of the ten conserved variables)."""
    ex, ey, ez = nrm.unbind(1)
    ds = torch.sqrt(ex * ex + ey * ey)
    polar = ds == 0
    ids = torch.where(polar, 0.0, 1.0 / torch.where(polar, 1.0, ds))
    cp, sp = torch.where(polar, 1.0, ex * ids), torch.where(polar, 0.0, ey * ids)
    A = ((cp * ds, ds * sp, ez), (-sp, cp, torch.zeros_like(sp)), (-ez * cp, -ez * sp, ds))
    rot = lambda v: [r[0] * v[:, 0] + r[1] * v[:, 1] + r[2] * v[:, 2] for r in A]  # noqa: E731
    w = rot(wij)[0]
    uL, vL, wL = rot(Wi[:, 1:4])
    uR, vR, wR = rot(Wj[:, 1:4])
    bxL, byL, bzL = rot(Wi[:, 5:8])
    bxR, byR, bzR = rot(Wj[:, 5:8])
    uR = torch.where(jbnd == 1, -uR, torch.where(jbnd == 3, torch.clamp(uR - 1.2 * w, min=0) + 1.2 * w, uR))
    dL, dR, eL, eR = Wi[:, 0], Wj[:, 0], Wi[:, E], Wj[:, E]
    pL, pR = (GAMMA - 1) * eL, (GAMMA - 1) * eR
    cL = torch.sqrt((GAMMA * pL + bxL ** 2 + byL ** 2 + bzL ** 2) / dL)
    cR = torch.sqrt((GAMMA * pR + bxR ** 2 + byR ** 2 + bzR ** 2) / dR)
    sL, sR = Wi[:, PSI], Wj[:, PSI]
    Bx = (bxL * cL + bxR * cR + (sL - sR)) / (cL + cR)
    psi = (sL * cR + sR * cL + cR * cL * (bxL - bxR)) / (cL + cR)
    sg, B2 = torch.sign(Bx), Bx * Bx
    q2L, q2R = B2 + byL ** 2 + bzL ** 2, B2 + byR ** 2 + bzR ** 2
    tL = eL + 0.5 * (dL * (uL ** 2 + vL ** 2 + wL ** 2) + q2L)
    tR = eR + 0.5 * (dR * (uR ** 2 + vR ** 2 + wR ** 2) + q2R)
    cf = torch.sqrt(torch.maximum((GAMMA * pL + q2L) / dL, (GAMMA * pR + q2R) / dR))
    SL, SR = torch.minimum(uL, uR) - cf, torch.maximum(uL, uR) + cf
    PL, PR = pL + 0.5 * q2L, pR + 0.5 * q2R
    i = 1.0 / ((SR - uR) * dR - (SL - uL) * dL)
    SM = i * ((SR - uR) * dR * uR - (SL - uL) * dL * uL - PR + PL)
    Ps = i * ((SR - uR) * dR * PL - (SL - uL) * dL * PR + dL * dR * (SR - uR) * (SL - uL) * (uR - uL))

    def star(S, d, u, v, z, by, bz, P, t):
        div = d * (S - u) * (S - SM) - B2
        idiv = torch.where(div != 0, 1.0 / torch.where(div != 0, div, 1.0), 0.0)
        vs, zs = v - Bx * by * (SM - u) * idiv, z - Bx * bz * (SM - u) * idiv
        f = (d * (S - u) ** 2 - B2) * idiv
        vb, vbs = u * Bx + v * by + z * bz, SM * Bx + vs * by * f + zs * bz * f
        return d * (S - u) / (S - SM), vs, zs, by * f, bz * f, vb, vbs, ((S - u) * t - P * u + Ps * SM + Bx * (vb - vbs)) / (S - SM)

    dLs, vLs, wLs, byLs, bzLs, vbL, vbLs, tLs = star(SL, dL, uL, vL, wL, byL, bzL, PL, tL)
    dRs, vRs, wRs, byRs, bzRs, vbR, vbRs, tRs = star(SR, dR, uR, vR, wR, byR, bzR, PR, tR)
    rL, rR = torch.sqrt(dLs), torch.sqrt(dRs)
    SLs, SRs = SM - (Bx / rL).abs(), SM + (Bx / rR).abs()
    q = 1.0 / (rL + rR)
    v2, w2 = q * (rL * vLs + rR * vRs + (byRs - byLs) * sg), q * (rL * wLs + rR * wRs + (bzRs - bzLs) * sg)
    y2, z2 = q * (rL * byRs + rR * byLs + rL * rR * (vRs - vLs) * sg), q * (rL * bzRs + rR * bzLs + rL * rR * (wRs - wLs) * sg)
    vb2 = SM * Bx + v2 * y2 + w2 * z2
    tL2, tR2 = tLs - rL * (vbLs - vb2) * sg, tRs + rR * (vbRs - vb2) * sg
    z = torch.zeros_like(w)
    left = w <= SM
    pick = lambda *p: torch.where(w <= SL, p[0], torch.where(w <= SLs, p[1], torch.where(left, p[2], torch.where(w <= SRs, p[3], torch.where(w <= SR, p[4], p[5])))))  # noqa: E731
    a = pick(z, z, SLs - w, SRs - w, z, z)
    b = pick(z, SL - w, SL - SLs, SR - SRs, SR - w, z)
    c = pick(-w, -SL, -SL, -SR, -SR, -w)
    sel = lambda x, y: torch.where(left, x, y)  # noqa: E731
    d, u, v, ww, by, bz, P, vb, t = (sel(x, y) for x, y in ((dL, dR), (uL, uR), (vL, vR), (wL, wR), (byL, byR), (bzL, bzR), (PL, PR), (vbL, vbR), (tL, tR)))
    ds_, vs, ws, bys, bzs, ts, t2 = (sel(x, y) for x, y in ((dLs, dRs), (vLs, vRs), (wLs, wRs), (byLs, byRs), (bzLs, bzRs), (tLs, tRs), (tL2, tR2)))
    Fd = d * u + (a + b) * ds_ + c * d
    Fx = d * u * u + P - B2 + (a + b) * ds_ * SM + c * d * u
    Fy = d * v * u - Bx * by + a * ds_ * v2 + b * ds_ * vs + c * d * v
    Fz = d * ww * u - Bx * bz + a * ds_ * w2 + b * ds_ * ws + c * d * ww
    Fe = t * u + P * u - Bx * vb + a * t2 + b * ts + c * t
    Gx, Gy, Gz = -w * Bx, by * u - Bx * v + a * y2 + b * bys + c * by, bz * u - Bx * ww + a * z2 + b * bzs + c * bz
    back = lambda k, x, y, zz: A[0][k] * x + A[1][k] * y + A[2][k] * zz  # noqa: E731
    up = Fd > 0
    return psi, Bx, torch.stack([Fd, back(0, Fx, Fy, Fz), back(1, Fx, Fy, Fz), back(2, Fx, Fy, Fz), Fe, back(0, Gx, Gy, Gz),
                                 back(1, Gx, Gy, Gz), back(2, Gx, Gy, Gz), Fd * torch.where(up, sL, sR),
                                 Fd * torch.where(up, Wi[:, ENTR], Wj[:, ENTR])], 1)


def _phi_min(dW, mn, mx):
    """The limiter of one extrapolated difference: Phi of the allowed over the extrapolated difference."""
    flat = dW.abs() <= 1e-16 * torch.maximum(mn.abs(), mx.abs())
    x = torch.where(dW < 0, mn, mx) / torch.where(flat, 1.0, dW)
    e = 0.2e-16
    return torch.where(flat, 1.0, (x * x + 2 * x + e) / (x * x + x + 2 + e))


def _exp2(x):
    return math.frexp(x)[1]


class _Gas:
    """Global steps of an ideal gas on a fixed mesh without boundaries."""

    def __init__(self, m, W, static):
        dev = _dev()
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
        self.static, self.n = static, m.ncell
        self.s1, self.s2, box = t(m.s1).long(), t(m.s2).long(), t(m.box)
        self.cell = torch.cat([self.s1, self.s2])
        nv = t(m.n)
        self.A = nv.norm(dim=1)
        self.nh = nv / self.A[:, None]
        self.V, self.pos, self.cc = t(m.volume), t(m.pos), t(m.cell_centroid)
        self.R = (self.V / (4 * math.pi / 3)) ** (1 / 3)
        wrap = lambda d: torch.where(d > 0.5 * box, d - box, torch.where(d < -0.5 * box, d + box, d))  # noqa: E731
        self.dr1 = t(m.centroid) - self.pos[self.s1]
        dr2 = wrap(t(m.centroid) - self.pos[self.s2])
        self.dsh = (self.dr1 * self.nh).sum(1)
        self.ext = torch.cat([self.dr1, self.dr1 - 2 * self.dsh[:, None] * self.nh])  # offsets of the extrapolated states
        self.d = torch.cat([wrap(self.dr1), dr2])
        sg = torch.where((self.d * torch.cat([self.nh, self.nh])).sum(1) < 0, -1.0, 1.0)[:, None]
        nd = torch.cat([self.nh, self.nh]) * sg
        sh = (self.d * nd).sum(1, keepdim=True)
        ia = torch.cat([self.A, self.A])[:, None] * 0.5 / sh
        self.wa, self.wb = nd * sh * ia, (self.d - nd * sh) * ia
        W = t(W)
        self.w, self.grad, self.t = W.clone(), torch.zeros(self.n, 3, 10, device=dev, dtype=torch.float64), torch.zeros_like(W)
        self.U = _cons(W, self.V)
        self.vel = self._pvel()
        cs, v = self._speeds(W), W[:, 1:4].norm(dim=1)
        self.rung = self._rung_of(float((self.R / (cs + v + 1 / HUGE)).min()) * COURANT, 0)
        self.ticks, self.time = 0, 0.0
        self.tend = self._dt(self.rung)

    def _rung_of(self, dt, least):
        return max(least, _exp2(DTMAX) - _exp2(dt))

    def _dt(self, rung):
        return DTMAX / 2.0 ** 31 * 2.0 ** (31 - rung)

    def _speeds(self, W):
        return torch.sqrt((GAMMA * (GAMMA - 1) * W[:, E] + (W[:, 5:8] ** 2).sum(1)) / W[:, 0])

    def _pvel(self):
        if self.static:
            return torch.zeros(self.n, 3, dtype=torch.float64, device=self.V.device)
        W = _prim(self.U, self.V)
        vabs = torch.sqrt(self._speeds(W) ** 2 + (W[:, 1:4] ** 2).sum(1))
        d3 = self.cc - self.pos
        d = d3.norm(dim=1)
        f1, f2 = float(np.float32(0.9)), float(np.float32(1.1))
        eR = 0.25 * self.R
        f = torch.where(d / eR < f1, 0.0, torch.where(d / eR < f2, (d - f1 * eR) / ((f2 - f1) * eR), 1.0))
        return W[:, 1:4] + torch.where(d > 0, f * vabs / torch.where(d > 0, d, 1.0), 0.0)[:, None] * d3

    def _sum(self, s1, s2):
        out = torch.zeros((self.n,) + s1.shape[1:], dtype=torch.float64, device=s1.device)
        return out.index_add_(0, self.s1, s1).index_add_(0, self.s2, s2)

    def _range(self, w):
        """Least and largest neighbour difference, zero among them."""
        d = w[self.s2] - w[self.s1]
        z = torch.zeros_like(w)
        mn = z.index_reduce(0, self.s1, d, "amin").index_reduce_(0, self.s2, -d, "amin")
        return mn, z.index_reduce(0, self.s1, d, "amax").index_reduce_(0, self.s2, -d, "amax")

    def _limit(self, off, grad, t, mn, mx):
        """The least limiter over a cell's faces of grad . off + t."""
        tau = torch.ones_like(mn)
        nf = self.s1.shape[0]
        for side, c in ((slice(0, nf), self.s1), (slice(nf, None), self.s2)):
            dW = (grad[c] * off[side][:, :, None]).sum(1) + t[c]
            tau.index_reduce_(0, c, _phi_min(dW, mn[c], mx[c]), "amin")
        return tau

    def _fluxes(self, Wi, Wj, scale):
        """What the cells of each face get: area and scale times flux, gradPsi and divB, summed per cell."""
        vi, vj = self.vel[self.s1], self.vel[self.s2]
        fij = self.dr1 - self.nh * self.dsh[:, None]
        x = -0.5 * ((vj - vi) * fij).sum(1) / self.dsh ** 2
        psi, Bn, f = _flux(0.5 * (vi + vj) + self.dr1 * x[:, None], Wi, Wj, torch.zeros_like(self.s1), self.nh)
        a = (self.A * scale)[:, None]
        v = torch.cat([-f * a, self.nh * psi[:, None] * a, Bn[:, None] * a], 1)
        return self._sum(v, -v)

    def _source(self, U, W, s, dt):
        """The Powell and Dedner terms: s times dt with the speeds of W."""
        divB, c2 = s[:, 13] * dt, GAMMA * (GAMMA - 1) * W[:, E] + (W[:, 5:8] ** 2).sum(1)
        return divB, c2, torch.sqrt(c2 / W[:, 0])

    def _update(self, U, W, s, dt, scale):
        U = U + s[:, :10] * scale
        divB, c2, ch = self._source(U, W, s, scale)
        U[:, 5:8] -= W[:, 1:4] * divB[:, None] + s[:, 10:13] * scale
        U[:, 8] = (U[:, 8] - c2 * divB) * torch.exp(-0.5 * ch / self.R * dt)
        return _prim(U, self.V)

    def step(self):
        nxt = (self.ticks // (1 << (31 - self.rung)) + 1) * (1 << (31 - self.rung))
        least = 31 - ((self.ticks ^ nxt).bit_length() - 1)
        now = DTMAX / 2.0 ** 31 * nxt
        dt = now - self.time
        mn, mx = self._range(self.w)
        tau = self._limit(self.ext, self.grad, self.t * (0.5 * dt), mn, mx)
        ex = lambda c, o: self.w[c] + tau[c] * ((self.grad[c] * o[:, :, None]).sum(1) + self.t[c] * (0.5 * dt))  # noqa: E731
        nf = self.s1.shape[0]
        s = self._fluxes(ex(self.s1, self.ext[:nf]), ex(self.s2, self.ext[nf:]), dt)
        W1 = self._update(self.U, self.w + tau * self.t * (0.5 * dt), s, dt, 1.0)
        cold = W1[:, E] <= 0
        rg = W1[:, 0] ** GAMMA
        W1[:, E], W1[:, ENTR] = (torch.where(cold, W1[:, ENTR] * rg / (GAMMA - 1), W1[:, E]),
                                 torch.where(cold, W1[:, ENTR], (GAMMA - 1) * W1[:, E] / rg))
        self.U = _cons(W1, self.V)
        self.vel = self._pvel()
        W = _prim(self.U, self.V)
        cs = self._speeds(W)
        x = cs + (W[:, 1:4] - self.vel).norm(dim=1) + 1 / HUGE
        for c, o in ((self.s1, self.s2), (self.s2, self.s1)):
            rel = cs[c] + (W[c, 1:4] - 0.5 * (self.vel[c] + self.vel[o])).norm(dim=1)
            x.index_reduce_(0, c, torch.maximum(rel, (self.vel[o] - self.vel[c]).norm(dim=1) + 1 / HUGE), "amax")
        rung = self._rung_of(float((self.R / x).min()) * COURANT, least)
        self.ticks, self.time = nxt, now
        s = self._fluxes(W[self.s1], W[self.s2], 1.0)
        while rung < 31 and bool((self.U[:, 0] + s[:, 0] * self._dt(rung) <= 0).any()):
            rung += 1
        ndt = self._dt(rung)
        Wp = self._update(self.U, W, s, ndt, ndt)
        Wp[:, E], Wp[:, ENTR] = (torch.where(Wp[:, E] <= 0, W[:, E], Wp[:, E]),
                                 torch.where(Wp[:, E] <= 0, Wp[:, ENTR], (GAMMA - 1) * Wp[:, E] / Wp[:, 0] ** GAMMA))
        t = (Wp - W) / ndt
        sm, df = W[self.s1] + W[self.s2], W[self.s2] - W[self.s1]
        g1 = self.wa[:nf, :, None] * sm[:, None] + self.wb[:nf, :, None] * df[:, None]
        g2 = self.wa[nf:, :, None] * sm[:, None] - self.wb[nf:, :, None] * df[:, None]
        grad = self._sum(g1, g2) / self.V[:, None, None]
        mn, mx = self._range(W)
        lim = self._limit(self.d, grad, torch.zeros_like(t), mn, mx)
        grad, t = grad * lim[:, None], t * lim
        sc = self._sum(self.d[:nf], self.d[nf:])
        dx = (grad[:, :, 0] * sc).sum(1)
        dw = torch.maximum(dx, dx + t[:, 0] * ndt)
        alpha = torch.where(dw > 0, torch.clamp(0.9 * W[:, 0] / torch.where(dw > 0, dw, 1.0), max=1.0), 1.0)
        grad[:, :, 0] *= alpha[:, None]
        t[:, 0] *= alpha
        self.w, self.grad, self.t, self.rung = W, grad, t, rung
        self.tend = now + self._dt(rung)


def _network(params, X, dev):
    shapes = ((128, 16), (128,), (128, 128), (128,), (128, 128), (128,), (8, 128), (8,))
    p = torch.from_numpy(np.asarray(params, np.float64)).to(dev).requires_grad_(True)
    parts, o = [], 0
    for s in shapes:
        parts.append(p[o:o + math.prod(s)].reshape(s))
        o += math.prod(s)
    h = X
    for k in range(4):
        h = h @ parts[2 * k].T + parts[2 * k + 1]
        h = torch.nn.functional.gelu(h, approximate="tanh") if k < 3 else h
    return p, h


def _mix64(x):
    x = x + np.uint64(0x9E3779B97F4A7C15)
    x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return x ^ (x >> np.uint64(31))


def _exact_network(case, seed):
    dev = _dev()
    X, T = rows(case, seed)
    params = weights(case, seed).astype(np.float64)
    t = lambda a: torch.from_numpy(np.asarray(a, np.float64)).to(dev)  # noqa: E731
    if case["kind"] == "eval":
        return {"Y": _network(params, t(X), dev)[1].detach()}
    wt, m, v, loss = t(learned.OUTPUT_WEIGHTS), 0.0, 0.0, []
    for it in range(case.get("steps", 1)):
        if case["kind"] == "train":
            r = np.arange(case["batch"], dtype=np.uint64)
            at = (_mix64(np.uint64(5) ^ np.uint64(it << 32) ^ r) % np.uint64(case["rows"])).astype(np.int64)
            x, y = t(X[at]), t(T[at])
        else:
            x, y = t(X), t(T)
        p, out = _network(params, x, dev)
        L = (wt * (out - y) ** 2).mean()
        L.backward()
        loss.append(float(L.detach()))
        g = p.grad.cpu().numpy()
        if case["kind"] == "grad":
            return {"loss": np.array(loss[0]), "grad": g}
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        params = params - 1e-3 * (m / (1 - 0.9 ** (it + 1))) / (np.sqrt(v / (1 - 0.999 ** (it + 1))) + 1e-8)
    return {"loss": np.array(loss), "params": params}


def exact(case, seed):
    if case["kind"] in ("train", "grad", "eval"):
        return _exact_network(case, seed)
    if case["kind"] == "flux":
        dev = _dev()
        psi, Bn, f = _flux(*[torch.from_numpy(a).to(dev) for a in faces(case, seed)])
        return {"psi": psi, "Bn": Bn, "flux": f}
    if not case["shared"] or case["learned"]:
        return None  # a sequential relaxation over sites; a network in the place of the solver
    m, W, _, args = inputs(case, seed)
    with torch.no_grad():
        g = _Gas(m, W, args["static_mesh"])
        for _ in range(case["steps"]):
            g.step()
    one = torch.ones(g.n, dtype=torch.float64)
    wrec = torch.cat([g.w, g.grad.reshape(g.n, 30), g.t], 1)
    return {"vel": g.vel, "tlast": one * g.time, "tend": one * g.tend, "rung": None, "U": g.U,
            "dU": None, "wrec": wrec, "cells": None, "faces": None}
