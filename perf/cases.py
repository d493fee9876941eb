"""Performance cases of the evaluator: what a program that uses it does, call by call.

Single structures on host buffers (a relaxation, a Monte Carlo step, a phonon displacement),
single structures that stay on the GPU (molecular dynamics), batches of structures of uneven
size (screening, labelling, parallel rare-event sampling), resident structures served step by
step, descriptor vectors, a LAMMPS pair style's force call, NEP potentials, and the parameter
gradients of force training.  Every pass is a call of the package's Python class or of its C
ABI.  The library computes its descriptors, networks and gradients in 32 bits and delivers
them in double buffers; the programs here keep the results as 32-bit numbers, the type they
were computed in.

Structures are made from a seed: a simple-cubic grid with Gaussian displacements at the
densities of the repository's workloads, species at random, atoms in random memory order, a
few of them just outside the box as in a running simulation.  ``exact`` is the same potential
in 64 bits, written with torch alone.
"""
import ctypes
import itertools
import json
import math
from functools import lru_cache

import numpy as np
import torch

from jse_gb300 import nnap as J
from jse_gb300.nep import NEP
from jse_gb300.serve import NNAPServer
from jse_gb300.workloads import Structure

# Potentials by name.  "copper": radial Chebyshev descriptors, two hidden layers of 32;
# "liquid": the ternary alloy potential (nmax 8, lmax 6, cutoff 6); "glass": the binary one
# (nmax 8, lmax 4, cutoff 5.5); "plain": the model format's defaults (nmax 5, lmax 6, cutoff
# 6) for a binary; "fused": trainable radial weights, as in training; "nep": a nep4 file with
# default hyperparameters (cutoffs 8 / 4).  density (1/A^3) is that of the systems they are for.
POTENTIALS = {
    "copper": dict(kind="radial", fractions=[1.0], nmax=10, lmax=-1, rcut=6.0, hidden=[32, 32], density=0.085),
    "liquid": dict(kind="spherical", fractions=[0.46, 0.46, 0.08], nmax=8, lmax=6, rcut=6.0, hidden=[64, 64],
                   density=0.060),
    "glass": dict(kind="spherical", fractions=[0.64, 0.36], nmax=8, lmax=4, rcut=5.5, hidden=[64, 64], density=0.058),
    "plain": dict(kind="spherical", fractions=[0.5, 0.5], nmax=5, lmax=6, rcut=6.0, hidden=[32, 32], density=0.060),
    "fused": dict(kind="spherical", fractions=[0.5, 0.5], nmax=4, lmax=4, rcut=6.0, hidden=[32, 32], density=0.060,
                  fuse=2),
    "nep": dict(kind="nep", fractions=[0.5, 0.5], nmax=4, lmax=4, rcut=8.0, hidden=[30], density=0.060),
}
SKIN = 0.5  # of resident rows and of a LAMMPS neighbour list


def listed():
    """The calls that stand for everyday use, smallest to largest."""
    return [
        # one step of a relaxation or rare-event search in a small skewed cell: launches and latency
        dict(name="cell33_mixed", call="host", potential="liquid", precision="mixed", atoms=33, box="prism", virials=True),
        # the plain drop-in call (32-bit network) on an ordinary supercell, energy, forces and stress
        dict(name="cell500_fp32", call="host", potential="liquid", precision="fp32", atoms=500, box="ortho", virials=False),
        # a fitted model in the format's default shape, an odd mid-size box
        dict(name="plain4099_fp32", call="host", potential="plain", precision="fp32", atoms=4099, box="lmp", virials=True),
        # radial descriptors alone, a 4000-atom metal kept on the GPU
        dict(name="copper4000_fp32", call="device", potential="copper", precision="fp32", atoms=4000, box="ortho",
             virials=False),
        # molecular dynamics of a liquid on the GPU
        dict(name="liquid32000_mixed", call="device", potential="liquid", precision="mixed", atoms=32000, box="ortho",
             virials=False),
        # large-scale molecular dynamics of a glass, skewed box, atomic stresses
        dict(name="glass1048573_mixed", call="device", potential="glass", precision="mixed", atoms=1048573, box="lmp",
             virials=True),
        # screening: a thousand structures of 32 to 2048 atoms on the GPU in one call
        dict(name="batch1024_mixed", call="batch_device", potential="liquid", precision="mixed", structures=1024,
             smallest=32, largest=2048),
        # labelling from a host program: dozens of structures through the C ABI's host buffers
        dict(name="batch48_host", call="batch_host", potential="liquid", precision="mixed", structures=48, smallest=32,
             largest=2048),
        # serving: resident structures, one step of all of them
        dict(name="serve64_mixed", call="serve", potential="liquid", precision="mixed", structures=64, smallest=50,
             largest=3000),
        # a pair style's force call between neighbour-list rebuilds
        dict(name="lammps8000_mixed", call="lammps", potential="liquid", precision="mixed", atoms=8000, box="ortho",
             rebuilt=False),
        # a NEP potential, molecular dynamics on the GPU
        dict(name="nep32000", call="device", potential="nep", precision="fp32", atoms=32000, box="ortho", virials=False),
        # one training step: gradients of an energy + force + virial loss, radial weights trained too
        dict(name="train24_fused", call="train", potential="fused", precision="fp32", structures=24, smallest=40,
             largest=250),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges: any call, potential, precision and box, sizes over the logarithm."""
    call = rng.choice(["host", "host", "device", "device", "batch_device", "batch_host", "serve", "lammps", "train", "fp"])
    case = dict(call=call, potential=rng.choice(["copper", "liquid", "glass", "plain", "nep"]),
                precision=rng.choice(["fp32", "mixed"]))
    if call in ("host", "device", "fp"):
        case.update(atoms=_log_int(rng, 32, {"host": 30000, "device": 1000000, "fp": 16000}[call]),
                    box=rng.choice(["ortho", "lmp", "prism"]), virials=rng.random() < 0.5)
        if case["potential"] in ("nep", "plain"):
            case["atoms"] = min(case["atoms"], 100000 + case["atoms"] % 1000)
        if call == "fp":
            case["potential"] = rng.choice(["liquid", "glass", "plain"])
            case["virials"] = False
    elif call == "lammps":
        case.update(atoms=_log_int(rng, 500, 12000), box=rng.choice(["ortho", "lmp"]), rebuilt=rng.random() < 0.3)
    else:
        if call == "train":
            case["potential"] = rng.choice(["fused", "liquid", "glass"])
            case["precision"] = "fp32"
        lo = rng.randint(32, 64)
        case.update(structures=_log_int(rng, 2, {"batch_device": 700, "batch_host": 96, "serve": 128, "train": 32}[call]),
                    smallest=lo, largest=_log_int(rng, 80, 250 if call == "train" else 2048))
    return case


# ------------------------------------------------------------------------------- inputs
def _sizes(case):
    """Atom counts of a case's structures, log-uniform between its bounds (fixed by the case)."""
    if "structures" not in case:
        return [case["atoms"]]
    g = np.random.default_rng(case["structures"] * 1009 + case["largest"])
    return [int(v) for v in np.rint(np.exp(g.uniform(math.log(case["smallest"]), math.log(case["largest"]), case["structures"])))]


def _structure(n, fractions, density, box, rng):
    m = max(1, round(n ** (1 / 3)))
    grid = (m, m, -(-n // (m * m)))
    spacing = (n / density / (grid[0] * grid[1] * grid[2])) ** (1 / 3)
    h = np.diag([spacing * g for g in grid])
    if box in ("lmp", "prism"):
        h[1, 0], h[2, 0], h[2, 1] = 0.1 * h[0, 0], 0.1 * h[0, 0], 0.1 * h[1, 1]
    if box == "prism":  # the same cell, turned
        c, s = math.cos(0.4), math.sin(0.4)
        h = h @ np.array([[c, s, 0.0], [-s, c, 0.0], [0.0, 0.0, 1.0]])
    sites = rng.permutation(grid[0] * grid[1] * grid[2])[:n]
    f = np.stack([sites % grid[0], sites // grid[0] % grid[1], sites // (grid[0] * grid[1])], 1) / np.array(grid)
    x = f @ h + rng.normal(0.0, 0.13, (n, 3)).clip(-0.4, 0.4)
    t = 1 + np.searchsorted(np.cumsum(fractions)[:-1], rng.random(n)).astype(np.int32)
    return Structure(x, t.astype(np.int32), h, {"ortho": 0, "lmp": 1, "prism": 2}[box])


def _structures(case, seed):
    rng = np.random.default_rng(seed)
    p = POTENTIALS[case["potential"]]
    boxes = itertools.cycle(["ortho", "lmp"]) if "structures" in case else itertools.repeat(case["box"])
    return [_structure(n, p["fractions"], p["density"] * (rng.uniform(0.95, 1.05) if "structures" in case else 1.0),
                       b, rng) for n, b in zip(_sizes(case), boxes)]


def _upstream(case, seed, structures):
    """A loss's gradients by energies, forces and virials."""
    rng = np.random.default_rng(seed + 77)
    n = sum(s.natoms for s in structures)
    return rng.normal(0, 1, n), rng.normal(0, 1, (n, 3)), rng.normal(0, 0.1, (len(structures), 9))


@lru_cache(None)
def _parameters(name):
    """A potential's numbers (float64): radial weights, networks and, for "nep", its file's values."""
    p = POTENTIALS[name]
    T, N1 = len(p["fractions"]), p["nmax"] + 1
    rng = np.random.default_rng(11)
    if p["kind"] == "nep":
        dim, H = N1 + N1 * 6, p["hidden"][0]
        nann, ndesc = (dim + 2) * H * T + 1, 2 * T * T * N1 * 9
        scale = rng.uniform(0.005, 0.02, dim)  # a trained file's scales bring every column near one
        scale[N1:] *= 30.0
        scale[N1 * 5:] *= 10.0
        return dict(dim=dim, ann=rng.normal(0, 1 / math.sqrt(dim), nann), c=rng.uniform(-1, 1, ndesc), scale=scale)
    if "fuse" in p:
        fuse = rng.normal(0, 1, (T, T, p["fuse"]))
        W = np.zeros((T, T, p["fuse"] * N1, N1))
        for k in range(p["fuse"]):
            W[:, :, np.arange(N1) + k * N1, np.arange(N1)] = fuse[:, :, k, None]
    else:  # the "default" weights: unweighted functions, then weighted by +-species
        fuse = None
        W = np.zeros((T, T, N1 * (2 if T > 1 else 1), N1))
        W[:, :, np.arange(N1), np.arange(N1)] = 1.0
        if T > 1:
            for t in range(T):
                W[:, t, N1 + np.arange(N1), np.arange(N1)] = t + 1 if t % 2 == 0 else -(t + 1)
    D = W.shape[2] * (p["lmax"] + 1 if p["lmax"] >= 0 else 1)
    nets = []
    for _ in range(T):
        dims = [D] + p["hidden"]
        nets.append(dict(W=[rng.normal(0, 1 / math.sqrt(a), (b, a)) for a, b in zip(dims, dims[1:])],
                         b=[rng.normal(0, 1 / math.sqrt(a), b) for a, b in zip(dims, dims[1:])],
                         ow=rng.normal(0, 1 / math.sqrt(dims[-1]), dims[-1]), ob=float(rng.normal(0, 0.1)),
                         mu=np.zeros(D), sigma=np.ones(D)))
    q = dict(W=W, fuse=fuse, nets=nets, D=D)
    # descriptors are normalised by their mean and spread over a sample structure, as a trainer does
    s = _structure(300, p["fractions"], p["density"], "ortho", np.random.default_rng(5))
    fp = _Exact(name, q, "cpu").descriptors(s).numpy()
    for t in range(T):
        f = fp[s.types == t + 1]
        nets[t]["mu"], nets[t]["sigma"] = f.mean(0), f.std(0) + 1e-3 * np.abs(f).max(0) + 1e-3
    return q


@lru_cache(None)
def _model_text(name):
    """The potential as the text that a handle reads."""
    p, q = POTENTIALS[name], _parameters(name)
    if p["kind"] == "nep":
        head = ["nep4 2 Si O", "cutoff 8 4 100 100", "n_max 4 4", "basis_size 8 8", "l_max 4 2 1", "ANN 30 0"]
        return "\n".join(head + ["%.17g" % v for v in np.concatenate([q["ann"], q["c"], q["scale"]])]) + "\n"
    models = []
    for t, net in enumerate(q["nets"]):
        basis = {"type": "chebyshev" if p["kind"] == "radial" else "spherical_chebyshev", "nmax": p["nmax"], "rcut": p["rcut"]}
        if p["kind"] != "radial":
            basis["lmax"] = p["lmax"]
        if q["fuse"] is not None:
            basis.update(wtype="fuse", fuse_size=p["fuse"], fuse_weight=q["fuse"][t].reshape(-1).tolist())
        models.append({"symbol": "ABC"[t], "basis": basis, "norm_mu": net["mu"].tolist(), "norm_sigma": net["sigma"].tolist(),
                       "nn": {"type": "feed_forward", "input_dim": q["D"], "hidden_dims": p["hidden"],
                              "hidden_weights": [w.tolist() for w in net["W"]], "hidden_biases": [b.tolist() for b in net["b"]],
                              "output_weight": net["ow"].tolist(), "output_bias": net["ob"]}})
    models[0].update(norm_mu_eng=-3.0, norm_sigma_eng=0.1)
    return json.dumps({"version": 6, "units": "metal", "models": models})


def prepare(case, seed):
    """A handle and the inputs of one call."""
    text = _model_text(case["potential"])
    pot = (NEP if case["potential"] == "nep" else J.NNAP)(text, precision=case["precision"], device=0)
    structures = _structures(case, seed)
    st = dict(call=case["call"], pot=pot, structures=structures, virials=case.get("virials", False))
    if case["call"] in ("device", "batch_device", "batch_host"):
        x = np.concatenate([s.x for s in structures])
        t = np.concatenate([s.types for s in structures])
        st.update(natoms=np.array([s.natoms for s in structures], dtype=np.int32),
                  kinds=np.array([s.box_kind for s in structures], dtype=np.int32),
                  boxes=np.stack([s.box.reshape(9) for s in structures]))
        S, n = len(structures), len(t)
        shapes = dict(energy=(S,), energies=(n,), forces=(n, 3), virial=(S, 9))
        if st["virials"]:
            shapes["virials"] = (n, 9)
        if case["call"] == "batch_host":
            st.update(x=x, t=t, out={k: np.zeros(v) for k, v in shapes.items()})
        else:
            st.update(x=torch.from_numpy(x).cuda(), t=torch.from_numpy(t).cuda(),
                      out={k: torch.zeros(v, dtype=torch.float64, device="cuda") for k, v in shapes.items()})
        st["flags"] = sum({"energy": J.WANT_ENERGY, "energies": J.WANT_ENERGIES, "forces": J.WANT_FORCES,
                           "virial": J.WANT_VIRIAL, "virials": J.WANT_VIRIALS}[k] for k in shapes)
    elif case["call"] == "serve":
        st["server"] = NNAPServer(pot, skin=SKIN, memory_budget=40e9)
        st["slots"] = [st["server"].admit(s) for s in structures]
        st["xs"] = [np.ascontiguousarray(s.x) for s in structures]
    elif case["call"] == "train":
        st["upstream"] = _upstream(case, seed, structures)
    elif case["call"] == "lammps":
        st.update(_lammps(structures[0], POTENTIALS[case["potential"]]["rcut"]), rebuilt=case["rebuilt"])
        _run_lammps(st, True)
    return st


def run(state):
    """One call and its outputs."""
    call, pot = state["call"], state["pot"]
    if call == "host":
        out = pot.calEnergyForceVirials(state["structures"][0], per_atom_virial=state["virials"])
    elif call == "fp":
        out = {"fp": pot.calFp(state["structures"][0])}
    elif call in ("device", "batch_device"):
        out = state["out"]
        p = {k + "_ptr": v.data_ptr() for k, v in out.items()}
        stream = torch.cuda.current_stream().cuda_stream
        if call == "device":
            pot.computeDevice(int(state["natoms"][0]), state["x"].data_ptr(), state["t"].data_ptr(), state["boxes"][0],
                              int(state["kinds"][0]), state["flags"], stream=stream, **p)
        else:
            pot.computeBatchDevice(state["natoms"], state["x"].data_ptr(), state["t"].data_ptr(), state["kinds"],
                                   state["boxes"], state["flags"], stream=stream, **p)
        return {k: v.float() for k, v in out.items()}
    elif call == "batch_host":
        out = state["out"]
        pot._check(J.load_library().nnap_compute_batch(
            pot._handle(), len(state["natoms"]), J._iptr(state["natoms"]), J._dptr(state["x"]), J._iptr(state["t"]),
            J._iptr(state["kinds"]), J._dptr(state["boxes"]), state["flags"], J._dptr(out["energy"]),
            J._dptr(out["energies"]), J._dptr(out["forces"]), J._dptr(out["virial"]), None))
    elif call == "serve":
        out = state["server"].step(state["slots"], state["xs"], energies=True)
    elif call == "train":
        be, bf, bw = state["upstream"]
        r = pot.backwardEnergyForceBatch(state["structures"], be, bf, bw, want_fp=True)
        out = {k: np.concatenate(v) for k, v in r.items()}
    else:
        out = _run_lammps(state, state["rebuilt"])
    return {k: np.float32(v) for k, v in out.items()}


def _lammps(s, rcut):
    """The arrays that LAMMPS hands a pair style: wrapped local atoms, then ghosts, full lists with a skin."""
    nl = _Neighbours(s, rcut + SKIN, "cuda" if torch.cuda.is_available() else "cpu")
    idx = nl.idx.to(torch.int32).cpu().numpy()
    num = nl.count.to(torch.int32).cpu().numpy()
    nall = len(nl.owner)
    owner = nl.owner.cpu().numpy()
    rows = np.ascontiguousarray(idx)
    most = _room(s, rcut)
    first = (ctypes.POINTER(ctypes.c_int) * nall)()
    base = rows.ctypes.data
    for i in range(s.natoms):
        first[i] = ctypes.cast(base + 4 * i * rows.shape[1], ctypes.POINTER(ctypes.c_int))
    numneigh = np.zeros(nall, dtype=np.int32)
    numneigh[:s.natoms] = num
    return dict(x=nl.pos.cpu().numpy().copy(), t=np.ascontiguousarray(s.types[owner]), rows=rows, first=first, numneigh=numneigh,
                ilist=np.arange(s.natoms, dtype=np.int32), nall=nall, most=most)


def _room(s, rcut):
    """Rows of a pair style's per-atom arrays, which LAMMPS allocates with room to spare: the grid sites of the box and of
    the ghosts' layer around it."""
    m = max(1, round(s.natoms ** (1 / 3)))
    reach = (rcut + SKIN) * np.linalg.norm(np.linalg.inv(s.box), axis=0)
    return int(np.prod([g + 2 * math.ceil(g * r) + 4 for g, r in zip((m, m, -(-s.natoms // (m * m))), reach)]))


def _run_lammps(st, rebuilt):
    n, nall, pot = len(st["ilist"]), st["nall"], st["pot"]
    out = dict(forces=np.zeros((st["most"], 3)), eng=np.zeros(1), eatom=np.zeros(st["most"]), virial=np.zeros(6))
    pot._check(J.load_library().nnap_compute_lammps_nl(
        pot._handle(), int(rebuilt), n, nall, J._iptr(st["ilist"]), J._iptr(st["numneigh"]), st["first"], J._dptr(st["x"]),
        J._iptr(st["t"]), None, 1, 1, 1, 0, 0, J._dptr(out["forces"]), J._dptr(out["eng"]), J._dptr(out["eatom"]),
        J._dptr(out["virial"]), None, None))
    return out


# ------------------------------------------------------------------------------- the work of a pass
def work(case):
    """Positions and species in, results out; the arithmetic of harmonics, expansion, power
    spectrum, network and their gradients, per pair and per atom."""
    p, sizes = POTENTIALS[case["potential"]], _sizes(case)
    n, S = sum(sizes), len(sizes)
    N1, T, K = p["nmax"] + 1, len(p["fractions"]), (p["lmax"] + 1) ** 2
    near = p["density"] * 4 / 3 * math.pi * p["rcut"] ** 3
    P = N1 * p.get("fuse", 2 if T > 1 else 1)
    D = P * (p["lmax"] + 1) if K else P
    pair = near * (4 * N1 + 10)
    if p["kind"] == "nep":  # both bases expand nine functions; the angular one reaches half as far
        P, D = N1, N1 * 7
        pair += near * 2 * 9 * N1 + near / 8 * (2 * 9 * N1 + 2 * N1 * K + 6 * K)
    elif K:
        pair += near * (2 * N1 * K + 6 * K)  # one product per radial function and harmonic
    hidden = [D] + p["hidden"]
    net = 2 * sum(a * b for a, b in zip(hidden, hidden[1:] + [1]))
    flops = n * (pair + 2 * P * max(K, 1) + net)
    if case["call"] == "fp":
        return {"bytes": n * (24 + 4 + 8 * D) + 72, "flops": n * (pair + 2 * P * max(K, 1))}
    flops *= 3 if case["call"] != "train" else 9
    if case["call"] == "train":
        return {"bytes": n * (24 + 4 + 8 + 24) + S * 144 + 16 * T * net / 2, "flops": flops}
    nbytes = n * (24 + 4 + 8 + 24 + (72 if case.get("virials") else 0)) + S * (72 + 8 + 72)
    if case.get("rebuilt"):
        nbytes += 4 * n * near * (1 + SKIN / p["rcut"]) ** 3
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------------------- 64 bits
class _Neighbours:
    """Full neighbour lists by cells: wrapped atoms then the ghosts within rc of the box (``pos``, ``owner``), and per atom
    the padded row ``idx`` of its neighbours' numbers there (-1: none)."""

    def __init__(self, s, rc, device):
        box, inverse = (torch.as_tensor(a, dtype=torch.float64, device=device) for a in (s.box, np.linalg.inv(s.box)))
        f = torch.as_tensor(s.x, dtype=torch.float64, device=device) @ inverse
        f = f - torch.floor(f)
        reach = rc * inverse.square().sum(0).sqrt()
        R = [int(math.ceil(float(v))) for v in reach]
        n = len(f)
        pos, owner = [f], [torch.arange(n, device=device)]
        for im in itertools.product(*(range(-r, r + 1) for r in R)):
            if any(im):
                g = f + torch.tensor(im, dtype=torch.float64, device=device)
                keep = ((g > -reach - 1e-9) & (g < 1 + reach + 1e-9)).all(1).nonzero()[:, 0]
                pos.append(g[keep])
                owner.append(keep)
        pos, self.owner = torch.cat(pos) @ box, torch.cat(owner)
        self.pos = pos
        lo = pos.min(0).values
        c = torch.floor((pos - lo) / rc).long() + 1
        dims = c.max(0).values + 2
        cid = c[:, 0] + dims[0] * (c[:, 1] + dims[1] * c[:, 2])
        order = torch.argsort(cid)
        start = torch.searchsorted(cid[order], torch.arange(int(dims.prod()) + 1, device=device))
        cap = int((start[1:] - start[:-1]).max())
        off = torch.tensor([a + int(dims[0]) * (b + int(dims[1]) * d) for a, b, d in itertools.product((-1, 0, 1), repeat=3)],
                           device=device)
        rows, self.count = [], []
        step = max(1, 30_000_000 // (27 * cap))
        for b in range(0, n, step):
            i = torch.arange(b, min(n, b + step), device=device)
            cells = cid[i][:, None] + off
            k = start[cells][:, :, None] + torch.arange(cap, device=device)
            ok = (k < start[cells + 1][:, :, None]).reshape(len(i), -1)
            j = order[k.clamp(max=len(order) - 1)].reshape(len(i), -1)
            ok &= (pos[j] - pos[i][:, None]).square().sum(-1) < rc * rc
            ok &= j != i[:, None]
            cnt = ok.sum(1)
            m = int(cnt.max())
            rows.append(torch.where(ok, j, -1).sort(1, descending=True).values[:, :m])
            self.count.append(cnt)
        m = max(1, max(r.shape[1] for r in rows))
        self.idx = torch.cat([torch.nn.functional.pad(r, (0, m - r.shape[1]), value=-1) for r in rows])
        self.count = torch.cat(self.count)


def _chebyshev(x, count):
    t = [torch.ones_like(x), x]
    while len(t) < count:
        t.append(2 * x * t[-1] - t[-2])
    return torch.stack(t[:count], -1)


def _harmonics(L, u):
    """Orthonormal real spherical harmonics of unit vectors, as polynomials (no poles); m = 0, then cos and sin of each m."""
    x, y, z = u.unbind(-1)
    by_l = [[] for _ in range(L + 1)]
    c, s = torch.ones_like(x), torch.zeros_like(x)
    for m in range(L + 1):
        if m:
            c, s = x * c - y * s, x * s + y * c
        q = [torch.full_like(x, float(np.prod(np.arange(2 * m - 1, 0, -2, dtype=np.float64))))]  # P_mm / sin^m
        for l in range(m, L + 1):
            if l > m:
                last = q[-2] if l > m + 1 else 0.0
                q.append(((2 * l - 1) * z * q[-1] - (l + m - 1) * last) / (l - m))
            N = math.sqrt((2 * l + 1) / (4 * math.pi) * math.factorial(l - m) / math.factorial(l + m))
            by_l[l] += [N * q[-1]] if m == 0 else [math.sqrt(2) * N * q[-1] * c, math.sqrt(2) * N * q[-1] * s]
    return torch.stack([v for l in by_l for v in l], -1)


class _Exact:
    """A potential in 64 bits."""

    def __init__(self, name, q, device):
        self.p, self.name, self.device = POTENTIALS[name], name, device
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=device)  # noqa: E731
        self.T = len(self.p["fractions"])
        if self.p["kind"] == "nep":
            N1, T, H = self.p["nmax"] + 1, self.T, self.p["hidden"][0]
            c = t(q["c"]).reshape(2, N1, 9, T, T).permute(0, 3, 4, 1, 2)  # radial, angular: [centre][neighbour][n][k]
            self.Wr, self.W, self.scale = c[0], c[1], t(q["scale"])
            ann, per = t(q["ann"]), (q["dim"] + 2) * H
            self.nets = [(ann[k * per:][:H * q["dim"]].reshape(H, -1), ann[k * per + H * q["dim"]:][:H],
                          ann[k * per + H * q["dim"] + H:][:H]) for k in range(T)]
            self.b1 = ann[-1]
        else:
            self.W = t(q["W"])
            self.nets = [{k: [t(a) for a in v] if isinstance(v, list) else t(v) for k, v in n.items()} for n in q["nets"]]

    def fingerprint(self, d, pad, tc, tn):
        """Descriptors [centres, D] from displacements [centres, M, 3], padding, and species from 0."""
        p = self.p
        r = d.square().sum(-1).sqrt()
        u = d / r[..., None]
        weigh = lambda f, W: torch.einsum("cmk,cmpk->cmp", f, W[tc[:, None], tn])  # noqa: E731
        if p["kind"] == "nep":
            def radial(rc):
                f = 0.5 * (_chebyshev(2 * (r / rc - 1) ** 2 - 1, 9) + 1) * (0.5 * torch.cos(math.pi * r / rc) + 0.5)[..., None]
                return f * (~pad & (r < rc))[..., None]
            g = weigh(radial(4.0), self.W)
            A = torch.einsum("cmp,cmk->cpk", g, _harmonics(4, u))
            out = [weigh(radial(8.0), self.Wr).sum(1)]
            out += [A[..., l * l:(l + 1) ** 2].square().sum(-1) for l in range(1, 5)]
            # the four- and five-body columns: the determinant of the quadrupole, the square of the dipole's square
            Q = torch.einsum("cmp,cmab->cpab", g, 1.5 * u[..., :, None] * u[..., None, :] - 0.5 * torch.eye(3, dtype=u.dtype, device=u.device))
            det = (Q[..., 0, :] * torch.linalg.cross(Q[..., 1, :], Q[..., 2, :])).sum(-1)
            out.append(-4 * math.sqrt(2 / 35) * (5 / 4 / math.pi) ** 1.5 * det)
            out.append(7 / 15 * out[1].square())
            return torch.cat(out, -1)
        rc = p["rcut"]
        fc = torch.where(pad | (r >= rc), 0.0, (1 - (r / rc) ** 2) ** 4)
        c = weigh(_chebyshev(1 - 2 * r / rc, p["nmax"] + 1) * fc[..., None], self.W)
        if p["kind"] == "radial":
            return c.sum(1)
        A = torch.bmm(c.transpose(1, 2), _harmonics(p["lmax"], u))
        return torch.stack([4 * math.pi / (2 * l + 1) * A[..., l * l:(l + 1) ** 2].square().sum(-1)
                            for l in range(p["lmax"] + 1)], -1).flatten(1)

    def energy(self, fp, tc):
        e = fp.new_zeros(len(fp))
        for t, net in enumerate(self.nets):
            k = (tc == t).nonzero()[:, 0]
            if self.p["kind"] == "nep":
                w0, b0, w1 = net
                v = torch.tanh((fp[k] * self.scale) @ w0.T - b0) @ w1 - self.b1
            else:
                a = (fp[k] - net["mu"]) / net["sigma"]
                for w, b in zip(net["W"], net["b"]):
                    a = torch.nn.functional.silu(a @ w.T + b)
                v = 0.1 * (a @ net["ow"] + net["ob"]) - 3.0
            e = e.index_add(0, k, v)
        return e

    def chunks(self, s, nl):
        """(centres, displacements, padding, species of centres and neighbours, neighbours' numbers)."""
        types = torch.as_tensor(s.types, device=self.device).long() - 1
        M = nl.idx.shape[1]
        step = max(1, (250_000 if self.p["lmax"] > 4 or self.p["kind"] == "nep" else 500_000) // M)
        for b in range(0, s.natoms, step):
            idx = nl.idx[b:b + step]
            pad = idx < 0
            j = idx.clamp(min=0)
            i = torch.arange(b, b + len(idx), device=self.device)
            d = nl.pos[j] - nl.pos[i][:, None]
            d = torch.where(pad[..., None], torch.full_like(d, self.p["rcut"]), d)
            yield i, d, pad, types[i], types[nl.owner[j]], j

    def descriptors(self, s):
        nl = _Neighbours(s, self.p["rcut"], self.device)
        return torch.cat([self.fingerprint(d, pad, tc, tn) for _, d, pad, tc, tn, _ in self.chunks(s, nl)])

    def evaluate(self, s, fold=True):
        """Energies, forces and atomic virials; ``fold``: on the atoms, else on atoms and ghosts."""
        nl = _Neighbours(s, self.p["rcut"] if fold else self.p["rcut"] + SKIN, self.device)
        size = s.natoms if fold else len(nl.owner)
        e = torch.zeros(size, dtype=torch.float64, device=self.device)
        f, v = e.new_zeros(size, 3), e.new_zeros(size, 9)
        for i, d, pad, tc, tn, j in self.chunks(s, nl):
            d.requires_grad_(True)
            ei = self.energy(self.fingerprint(d, pad, tc, tn), tc)
            g = torch.autograd.grad(ei.sum(), d)[0].masked_fill(pad[..., None], 0.0)
            with torch.no_grad():
                to = (nl.owner[j] if fold else j).flatten()
                e[i] = ei.detach()
                f.index_add_(0, i, g.sum(1))
                f.index_add_(0, to, -g.reshape(-1, 3))
                w = -(d[..., :, None] * g[..., None, :]).reshape(-1, 9)
                v.index_add_(0, to, w[:, [0, 4, 8, 1, 2, 5, 3, 6, 7]])
        return e, f, v

    def gradients(self, structures, be, bf, bw):
        """Gradients of sum be E + bf F + bw W by network and radial weights, in the C layout."""
        leaves = []
        for net in self.nets:
            leaves += net["W"] + [net["ow"]] + net["b"] + [net["ob"]]
        leaves.append(self.W)
        for q in leaves:
            q.requires_grad_(True)
        total = [torch.zeros_like(q) for q in leaves]
        a0 = 0
        for k, s in enumerate(structures):
            nl = _Neighbours(s, self.p["rcut"], self.device)
            B = torch.as_tensor(bw[k], device=self.device)[[0, 3, 4, 6, 1, 5, 7, 8, 2]].reshape(3, 3)
            E = torch.as_tensor(be[a0:a0 + s.natoms], device=self.device)
            F = torch.as_tensor(bf[a0:a0 + s.natoms], device=self.device)
            for i, d, pad, tc, tn, j in self.chunks(s, nl):
                d.requires_grad_(True)
                ei = self.energy(self.fingerprint(d, pad, tc, tn), tc)
                g = torch.autograd.grad(ei.sum(), d, create_graph=True)[0].masked_fill(pad[..., None], 0.0)
                up = F[i][:, None] - F[nl.owner[j]] - d.detach() @ B
                loss = (ei * E[i]).sum() + (g * up).sum()
                for t, q in zip(total, torch.autograd.grad(loss, leaves, allow_unused=True)):
                    if q is not None:
                        t += q
            a0 += s.natoms
        nn = torch.cat([t.reshape(-1) for t in total[:-1]])
        fuse = total[-1].reshape(-1) if "fuse" in self.p else torch.zeros_like(total[-1]).reshape(-1)
        return {"grad_nn": nn.cpu().numpy(), "grad_fp": fuse.cpu().numpy()}


def exact(case, seed):
    """What run returns, in 64 bits."""
    device = "cuda" if torch.cuda.is_available() else "cpu"
    X = _Exact(case["potential"], _parameters(case["potential"]), device)
    structures = _structures(case, seed)
    call = case["call"]
    if call == "fp":
        return {"fp": X.descriptors(structures[0]).cpu().numpy()}
    if call == "train":
        return X.gradients(structures, *_upstream(case, seed, structures))
    if call == "lammps":
        e, f, v = X.evaluate(structures[0], fold=False)
        spare = _room(structures[0], POTENTIALS[case["potential"]]["rcut"]) - len(e)
        return {"forces": np.pad(f.cpu().numpy(), ((0, spare), (0, 0))), "eng": e.sum().reshape(1).cpu().numpy(),
                "eatom": np.pad(e.cpu().numpy(), (0, spare)), "virial": v.sum(0)[:6].cpu().numpy()}
    parts = [X.evaluate(s) for s in structures]
    out = {"energies": torch.cat([e for e, _, _ in parts]), "forces": torch.cat([f for _, f, _ in parts])}
    if call == "host":
        out.update(energy=parts[0][0].sum(), virial=parts[0][2].sum(0))
    else:
        out.update(energy=torch.stack([e.sum() for e, _, _ in parts]), virial=torch.stack([v.sum(0) for _, _, v in parts]))
    if case.get("virials"):
        out["virials"] = parts[0][2]
    return {k: v.cpu().numpy() for k, v in out.items()}
