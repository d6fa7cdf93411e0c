"""Performance cases of the NNP energy/force library: the calls a user's
program makes, through the public entry points of ``ace_b200.NNP``.

A case is one call: a family of structures (a small periodic cell, an FCC
crystal, a batch of sheared random cells, free clusters, one domain with its
ghost atoms), a potential (elements, basis, networks) and an entry point.
Sizes, densities and bases are those of the benchmark's workloads; the listed
cases run from one 64-atom cell to the 4096-structure batch, and ``draw``
spreads over the same ranges.

Outputs are handed on in FP32: the basis, the networks and the force terms
are FP32 arithmetic (the ABI's FP64 arrays hold their sums), and FP32 is what
a torch program keeps of them.

``exact`` restates the path (neighbour list, symmetry functions, networks,
forces, virial, loss gradient) with plain torch operations in FP64.
"""
from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch

from ace_b200 import NNP
from ace_b200 import potential as potfile

DENSITY = 0.05            # atoms per cubic A of the batched random cells
FCC_A = 4.05              # lattice constant of the crystals, A
PREC = {"fp32": 0, "bf16x3": 2}

# potentials of the benchmark's workloads: elements, cutoff radius, radial
# functions per neighbour element, angular functions per element pair, hidden layers
ONE = dict(ntypes=1, rc=6.0, nrad=16, ang="16", hid="20,20")
THREE = dict(ntypes=3, rc=6.0, nrad=8, ang="6,5,5,6,5,5", hid="32,32")
TWO = dict(ntypes=2, rc=6.0, nrad=12, ang="8,8,8", hid="32,32")
ALLOY = dict(ntypes=2, rc=6.5, nrad=16, ang="16,16,16", hid="64,64")
FOUR = dict(ntypes=4, rc=6.0, nrad=6, ang="4,4,4,4,4,4,4,4,4,4", hid="48,48")
GAUSS = dict(cut="COS", rform="GAUSSIAN", aform="GAUSS", neuron="TANH")
OTHER = dict(cut="TANH", rform="SECH", aform="GAUSS2", neuron="SIGMOID")


def listed():
    return [
        # molecular dynamics or relaxation of one small cell: the shortest call, latency counts
        dict(name="md cell 64", api="device", family="cell", n_struct=1, nmin=64, nmax=64, prec="fp32", **ONE, **GAUSS),
        # one free molecule or cluster through NNP.compute with host arrays (a script, a geometry optimiser)
        dict(name="cluster 57 host", api="host", family="free", n_struct=1, nmin=57, nmax=57, prec="fp32", **TWO, **GAUSS),
        # crystal MD with stress and per-atom energies (barostat, analysis), host arrays
        dict(name="md crystal 4000 virial", api="md", family="fcc", n_struct=1, nmin=10, nmax=10, prec="fp32", **ALLOY, **GAUSS),
        # one spatial domain of a domain-decomposed MD code with its ghost atoms (pair style)
        dict(name="domain 256 ghosts", api="ghost", family="fcc", n_struct=1, nmin=4, nmax=4, prec="fp32", **ALLOY, **GAUSS),
        # MD of a large crystal on device-resident arrays
        dict(name="md crystal 131072", api="device", family="fcc", n_struct=1, nmin=32, nmax=32, prec="bf16x3", **ALLOY, **GAUSS),
        # evaluation of a validation batch of uneven cells, FP32 networks
        dict(name="batch 256 fp32", api="device", family="random", n_struct=256, nmin=16, nmax=512, prec="fp32", **THREE, **GAUSS),
        # screening: the largest batch, tensor-core networks
        dict(name="batch 4096", api="device", family="random", n_struct=4096, nmin=16, nmax=512, prec="bf16x3", **THREE, **GAUSS),
        # a stream of very uneven structures from host buffers, four elements
        dict(name="stream 1000 host", api="host", family="loguniform", n_struct=1000, nmin=8, nmax=2048, prec="bf16x3", **FOUR, **GAUSS),
        # symmetry functions of a data set, for fitting outside the library
        dict(name="symm 32", api="symm", family="random", n_struct=32, nmin=16, nmax=512, prec="fp32", **THREE, **GAUSS),
        # training: gradient of the energy+force loss of one batch on the device
        dict(name="train 256", api="train", family="random", n_struct=256, nmin=64, nmax=256, prec="fp32", **TWO, **GAUSS),
        # a small mini-batch from host arrays
        dict(name="train 8 host", api="train_host", family="random", n_struct=8, nmin=64, nmax=256, prec="fp32", **TWO, **GAUSS),
        # the other basis forms, cutoff and activation
        dict(name="batch 128 other forms", api="device", family="random", n_struct=128, nmin=16, nmax=512, prec="fp32",
             **dict(TWO, nrad=6, ang="4,4,4", hid="16,16"), **OTHER),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def blocks(ntypes, lo, hi):
        return ",".join(str(rng.randint(lo, hi)) for _ in range(ntypes * (ntypes + 1) // 2))

    forms = OTHER if rng.random() < 0.1 else GAUSS
    prec = rng.choice(["fp32", "bf16x3"])
    kind = rng.choice(["cell", "free", "fcc", "ghost", "random", "random", "stream", "symm", "train", "train"])
    nt = rng.randint(1, 4)
    pot = dict(ntypes=nt, rc=rng.choice([6.0, 6.5]), nrad=rng.randint(4, 16),
               ang=blocks(nt, 4, 16 if nt < 3 else 8), hid=rng.choice(["20,20", "32,32", "48,48", "64,64"]))
    if kind == "cell":
        n = rng.randint(32, 110)
        return dict(api=rng.choice(["device", "md"]), family="cell", n_struct=1, nmin=n, nmax=n, prec=prec,
                    **dict(pot, ntypes=1, ang=str(rng.randint(4, 16))), **forms)
    if kind == "free":
        n = log(12, 250)
        return dict(api="host", family="free", n_struct=1, nmin=n, nmax=n, prec=prec, **dict(pot, rc=5.0), **forms)
    if kind in ("fcc", "ghost"):
        n = rng.randint(5, 26) if kind == "fcc" else 4
        return dict(api="ghost" if kind == "ghost" else rng.choice(["device", "md"]), family="fcc", n_struct=1, nmin=n, nmax=n,
                    prec=prec, **pot, **forms)
    if kind in ("random", "stream"):
        lu = kind == "stream"
        return dict(api=rng.choice(["device", "host"]), family="loguniform" if lu else "random", n_struct=log(4, 1500 if forms is GAUSS else 300),
                    nmin=rng.randint(8, 32), nmax=rng.randint(300, 600) if not lu else rng.randint(500, 2048), prec=prec, **pot, **forms)
    if kind == "symm":
        return dict(api="symm", family="random", n_struct=log(2, 100), nmin=rng.randint(8, 32), nmax=rng.randint(200, 512),
                    prec="fp32", **pot, **forms)
    return dict(api=rng.choice(["train", "train_host"]), family="random", n_struct=log(4, 300), nmin=rng.randint(32, 64),
                nmax=rng.randint(128, 256), prec="fp32", **dict(pot, ntypes=min(nt, 3), ang=blocks(min(nt, 3), 4, 8)), **GAUSS)


# ---------------------------------------------------------------- structures

def _cells(case, rng):
    """(atom offsets, positions, types, cells with the lattice vectors as rows) of the case's structures."""
    nt, fam = case["ntypes"], case["family"]
    if fam == "fcc":
        n = case["nmin"]
        base = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
        g = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 1, 3)
        pos = ((g + base) * FCC_A).reshape(-1, 3)
        pos = pos + rng.normal(0.0, 0.1, size=pos.shape)
        typ = rng.permutation(np.arange(len(pos)) % nt).astype(np.int32)
        return np.array([0, len(pos)]), pos, typ, np.eye(3)[None] * (FCC_A * n)
    if fam == "cell":                       # uniform positions at least 1.8 A apart, the density of 64 atoms in (8.5 A)^3
        n = case["nmin"]
        L = 8.5 * (n / 64.0) ** (1.0 / 3.0)
        pos = np.zeros((n, 3))
        k = 0
        while k < n:
            p = rng.uniform(0.0, L, 3)
            d = pos[:k] - p
            d -= L * np.round(d / L)
            if k == 0 or (d * d).sum(1).min() >= 1.8 ** 2:
                pos[k] = p
                k += 1
        return np.array([0, n]), pos, rng.integers(0, nt, n).astype(np.int32), np.eye(3)[None] * L
    sizes = np.random.default_rng([case["n_struct"], case["nmin"], case["nmax"]])   # the case's sizes; the seed sets the rest
    if fam == "loguniform":
        cnt = np.exp(sizes.uniform(math.log(case["nmin"]), math.log(case["nmax"] + 1), case["n_struct"])).astype(np.int64)
    else:
        cnt = sizes.integers(case["nmin"], case["nmax"] + 1, case["n_struct"])
    off = np.concatenate([[0], np.cumsum(cnt)])
    pos, typ, cell = np.zeros((off[-1], 3)), np.zeros(off[-1], np.int32), np.zeros((len(cnt), 3, 3))
    for s, n in enumerate(cnt):             # a random subset of a jittered grid in a sheared cell
        L = (n / DENSITY) ** (1.0 / 3.0)
        shear = rng.uniform(-0.1, 0.1, (3, 3)) if fam != "free" else np.zeros((3, 3))
        np.fill_diagonal(shear, 0.0)
        cell[s] = L * (np.eye(3) + shear).T
        m = int(math.ceil((1.5 * n) ** (1.0 / 3.0)))
        pick = rng.permutation(m ** 3)[:n]
        g = np.stack([pick // (m * m), pick // m % m, pick % m], 1)
        pos[off[s]:off[s + 1]] = ((g + 0.5 + rng.uniform(-0.3, 0.3, (n, 3))) / m) @ cell[s]
        typ[off[s]:off[s + 1]] = rng.choice(nt, n, p=rng.dirichlet(np.ones(nt)))
    return off, pos, typ, cell


def _ghosts(pos, L, rc):
    """Periodic images within rc and a skin of 0.5 A of the box [0, L)^3: their positions and the atoms they image."""
    rc = rc + 0.5
    gp, go = [], []
    for q in np.ndindex(3, 3, 3):
        sh = np.array(q) - 1
        if sh.any():
            x = pos + sh * L
            near = ((x >= -rc) & (x < L + rc)).all(1)
            gp.append(x[near])
            go.append(np.nonzero(near)[0])
    return np.concatenate(gp), np.concatenate(go)


# ---------------------------------------------------------------- potentials

_pots = {}
_dir = tempfile.TemporaryDirectory(prefix="nnp_perf_")


def _potential(case):
    """(potential, its file): random networks whose inputs are scaled to the spread of
    the symmetry functions over a fixed sample, as a potential is before training."""
    key = tuple(case[k] for k in ("ntypes", "rc", "nrad", "ang", "hid", "cut", "rform", "aform", "neuron")) + (case["family"],)
    if key in _pots:
        return _pots[key]
    rng = np.random.default_rng(1234)
    T, rc = case["ntypes"], case["rc"]
    sizes, hidden = [int(x) for x in case["ang"].split(",")], [int(x) for x in case["hid"].split(",")]
    full = [(e, z, l) for e in (14.142136, 7.071068) for z in (1.0, 2.0, 4.0, 8.0) for l in (1, -1)]
    rs = np.round(np.linspace(0.5, min(6.0, rc), case["nrad"]), 6)

    def angular(m):
        p = [full[k] for k in np.round(np.linspace(0, len(full) - 1, m)).astype(int)]
        return potfile.BasisA(case["cut"], rc, case["aform"], np.array([x[0] for x in p]), np.array([x[1] for x in p]),
                              np.array([x[2] for x in p], dtype=np.int32))

    nin = T * case["nrad"] + sum(sizes)
    nets = []
    for _ in range(T):
        nodes, b, w = [nin] + hidden + [1], [], []
        for l in range(len(nodes) - 1):
            s = math.sqrt(2.0 / (nodes[l] + nodes[l + 1]))
            b.append(np.round(rng.normal(0.0, 0.1 * s, nodes[l + 1]), 12))
            w.append(np.round(rng.normal(0.0, s, (nodes[l + 1], nodes[l])), 12))
        b[-1] -= 3.0                        # a cohesive energy of a few eV per atom
        nets.append(potfile.Network(nodes, case["neuron"], 1.0, np.ones(nin), np.zeros(nin), np.ones(1), np.zeros(1), b, w))
    pot = potfile.Potential([potfile.ElementType(name="ABCD"[i], energy=-1.0 - 0.5 * i, mass=1.0 + i) for i in range(T)], rc,
                            [[potfile.BasisR(case["cut"], rc, case["rform"], rs.copy(), np.ones(case["nrad"])) for _ in range(T)]
                             for _ in range(T)],
                            [[angular(m) for m in sizes] for _ in range(T)], nets)
    # inpb = -mean(G), inpw = 1 / dev(G) over the sample
    sample = dict(case, n_struct=1 if case["family"] == "fcc" else 6)
    sample["nmin"] = sample["nmax"] = 4 if case["family"] == "fcc" else 64
    G, typ = [], []
    for s in range(1 if sample["family"] == "fcc" else 6):
        off, pos, t, cell = _cells(dict(sample, n_struct=1), np.random.default_rng(997 + s))
        for II, idx, _, _, g in _Exact(pot, off, pos, t, cell, case["family"] != "free").rows(False):
            G.append(g.cpu().numpy())
            typ.append(np.full(len(g), II))
    G, typ = np.concatenate(G), np.concatenate(typ)
    for II in range(T):
        g = G[typ == II]
        if len(g):
            dev = g.std(0)
            nets[II].inpb = np.round(-g.mean(0), 9)
            nets[II].inpw = np.round(1.0 / np.where(dev > 1e-6, dev, 1.0), 9)
    path = os.path.join(_dir.name, "%d.nnp" % len(_pots))
    potfile.write(path, pot)
    _pots[key] = pot, path
    return _pots[key]


# ---------------------------------------------------------------- the calls

_shared = {}


def _handle(case, path, own):
    """The potential on the GPU, on a stream of the program. An MD program has one handle that works
    on the same arrays at each step; a program that evaluates batch after batch uses one for all of them."""
    key = (path, case["prec"], case["api"])
    if own or key not in _shared:
        nn = NNP.read(path)
        nn.set_precision(PREC[case["prec"]])
        stream = torch.cuda.Stream()
        nn.set_stream(stream.cuda_stream)
        if own:
            return nn, stream
        _shared[key] = nn, stream
    return _shared[key]


def prepare(case, seed):
    pot, path = _potential(case)
    rng = np.random.default_rng(seed)
    off, pos, typ, cell = _cells(case, rng)
    own = case["n_struct"] == 1
    nn, stream = _handle(case, path, own)
    st = dict(api=case["api"], nn=nn, stream=stream, pbc=case["family"] != "free", n=len(pos), S=len(cell))
    st.update(off=off.astype(np.int64), pos=pos, typ=typ, cell=np.ascontiguousarray(cell))
    if case["api"] == "ghost":
        L = float(cell[0, 0, 0])
        st["pos"] = pos - L * np.floor(pos / L)
        st["gpos"], own_of = _ghosts(st["pos"], L, case["rc"])
        st["gtyp"] = typ[own_of]
    if case["api"] == "host":               # pinned result arrays, reused from call to call
        st["e"] = torch.zeros(len(cell), dtype=torch.float64).pin_memory().numpy()
        st["f"] = torch.zeros(len(pos), 3, dtype=torch.float64).pin_memory().numpy()
        st["pos"] = torch.from_numpy(st["pos"]).pin_memory().numpy()
    if case["api"].startswith("train"):     # labels as at the start of a training run
        st["e_ref"] = rng.normal(0.0, 0.3, len(cell)) * np.diff(off)
        st["f_ref"] = rng.normal(0.0, 1.0, (len(pos), 3))
    if case["api"] in ("device", "train"):
        for k in ("off", "pos", "typ", "cell") + (("e_ref", "f_ref") if case["api"] == "train" else ()):
            st[k] = torch.from_numpy(st[k]).cuda()
        st["e"] = torch.zeros(len(cell), dtype=torch.float64, device="cuda")
        st["f"] = torch.zeros(len(pos), 3, dtype=torch.float64, device="cuda")
        if case["api"] == "train":
            st["loss"] = torch.zeros(1, dtype=torch.float64, device="cuda")
            st["grad"] = torch.zeros(nn.nparams(), dtype=torch.float64, device="cuda")
    return st


W_FORCE = 0.1


def run(st):
    nn, api = st["nn"], st["api"]
    f32 = np.float32
    if api == "device":
        nn.compute_device(st["off"].data_ptr(), st["pos"].data_ptr(), st["typ"].data_ptr(), st["cell"].data_ptr(), st["S"],
                          st["e"].data_ptr(), st["f"].data_ptr(), pbc=st["pbc"])
        with torch.cuda.stream(st["stream"]):
            return {"energy": st["e"].float(), "forces": st["f"].float()}
    if api == "host":
        e, f = nn.compute_batch(st["off"], st["pos"], st["typ"], st["cell"], pbc=st["pbc"], out_e=st["e"], out_f=st["f"])
        return {"energy": e.astype(f32), "forces": f.astype(f32)}
    if api == "md":
        e, f, a, w = nn.compute_md(st["off"], st["pos"], st["typ"], st["cell"], pbc=st["pbc"])
        return {"energy": e.astype(f32), "forces": f.astype(f32), "atom_energy": a.astype(f32), "virial": w.astype(f32)}
    if api == "ghost":
        e, f, a, w = nn.compute_local_ghost(st["pos"], st["typ"], st["gpos"], st["gtyp"])
        return {"energy": f32(e), "forces": f.astype(f32), "atom_energy": a.astype(f32), "virial": w.astype(f32)}
    if api == "symm":
        _, _, g = nn.compute_batch(st["off"], st["pos"], st["typ"], st["cell"], pbc=st["pbc"], energy=False, forces=False, symm=True)
        return {"symm": g.astype(f32)}
    if api == "train":
        nn.train_grad_device(st["off"].data_ptr(), st["pos"].data_ptr(), st["typ"].data_ptr(), st["cell"].data_ptr(), st["S"],
                             st["e_ref"].data_ptr(), st["f_ref"].data_ptr(), W_FORCE, st["loss"].data_ptr(), st["grad"].data_ptr())
        with torch.cuda.stream(st["stream"]):
            return {"loss": st["loss"].float(), "grad": st["grad"].float()}
    loss, g, e, f = nn.train_grad(st["off"], st["pos"], st["typ"], st["cell"], st["e_ref"], st["f_ref"], W_FORCE)
    return {"loss": f32(loss), "grad": g.astype(f32), "energy": e.astype(f32), "forces": f.astype(f32)}


# ---------------------------------------------------------------- what a pass needs

def work(case):
    """Bytes: positions, types and cells in, results out.  Operations: per pair the distance, the cutoff and
    the radial functions with their slopes; per atom the networks; the angular functions in the cheaper of
    two forms: a term for each triplet, or (GAUSS, powers zeta <= 8 of the cosine) the 81 moments of the
    neighbours' directions for each element and width, with their adjoint."""
    n, S, T = _atoms(case), case["n_struct"], case["ntypes"]
    dens = {"fcc": 4.0 / FCC_A ** 3, "cell": 64 / 8.5 ** 3}.get(case["family"], DENSITY)
    P = dens * 4.18879 * case["rc"] ** 3
    if case["family"] == "free":
        P = min(P, n - 1)
    sizes, hidden = [int(x) for x in case["ang"].split(",")], [int(x) for x in case["hid"].split(",")]
    nin = T * case["nrad"] + sum(sizes)
    nodes = [nin] + hidden + [1]
    net = sum(a * b for a, b in zip(nodes[:-1], nodes[1:]))
    grad = case["api"] != "symm"
    back = (3 if case["api"].startswith("train") else 2) if grad else 1
    nf = sum(sizes) / len(sizes)
    triplets = P * (P - 1) / 2 * (25 + 10 * nf)
    moments = P * 81 * 2 * 2 + 81 * 2 * 2 * len(sizes)
    ang = min(triplets, moments) if case["aform"] == "GAUSS" else triplets
    flops = n * (P * (10 + 8 * case["nrad"]) * back + ang * (2 * back - 1) + 2 * net * back * (2 if back == 3 else 1))
    out = 4 * nin * n if not grad else 24 * n + 8 * S
    if case["api"].startswith("train"):
        out = 8 * T * (net + sum(nodes[1:])) + 8
    return {"bytes": n * 28 + S * 72 + out, "flops": flops}


def _atoms(case):
    """Atoms of a case, by expectation."""
    if case["family"] == "fcc":
        return 4 * case["nmin"] ** 3
    a, b = case["nmin"], case["nmax"]
    return case["n_struct"] * ((b - a) / math.log(b / a) if case["family"] == "loguniform" else (a + b) / 2)


# ---------------------------------------------------------------- the path in FP64

def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Exact:
    def __init__(self, pot, off, pos, typ, cell, pbc, ghosts=None):
        self.pot, self.S, self.off = pot, len(off) - 1, off
        d = _dev()
        self.n = len(pos)
        self.typ = torch.as_tensor(np.asarray(typ), device=d).long()
        self.struct = torch.as_tensor(np.repeat(np.arange(self.S), np.diff(off)), device=d)
        gp, go = ghosts if ghosts is not None else (None, None)
        I, J, D = [], [], []
        for s in range(self.S):
            i, j, x = self._pairs(pos[off[s]:off[s + 1]], cell[s], pbc, gp)
            I.append(i + int(off[s]))
            J.append(j + int(off[s]))
            D.append(x)
        self.i, self.j, self.d = torch.cat(I), torch.cat(J), torch.cat(D)
        self.tj = (self.typ if go is None else torch.cat([self.typ, self.typ[torch.as_tensor(go, device=d)]]))[self.j]

    def _pairs(self, pos, cell, pbc, gp):
        """Ordered pairs within the cutoff: centre, neighbour, displacement x_i - x_j - image."""
        dev, rc = _dev(), self.pot.rc
        x = torch.as_tensor(np.asarray(pos), device=dev)
        y = x if gp is None else torch.cat([x, torch.as_tensor(gp, device=dev)])
        c = torch.as_tensor(np.asarray(cell), device=dev)
        inv = torch.linalg.inv(c)
        width = 1.0 / inv.norm(dim=0)
        periodic = pbc and gp is None
        nearest = periodic and bool(width.min() >= 2.0 * rc)
        shifts = torch.zeros(1, 3, dtype=torch.float64, device=dev)
        if periodic and not nearest:
            frac = x @ inv
            base = torch.floor(frac)
            x = x - base @ c
            y = x
            m = [int(math.ceil(rc / float(w))) for w in width]
            q = torch.tensor([[a, b, e] for a in range(-m[0], m[0] + 1) for b in range(-m[1], m[1] + 1)
                              for e in range(-m[2], m[2] + 1)], dtype=torch.float64, device=dev)
            shifts = q @ c
        rows = max(1, int(3e7 / (len(y) * len(shifts))))
        I, J, D = [], [], []
        for a in range(0, len(x), rows):
            d = x[a:a + rows, None, None] - y[None, :, None] - shifts
            if nearest:
                d = d - torch.round(d @ inv) @ c
            r2 = (d * d).sum(-1)
            k = torch.nonzero((r2 < rc * rc) & (r2 > 1e-12))
            I.append(k[:, 0] + a)
            J.append(k[:, 1])
            D.append(d[k[:, 0], k[:, 1], k[:, 2]])
        return torch.cat(I), torch.cat(J), torch.cat(D)

    @staticmethod
    def _cut(name, r, rc):
        f = 0.5 * (torch.cos(math.pi * r / rc) + 1.0) if name == "COS" else torch.tanh(1.0 - r / rc) ** 3
        return torch.where(r < rc, f, torch.zeros_like(f))

    def _symm(self, d, II):
        """Symmetry functions of a chunk of centres of element II; d[J]: [C, P_J, 3] displacements, padded beyond the cutoff."""
        pot, G = self.pot, []
        r = [x.square().sum(-1).sqrt() for x in d]
        u = [x / q[..., None] for x, q in zip(d, r)]
        for J in range(pot.ntypes):
            b = pot.basis_r[II][J]
            fc = self._cut(b.cut, r[J], b.rc)
            for rs, eta in zip(b.rs, b.eta):
                a = eta * (r[J] - rs)
                v = torch.exp(-a * a) if b.form == "GAUSSIAN" else 1.0 / torch.cosh(a)
                G.append((v * fc).sum(-1))
        for K in range(pot.ntypes):
            for J in range(K + 1):
                b = pot.basis_a[II][K * (K + 1) // 2 + J]
                cs = (u[J][:, :, None] * u[K][:, None]).sum(-1)
                cc = self._cut(b.cut, r[J], b.rc)[:, :, None] * self._cut(b.cut, r[K], b.rc)[:, None]
                if J == K:
                    cc = cc * 0.5 * (1.0 - torch.eye(cs.shape[1], dtype=cc.dtype, device=cc.device))
                r2 = r[J].square()[:, :, None] + r[K].square()[:, None]
                rad = {}
                for eta, zeta, lam in zip(b.eta, b.zeta, b.lam):
                    if eta not in rad:
                        if b.form == "GAUSS":
                            rad[eta] = torch.exp(-r2 / eta ** 2) * cc
                        else:
                            e = torch.exp(-0.5 * math.pi * r2 / eta ** 2)
                            rad[eta] = 2.0 * e / (1.0 + e) * cc
                    x = 0.5 + 0.5 * float(lam) * cs
                    for _ in range(int(round(math.log2(zeta)))):
                        x = x * x
                    G.append((x * rad[eta]).sum((1, 2)))
        return torch.stack(G, 1)

    def rows(self, graph):
        """Per chunk of centres of one element: (element, centres, edge indices and displacements by neighbour element, G)."""
        T = self.pot.ntypes
        key = self.i * T + self.tj
        order = torch.argsort(key, stable=True)
        cnt = torch.bincount(key, minlength=self.n * T).reshape(self.n, T)
        start = (torch.cumsum(cnt.reshape(-1), 0) - cnt.reshape(-1)).reshape(self.n, T)
        for II in range(T):
            centres = torch.nonzero(self.typ[:self.n] == II)[:, 0]
            if not len(centres):
                continue
            P = int(cnt[centres].sum(1).max()) + T
            nf = sum(b.size for b in self.pot.basis_a[II])
            step = max(1, int((3e10 if _dev() == "cuda" else 2e9) / (8.0 * P * P * (4 * nf if graph else 12) + 1)))
            for a in range(0, len(centres), step):
                c = centres[a:a + step]
                edge, disp = [], []
                for J in range(T):
                    k = torch.arange(max(1, int(cnt[c, J].max())), device=c.device)
                    ok = k[None] < cnt[c, J][:, None]
                    e = order[torch.where(ok, start[c, J][:, None] + k[None], torch.zeros_like(ok, dtype=torch.long))] if len(order) else torch.zeros_like(ok, dtype=torch.long)
                    far = torch.tensor([3.0 * self.pot.rc, 0.0, 0.0], dtype=torch.float64, device=c.device)
                    x = torch.where(ok[..., None], self.d[e], far) if len(order) else far.expand(*ok.shape, 3)
                    edge.append((e, ok))
                    disp.append(x.clone().requires_grad_(graph))
                with torch.set_grad_enabled(graph):
                    yield II, c, edge, disp, self._symm(disp, II)

    def net(self, II, G, params=None):
        """Energies of rows G by element II's network."""
        nn = self.pot.nets[II]
        t = lambda v: torch.as_tensor(v, device=G.device)  # noqa: E731
        b, w = params if params is not None else ([t(v) for v in nn.b], [t(v) for v in nn.w])
        x = t(nn.inpw) * (G + t(nn.inpb))
        for l in range(len(b)):
            x = x @ w[l].T + b[l]
            if l < len(b) - 1:
                x = torch.tanh(x) if nn.neuron == "TANH" else torch.sigmoid(x)
        return t(nn.outb)[0] + t(nn.outw)[0] * x[:, 0]

    def energy_forces(self):
        dev = _dev()
        nall = max(self.n, int(self.j.max()) + 1 if len(self.j) else 0)
        E, F = torch.zeros(self.S, dtype=torch.float64, device=dev), torch.zeros(nall, 3, dtype=torch.float64, device=dev)
        A, W = torch.zeros(self.n, dtype=torch.float64, device=dev), torch.zeros(self.S, 9, dtype=torch.float64, device=dev)
        for II, c, edge, disp, G in self.rows(True):
            e = self.net(II, G)
            g = torch.autograd.grad(e.sum(), disp)
            A[c] = e.detach()
            for (k, ok), x, gx in zip(edge, disp, g):
                gx = torch.where(ok[..., None], gx, torch.zeros_like(gx))
                F.index_add_(0, c, -gx.sum(1))
                if len(self.j):
                    F.index_add_(0, self.j[k].reshape(-1), gx.reshape(-1, 3))
                W.index_add_(0, self.struct[c], -(gx[..., :, None] * x.detach()[..., None, :]).sum(1).reshape(-1, 9))
        E.index_add_(0, self.struct, A)
        return E, F, A, W.reshape(-1, 3, 3)

    def train(self, e_ref, f_ref, wf):
        """Loss, gradient (per element: biases by layer, then the weights column by column), energies, forces."""
        E, F, _, _ = self.energy_forces()
        dev = E.device
        nat = torch.bincount(self.struct, minlength=self.S).double()
        dE, dF = E - torch.as_tensor(e_ref, device=dev), F - torch.as_tensor(f_ref, device=dev)
        per = torch.zeros(self.S, dtype=torch.float64, device=dev).index_add_(0, self.struct, dF.square().sum(1))
        loss = (0.5 * (dE / nat).square() + wf * 0.5 / (3 * nat) * per).sum() / self.S
        gE = (dE / nat ** 2 / self.S)[self.struct]
        V = wf * dF / (3 * nat[self.struct] * self.S)[:, None]
        nets = [([torch.as_tensor(v, device=dev).requires_grad_() for v in nn.b], [torch.as_tensor(v, device=dev).requires_grad_() for v in nn.w])
                for nn in self.pot.nets]
        grad = [[torch.zeros_like(v) for v in b + w] for b, w in nets]
        for II, c, edge, disp, G in self.rows(False):
            dv = [torch.where(ok[..., None], V[c][:, None] - V[self.j[k]], torch.zeros(1, dtype=torch.float64, device=dev)) for k, ok in edge]
            _, C = torch.func.jvp(lambda *x: self._symm(x, II), tuple(x.detach() for x in disp), tuple(dv))
            g = G.detach().requires_grad_()
            with torch.enable_grad():
                e = self.net(II, g, nets[II])
                dg, = torch.autograd.grad(e.sum(), g, create_graph=True)
                part = torch.autograd.grad((gE[c] * e).sum() - (dg * C).sum(), nets[II][0] + nets[II][1], allow_unused=True)
            for t, p in zip(grad[II], part):
                if p is not None:
                    t += p
        flat = [(t if t.dim() == 1 else t.T).reshape(-1) for ts in grad for t in ts]
        return loss, torch.cat(flat), E, F


EXACT_ATOMS = 150_000     # beyond this the FP64 restatement takes too long


def exact(case, seed):
    pot, _ = _potential(case)
    rng = np.random.default_rng(seed)
    off, pos, typ, cell = _cells(case, rng)
    if len(pos) > EXACT_ATOMS:
        return None
    if case["api"] == "ghost":
        L = float(cell[0, 0, 0])
        pos = pos - L * np.floor(pos / L)
        e, f, a, w = _Exact(pot, off, pos, typ, cell, False, _ghosts(pos, L, case["rc"])).energy_forces()
        f = torch.nn.functional.pad(f, (0, 0, 0, len(pos) + len(_ghosts(pos, L, case["rc"])[0]) - len(f)))
        return {"energy": e[0], "forces": f, "atom_energy": a, "virial": w[0]}
    X = _Exact(pot, off, pos, typ, cell, case["family"] != "free")
    if case["api"] == "symm":
        G = torch.zeros(len(pos), (max(pot.n_input(t) for t in range(pot.ntypes)) + 3) & ~3, dtype=torch.float64, device=_dev())
        for _, c, _, _, g in X.rows(False):
            G[c, :g.shape[1]] = g
        return {"symm": G}
    if case["api"].startswith("train"):
        e_ref = rng.normal(0.0, 0.3, len(cell)) * np.diff(off)
        f_ref = rng.normal(0.0, 1.0, (len(pos), 3))
        loss, g, e, f = X.train(e_ref, f_ref, W_FORCE)
        if case["api"] == "train":
            return {"loss": loss.reshape(1), "grad": g}
        return {"loss": loss, "grad": g, "energy": e, "forces": f}
    e, f, a, w = X.energy_forces()
    return {"energy": e, "forces": f, "atom_energy": a, "virial": w} if case["api"] == "md" else {"energy": e, "forces": f}
