"""Atoms whose neighbours lie to one side (an adatom over a sheet or a slab, a
cluster's tip, a free surface): there the angular functions of lambda = -1 and
large zeta are 1e-4 to 1e-8 of the (sum of the damping factors)^2 that the
moments' terms have (nnp_moments.cuh), with any number of pairs.  The inputs
are scaled by their spread over these environments, as a potential that was
trained on them has it (a spread of at least 4 % of the largest value: below,
FP32 rows of G themselves are too coarse).

Tolerances, those of the FP32 path: G within 2e-5 of each function's spread,
forces within 1e-5 eV/A of the FP64 oracle with dE/d(scaled input) below 0.1 eV,
or twice the error of the generic pair loops where those are further off; the
training gradient within 1e-5 of its largest entry of the generic pair loops
(rows to 2e-5 of the spread, summed over atoms)."""
import numpy as np
import pytest

from ace_b200 import NNP, potential, synth
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def fcc(nx, ny, nz, a):
    base = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
    g = np.stack(np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij"), -1).reshape(-1, 1, 3)
    return ((g + base) * a).reshape(-1, 3)


def sheet(rng):
    """an adatom 3.2 to 4.5 A over a graphene sheet of 24 atoms"""
    base = np.array([[0, 0], [1.23, 0.71], [1.23, 2.13], [0, 2.84]])
    g = np.stack(np.meshgrid(np.arange(3) * 2.46, np.arange(2) * 4.26, indexing="ij"), -1).reshape(-1, 1, 2)
    p = (g + base).reshape(-1, 2)
    pos = np.column_stack([p, np.full(len(p), 5.0)]) + rng.normal(0, 0.03, (len(p), 3))
    ad = [rng.uniform(0, 7.38), rng.uniform(0, 8.52), 5.0 + rng.uniform(3.2, 4.5)]
    return np.vstack([pos, ad]), np.array([0] * len(p) + [1]), np.diag([7.38, 8.52, 24.0])


def slab(rng):
    """an adatom 1.8 to 4.5 A over a (100) face of 72 atoms"""
    pos = fcc(3, 3, 2, 3.6) + rng.normal(0, 0.05, (72, 3)) + [0, 0, 2.0]
    top = pos[:, 2].max()
    ad = [rng.uniform(0, 10.8), rng.uniform(0, 10.8), top + rng.uniform(1.8, 4.5)]
    return np.vstack([pos, ad]), np.array([0] * 72 + [1]), np.diag([10.8, 10.8, 24.0])


def tip(rng):
    """a pyramid with its tip a second element, in a large cell"""
    p = fcc(6, 6, 3, 3.6)
    p = p - p.mean(0)
    h = p[:, 2].max() - p[:, 2]
    p = p[np.abs(p[:, :2]).max(1) <= 0.8 * h + 0.1]
    ad = [0.0, 0.0, p[:, 2].max() + rng.uniform(1.8, 2.6)]
    pos = np.vstack([p, ad])
    return pos + rng.normal(0, 0.06, pos.shape), np.array([0] * len(p) + [1]), np.diag([36.0, 36.0, 24.0])


def surface(rng):
    """a free (111)-like face: the outermost layer is the second element"""
    pos = fcc(3, 3, 2, 3.6)
    typ = (pos[:, 2] > pos[:, 2].max() - 0.1).astype(int)
    return pos + rng.normal(0, 0.12, pos.shape) + [0, 0, 3.0], typ, np.diag([10.8, 10.8, 24.0])


KINDS = {"sheet": sheet, "slab": slab, "tip": tip, "surface": surface}


def conditioned(s, tmp_path):
    """the structures as a batch, a potential conditioned on them, the oracle's results"""
    off = np.concatenate([[0], np.cumsum([len(x[1]) for x in s])]).astype(np.int64)
    b = synth.Batch(off, np.concatenate([x[0] for x in s]), np.concatenate([x[1] for x in s]).astype(np.int32),
                    np.array([x[2] for x in s]))
    full = [(e, z, l) for e in synth.ETA_A for z in (1.0, 2.0, 4.0, 8.0) for l in (1, -1)]
    pot = synth.make_potential(2, 6.0, 8, [16, 16, 16], [12], 3)
    for row in pot.basis_a:
        for q in row:
            q.eta, q.zeta, q.lam = np.array([f[0] for f in full]), np.array([f[1] for f in full]), np.array([f[2] for f in full], dtype=np.int32)
    path = str(tmp_path / "pot.nnp")
    potential.write(path, pot)
    op = orc.OraclePot.from_file(path)
    G = np.concatenate([orc.compute_symm(op, *b.structure(k)) for k in range(len(s))])
    synth.condition(pot, G, b.type)
    for II, net in enumerate(pot.nets):
        net.inpw = np.minimum(net.inpw, 1.0 / np.maximum(0.04 * np.abs(G[b.type == II]).max(0), 1e-300))
        net.outw = np.array([0.07])
    potential.write(path, pot)
    return b, path, G, pot, orc.compute_batch(orc.OraclePot.from_file(path), b)[1]


def workload(kind, tmp_path, n=24):
    rng = np.random.default_rng(5)
    return conditioned([KINDS[kind](rng) for _ in range(n)], tmp_path)


def tiled(b, atoms):
    """the batch's structures again and again, at least that many atoms"""
    k = -(-atoms // b.n_atoms)
    return b.subset(list(range(b.n_struct)) * k), k


def errors(w, nn, atoms):
    """largest error of the scaled inputs and of the forces"""
    b, _, G, pot, Fo = w
    B, k = tiled(b, atoms) if atoms else (b, 1)
    E, F, g = nn.compute_batch(B.atom_off, B.pos, B.type, B.cell, symm=True)
    scale = np.array([net.inpw for net in pot.nets])[B.type]
    return np.array([(np.abs(g[:, :G.shape[1]] - np.tile(G, (k, 1))) * scale).max(), np.abs(F - np.tile(Fo, (k, 1))).max()])


def check(w, sizes):
    """Each size, with FP32 and with FP64 symmetry functions: the tolerances, or twice
    what the generic pair loops are off on these inputs."""
    nn = NNP.read(w[1])
    assert "JitMoments" in nn.specialization()[1]
    nn.set_specialization(False)
    bound = np.maximum([2e-5, 1e-5], 2.0 * errors(w, nn, 0))
    nn.set_specialization(True)
    for atoms in sizes:
        for mode in (0, 2):
            nn.set_accumulation(mode)
            e = errors(w, nn, atoms)
            assert (e < bound).all(), (atoms, mode, e, bound)
    nn.close()
    return bound


@pytest.mark.parametrize("kind", KINDS)
def test_one_sided_environments_match_oracle(tmp_path, kind):
    """a warp per atom, a thread per atom for the symmetry functions (16000) and for
    the forces too (40000), and the forces of FP64 symmetry functions"""
    w = workload(kind, tmp_path)
    bound = check(w, (0, 16000, 40000))
    # with the virial a warp per atom follows the marks that a thread per atom left
    b, path, _, _, Fo = w
    nn = NNP.read(path)
    B, k = tiled(b, 16000)
    _, F, _, W = nn.compute_md(B.atom_off, B.pos, B.type, B.cell)
    nn.set_specialization(False)
    _, _, _, W0 = nn.compute_md(b.atom_off, b.pos, b.type, b.cell)
    nn.close()
    assert np.abs(F - np.tile(Fo, (k, 1))).max() < bound[1]
    assert (np.abs(W - np.tile(W0, (k, 1, 1))).reshape(B.n_struct, -1).max(1) / np.diff(B.atom_off)).max() < 5e-5


@pytest.mark.parametrize("kind", KINDS)
def test_one_sided_training_gradient(tmp_path, kind):
    b, path, _, _, _ = workload(kind, tmp_path)
    B, _ = tiled(b, 16000)
    rng = np.random.default_rng(1)
    e_ref, f_ref = rng.normal(0, 1, B.n_struct), rng.normal(0, 1, (B.n_atoms, 3))
    nn = NNP.read(path)
    loss, g, _, _ = nn.train_grad(B.atom_off, B.pos, B.type, B.cell, e_ref, f_ref, 0.5)
    nn.set_specialization(False)
    loss0, g0, _, _ = nn.train_grad(B.atom_off, B.pos, B.type, B.cell, e_ref, f_ref, 0.5)
    nn.close()
    assert abs(loss - loss0) < 1e-5 * abs(loss0)
    assert np.abs(g - g0).max() < 1e-5 * np.abs(g0).max()


@pytest.mark.parametrize("n", [16, 31, 33, 70])
@pytest.mark.parametrize("nb", [0, 1, 2, 40])
def test_blocks_of_many_pairs(tmp_path, n, nb):
    """Blocks that cancel, at the edges of the 32 lanes that take one: n neighbours of
    one element and nb of the other within 35 degrees of an axis, 2 to 5.8 A from the
    centre (the other atoms see them from the inside and the rim)."""
    rng = np.random.default_rng(n + 100 * nb)
    s = []
    for _ in range(4):
        pts = np.zeros((0, 3))
        while len(pts) < n + nb:                                  # at least 0.4 A apart
            c = rng.uniform(np.cos(np.radians(35)), 1)
            ph, r = rng.uniform(0, 2 * np.pi), rng.uniform(2, 5.8)
            p = r * np.array([np.sqrt(1 - c * c) * np.cos(ph), np.sqrt(1 - c * c) * np.sin(ph), c])
            if not len(pts) or np.linalg.norm(pts - p, axis=1).min() > 0.4:
                pts = np.vstack([pts, p])
        s.append((np.vstack([[0, 0, 0], pts]) + 10.0, np.array([1] + [0] * n + [1] * nb), np.eye(3) * 40.0))
    check(conditioned(s, tmp_path), (0, 16000))
