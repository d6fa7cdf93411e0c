"""Moment form of the GAUSS angular functions (ace_b200/csrc/nnp_moments.cuh).

CPU: the component numbering, the monic harmonics with their factors, the
Legendre coefficients and the gradient formulas of the kernels, restated here,
against the pair sums they replace, and the shared-memory layout's bounds.

GPU: symmetry functions and forces of the kernels against the FP64 oracle over
the sizes that set the code's shape: largest zeta (row length, odd and even
component counts), damping factors, elements, radial functions, neighbour
counts around the 32-row chunk, a structure with one neighbour of an element
(no pair); and the forms for many atoms (thread per atom, two atoms per warp)
against the small call on some of the batch's structures.  Tolerances as for the FP32 path (G 2e-5 of the row's largest,
energies 2e-6 eV/atom, forces 1e-5 eV/A times the networks' input scale, which
is 1 here)."""
import math

import numpy as np
import pytest

from ace_b200 import NNP, potential, synth
from oracle import oracle as orc


def m0(L):
    return (L + 2) & ~1


def base(L, m):
    return m0(L) + 2 * ((m - 1) * (L + 1) - (m * (m - 1)) // 2)


def comps(L):
    return base(L, L) + 2


def norm(l, m):
    n, lead = (2.0 if m else 1.0), 1.0
    for q in range(l - m + 1, l + m + 1):
        n /= q
    for q in range(1, l + 1):
        lead *= (2.0 * q - 1.0) / q
    for q in range(l - m + 1, l + 1):
        lead *= q
    return math.sqrt(n) * lead


def monic(L, m, z):
    """Q_lm(z) for l = m .. L"""
    q, p, out = np.ones_like(z), np.zeros_like(z), []
    for l in range(m, L + 1):
        out.append(q)
        q, p = z * q - ((l * l - m * m) / (4 * l * l - 1) * p if l > m else 0), q
    return out


def harmonics(L, u):
    """normalised components [n, comps] and their gradients [n, comps, 3]"""
    x, y, z = u.T
    Y, G = np.zeros((len(u), comps(L))), np.zeros((len(u), comps(L), 3))
    c, s, cp, sp = np.ones_like(x), np.zeros_like(x), np.zeros_like(x), np.zeros_like(x)
    for m in range(L + 1):
        Q, R = monic(L, m, z), [np.zeros_like(z)] + monic(L, m + 1, z)
        for l in range(m, L + 1):
            q, dq, n = Q[l - m], (l - m) * R[l - m], norm(l, m)
            k = l if m == 0 else base(L, m) + 2 * (l - m)
            Y[:, k], G[:, k] = n * q * c, n * np.stack([m * q * cp, -m * q * sp, dq * c], 1)
            if m:
                Y[:, k + 1], G[:, k + 1] = n * q * s, n * np.stack([m * q * sp, m * q * cp, dq * s], 1)
        c, s, cp, sp = c * x - s * y, s * x + c * y, c, s
    return Y, G


def degree(L):
    d = np.full(comps(L), -1)
    d[:L + 1] = np.arange(L + 1)
    for m in range(1, L + 1):
        for l in range(m, L + 1):
            d[base(L, m) + 2 * (l - m):][:2] = l
    return d


def legendre_power(lf, zeta, L):
    c = np.zeros(L + 1)
    for k in range(zeta + 1):
        x = 0.5 ** (zeta - k) * lf ** k * math.comb(zeta, k)
        for l in range(k, -1, -2):
            t = (2 * l + 1) * math.factorial(k) / 2.0 ** ((k - l) // 2) / math.factorial((k - l) // 2)
            for q in range(k + l + 1, 1, -2):
                t /= q
            c[l] += x * t
    return c


@pytest.mark.parametrize("L", range(1, 9))
def test_components_cover_the_row_once(L):
    seen = list(range(L + 1))
    for m in range(1, L + 1):
        for l in range(m, L + 1):
            k = base(L, m) + 2 * (l - m)
            assert k % 2 == 0                      # 16-byte loads of a cos/sin pair of two factors
            seen += [k, k + 1]
    assert len(set(seen)) == len(seen) == (L + 1) ** 2 and max(seen) == comps(L) - 1
    assert comps(L) % 2 == 0 and comps(L) - len(seen) in (0, 1)
    for NR in (1, 8, 16, 32):
        for ND in (1, 2, 3, 4):
            row = (comps(L) + NR + ND) | 1
            nq = (comps(L) + NR + ND + 31) // 32
            # the last component group of row 31 reads past the rows, into the factors' array
            assert 31 * row + 32 * nq <= ((32 * row + 3) & ~3) + 64 * ((ND + 1) // 2)


@pytest.mark.parametrize("zeta", [0, 1, 2, 3, 4, 5, 7, 8])
@pytest.mark.parametrize("lam", [1, -1])
def test_pair_sums_from_moments(zeta, lam):
    rng = np.random.default_rng(zeta)
    L = max(zeta, 1)
    u = rng.normal(size=(9, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    w, J = rng.uniform(0.1, 1.0, 9), np.array([0, 0, 0, 0, 1, 1, 1, 1, 1])
    Y, dY = harmonics(L, u)
    c, d = legendre_power(0.5 * lam, zeta, L), degree(L)
    cc = np.where(d >= 0, c[d], 0.0)
    A = [(w[:, None] * Y)[J == t].sum(0) for t in (0, 1)]
    f = (0.5 + 0.5 * lam * (u @ u.T)) ** zeta * np.outer(w, w)
    iu = np.triu_indices(9, 1)
    pair = {(0, 1): f[J == 0][:, J == 1].sum()}
    for t in (0, 1):
        pair[t, t] = sum(f[a, b] for a, b in zip(*iu) if J[a] == t == J[b])
    f1 = (0.5 + 0.5 * lam) ** zeta
    assert abs((cc * A[0] * A[1]).sum() - pair[0, 1]) < 1e-12
    for t in (0, 1):
        assert abs(0.5 * ((cc * A[t] * A[t]).sum() - f1 * (w[J == t] ** 2).sum()) - pair[t, t]) < 1e-12
    # gradient of e00 G00 + e01 G01 with respect to u_a, tangential part
    e00, e01, h = 0.7, -1.3, 1e-6
    B0 = cc * (e00 * A[0] + e01 * A[1])

    def energy(v):
        v = v / np.linalg.norm(v, axis=1)[:, None]
        g = (0.5 + 0.5 * lam * (v @ v.T)) ** zeta * np.outer(w, w)
        return e01 * g[J == 0][:, J == 1].sum() + e00 * sum(g[a, b] for a, b in zip(*iu) if J[a] == 0 == J[b])

    for a in range(4):
        g = w[a] * (B0[:, None] * dY[a]).sum(0)
        g -= u[a] * (u[a] @ g)
        for k in range(3):
            p, q = u.copy(), u.copy()
            p[a, k] += h
            q[a, k] -= h
            assert abs((energy(p) - energy(q)) / (2 * h) - g[k]) < 1e-7


def basis(nt, nrad, zetas, etas, cuts, rc):
    rng = np.random.default_rng(3)
    TT = nt * (nt + 1) // 2
    fs = [(e, z, l) for e in etas for z in zetas for l in (1, -1)]
    types = [potential.ElementType(name=synth.NAMES[i], energy=-1.0, mass=1.0) for i in range(nt)]
    br = [[potential.BasisR(cuts[(i + j) % len(cuts)], rc, "GAUSSIAN" if (i + j) % 2 == 0 else "SECH",
                            np.round(np.linspace(0.5, rc, nrad - j % 2 * (nrad > 1)), 6),
                            np.ones(nrad - j % 2 * (nrad > 1))) for j in range(nt)] for i in range(nt)]
    ba = [[potential.BasisA(cuts[t % len(cuts)], rc, "GAUSS", np.array([f[0] for f in fs]),
                            np.array([float(f[1]) for f in fs]), np.array([f[2] for f in fs], dtype=np.int32))
           for t in range(TT)] for _ in range(nt)]
    pot = potential.Potential(types, rc, br, ba, [])
    for i in range(nt):
        pot.nets.append(synth.xavier_net(rng, [pot.n_input(i), 12, 1]))
        pot.nets[i].inpw = np.full(pot.n_input(i), 0.25)
    return pot


# elements, radial functions, zetas, widths, cutoffs, atoms, density
SHAPES = [
    (1, 1, [1], [7.0], ["COS"], 20, 0.03),
    (1, 6, [2], [7.0], ["COS"], 33, 0.036),                      # ~32 neighbours: around one chunk
    (2, 5, [1, 3], [7.0, 14.0], ["POLY3"], 65, 0.07),            # ~64: around two
    (3, 8, [0, 4], [5.0, 7.0, 14.0], ["COS"], 40, 0.05),
    (4, 14, [5], [7.0, 14.0], ["TANH", "COS"], 60, 0.05),        # two cutoffs: four damping factors
    (2, 32, [1, 2, 7], [14.0], ["COS"], 50, 0.1),
    (5, 3, [8], [7.0], ["COS"], 30, 0.01),                       # elements with no or one neighbour
    (8, 2, [6], [9.0], ["STEP"], 120, 0.05),
    (2, 13, [1, 8], [7.0, 14.0], ["COS"], 3, 0.001),             # two or no neighbours
]


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "T%d-R%d-z%d-w%d" % (s[0], s[1], max(s[2]), len(s[3]) * len(s[4])))
def test_moment_kernels_match_oracle(tmp_path, shape):
    nt, nrad, zetas, etas, cuts, n, dens = shape
    pot = basis(nt, nrad, zetas, etas, cuts, 6.0)
    path = str(tmp_path / "pot.nnp")
    potential.write(path, pot)
    b = synth.batch_random(7, [n, max(2, n // 2), n + 5], nt, density=dens, dirichlet=False)
    op = orc.OraclePot.from_file(path)
    Eo, Fo = orc.compute_batch(op, b)
    Go = np.concatenate([orc.compute_symm(op, *b.structure(s)) for s in range(b.n_struct)])
    nn = NNP.read(path)
    assert "JitMoments" in nn.specialization()[1]
    E, F, G = nn.compute_batch(b.atom_off, b.pos, b.type, b.cell, symm=True)
    nn.set_accumulation(2)                                        # FP64 symmetry functions, the same force kernel
    E2, F2 = nn.compute_batch(b.atom_off, b.pos, b.type, b.cell)
    nn.close()
    G = G[:, :Go.shape[1]]
    assert (np.abs(G - Go).max(1) / np.maximum(np.abs(Go).max(1), 1e-30)).max() < 2e-5
    assert (np.abs(E - Eo) / np.diff(b.atom_off)).max() < 2e-6
    assert np.abs(F - Fo).max() < 1e-5 and np.abs(F2 - Fo).max() < 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [s for s in SHAPES if s[0] <= 5 and s[5] > 3] , ids=lambda s: "T%d-R%d-z%d-w%d" % (s[0], s[1], max(s[2]), len(s[3]) * len(s[4])))
def test_forms_for_many_atoms_match_the_small_call(tmp_path, shape):
    """A batch of more than 40000 atoms (an odd count) and a subset of its
    structures: the same terms in another summation order, so G within 1e-6 of
    the row's largest, energies within 1e-6 eV/atom, forces within 5e-6 eV/A."""
    nt, nrad, zetas, etas, cuts, _, dens = shape
    pot = basis(nt, nrad, zetas, etas, cuts, 6.0)
    path = str(tmp_path / "pot.nnp")
    potential.write(path, pot)
    rng = np.random.default_rng(1)
    counts = list(rng.integers(40, 400, 190))
    counts[-1] += 1 - sum(counts) % 2
    b = synth.batch_random(8, counts, nt, density=dens)
    assert b.n_atoms > 40000 and b.n_atoms % 2 == 1
    some = [0, 7, 100, 188, 189]
    sub = b.subset(some)
    nn = NNP.read(path)
    E, F, G = nn.compute_batch(b.atom_off, b.pos, b.type, b.cell, symm=True)
    Es, Fs, Gs = nn.compute_batch(sub.atom_off, sub.pos, sub.type, sub.cell, symm=True)
    nn.close()
    at = np.concatenate([np.arange(b.atom_off[s], b.atom_off[s + 1]) for s in some])
    assert (np.abs(G[at] - Gs).max(1) / np.maximum(np.abs(Gs).max(1), 1e-30)).max() < 1e-6
    assert (np.abs(E[some] - Es) / np.diff(sub.atom_off)).max() < 1e-6
    assert np.abs(F[at] - Fs).max() < 5e-6


@pytest.mark.gpu
@pytest.mark.parametrize("n", [16000, 16033, 40000, 40033])
@pytest.mark.parametrize("shape", [(1, 20, [8], [9.0]), (2, 3, [3, 8], [7.0]), (3, 5, [1, 8], [7.0, 14.0]), (4, 4, [2, 8], [7.0, 14.0])],
                         ids=lambda s: "T%d" % s[0])
def test_thread_forms_at_their_limits(tmp_path, shape, n):
    """The fewest atoms of the thread-per-atom kernels (symmetry functions, then
    forces too) and a last group of one row, elements in every proportion (blocks without pairs, of few pairs, lists
    of one element), forces also with the virial (a warp per atom reads what a
    thread per atom wrote); tolerances as above."""
    nt, nrad, zetas, etas = shape
    pot = basis(nt, nrad, zetas, etas, ["COS"], 6.0)
    path = str(tmp_path / "pot.nnp")
    potential.write(path, pot)
    rng = np.random.default_rng(2)
    counts = [1, 2, 5] + list(rng.integers(20, 300, 400))
    counts = counts[:int(np.searchsorted(np.cumsum(counts), n))]
    counts.append(n - sum(counts))
    b = synth.batch_random(8, counts, nt, density=0.05)
    assert b.n_atoms == n
    some = [0, 1, 2, 9, len(counts) - 2, len(counts) - 1]
    sub = b.subset(some)
    nn = NNP.read(path)
    E, F, G = nn.compute_batch(b.atom_off, b.pos, b.type, b.cell, symm=True)
    Em, Fm, _, Wm = nn.compute_md(b.atom_off, b.pos, b.type, b.cell)
    Es, Fs, Gs = nn.compute_batch(sub.atom_off, sub.pos, sub.type, sub.cell, symm=True)
    _, _, _, Ws = nn.compute_md(sub.atom_off, sub.pos, sub.type, sub.cell)
    nn.close()
    at = np.concatenate([np.arange(b.atom_off[s], b.atom_off[s + 1]) for s in some])
    assert (np.abs(G[at] - Gs).max(1) / np.maximum(np.abs(Gs).max(1), 1e-30)).max() < 1e-6
    assert (np.abs(E[some] - Es) / np.diff(sub.atom_off)).max() < 1e-6
    assert np.abs(F[at] - Fs).max() < 5e-6 and np.abs(F - Fm).max() < 5e-6
    assert (np.abs(Wm[some] - Ws).reshape(len(some), -1).max(1) / np.diff(sub.atom_off)).max() < 5e-5


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 20, [8], [9.0]), (2, 3, [3, 8], [7.0]), (3, 5, [1, 8], [7.0, 14.0]), (4, 4, [2, 8], [7.0, 14.0])],
                         ids=lambda s: "T%d" % s[0])
def test_training_gradient_from_moments(tmp_path, shape):
    """Tangent symmetry functions of a thread per atom (16033 atoms, blocks of no
    and of few pairs) against the generic pair loops: the gradient within 1e-5 of
    its largest entry (FP32 rows to 2e-5 of their largest value, summed over
    atoms)."""
    nt, nrad, zetas, etas = shape
    pot = basis(nt, nrad, zetas, etas, ["COS"], 6.0)
    path = str(tmp_path / "pot.nnp")
    potential.write(path, pot)
    rng = np.random.default_rng(2)
    counts = [1, 2, 5] + list(rng.integers(20, 300, 400))
    counts = counts[:int(np.searchsorted(np.cumsum(counts), 16033))]
    counts.append(16033 - sum(counts))
    b = synth.batch_random(8, counts, nt, density=0.05)
    e_ref, f_ref = rng.normal(0, 1, len(counts)), rng.normal(0, 1, (b.n_atoms, 3))
    nn = NNP.read(path)
    loss, g, _, _ = nn.train_grad(b.atom_off, b.pos, b.type, b.cell, e_ref, f_ref, 0.5)
    nn.set_specialization(False)
    loss0, g0, _, _ = nn.train_grad(b.atom_off, b.pos, b.type, b.cell, e_ref, f_ref, 0.5)
    nn.close()
    assert abs(loss - loss0) < 1e-5 * abs(loss0)
    assert np.abs(g - g0).max() < 1e-5 * np.abs(g0).max()
