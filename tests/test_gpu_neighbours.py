"""Neighbour lists against the oracle, count for count: per atom and
element, the neighbours found by the cell-list search (nnp_neighbor_counts
after a compute call) equal the oracle's list (orc_nlist: every atom and
every image within rc, the displacement test of neighbor.cpp:46-88) exactly.
The cases go through both prologue forms (one thread block for a periodic
batch of at most 2048 atoms and 32 structures, the launch sequence above),
the work items that split a big cell over several blocks (periodic
structures small enough to be one cell, seen through 27 images; a free
cluster that is one cell), triclinic shear and several elements."""
import numpy as np
import pytest

from ace_b200 import NNP, potential, synth
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def oracle_counts(rc, b, ntypes):
    out = []
    for s in range(b.n_struct):
        pos, typ, cell = b.structure(s)
        nl = orc.nlist(rc, pos, cell, pbc=b.pbc, cap=4096)
        c = np.zeros((len(pos), ntypes), np.int32)
        for i, (idx, _) in enumerate(nl):
            np.add.at(c[i], typ[idx], 1)
        out.append(c)
    return np.concatenate(out)


def batches():
    big = synth.config2(seed=31, n_struct=40, nmin=16, nmax=512)
    counts = np.diff(big.atom_off)
    k = int(max(2, min(20, np.searchsorted(np.cumsum(counts), 1800))))
    free = synth.batch_random(62, [700, 40, 1900], 3)
    return {
        "config1_cell": (1, synth.config1()),
        "mixed_one_block": (2, big.subset(range(k))),
        "mixed_launch_sequence": (2, big),
        "free_clusters": (2, synth.Batch(free.atom_off, free.pos, free.type, free.cell, pbc=False)),
    }


@pytest.mark.parametrize("name", ["config1_cell", "mixed_one_block", "mixed_launch_sequence", "free_clusters"])
def test_neighbour_counts_match_oracle(tmp_path, name):
    k, b = batches()[name]
    pot = synth.potential_config(k)
    path = str(tmp_path / "pot.nnp")
    potential.write(path, pot)
    nn = NNP.read(path)
    if b.pbc:
        nn.compute_batch(b.atom_off, b.pos, b.type, b.cell)
    else:
        nn.compute_batch(b.atom_off, b.pos, b.type, None, pbc=False)
    got = nn.neighbor_counts(b.n_atoms)
    nn.close()
    want = oracle_counts(pot.rc, b, len(pot.types))
    assert got.shape == want.shape
    bad = np.argwhere(got != want)
    assert bad.size == 0, "first mismatches (atom, element): %s" % bad[:5].tolist()


def slab(n, vacuum, seed):
    """n atoms in the lower part of a cell whose upper part, `vacuum` times as high, is empty"""
    b = synth.batch_random(seed, [n], 3, shear=0.0)
    cell = b.cell.copy()
    cell[0, 2, 2] *= 1.0 + vacuum
    return synth.Batch(b.atom_off, b.pos, b.type, cell, True)


@pytest.mark.parametrize("n, free", [(600, False), (3000, False), (2600, True)])
def test_empty_cells_have_no_candidates(tmp_path, n, free):
    """Cells without atoms, in the one-block prologue (600 atoms), the launch
    sequence and the grid over a large free structure's box, on a handle whose
    previous batch had atoms in every cell: the counts of the earlier batch
    must not be seen."""
    pot = synth.potential_config(2)
    path = str(tmp_path / "pot.nnp")
    potential.write(path, pot)
    nn = NNP.read(path)
    full = synth.batch_random(5, [4 * n], 3)
    nn.compute_batch(full.atom_off, full.pos, full.type, full.cell)
    b = slab(n, 2.0, 6)
    if free:
        b = synth.Batch(b.atom_off, b.pos, b.type, b.cell, pbc=False)
        nn.compute_batch(b.atom_off, b.pos, b.type, None, pbc=False)
    else:
        nn.compute_batch(b.atom_off, b.pos, b.type, b.cell)
    got = nn.neighbor_counts(b.n_atoms)
    nn.close()
    assert np.array_equal(got, oracle_counts(pot.rc, b, 3))


@pytest.mark.parametrize("n, shift", [(512, 0.0), (513, 0.0), (300, 5000.0), (700, -3000.0)])
def test_free_structures_around_the_grid_limit(tmp_path, n, shift):
    """Free structures up to 512 atoms are one cell, larger ones searched
    through a grid; far from the origin the candidates' FP32 box test has its
    coordinates rounded to 2^-12 A."""
    pot = synth.potential_config(2)
    path = str(tmp_path / "pot.nnp")
    potential.write(path, pot)
    b = synth.batch_random(17, [n, 5], 3)
    b = synth.Batch(b.atom_off, b.pos + shift, b.type, b.cell, pbc=False)
    nn = NNP.read(path)
    nn.compute_batch(b.atom_off, b.pos, b.type, None, pbc=False)
    got = nn.neighbor_counts(b.n_atoms)
    nn.close()
    assert np.array_equal(got, oracle_counts(pot.rc, b, 3))


def brute_counts(rc, pos, typ, cell, ntypes, images):
    """Counts over wrapped positions and all images up to `images` (the oracle
    takes its range from the edges' lengths, too few for a strong shear)."""
    frac = pos @ np.linalg.inv(cell)
    q = (frac - np.floor(frac)) @ cell
    sh = np.array(list(np.ndindex(*[2 * m + 1 for m in images]))) - np.array(images)
    out = np.zeros((len(pos), ntypes), np.int32)
    for i in range(len(pos)):
        r2 = ((q[i] - (q[None] + (sh @ cell)[:, None])) ** 2).sum(-1)
        np.add.at(out[i], typ[np.nonzero((r2 < rc * rc) & (r2 > 1e-12))[1]], 1)
    return out


def test_thin_and_skewed_cells(tmp_path):
    """A cell thinner than the cutoff (many images) and a strongly sheared one."""
    pot = synth.potential_config(2)
    path = str(tmp_path / "pot.nnp")
    potential.write(path, pot)
    rng = np.random.default_rng(3)
    cells = np.array([np.diag([2.2, 14.0, 30.0]), [[15.0, 0, 0], [9.0, 13.0, 0], [-8.0, 7.0, 14.0]]])
    off = np.array([0, 40, 170])
    pos = np.concatenate([rng.uniform(0, 1, (40, 3)) @ cells[0], rng.uniform(-1, 2, (130, 3)) @ cells[1]])
    b = synth.Batch(off, pos, rng.integers(0, 3, 170).astype(np.int32), cells, True)
    nn = NNP.read(path)
    nn.compute_batch(b.atom_off, b.pos, b.type, b.cell)
    got = nn.neighbor_counts(b.n_atoms)
    nn.close()
    want = np.concatenate([brute_counts(pot.rc, *b.structure(s), 3, m) for s, m in ((0, (4, 2, 2)), (1, (3, 3, 3)))])
    assert np.array_equal(got, want)


@pytest.mark.parametrize("n, side", [(38, 6.0), (96, 8.2), (150, 9.5), (9, 3.7)])
def test_candidate_lists_longer_than_the_buffers(tmp_path, n, side):
    """Dense cells one cell wide: candidate lists that end inside a round of 256, longer
    than the segment window (1024) and with more kept candidates than the list
    holds (640), segments short and long.  In the 6 A cell every atom's own images
    lie at the cutoff itself, where the rounding of either side decides: counts
    between those at rc -+ 1e-10, which are equal for the other cells."""
    pot = synth.potential_config(2)
    path = str(tmp_path / "pot.nnp")
    potential.write(path, pot)
    rng = np.random.default_rng(5)
    cells = np.array([np.eye(3) * side, np.eye(3) * side])
    pos = rng.uniform(0, side, (2 * n, 3))
    typ = np.concatenate([rng.integers(0, 3, n), np.zeros(n)]).astype(np.int32)
    b = synth.Batch(np.array([0, n, 2 * n]), pos, typ, cells, True)
    low, high = (np.concatenate([brute_counts(pot.rc + d, *b.structure(s), 3, (3, 3, 3)) for s in (0, 1)])
                 for d in (-1e-10, 1e-10))
    assert np.array_equal(low, high) == (side != pot.rc)
    nn = NNP.read(path)
    nn.compute_batch(b.atom_off, b.pos, b.type, b.cell)
    got = nn.neighbor_counts(b.n_atoms)
    nn.close()
    assert (low <= got).all() and (got <= high).all()
