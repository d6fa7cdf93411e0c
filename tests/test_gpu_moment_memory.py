"""Device memory of the moments (nnp_set_moment_memory): a batch that needs more is
worked off part by part, an allocation that fails is remembered, and with too
little for a useful part the pair kernels run.  Results against a handle without
limit: the same terms, so energies and forces within 1e-9 where the same kernels
run on each atom, else the tolerances between the kernels' forms (G 1e-6 of the
row's largest, energies 1e-6 eV/atom, forces 5e-6 eV/A)."""
import numpy as np
import pytest
import torch

from ace_b200 import NNP, potential, synth

pytestmark = pytest.mark.gpu

ROW = 3 * 82 * 8 + 16 + 8 + 6 * 8      # three elements, one pair of damping factors, zeta up to 8


def handles(tmp_path):
    pot = synth.potential_config(2)
    path = str(tmp_path / "pot.nnp")
    potential.write(path, pot)
    out = []
    for _ in range(2):
        nn = NNP.read(path)
        s = torch.cuda.Stream()
        nn.set_stream(s.cuda_stream)
        nn.set_autotune(False)
        out.append((nn, s))
    return out


def same(a, b, n, tol_e=1e-9, tol_f=1e-9):
    assert (np.abs(a[0] - b[0]) / n).max() < tol_e and np.abs(a[1] - b[1]).max() < tol_f


@pytest.mark.parametrize("mode", [0, 2])
@pytest.mark.parametrize("rows", [1024, 1100, 2999, 3000])
def test_small_batch_in_parts(tmp_path, rows, mode):
    (nn, _), (ref, _) = handles(tmp_path)
    b = synth.batch_random(3, [100] * 30, 3)
    n = np.diff(b.atom_off)
    nn.set_moment_memory(rows * ROW)
    nn.set_accumulation(mode)
    ref.set_accumulation(mode)
    rng = np.random.default_rng(1)
    pos = b.pos
    for _ in range(5):                                            # eager, captured, replayed
        pos = pos + rng.normal(0, 0.01, pos.shape)
        same(nn.compute_batch(b.atom_off, pos, b.type, b.cell), ref.compute_batch(b.atom_off, pos, b.type, b.cell), n)
    e, f, _, w = nn.compute_md(b.atom_off, pos, b.type, b.cell)
    e0, f0, _, w0 = ref.compute_md(b.atom_off, pos, b.type, b.cell)
    same((e, f), (e0, f0), n)
    assert np.abs(w - w0).max() < 1e-6
    nn.close()
    ref.close()


@pytest.mark.parametrize("rows", [17000, 20000, 33333])
def test_large_batch_in_parts(tmp_path, rows):
    """parts of a thread per atom, a last one of a warp per atom, the order by neighbour counts"""
    (nn, _), (ref, _) = handles(tmp_path)
    b = synth.batch_random(4, [201] * 250, 3)
    n = np.diff(b.atom_off)
    nn.set_moment_memory(rows * ROW)
    for _ in range(3):
        e, f, g = nn.compute_batch(b.atom_off, b.pos, b.type, b.cell, symm=True)
        e0, f0, g0 = ref.compute_batch(b.atom_off, b.pos, b.type, b.cell, symm=True)
        same((e, f), (e0, f0), n, 1e-6, 5e-6)
        assert (np.abs(g - g0).max(1) / np.abs(g0).max(1)).max() < 1e-6
    nn.close()
    ref.close()


def test_failed_allocation_is_remembered(tmp_path):
    """12000 atoms' worth of memory for 50250: parts of a quarter, call after call with
    the same memory, and the step still replays"""
    (nn, _), (ref, _) = handles(tmp_path)
    b = synth.batch_random(4, [201] * 250, 3)
    n = np.diff(b.atom_off)
    ref.set_graphs(False)
    nn.set_moment_memory(8 << 30, 13000 * ROW)
    free, launches = [], []
    for _ in range(6):
        l0 = nn.launch_count()
        same(nn.compute_batch(b.atom_off, b.pos, b.type, b.cell), ref.compute_batch(b.atom_off, b.pos, b.type, b.cell), n, 1e-6, 5e-6)
        free.append(torch.cuda.mem_get_info()[0])
        launches.append(nn.launch_count() - l0)
    assert len(set(free[2:])) == 1 and len(set(launches[1:])) == 1
    rng = np.random.default_rng(1)
    e_ref, f_ref = rng.normal(0, 1, b.n_struct), rng.normal(0, 1, (b.n_atoms, 3))
    loss, g, _, _ = nn.train_grad(b.atom_off, b.pos, b.type, b.cell, e_ref, f_ref, 0.5)
    loss0, g0, _, _ = ref.train_grad(b.atom_off, b.pos, b.type, b.cell, e_ref, f_ref, 0.5)
    assert abs(loss - loss0) < 1e-5 * abs(loss0) and np.abs(g - g0).max() < 1e-5 * np.abs(g0).max()
    nn.close()
    ref.close()


def test_pair_kernels_without_moments(tmp_path):
    (nn, _), (ref, _) = handles(tmp_path)
    b = synth.batch_random(3, [100] * 30, 3)
    n = np.diff(b.atom_off)
    nn.set_moment_memory(0)
    ref.set_specialization(False)
    for _ in range(4):
        same(nn.compute_batch(b.atom_off, b.pos, b.type, b.cell), ref.compute_batch(b.atom_off, b.pos, b.type, b.cell), n)
    nn.set_moment_memory()                                        # and back
    ref.set_specialization(True)
    for _ in range(2):
        same(nn.compute_batch(b.atom_off, b.pos, b.type, b.cell), ref.compute_batch(b.atom_off, b.pos, b.type, b.cell), n)
    nn.close()
    ref.close()
