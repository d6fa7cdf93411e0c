"""A replayed call takes its sizes from its own arguments, whatever ran on the
handle in between: a device batch is called until its graph replays, then
nnp_compute_energy_symm runs on another structure (which has its own numbers of
atoms and structures and drops no graph), then the batch is called again on new
positions.  Energies and forces are those of a fresh handle, and nothing is
written behind the caller's arrays."""
import numpy as np
import pytest
import torch

from ace_b200 import NNP, potential, synth
from ace_b200.nnp import NNPError

pytestmark = pytest.mark.gpu

GUARD = 4096


class Device:
    """a batch on the device, with guard words behind its result arrays"""

    def __init__(self, b):
        self.b = b
        self.off, self.typ, self.cell = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (b.atom_off, b.type, b.cell))
        self.pos = torch.from_numpy(b.pos).cuda()
        self.e = torch.full((b.n_struct + GUARD,), 7.0, dtype=torch.float64, device="cuda")
        self.f = torch.full((3 * b.n_atoms + GUARD,), 7.0, dtype=torch.float64, device="cuda")

    def call(self, nn):
        nn.compute_device(self.off.data_ptr(), self.pos.data_ptr(), self.typ.data_ptr(), self.cell.data_ptr(), self.b.n_struct,
                          self.e.data_ptr(), self.f.data_ptr())

    def results(self):
        S, N = self.b.n_struct, self.b.n_atoms
        e, f = self.e.cpu().numpy(), self.f.cpu().numpy()
        assert (e[S:] == 7.0).all() and (f[3 * N:] == 7.0).all()
        return e[:S], f[:3 * N].reshape(N, 3)


def make(tmp_path):
    pot = synth.potential_config(2)
    path = str(tmp_path / "pot.nnp")
    potential.write(path, pot)
    return path


@pytest.mark.parametrize("other", [30, 900])
def test_replay_after_energies_of_another_structure(tmp_path, other):
    path = make(tmp_path)
    rng = np.random.default_rng(4)
    b = synth.batch_random(5, rng.integers(20, 60, 6), 3)
    big = synth.batch_random(6, [300] * 4, 3)
    nn, ref = NNP.read(path), NNP.read(path)
    s = torch.cuda.Stream()
    nn.set_stream(s.cuda_stream)
    nn.set_autotune(False)
    ref.set_graphs(False)
    nn.compute_batch(big.atom_off, big.pos, big.type, big.cell)       # buffers for the largest call
    typ = rng.integers(0, 3, other).astype(np.int32)
    G = rng.uniform(0.0, 1.0, (other, nn.gstride))
    e_other = ref.compute_energy(typ, G)
    d = Device(b)
    for k in range(6):
        if k == 4:
            assert abs(nn.compute_energy(typ, G) - e_other) < 1e-6 * other
        d.pos += torch.from_numpy(rng.normal(0, 0.01, b.pos.shape)).cuda()
        torch.cuda.synchronize()
        d.call(nn)
        e, f = d.results()
        e0, f0 = ref.compute_batch(b.atom_off, d.pos.cpu().numpy(), b.type, b.cell)
        assert np.abs(e - e0).max() < 1e-9 and np.abs(f - f0).max() < 1e-9
        n = nn.neighbor_counts(b.n_atoms)
        assert (n == ref.neighbor_counts(b.n_atoms)).all()
    nn.close()
    ref.close()


def test_gradient_of_a_replayed_step(tmp_path):
    """the training step's forward pass replays too: loss and gradient take the batch's own sizes"""
    path = make(tmp_path)
    rng = np.random.default_rng(4)
    b = synth.batch_random(5, rng.integers(20, 60, 6), 3)
    e_ref, f_ref = rng.normal(0, 1, b.n_struct), rng.normal(0, 1, (b.n_atoms, 3))
    typ = rng.integers(0, 3, 30).astype(np.int32)
    G = rng.uniform(0.0, 1.0, (30, 56))
    nn, ref = NNP.read(path), NNP.read(path)
    s = torch.cuda.Stream()
    nn.set_stream(s.cuda_stream)
    nn.set_autotune(False)
    ref.set_graphs(False)
    loss0, g0, e0, f0 = ref.train_grad(b.atom_off, b.pos, b.type, b.cell, e_ref, f_ref, 0.5)
    for k in range(6):
        if k == 4:
            nn.compute_energy(typ, G)
        loss, g, e, f = nn.train_grad(b.atom_off, b.pos, b.type, b.cell, e_ref, f_ref, 0.5)
        assert abs(loss - loss0) < 1e-9 * abs(loss0) and np.abs(g - g0).max() < 1e-6 * np.abs(g0).max()
        assert np.abs(e - e0).max() < 1e-9 and np.abs(f - f0).max() < 1e-9
    nn.close()
    ref.close()


@pytest.mark.parametrize("shift", [1, 4])
def test_result_arrays_at_any_address(tmp_path, shift):
    """device results into arrays that are not aligned to doubles"""
    path = make(tmp_path)
    b = synth.batch_random(5, [30, 50], 3)
    nn = NNP.read(path)
    e0, f0 = nn.compute_batch(b.atom_off, b.pos, b.type, b.cell)
    d = Device(b)
    e = torch.zeros(8 * b.n_struct + 16, dtype=torch.uint8, device="cuda")
    f = torch.zeros(24 * b.n_atoms + 16, dtype=torch.uint8, device="cuda")
    for _ in range(4):
        nn.compute_device(d.off.data_ptr(), d.pos.data_ptr(), d.typ.data_ptr(), d.cell.data_ptr(), b.n_struct,
                          e.data_ptr() + shift, f.data_ptr() + shift)
        e1 = e.cpu().numpy()[shift:shift + 8 * b.n_struct].copy().view(np.float64)
        f1 = f.cpu().numpy()[shift:shift + 24 * b.n_atoms].copy().view(np.float64).reshape(-1, 3)
        assert np.abs(e1 - e0).max() < 1e-9 and np.abs(f1 - f0).max() < 1e-9
    nn.close()


@pytest.mark.parametrize("other", [10, 5000])
def test_neighbour_counts_are_the_last_compute_calls(tmp_path, other):
    """after energies of another structure: the same counts, or an error when its larger
    buffers replaced the lists"""
    path = make(tmp_path)
    b = synth.batch_random(5, [30, 50], 3)
    nn = NNP.read(path)
    nn.compute_batch(b.atom_off, b.pos, b.type, b.cell)
    want = nn.neighbor_counts(b.n_atoms)
    rng = np.random.default_rng(4)
    nn.compute_energy(rng.integers(0, 3, other).astype(np.int32), rng.uniform(0.0, 1.0, (other, nn.gstride)))
    if other < b.n_atoms:
        assert (nn.neighbor_counts(b.n_atoms) == want).all()
    else:
        with pytest.raises(NNPError):
            nn.neighbor_counts(b.n_atoms)
    nn.compute_batch(b.atom_off, b.pos, b.type, b.cell)
    assert (nn.neighbor_counts(b.n_atoms) == want).all()
    nn.close()
