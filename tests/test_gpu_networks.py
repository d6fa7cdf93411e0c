"""FP32 network tiles against the oracle at the shapes that set their code:
no hidden layer up to four, widths around the 2- and 4-neuron register blocks
and their limits (1, 32, 33, 64, 65, 128), tiles of 32 atoms with remainders, an
element without atoms, elements with different networks.  Tolerances of the
FP32 path: energies 2e-6 eV/atom, forces 1e-5 eV/A."""
import numpy as np
import pytest

from ace_b200 import NNP, potential, synth
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

NETS = [[[]], [[1]], [[33], [5]], [[32, 64], [65, 7]], [[128]], [[17, 40, 9], [20, 20, 20]], [[12, 13, 14, 15], [16]],
        [[20, 20], [20, 20], [20, 20]]]


@pytest.mark.parametrize("hidden", NETS, ids=str)
@pytest.mark.parametrize("counts", [[1, 30, 33], [64, 97, 160]], ids=str)
def test_network_tiles_match_oracle(tmp_path, hidden, counts):
    nt = len(hidden)
    pot = synth.make_potential(nt, 5.0, 5, [4] * (nt * (nt + 1) // 2), [4], 3)
    rng = np.random.default_rng(4)
    for i, h in enumerate(hidden):
        pot.nets[i] = synth.xavier_net(rng, [pot.n_input(i)] + h + [1], ["TANH", "SIGMOID", "SOFTPLUS"][i])
        pot.nets[i].inpw = np.full(pot.n_input(i), 0.25)
        pot.nets[i].outw, pot.nets[i].outb = np.array([1.5]), np.array([-0.5])
    path = str(tmp_path / "pot.nnp")
    potential.write(path, pot)
    b = synth.batch_random(9, counts, max(nt - 1, 1))          # the last of several elements has no atoms
    Eo, Fo = orc.compute_batch(orc.OraclePot.from_file(path), b)
    nn = NNP.read(path)
    E, F, G = nn.compute_batch(b.atom_off, b.pos, b.type, b.cell, symm=True)
    assert (np.abs(E - Eo) / np.diff(b.atom_off)).max() < 2e-6 and np.abs(F - Fo).max() < 1e-5
    # energies from the symmetry functions alone, after a call on other atoms and with ghosts
    nn.compute_local_ghost(b.pos[:5], b.type[:5], b.pos[5:20], b.type[5:20])
    s = slice(int(b.atom_off[2]), int(b.atom_off[3]))
    vac = sum(pot.types[t].energy for t in b.type[s])
    assert abs(nn.compute_energy(b.type[s], G[s]) - vac - E[2]) < 2e-6 * counts[2] + 1e-6 * abs(vac)
    nn.close()


@pytest.mark.parametrize("hidden", [[[32, 32]], [[48, 48], [16]], [[64, 64], [20, 20], [7, 33, 9]]], ids=str)
@pytest.mark.parametrize("n_struct", [1, 120, 330])
def test_tensor_core_tiles_in_flight(tmp_path, hidden, n_struct):
    """One to four tiles of 128 atoms in flight per SM, elements with different
    layer counts, the last element's last tile ragged: BF16X3 against FP32
    networks.  ~16 significant bits of operands of order 1 through two or three
    layers: 2e-5 eV/atom, 2e-4 eV/A as against the reference's outputs."""
    nt = len(hidden)
    pot = synth.make_potential(nt, 4.5, 16, [8] * (nt * (nt + 1) // 2), [4], 3)
    rng = np.random.default_rng(6)
    for i, h in enumerate(hidden):
        pot.nets[i] = synth.xavier_net(rng, [pot.n_input(i)] + h + [1], "TANH")
        pot.nets[i].inpw = np.full(pot.n_input(i), 0.25)
    path = str(tmp_path / "pot.nnp")
    potential.write(path, pot)
    b = synth.batch_random(3, [201] * n_struct, nt)
    nn = NNP.read(path)
    E0, F0 = nn.compute_batch(b.atom_off, b.pos, b.type, b.cell)
    nn.set_precision(2)
    E, F = nn.compute_batch(b.atom_off, b.pos, b.type, b.cell)
    assert (np.abs(E - E0) / 201).max() < 2e-5 and np.abs(F - F0).max() < 2e-4
    assert np.abs(F - F0).max() > 0                             # the tensor cores ran
    nn.close()
