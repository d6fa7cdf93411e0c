"""Tensor-core networks of one and of three hidden layers (register plans of their
own): BF16X3 against FP32 networks with one to four tiles in flight per SM.
Tolerances as for two hidden layers: ~16 significant bits of operands of order 1,
2e-5 eV/atom, 2e-4 eV/A."""
import numpy as np
import pytest

from ace_b200 import NNP, potential, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden", [[[32]], [[64], [7]], [[24, 24, 24]], [[33, 9, 17], [16, 48, 16]]], ids=str)
@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("n_struct", [1, 120, 330])
def test_layer_counts(tmp_path, hidden, n_struct, precision):
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
    nn.set_precision(precision)
    E, F = nn.compute_batch(b.atom_off, b.pos, b.type, b.cell)
    nn.close()
    # BF16 alone: 8 bits instead of 16
    scale = 1.0 if precision == 2 else 256.0
    assert (np.abs(E - E0) / 201).max() < 2e-5 * scale and np.abs(F - F0).max() < 2e-4 * scale
    assert np.abs(F - F0).max() > 0                             # the tensor cores ran
