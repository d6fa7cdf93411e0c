"""Handles of one potential share their loaded kernels: created, used and closed from
several threads at once and in any order, with other neighbour capacities and sizes,
each gives the results of a handle of its own."""
import threading

import numpy as np
import pytest

from ace_b200 import NNP, potential, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pot", [synth.potential_config(2), synth.potential_forms("forms_logistic_sech")], ids=["moments", "pairs"])
def test_handles_in_threads(tmp_path, pot):
    path = str(tmp_path / "pot.nnp")
    potential.write(path, pot)
    nt = pot.ntypes
    batches = [synth.batch_random(s, [60] * n, nt, density=d) for s, (n, d) in enumerate([(3, 0.05), (8, 0.02), (150, 0.05), (20, 0.09)])]
    want = []
    for b in batches:
        nn = NNP.read(path)
        want.append(nn.compute_batch(b.atom_off, b.pos, b.type, b.cell))
        nn.close()
    errors = []

    def work(k):
        try:
            for r in range(4):
                nn = NNP.read(path)
                for q in range(3):
                    b, w = batches[(k + q + r) % 4], want[(k + q + r) % 4]
                    e, f = nn.compute_batch(b.atom_off, b.pos, b.type, b.cell)
                    # the same terms (a larger capacity changes no list); FP64 atomics may reorder
                    assert np.abs(e - w[0]).max() < 1e-9 and np.abs(f - w[1]).max() < 1e-9
                nn.close()
        except BaseException as ex:
            errors.append(ex)

    th = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not errors, errors
