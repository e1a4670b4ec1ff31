"""The order of equal keys in nrg_prepare_basis against the exchange sort itself (module.F90:531-602:
for every i, for every j > i, swap when the key at j is smaller), swap by swap, on the CPU."""
import numpy as np
import pytest

from nrg_b200 import prepare_basis


def _exchange_sort(rec, nkey):
    rec = [tuple(r) for r in rec.tolist()]
    for i in range(len(rec)):
        for j in range(i + 1, len(rec)):
            if rec[j][:nkey] < rec[i][:nkey]:
                rec[i], rec[j] = rec[j], rec[i]
    return np.array(rec, dtype=np.int32)


@pytest.mark.parametrize("nb_old", [1, 2, 3, 7, 16, 33])
@pytest.mark.parametrize("distinct", [1, 2, 3])   # quantum-number changes among the operations
@pytest.mark.parametrize("n_ops", [2, 3, 4, 9])
def test_ties_are_ordered_as_by_the_swaps(nb_old, distinct, n_ops):
    rng = np.random.default_rng(100 * nb_old + 10 * distinct + n_ops)
    nVar = 2
    ops = rng.integers(-1, 2, size=(distinct, nVar))[rng.integers(0, distinct, size=n_ops)].astype(np.int32)
    ops = np.hstack([ops, np.zeros((n_ops, 1), dtype=np.int32)])
    bo = np.zeros((nb_old, nVar + 3), dtype=np.int32)
    bo[:, :nVar] = rng.integers(-1, 2, size=(nb_old, nVar))
    bo[:, nVar] = np.arange(1, nb_old + 1)
    bi, _ = prepare_basis(ops, nVar, bo)
    rec = []
    for i in range(nb_old):
        for a in range(n_ops):
            rec.append(list(bo[i, :nVar] - ops[a, :nVar]) + [i + 1, bo[i, nVar], a + 1])
    assert np.array_equal(bi, _exchange_sort(np.array(rec, dtype=np.int32), nVar + 1))
