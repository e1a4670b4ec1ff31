"""The tridiagonalisation at the edges of its plans (on chip: orders 64, 128, 160, 256, 320,
384, 512 and one beyond each, the smallest orders; streamed: one column, fewer and more
columns than updates are kept back, and orders that keep fewer back), through the entries
that use it: nrg_diagonalization on a synthetic iteration and nrg_block_eigh_noalloc.

Tolerances: a backward stable solver's residual and loss of orthogonality are a small
multiple of n eps (times the norm of H for the residual); 20 n eps is allowed, for the
eigenvalues against LAPACK as well."""
import ctypes
import math

import numpy as np
import pytest
import torch

from nrg_b200 import load_library, model, prepare_basis

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def check(H, E, V):
    n = len(E)
    norm = np.linalg.norm(H, 2) if n > 1 else abs(H[0, 0])
    tol = 20 * max(n, 4) * EPS
    assert np.all(np.diff(E) >= 0)
    assert np.max(np.abs(E - np.linalg.eigvalsh(H))) <= tol * norm
    assert np.max(np.abs(V.T @ V - np.eye(n))) <= tol
    assert np.max(np.abs(H @ V - V * E)) <= tol * norm


@pytest.mark.parametrize("n", [1, 2, 3, 5, 31, 32, 33, 63, 64, 65, 100, 127, 128])
@pytest.mark.parametrize("kind", ["dense", "tridiagonal", "decoupled", "tiny", "huge"])
def test_block(n, kind):
    rng = np.random.default_rng(n)
    H = rng.standard_normal((n, n))
    H = (H + H.T) / 2
    if kind == "tridiagonal":          # columns that need no reflector
        H = np.triu(np.tril(H, 1), -1)
    elif kind == "decoupled":          # zero columns inside
        H[n // 2:, :n // 2] = 0.0
        H[:n // 2, n // 2:] = 0.0
    elif kind == "tiny":               # squares far below one: the normalised reflectors
        H *= 1e-90
    elif kind == "huge":
        H *= 1e90
    lib = load_library()
    fn = lib.nrg_block_eigh_noalloc
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int32, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    h = torch.from_numpy(H).cuda()
    E = torch.zeros(n, dtype=torch.float64, device="cuda")
    V = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    assert fn(h.data_ptr(), n, E.data_ptr(), V.data_ptr(), None) == 0
    check(H, E.cpu().numpy(), V.cpu().numpy().T)


@pytest.mark.parametrize("n", [129, 159, 160, 161, 255, 256, 257, 319, 320, 321, 383, 384, 385, 511, 512, 513, 545, 640, 1500, 2100])
def test_sector(n, ctx_factory):
    """One iteration whose old states are a sector of n // 2 and one of n - n // 2 states that
    f-dagger-up connects: the new sectors have orders n, n // 2 and n - n // 2."""
    it = 8
    rng = np.random.default_rng(n)
    inp = model.siam(U=0.2, Gamma=0.02, eps_d=-0.1, Lambda=2.0, n_keep=64, n_iterations=20)
    ctx = ctx_factory(inp)
    ka, kb = n // 2, n - n // 2
    rec = np.zeros((n, 5), dtype=np.int32)
    rec[:ka, 2], rec[ka:, :2], rec[ka:, 2] = np.arange(1, ka + 1), (1, 1), np.arange(1, kb + 1)
    E_old = np.concatenate([np.sort(7 * rng.random(ka)), np.sort(7 * rng.random(kb))])
    im = np.zeros((n, n, 2), order="F")
    im[:ka, ka:, 0] = rng.standard_normal((ka, kb)) / math.sqrt(n)
    bi, si = prepare_basis(inp.operation, 2, rec)
    assert si[:, 2].max() == n
    E, V, _, ground = ctx.diagonalization(it, si, bi, E_old, im)
    hop = inp.rescaled_chains()[1][it - inp.indexOfFirstIteration, 0]
    shift = None
    for q in si:
        d, c0, b0 = int(q[2]), int(q[3]) - 1, int(q[4]) - 1
        ref, op = bi[b0:b0 + d, 2] - 1, bi[b0:b0 + d, 4]
        H = np.diag(math.sqrt(inp.Lambda) * E_old[ref])
        for (a, b, t, _), c in zip(inp.coefficient_diagonalization_type, inp.coefficient_diagonalization):
            I, J = np.nonzero(op == a)[0], np.nonzero(op == b)[0]
            B = hop * c * im[np.ix_(ref[J], ref[I], [t - 1])][:, :, 0].T
            H[np.ix_(I, J)], H[np.ix_(J, I)] = B, B.T
        if shift is None:
            shift = ground - E[b0]      # the entry returns energies above the lowest one
        check(H, E[b0:b0 + d] + shift, V[c0:c0 + d * d].reshape((d, d), order="F"))
