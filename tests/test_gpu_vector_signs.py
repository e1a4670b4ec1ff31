"""The signs of the eigenvectors that a caller receives do not change from one version of the
code to the next.  golden/sector_signs.npz holds, for every column of six random sectors, the
index of its entry of largest magnitude and whether that entry is negative, as
nrg_diagonalization returned them before the reduction of the device-resident runs was
replaced; the solver of those runs returns columns 4 and 849 of the first one (and others) with
the opposite sign."""
import ctypes
import math
import os

import numpy as np
import pytest
import torch

from nrg_b200 import load_library, model, prepare_basis

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "sector_signs.npz")


@pytest.mark.parametrize("n,seed", [(200, 0), (900, 0), (900, 3), (900, 5), (1300, 1), (1300, 5)])
def test_sector_signs(n, seed, ctx_factory):
    """An iteration whose old states are two sectors that f-dagger-up connects (see
    test_gpu_tri_resident.test_sector)."""
    rng = np.random.default_rng(seed)
    inp = model.siam(U=0.2, Gamma=0.02, eps_d=-0.1, Lambda=2.0, n_keep=64, n_iterations=20)
    ctx = ctx_factory(inp)
    ka, kb = n // 2, n - n // 2
    rec = np.zeros((n, 5), dtype=np.int32)
    rec[:ka, 2], rec[ka:, :2], rec[ka:, 2] = np.arange(1, ka + 1), (1, 1), np.arange(1, kb + 1)
    E_old = np.concatenate([np.sort(7 * rng.random(ka)), np.sort(7 * rng.random(kb))])
    im = np.zeros((n, n, 2), order="F")
    im[:ka, ka:, 0] = rng.standard_normal((ka, kb)) / math.sqrt(n)
    bi, si = prepare_basis(inp.operation, 2, rec)
    _, V, _, _ = ctx.diagonalization(8, si, bi, E_old, im)
    q = [q for q in si if q[2] == n][-1]      # the last of the sectors of order n
    c0 = int(q[3]) - 1
    V = V[c0:c0 + n * n].reshape((n, n), order="F")
    with np.load(GOLDEN) as g:
        entry = g[f"entry_{n}_{seed}"]
        negative = np.unpackbits(g[f"negative_{n}_{seed}"], count=n).astype(bool)
    assert np.array_equal(np.nonzero((V[entry, np.arange(n)] < 0) != negative)[0], [])


@pytest.mark.parametrize("n,seed", [(17, 3), (64, 2), (100, 1), (128, 0), (128, 2456)])
@pytest.mark.parametrize("in_place", [False, True])
def test_block_signs(n, seed, in_place):
    """The same of nrg_block_eigh_noalloc (golden/block_signs.npz); the faster solver alone
    returns column 6 of the last block with the opposite sign."""
    rng = np.random.default_rng(10000 + seed)
    H = rng.standard_normal((n, n)) / math.sqrt(n)
    H = (H + H.T) / 2 + np.diag(np.sort(7.0 * rng.random(n) ** 0.45))
    fn = load_library().nrg_block_eigh_noalloc
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int32, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    h = torch.from_numpy(H).cuda()
    E = torch.zeros(n, dtype=torch.float64, device="cuda")
    V = h if in_place else torch.zeros_like(h)
    assert fn(h.data_ptr(), n, E.data_ptr(), V.data_ptr(), None) == 0
    V = V.cpu().numpy().T
    assert np.max(np.abs(H @ V - V * E.cpu().numpy())) < 20 * n * np.finfo(np.float64).eps * np.linalg.norm(H, 2)
    with np.load(os.path.join(os.path.dirname(GOLDEN), "block_signs.npz")) as g:
        entry = g[f"entry_{n}_{seed}"]
        negative = np.unpackbits(g[f"negative_{n}_{seed}"], count=n).astype(bool)
    assert np.array_equal(np.nonzero((V[entry, np.arange(n)] < 0) != negative)[0], [])


@pytest.mark.parametrize("n,seed,at", [(5, 1, 0), (17, 3, 0), (128, 2456, 0), (128, 2456, 128 * 128 - 128)])
def test_eigenvalues_over_the_block(n, seed, at):
    """The eigenvalues may take the block's own storage: the last blocks are solved a second time, from
    the block as it was given."""
    rng = np.random.default_rng(10000 + seed)
    H = rng.standard_normal((n, n)) / math.sqrt(n)
    H = (H + H.T) / 2 + np.diag(np.sort(7.0 * rng.random(n) ** 0.45))
    fn = load_library().nrg_block_eigh_noalloc
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int32, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    h = torch.from_numpy(H).cuda()
    E = h.view(-1)[at:at + n]
    V = torch.zeros_like(h)
    assert fn(h.data_ptr(), n, E.data_ptr(), V.data_ptr(), None) == 0
    E, V = E.cpu().numpy(), V.cpu().numpy().T
    tol = 20 * n * np.finfo(np.float64).eps
    assert np.max(np.abs(H @ V - V * E)) < tol * np.linalg.norm(H, 2)
    assert np.max(np.abs(V.T @ V - np.eye(n))) < tol
