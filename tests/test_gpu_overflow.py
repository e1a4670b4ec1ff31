"""Finite blocks whose squares overflow (entries of 1e160): the reduction's norms are infinite and
its results NaN, which the divide and conquer must report, not use: it ranks the values and
indexes by the ranks.  Both entries, both solvers."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from nrg_b200 import NrgError, load_library, model, prepare_basis

pytestmark = pytest.mark.gpu

NUMERIC = 8


@pytest.mark.parametrize("n", [3, 5, 33, 65, 128])
def test_block(n):
    rng = np.random.default_rng(n)
    H = rng.standard_normal((n, n))
    H = H + H.T
    fn = load_library().nrg_block_eigh_noalloc
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int32, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    E = torch.zeros(n, dtype=torch.float64, device="cuda")
    V = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    h = torch.from_numpy(H * 1e160).cuda()
    assert fn(h.data_ptr(), n, E.data_ptr(), V.data_ptr(), None) == NUMERIC
    h = torch.from_numpy(H).cuda()      # the next call is not affected
    assert fn(h.data_ptr(), n, E.data_ptr(), V.data_ptr(), None) == 0
    assert np.max(np.abs(E.cpu().numpy() - np.linalg.eigvalsh(H))) <= 20 * max(n, 4) * np.finfo(np.float64).eps * np.linalg.norm(H, 2)


@pytest.mark.parametrize("n", [100, 200, 400, 600])
def test_sector(n, ctx_factory):
    rng = np.random.default_rng(n)
    inp = model.siam(U=0.2, Gamma=0.02, eps_d=-0.1, Lambda=2.0, n_keep=64, n_iterations=20)
    ctx = ctx_factory(inp)
    ka, kb = n // 2, n - n // 2
    rec = np.zeros((n, 5), dtype=np.int32)
    rec[:ka, 2], rec[ka:, :2], rec[ka:, 2] = np.arange(1, ka + 1), (1, 1), np.arange(1, kb + 1)
    E_old = np.concatenate([np.sort(7 * rng.random(ka)), np.sort(7 * rng.random(kb))])
    im = np.zeros((n, n, 2), order="F")
    im[:ka, ka:, 0] = rng.standard_normal((ka, kb))
    bi, si = prepare_basis(inp.operation, 2, rec)
    with pytest.raises(NrgError) as e:
        ctx.diagonalization(8, si, bi, E_old, im * 1e160)
    assert e.value.status == NUMERIC
    E, V, _, _ = ctx.diagonalization(8, si, bi, E_old, im)
    assert np.all(np.isfinite(E)) and np.all(np.isfinite(V))


def test_sectors_through_the_device_solver():
    here = os.path.dirname(os.path.abspath(__file__))
    cmd = [sys.executable, "-m", "pytest", "-q", "-x", "-p", "no:cacheprovider",
           os.path.join(here, "test_gpu_overflow.py"), "-k", "test_sector and not through"]
    r = subprocess.run(cmd, env=dict(os.environ, NRG_ENTRY_SOLVER="device"), cwd=os.path.dirname(here),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
    assert "4 passed" in r.stdout
