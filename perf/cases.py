"""The measured work of this framework: what a program that uses it has it do.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges, ``prepare`` makes
what a program holds before the call, ``run`` is one pass through the public entry points of
the ``nrg_b200`` package, ``work`` the bytes and operations no implementation can do without
and ``exact`` the same results from plain numpy in 64 bits.

Kinds of work:

block            one symmetric block through nrg_block_eigh_noalloc, device arrays
diagonalization  one iteration's sector Hamiltonians through the drop-in entry (host arrays)
transforms       the two invariant-matrix routines after it (postprocess), drop-in entries
cfs              the complete-Fock-space spectrum step of one iteration, drop-in entry
broaden          log-Gaussian broadening of a binned spectrum
sweep            a whole device-resident run: forward only, with the T = 0 spectrum, or with
                 the full-density-matrix spectrum at T > 0
batch            independent impurity models side by side on one device

The inputs of the single-routine kinds are drawn with the structure an iteration has: sector
orders follow the Gaussian in (Q, 2Sz) that the kept states of a flat-band model show, the
old energies rise from zero with the density of a many-body spectrum, the matrix elements
fall off with the energy difference, and eigenvector blocks have the entries' size of
orthonormal columns.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nrg-mpi_b200"))
from nrg_b200 import Context, load_library, model, prepare_basis, run_batch  # noqa: E402

SECTOR_WIDTH = 2.0      # of the kept states' distribution over Q and over 2Sz
N_ITERATIONS = 40       # of the chain that the single-routine kinds stand in
ITERATION = 8           # the iteration they stand at


def listed():
    return [
        # the smallest call: one small block in a caller's own pipeline, launch latency
        dict(name="block_17", kind="block", n=17),
        # the largest block that entry takes
        dict(name="block_128", kind="block", n=128),
        # one diagonalization() call of a Fortran driver, a small and a large N_keep
        dict(name="diagonalization_333", kind="diagonalization", n_keep=333),
        dict(name="diagonalization_2048", kind="diagonalization", n_keep=2048),
        # the invariant-matrix calls of postprocess(), an ordinary N_keep
        dict(name="transforms_1000", kind="transforms", n_keep=1000),
        # one spikeCFS() call of the spectrum phase
        dict(name="cfs_777", kind="cfs", n_keep=777),
        # a broadened spectrum on a grid of 100 points per decade over eight decades
        dict(name="broaden_801", kind="broaden", points=801, width=0.6),
        # a quick look at a model: N_keep as small as it is used, T = 0 spectrum
        dict(name="sweep_250", kind="sweep", model="siam", n_keep=250, iterations=30, spectrum="cfs"),
        # a production run with the finite-temperature spectrum
        dict(name="sweep_2048_fdm", kind="sweep", model="siam", n_keep=2048, iterations=60, spectrum="fdm"),
        # the largest run, bench.py's workload: N_keep = 4096, 60 iterations, T = 0 spectrum
        dict(name="sweep_4096", kind="sweep", model="siam", n_keep=4096, iterations=60, spectrum="cfs"),
        # two orbitals (16 local states), thermodynamics and level flow only
        dict(name="two_orbital_600", kind="sweep", model="two_orbital", n_keep=600, iterations=8, spectrum="none"),
        # a parameter sweep: eight models of different sizes in flight at once
        dict(name="batch_8", kind="batch", instances=8, n_keep=512, iterations=30, spectrum="cfs"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["block", "diagonalization", "transforms", "cfs", "broaden", "sweep", "sweep", "sweep", "batch"])
    if kind == "block":
        return dict(kind=kind, n=_log_int(rng, 2, 128))
    if kind in ("diagonalization", "transforms", "cfs"):
        return dict(kind=kind, n_keep=_log_int(rng, 64, 2048))
    if kind == "broaden":
        return dict(kind=kind, points=_log_int(rng, 50, 4000), width=round(rng.uniform(0.2, 0.9), 3))
    if kind == "batch":
        return dict(kind=kind, instances=rng.randint(2, 12), n_keep=_log_int(rng, 128, 1024),
                    iterations=rng.randint(20, 50), spectrum=rng.choice(["none", "cfs", "fdm"]))
    if rng.random() < 0.25:
        return dict(kind=kind, model="two_orbital", n_keep=_log_int(rng, 100, 900), iterations=rng.randint(5, 9),
                    spectrum="none")
    return dict(kind=kind, model="siam", n_keep=_log_int(rng, 64, 4096), iterations=rng.randint(12, 50),
                spectrum=rng.choice(["none", "cfs", "fdm"]))


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------
def _siam(rng, n_keep, iterations):
    """One model of the ranges of nrg_b200.sweep (U, Gamma log-uniform, eps_d around -U/2)."""
    U = float(rng.uniform(0.05, 0.5))
    gamma = float(10.0 ** rng.uniform(math.log10(0.005), math.log10(0.05)))
    delta = float(rng.uniform(-0.02, 0.02))
    return model.siam(U=U, Gamma=gamma, eps_d=-U / 2 + delta, Lambda=2.0, n_keep=n_keep, n_iterations=iterations)


def _two_orbital(rng, n_keep, iterations):
    return model.two_orbital_hund(U=float(rng.uniform(0.1, 0.4)), J=float(rng.uniform(0.01, 0.03)),
                                  Gamma=float(rng.uniform(0.01, 0.03)), n_keep=n_keep, n_iterations=iterations)


def _sector_counts(n_keep, parity):
    """{(Q, 2Sz): states} of about n_keep kept states, Q + 2Sz of the given parity."""
    got = {}
    for Q in range(-9, 10):
        for S in range(-9, 10):
            if (Q + S) % 2 != parity:
                continue
            k = n_keep * math.exp(-(Q * Q + S * S) / (2 * SECTOR_WIDTH ** 2)) / (math.pi * SECTOR_WIDTH ** 2)
            if int(round(k)):
                got[(Q, S)] = int(round(k))
    return got


def _levels(rng, Q, S, k):
    """k ascending energies of one sector."""
    return np.sort(0.15 * (Q * Q + S * S) + 7.0 * rng.random(k) ** 0.45)


def _operator(rng, blocks, E, n_types, raised):
    """(n, n, n_types) matrices <l| op_t^dagger |r> stored at (r, l, t): nonzero between the
    sectors that op_t connects, falling with the energy difference."""
    n = len(E)
    M = np.zeros((n, n, n_types), order="F")
    for t in range(n_types):
        dQ, dS = raised[t]
        for (Q, S), (r0, kr) in blocks.items():
            hit = blocks.get((Q + dQ, S + dS))
            if hit is None:
                continue
            l0, kl = hit
            away = np.abs(E[r0:r0 + kr, None] - E[None, l0:l0 + kl])
            M[r0:r0 + kr, l0:l0 + kl, t] = rng.standard_normal((kr, kl)) * np.exp(-away) / math.sqrt(max(kr, kl))
    return M


def _blocks(counts):
    at, got = 0, {}
    for q in sorted(counts):
        got[q] = (at, counts[q])
        at += counts[q]
    return got, at


def _iteration_state(rng, n_keep):
    """The module arrays of one iteration: the kept states of the last one and the sectors
    that prepareBasis makes of them."""
    inp = _siam(rng, n_keep, N_ITERATIONS)
    blocks, nb = _blocks(_sector_counts(n_keep, 0))
    records = np.zeros((nb, 5), dtype=np.int32)
    E = np.zeros(nb)
    for (Q, S), (r0, k) in blocks.items():
        records[r0:r0 + k, 0], records[r0:r0 + k, 1] = Q, S
        records[r0:r0 + k, 2] = np.arange(1, k + 1)
        E[r0:r0 + k] = _levels(rng, Q, S, k)
    E -= E.min()
    raised = [tuple(int(x) for x in q) for q in inp.conservation_difference_spectrum]
    basis_input, sectors = prepare_basis(inp.operation, 2, records)
    return dict(inp=inp, blocks=blocks, nb=nb, E=E, raised=raised, basis_input=basis_input, sectors=sectors)


def _vectors(rng, sectors):
    return np.concatenate([rng.standard_normal(int(d) * int(d)) / math.sqrt(int(d)) for d in sectors[:, 2]])


def _kept_of(sectors, n_keep):
    """Kept states of every sector (its lowest ones)."""
    want = _sector_counts(n_keep, 1)
    return [min(int(s[2]), want.get((int(s[0]), int(s[1])), 0)) for s in sectors]


def _kept_records(sectors, kept):
    rows = []
    for s, k in zip(sectors, kept):
        r = np.zeros((k, 5), dtype=np.int32)
        r[:, 0], r[:, 1], r[:, 2] = s[0], s[1], np.arange(1, k + 1)
        rows.append(r)
    return np.concatenate(rows)


def _empty_bins(inp):
    """binnedSpikePositive / Negative as the driver initialises them."""
    nbin = int(int(math.log10(inp.scale(-1))) + 1.0 + 15.0) * 1000 + 1
    e = 10.0 ** (-15.0 + np.arange(nbin) / 1000.0)
    pos = np.zeros((nbin * inp.numberOfMatrix, 2), order="F")
    pos[:, 0] = np.tile(e, inp.numberOfMatrix)
    neg = pos.copy(order="F")
    neg[:, 0] *= -1.0
    return nbin, pos, neg


def _inputs(case, seed):
    """The inputs of one case, host side."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "block":
        n = case["n"]
        H = rng.standard_normal((n, n)) / math.sqrt(n)
        return dict(H=(H + H.T) / 2 + np.diag(np.sort(7.0 * rng.random(n) ** 0.45)))
    if kind == "broaden":
        inp = _siam(rng, 64, 20)
        nbin, bins, _ = _empty_bins(inp)
        nm = inp.numberOfMatrix
        e = bins[:nbin, 0]
        for m in range(nm):
            w = rng.random(nbin) * e / (e + 10.0 ** rng.uniform(-4, -2)) ** 2
            w[e > 2.0] = 0.0
            bins[m * nbin:(m + 1) * nbin, 1] = w / w.sum()
        omega = 10.0 ** np.linspace(-8.0, 0.0, case["points"])
        return dict(inp=inp, bins=bins, nbin=nbin, nm=nm, omega=omega)
    if kind == "sweep":
        make = _siam if case["model"] == "siam" else _two_orbital
        return dict(models=[make(rng, case["n_keep"], case["iterations"])],
                    T=float(10.0 ** rng.uniform(-6, -4)) if case["spectrum"] == "fdm" else 0.0)
    if kind == "batch":
        # sizes from half to twice the case's, largest first, as a caller sorts them
        sizes = sorted((max(32, int(case["n_keep"] * 2.0 ** (2.0 * i / (case["instances"] - 1) - 1.0)))
                        for i in range(case["instances"])), reverse=True)
        return dict(models=[_siam(rng, k, case["iterations"]) for k in sizes],
                    T=float(10.0 ** rng.uniform(-6, -4)) if case["spectrum"] == "fdm" else 0.0)
    s = _iteration_state(rng, case["n_keep"])
    inp = s["inp"]
    if kind == "diagonalization":
        s["im"] = _operator(rng, s["blocks"], s["E"], inp.numberOfConductionMatrix, s["raised"])
        return s
    s["kept"] = _kept_of(s["sectors"], case["n_keep"])
    s["V"] = _vectors(rng, s["sectors"])
    s["ims"] = _operator(rng, s["blocks"], s["E"], inp.numberOfMatrix, s["raised"])
    s["records"] = _kept_records(s["sectors"], s["kept"])
    s["n_kept"] = len(s["records"])
    if kind == "transforms":
        return s
    # cfs: energies, kept states first, the discarded ones in energy order, density matrices
    E, gone, gone_E, at = [], [], [], 0
    for q, k in zip(s["sectors"], s["kept"]):
        e = _levels(rng, int(q[0]), int(q[1]), int(q[2]))
        E.append(e[:k])
        r = np.zeros((len(e) - k, 5), dtype=np.int32)
        r[:, 0], r[:, 1], r[:, 2] = q[0], q[1], np.arange(k + 1, len(e) + 1)
        gone.append(r)
        gone_E.append(e[k:])
    gone, gone_E = np.concatenate(gone), np.concatenate(gone_E)
    order = np.argsort(gone_E, kind="stable")
    s["basis_output"] = np.concatenate([s["records"], gone[order]])
    s["eigenvalue"] = np.concatenate(E + [gone_E[order]])
    rows, rho, at, out = [], [], 1, 1
    share = np.array([math.exp(-float(e[0])) if len(e) else 0.0 for e in E])
    share /= share.sum()
    for q, k, e, part in zip(s["sectors"], s["kept"], E, share):
        if not k:
            continue
        X = rng.standard_normal((k, 8)) * np.exp(-e)[:, None]
        X = X @ X.T
        rho.append((X * (part / np.trace(X))).reshape(-1))
        rows.append([q[0], q[1], q[2], k, q[3], q[4], out, at])
        at += k * k
        out += k
    s["full"] = dict(fullSubspaceInfo=np.array(rows, dtype=np.int32), rdm=np.concatenate(rho),
                     map=np.where(np.arange(inp.numberOfIteration + 2) <= ITERATION + 1, 1, len(rows) + 1).astype(np.int32))
    s["nbin"], s["pos"], s["neg"] = _empty_bins(inp)
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    s["kind"], s["case"] = kind, case
    if kind == "block":
        lib = load_library()
        s["entry"] = lib.nrg_block_eigh_noalloc
        s["entry"].argtypes = [ctypes.c_void_p, ctypes.c_int32, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
        s["H"] = torch.from_numpy(np.asfortranarray(s["H"]).T.copy()).cuda()
        s["E"] = torch.zeros(case["n"], dtype=torch.float64, device="cuda")
        s["V"] = torch.zeros(case["n"], case["n"], dtype=torch.float64, device="cuda")
        return s
    models = s["models"] if "models" in s else [s["inp"]]
    s["ctx"] = []
    for m in models:
        c = Context(0)
        c.set_model(m)
        s["ctx"].append(c)
    return s


def _result(r):
    """A run's physical results, whole."""
    return {k: r[k] for k in ("kept", "numberOfBasisFull", "groundStateEnergy", "flow", "thermo", "finalEigenvalue",
                              "rdmTrace", "binPos", "binNeg")}


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "block":
        rc = s["entry"](s["H"].data_ptr(), case["n"], s["E"].data_ptr(), s["V"].data_ptr(), None)
        if rc:
            raise RuntimeError("nrg_block_eigh_noalloc: status %d" % rc)
        return s["E"], s["V"]
    ctx = s["ctx"][0]
    if kind == "diagonalization":
        return ctx.diagonalization(ITERATION, s["sectors"], s["basis_input"], s["E"], s["im"])
    if kind == "transforms":
        f = ctx.invariant_matrix_dgemm(ITERATION, s["sectors"], s["basis_input"], s["n_kept"], s["records"], s["V"])
        d = ctx.invariant_matrix_for_spectrum_dgemm(ITERATION, s["sectors"], s["basis_input"], s["n_kept"],
                                                    s["records"], s["V"], s["ims"])
        return f, d
    if kind == "cfs":
        R = dict(subspaceInfo=s["sectors"], basis_input=s["basis_input"], basis_output=s["basis_output"],
                 eigenvalue=s["eigenvalue"], eigenvector=s["V"], numberOfBasis=s["n_kept"])
        return ctx.spike_cfs(ITERATION, R, s["pos"].copy(order="F"), s["neg"].copy(order="F"), s["ims"], s["nb"],
                             s["full"])
    if kind == "broaden":
        return ctx.broaden_log_gaussian(s["bins"], s["nbin"], s["nm"], case["width"], s["omega"])
    spectrum = case["spectrum"] != "none"
    if kind == "sweep":
        return _result(ctx.run(spectrum=spectrum, flow_stride=256, final_capacity=1024, temperature=s["T"]))
    results, _ = run_batch(s["ctx"], spectrum=spectrum, concurrency=8, flow_stride=256, temperature=s["T"])
    results = [_result(r) for r in results]     # every instance has the same array sizes
    return {k: np.stack([r[k] for r in results]) for k in results[0]}


# ---------------------------------------------------------------------------------------
# work: what one pass cannot do without
# ---------------------------------------------------------------------------------------
def _step(n_keep, n_local):
    """Sum over the sectors of one full-size iteration of d, d^2 and d^3, and the number of
    kept states: the sectors of n_keep kept states times n_local local states."""
    width2 = SECTOR_WIDTH ** 2 * (1.0 if n_local == 4 else 2.0)
    n = n_keep * n_local
    d = [n * math.exp(-(Q * Q + S * S) / (2 * width2)) / (math.pi * width2)
         for Q in range(-12, 13) for S in range(-12, 13) if (Q + S) % 2]
    return sum(d), sum(x * x for x in d), sum(x ** 3 for x in d)


def _sweep_work(case, n_keep):
    n_local = 4 if case.get("model", "siam") == "siam" else 16
    full = max(0, case["iterations"] - (math.ceil(math.log(max(n_keep, 2), n_local)) - 1))
    one, two, three = _step(n_keep, n_local)
    # eigensolver (tridiagonalisation, its vectors, back-transformation) of every sector
    flops = full * (4.0 / 3.0 + 2.0) * three
    # the invariant matrices: kept x d x kept and kept x d x d products per sector pair and type
    types = 2 if n_local == 4 else 4
    flops += full * types * 2.0 * three / n_local * (1 + 1.0 / n_local)
    # eigenvectors and energies written once
    bytes_ = full * 8.0 * (two + one)
    if case["spectrum"] != "none":
        flops += full * (2.0 * three / n_local * (1 + 1.0 / n_local) + 2 * types * 2.0 * three / n_local)
        bytes_ += full * 8.0 * two
    return bytes_, flops


def work(case):
    kind = case["kind"]
    if kind == "block":
        n = case["n"]
        return dict(bytes=8.0 * (2 * n * n + n), flops=(4.0 / 3.0 + 2.0) * n ** 3)
    if kind == "broaden":
        return dict(bytes=8.0 * (2 * 2 * 15001 + 3 * case["points"]), flops=2.0 * 8.0 * 15001 * case["points"])
    if kind == "sweep":
        b, f = _sweep_work(case, case["n_keep"])
        return dict(bytes=b, flops=f)
    if kind == "batch":
        total = [0.0, 0.0]
        for i in range(case["instances"]):
            n = max(32, int(case["n_keep"] * 2.0 ** (2.0 * i / (case["instances"] - 1) - 1.0)))
            b, f = _sweep_work(case, n)
            total[0] += b
            total[1] += f
        return dict(bytes=total[0], flops=total[1])
    n_keep = case["n_keep"]
    one, two, three = _step(n_keep, 4)
    pair = 4.0 / (math.pi * SECTOR_WIDTH ** 2)          # share of the old states in one sector's neighbours
    if kind == "diagonalization":
        return dict(bytes=8.0 * (two + one) + 8.0 * 2 * n_keep * n_keep * pair / 4 + 40.0 * one,
                    flops=(4.0 / 3.0 + 2.0) * three)
    if kind == "transforms":
        return dict(bytes=8.0 * (two / 4 + 2 * 2 * n_keep * n_keep + 2 * n_keep * n_keep * pair / 4),
                    flops=2 * 2.0 * three / 16 + 2 * 2.0 * three / 4 * 1.25)
    return dict(bytes=8.0 * (two + n_keep * n_keep * pair + 4 * 2 * 15001), flops=4 * 2.0 * three * (1 / 16 + 3 / 16 + 3 / 16))


# ---------------------------------------------------------------------------------------
# the same results from plain numpy, 64 bits
# ---------------------------------------------------------------------------------------
def _rows(s, q):
    b0 = int(q[4]) - 1
    r = s["basis_input"][b0:b0 + int(q[2])]
    return r[:, 2] - 1, r[:, 3], r[:, 4] - 1        # reference, variation, operation (0-based)


def _vec(s, q):
    d, c0 = int(q[2]), int(q[3]) - 1
    return s["V"][c0:c0 + d * d].reshape((d, d), order="F")


def _exact_diagonalization(s):
    inp = s["inp"]
    _, hop, _ = inp.rescaled_chains()
    E, bo = [], []
    for q in s["sectors"]:
        d = int(q[2])
        ref, _, op = _rows(s, q)
        H = np.zeros((d, d))
        H[np.arange(d), np.arange(d)] = math.sqrt(inp.Lambda) * s["E"][ref]   # the flat band has no on-site term
        for (a, b, t, c), v in zip(inp.coefficient_diagonalization_type, inp.coefficient_diagonalization):
            I, J = np.nonzero(op == a - 1)[0], np.nonzero(op == b - 1)[0]
            B = hop[ITERATION - inp.indexOfFirstIteration, c - 1] * v * s["im"][np.ix_(ref[J], ref[I], [t - 1])][:, :, 0].T
            H[np.ix_(I, J)] = B
            H[np.ix_(J, I)] = B.T
        E.append(np.linalg.eigvalsh(H))
        r = np.zeros((d, 5), dtype=np.int32)
        r[:, 0], r[:, 1], r[:, 2] = q[0], q[1], np.arange(1, d + 1)
        bo.append(r)
    E = np.concatenate(E)
    ground = float(E[0])
    E = E - E.min()
    E[E <= 1e-12] = 0.0
    # the eigenvectors' signs are the solver's own: no value for them
    return E, None, np.concatenate(bo), ground


def _elements(s, left, right, m):
    """coefficient matrix of d_m^dagger between the product states of two sectors."""
    refL, _, opL = _rows(s, left)
    refR, _, opR = _rows(s, right)
    c = s["inp"].coefficient_invariant_matrix_spectrum[m]
    return np.where(opL[:, None] == opR[None, :], c[opL][:, None] * s["ims"][:, :, m].T[np.ix_(refL, refR)], 0.0)


def _exact_transforms(s):
    inp = s["inp"]
    n = s["n_kept"]
    f = np.zeros((n, n, inp.numberOfConductionMatrix))
    d = np.zeros((n, n, inp.numberOfMatrix))
    start = np.concatenate([[0], np.cumsum(s["kept"])])
    at = {(int(q[0]), int(q[1])): i for i, q in enumerate(s["sectors"])}
    for (Q, S), ir in at.items():
        kr = s["kept"][ir]
        for dS in (1, -1):
            il = at.get((Q + 1, S + dS))
            if il is None or not kr or not s["kept"][il]:
                continue
            L, R, kl = s["sectors"][il], s["sectors"][ir], s["kept"][il]
            VL, VR = _vec(s, L)[:, :kl], _vec(s, R)[:, :kr]
            _, varL, opL = _rows(s, L)
            _, varR, opR = _rows(s, R)
            cols = np.s_[start[ir]:start[ir] + kr, start[il]:start[il] + kl]
            for t in range(inp.numberOfConductionMatrix):
                C = np.zeros((len(opL), len(opR)))
                for (a, b, tt), v in zip(inp.coefficient_invariant_matrix_type, inp.coefficient_invariant_matrix):
                    if tt - 1 == t:
                        C[(opL[:, None] == a - 1) & (opR[None, :] == b - 1) & (varL[:, None] == varR[None, :])] = v
                f[cols + (t,)] = (VL.T @ C @ VR).T
            for m, (dq, ds) in enumerate(s["raised"]):
                if (dq, ds) == (1, dS):
                    d[cols + (m,)] = (VL.T @ _elements(s, L, R, m) @ VR).T
    return f, d


def _bin(container, nbin, m, energy, weight):
    """Every spike's weight, split between the two logarithmic bins around its energy."""
    position = (np.log10(np.abs(energy)) + 15.0) * 1000.0 + 1.0
    at = np.maximum(np.trunc(position).astype(np.int64), 1)
    low, high = position <= 0.0, position >= nbin
    at = np.where(low, 1, np.where(high, nbin, at))
    frac = np.where(low | high, 0.0, position - at)
    np.add.at(container[:, 1], m * nbin + at - 1, weight * (1.0 - frac))
    two = ~(low | high)
    np.add.at(container[:, 1], m * nbin + at[two], (weight * frac)[two])


def _exact_cfs(s):
    inp, nbin = s["inp"], s["nbin"]
    pos, neg = s["pos"].copy(order="F"), s["neg"].copy(order="F")
    total = np.zeros((inp.numberOfMatrix, 4))
    scale = inp.scale(ITERATION)
    at = {(int(q[0]), int(q[1])): i for i, q in enumerate(s["sectors"])}
    rho = {(int(r[0]), int(r[1])): s["full"]["rdm"][r[7] - 1:r[7] - 1 + r[3] * r[3]].reshape(r[3], r[3])
           for r in s["full"]["fullSubspaceInfo"]}
    start = np.concatenate([[0], np.cumsum(s["kept"])])
    gone, E = s["basis_output"][s["n_kept"]:], s["eigenvalue"]
    for (Q, S), il in at.items():
        L = s["sectors"][il]
        mine = np.nonzero((gone[:, 0] == Q) & (gone[:, 1] == S))[0]
        El = E[s["n_kept"] + mine]
        Vl = _vec(s, L)[:, gone[mine, 2] - 1]
        for m, (dQ, dS) in enumerate(s["raised"]):
            for up in (True, False):
                q = (Q + dQ, S + dS) if up else (Q - dQ, S - dS)
                ik = at.get(q)
                if ik is None or q not in rho or not len(mine):
                    continue
                k = s["kept"][ik]
                K, Ek = s["sectors"][ik], E[start[ik]:start[ik] + k]
                Vk = _vec(s, K)[:, :k]
                X = Vk.T @ _elements(s, K, L, m) @ Vl if up else (Vl.T @ _elements(s, L, K, m) @ Vk).T
                W = X * (rho[q] @ X)
                to, energy = (neg, Ek[:, None] - El) if up else (pos, El - Ek[:, None])
                _bin(to, nbin, m, (energy * scale).reshape(-1), W.reshape(-1))
                total[m, 0 if up else 1] += W.sum()
                total[m, 2 if up else 3] += W.sum()
    return pos, neg, total


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sweep", "batch"):
        return None     # a sweep's numpy replay takes from half a minute to many minutes
    s = _inputs(case, seed)
    if kind == "block":
        # the eigenvectors' signs are the solver's own: no value for them
        return np.linalg.eigvalsh(s["H"]), None
    if kind == "diagonalization":
        return _exact_diagonalization(s)
    if kind == "transforms":
        return _exact_transforms(s)
    if kind == "cfs":
        return _exact_cfs(s)
    b, out = case["width"], np.zeros((s["nm"], len(s["omega"])))
    for m in range(s["nm"]):
        E, W = (s["bins"][m * s["nbin"]:(m + 1) * s["nbin"], j] for j in (0, 1))
        E, W = E[W != 0.0], W[W != 0.0]
        for k, w in enumerate(s["omega"]):
            x = np.log(w / E) / b
            out[m, k] = math.exp(-b * b / 4) / (b * math.sqrt(math.pi)) * np.sum(W * np.exp(-x * x) / E)
    return out
