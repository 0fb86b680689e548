"""Several roots (block Davidson), batched solves and the request server.

Roots 2-4 have no reference counterpart (the reference is single-root): they
are checked against a dense diagonalisation of the Hamiltonian built column
by column from the oracle's matvec; the lowest root against the reference's
golden energy.  Batched results must be bit-identical to the same solve run
alone; served one-root results equal the same single-root solve run alone to
1e-9 Ha."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dg():
    import doci_gb300
    doci_gb300.lib()
    return doci_gb300


def dense_eigs(path, k):
    o = oracle.Ham(path)
    H = np.empty((o.D, o.D))
    e = np.zeros(o.D)
    for c in range(o.D):
        e[c] = 1.0
        H[:, c] = o.matvec(e, nthreads=1)
        e[c] = 0.0
    return np.linalg.eigvalsh(0.5 * (H + H.T))[:k]


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
@pytest.mark.parametrize("L,N,seed", [(12, 6, 51), (13, 5, 52), (14, 7, 1)])
def test_four_roots_vs_dense(L, N, seed, mode, synth, dg):
    p = synth(L, N, seed)
    ref = dense_eigs(p, 4)
    with dg.Hamiltonian.from_fcidump(p) as h:
        r = dg.solve_roots(h, nroots=4, tol=1e-7, mode=mode, max_vec=20)
    assert r["status"] == 0 and r["converged"] == 1
    assert np.allclose(r["energies"], ref, atol=1e-9), (r["energies"], ref)
    assert max(r["residuals"]) <= 1e-7


def test_lowest_root_matches_reference(fcidump, golden, dg):
    name = "synthetic_L14_N7_s1"
    with dg.Hamiltonian.from_fcidump(fcidump(name)) as h:
        r = dg.solve_roots(h, nroots=2, tol=1e-7, mode="mixed")
    assert abs(r["energies"][0] - golden["cases"][name]["davidson"]["energy"]) < 1e-8


def test_batch_same_as_alone(synth, dg):
    specs = [(L, L // 2 + d, 100 + i) for i, (L, d) in enumerate([(10, 0), (12, -1), (16, 0), (11, 1), (14, 0),
                                                                    (18, 0), (13, 0), (15, -2), (12, 0), (17, 1)])]
    hams = [dg.Hamiltonian.from_fcidump(synth(*s)) for s in specs]
    try:
        alone = [dg.solve_roots(h, nroots=4, tol=1e-6, mode="mixed") for h in hams]
        st, mixed = dg.batch_solve(hams, nroots=4, tol=1e-6, mode="mixed", workers=6)
        assert st == 0
        for a, b in zip(alone, mixed):
            assert a["energies"] == b["energies"]  # bit-identical
            assert a["iterations"] == b["iterations"]
    finally:
        for h in hams:
            h.close()


def test_server_continuous_batching(dg):
    from doci_gb300.fcidump import raw_integrals
    rng = np.random.default_rng(4)
    reqs = []
    for i in range(14):
        L = int(rng.integers(10, 19))
        N = L // 2 + int(rng.integers(-2, 3))
        reqs.append((L, N, 2000 + i))
    alone = {}
    for L, N, seed in reqs:
        one, two = raw_integrals(L, seed)
        with dg.Hamiltonian.from_integrals(L, N, 0.0, one, two) as h:
            # a one-root request runs the single-root device Davidson with the
            # server's options (doci_batch_opts defaults: MAX_VEC 16, mixed_tol 1e-4)
            r, _ = h.solve(solver="D", tol=1e-6, mode="mixed", mixed_tol=1e-4, davidson_max_vec=16,
                           davidson_keep=2, max_its=200)
            alone[seed] = r
    with dg.Server(nroots=1, tol=1e-6, mode="mixed", workers=5) as srv:
        tickets = {}
        for L, N, seed in reqs:
            one, two = raw_integrals(L, seed)
            tickets[seed] = srv.submit(L, N, one, two)
        st, _ = srv.poll(10_000)
        assert st == 10  # DOCI_ERR_NOT_FOUND
        results = {seed: srv.wait(t) for seed, t in tickets.items()}
        s = srv.stats()
        assert s["submitted"] == s["finished"] == len(reqs) and s["bytes_in_use"] == 0
    overlapped = 0
    for seed, r in results.items():
        assert r["status"] == 0 and r["converged"] == 1
        # same alone and in the mix, within the rounding of the FP32 sigma's atomic adds
        assert abs(r["energies"][0] - alone[seed]["energy"]) <= 1e-9
        assert r["queued_s"] <= r["start_s"] <= r["end_s"]
        overlapped += any(o is not r and o["start_s"] < r["end_s"] and r["start_s"] < o["end_s"]
                          for o in results.values())
    assert overlapped > 0  # requests ran concurrently


def test_server_admission_rejects_oversized(dg):
    from doci_gb300.fcidump import raw_integrals
    one, two = raw_integrals(12, 7)
    with dg.Server(nroots=1, workers=1, hbm_budget=1 << 20) as srv:
        t = srv.submit(12, 6, one, two)
        r = srv.wait(t)
    assert r["status"] == 9  # DOCI_ERR_ADMISSION


def test_engine_tile_autotune(synth, dg):
    """doci_engine_autotune picks, for one (L, N) shape, the batch engine's
    sigma path: a tile of 1, 2 or 4 determinants per thread of the batched
    gather (returned as 1, 2, 4), or the single-problem kernels (returned as
    0).  A tile shape changes which thread computes a determinant, not its
    sum; the single-problem kernels reduce in another order.  Either way the
    solve reaches the same energies, within the residual tolerance's
    quadratic energy error."""
    with dg.Hamiltonian.from_fcidump(synth(16, 8, 61)) as h:
        before = dg.solve_roots(h, nroots=2, tol=1e-6, mode="mixed")
        choice = h.engine_autotune(2)
        assert choice in (0, 1, 2, 4)
        after = dg.solve_roots(h, nroots=2, tol=1e-6, mode="mixed")
    assert before["converged"] == after["converged"] == 1
    assert np.allclose(before["energies"], after["energies"], rtol=0, atol=1e-9)


@pytest.mark.parametrize("nroots,max_vec", [(1, 7), (1, 8), (1, 9), (2, 15), (3, 31), (4, 17), (4, 32)])
def test_subspace_eigenproblem_sizes(nroots, max_vec, synth, dg):
    """Bases around the size from which the subspace eigenproblem goes through
    FP32 first (8), odd and even, up to the largest: every energy is an
    eigenvalue, to the square of the residual bound over the gap and FP64's
    rounding of the solve (1e-9, as above)."""
    p = synth(10, 5, 140 + max_vec)
    ref = dense_eigs(p, 252)
    with dg.Hamiltonian.from_fcidump(p) as h:
        r = dg.solve_roots(h, nroots=nroots, tol=1e-7, mode="fp64", max_vec=max_vec, max_its=400)
    assert r["status"] == 0 and r["converged"] == 1
    for e in r["energies"][:nroots]:
        assert np.abs(ref - e).min() < 1e-9


@pytest.mark.parametrize("mode", ["fp64", "mixed"])
@pytest.mark.parametrize("L,N,nroots", [(1, 1, 1), (2, 1, 4), (3, 1, 2), (4, 2, 4), (4, 2, 8), (9, 4, 1), (12, 6, 5)])
def test_orthogonalisation_step_edges(L, N, nroots, mode, synth, dg):
    """Few determinants (corrections with nothing left of them), one root (no next
    correction in a step), more than four: the lowest eigenvalues, each once,
    with orthonormal vectors; more roots than determinants are refused, as ever.
    Residuals below 1e-7 bound the energies' errors; vectors are FP64."""
    p = synth(L, N, 150 + L + nroots)
    with dg.Hamiltonian.from_fcidump(p) as h:
        k = nroots
        if k > h.D:
            with pytest.raises(dg.DociError, match="DOCI_ERR_INVALID"):
                dg.solve_roots(h, vectors=True, nroots=nroots, tol=1e-7, mode=mode, max_vec=32)
            return
        ref = dense_eigs(p, k)
        r = dg.solve_roots(h, vectors=True, nroots=nroots, tol=1e-7, mode=mode, max_vec=32)
        r, v = r if isinstance(r, tuple) else (r, r["vectors"])
        v = np.asarray(v).reshape(-1, h.D)[:k]
    assert r["status"] == 0 and r["converged"] == 1
    assert np.allclose(r["energies"][:k], ref, atol=1e-7)
    assert np.abs(v @ v.T - np.eye(k)).max() < 1e-6


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("nroots", [1, 2, 8])
def test_integrals_not_finite(nroots, bad, synth, dg):
    """An integral that is not finite makes the subspace matrix and its
    eigenvalues NaN: they are ordered all the same (every one has a place), the
    solve ends, and the next one on the device is as ever."""
    from doci_gb300.fcidump import raw_integrals
    one, two = raw_integrals(10, 160)
    two = np.array(two, dtype=np.float64).reshape(10, 10, 10, 10)
    for i, j, k, l in ((0, 9, 0, 9), (0, 9, 9, 0), (9, 0, 0, 9), (9, 0, 9, 0)):
        two[i, j, k, l] = bad
    with dg.Hamiltonian.from_integrals(10, 5, 0.0, one, two) as h:
        r = dg.solve_roots(h, nroots=nroots, tol=1e-7, mode="fp64", max_vec=16, max_its=20)
    assert r["status"] == 0 and not np.isfinite(r["energies"][0])
    p = synth(10, 5, 161)
    with dg.Hamiltonian.from_fcidump(p) as h:
        r = dg.solve_roots(h, nroots=2, tol=1e-7, mode="fp64")
    assert r["converged"] == 1 and np.allclose(r["energies"][:2], dense_eigs(p, 2), atol=1e-9)


@pytest.mark.parametrize("power", [0, 60, 63])
def test_mixed_solve_scales(power, dg):
    """A Hamiltonian and tolerances times a power of two give the same solve times
    that power, as long as the values' squares are in FP32's range (up to 2^126
    here): a thread's FP32 sums then are, and a block's, formed in FP64, are in any case."""
    L, N, s = 10, 5, 2.0 ** power
    rng = np.random.default_rng(170)
    K = rng.uniform(0.9, 0.99, (L, L))
    K = np.triu(K, 1) + np.triu(K, 1).T
    eri = np.zeros((L, L, L, L))
    i, j = np.nonzero(~np.eye(L, dtype=bool))
    eri[i, j, i, j] = eri[i, j, j, i] = K[i, j]
    h1 = np.diag(np.linspace(-4, 4, L))
    out = []
    for f in (1.0, s):
        with dg.Hamiltonian.from_integrals(L, N, 0.0, h1 * f, eri * f) as h:
            out.append(dg.solve_roots(h, nroots=2, tol=1e-7 * f, mixed_tol=1e-4 * f, mode="mixed", max_vec=16))
    a, b = out
    assert a["converged"] == b["converged"] == 1
    assert a["iterations_fp32"] == b["iterations_fp32"] > 3 and a["iterations"] == b["iterations"]
    assert np.allclose(np.array(b["energies"][:2]) / s, a["energies"][:2], rtol=1e-12, atol=0)


def nbr_table_bytes(L, N):
    import math
    n = math.comb(L, N) * N * (L - N)
    return 4 * n if n <= 1 << 23 else 0


@pytest.mark.parametrize("nroots", [1, 2])
@pytest.mark.parametrize("L,N", [(14, 7), (18, 8)])
def test_admission_leaves_room_for_the_solve_alone(L, N, nroots, dg):
    """A budget that holds the solve but not the neighbour table beside it admits
    the request (which runs without the table), and a batch of handles that
    exist already, tables and all, needs room for its solves alone."""
    import ctypes as C
    from doci_gb300.fcidump import raw_integrals
    one, two = raw_integrals(L, 180)
    opts = dict(nroots=nroots, tol=1e-6, mode="mixed", max_vec=16)
    fp = dg.lib().doci_roots_footprint(L, N, C.byref(dg.batch_opts(**opts)))
    table = nbr_table_bytes(L, N)
    assert 0 < table < fp
    got = {}
    for budget in (fp, fp - table, fp - table - 1):
        with dg.Server(workers=1, hbm_budget=budget, **opts) as srv:
            got[budget] = srv.wait(srv.submit(L, N, one, two))
    assert got[fp - table - 1]["status"] == 9  # DOCI_ERR_ADMISSION
    for b in (fp, fp - table):
        assert got[b]["status"] == 0 and got[b]["converged"] == 1
        assert np.allclose(got[b]["energies"][:nroots], got[fp]["energies"][:nroots], rtol=0, atol=1e-9)
    if nroots > 1:  # (the footprint of one root is that of the single-root solver)
        with dg.Hamiltonian.from_integrals(L, N, 0.0, one, two) as h:
            solve = fp - 12 * h.D - table
            for budget, want in ((solve, 0), (solve - 1, 9)):
                st, res = dg.batch_solve([h], hbm_budget=budget, **opts)
                assert st == res[0]["status"] == want
            assert np.allclose(dg.batch_solve([h], hbm_budget=solve, **opts)[1][0]["energies"][:nroots],
                               got[fp]["energies"][:nroots], rtol=0, atol=1e-9)
