"""doci_multidot (the Davidson projection / subspace-column reduction) on
device buffers: FP64 accumulation, deterministic, both storage types."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 7, 16, 32])
@pytest.mark.parametrize("dtype,prec", [("float64", 0), ("float32", 1)])
def test_multidot(m, dtype, prec):
    import torch
    import doci_gb300
    L = doci_gb300.lib()
    tdt = getattr(torch, dtype)
    n, ld = 1_000_003, 1_000_011
    g = torch.Generator(device="cuda").manual_seed(m + 100 * prec)
    V = torch.randn(m, ld, dtype=tdt, device="cuda", generator=g)
    w = torch.randn(n, dtype=tdt, device="cuda", generator=g)
    out = torch.empty(m, dtype=torch.float64, device="cuda")
    out2 = torch.empty_like(out)
    for o in (out, out2):
        assert L.doci_multidot(C.c_void_p(V.data_ptr()), ld, m, C.c_void_p(w.data_ptr()), n, prec,
                               C.c_void_p(o.data_ptr()), None) == 0
    torch.cuda.synchronize()
    exact = (V[:, :n].double() @ w.double()).cpu().numpy()
    got = out.cpu().numpy()
    scale = V[:, :n].abs().max().item() * w.abs().max().item()
    assert np.abs(got - exact).max() <= 1e-12 * np.sqrt(n) * scale
    assert np.array_equal(got, out2.cpu().numpy())  # fixed reduction order


def test_multidot_invalid():
    import doci_gb300
    L = doci_gb300.lib()
    assert L.doci_multidot(None, 10, 3, None, 10, 0, None, None) == 5


@pytest.mark.parametrize("n", [1, 31, 257, 9_973, 700_001])
@pytest.mark.parametrize("m", [1, 3, 8, 9, 17])
def test_multidot_f32_exact_products(n, m):
    """FP32 storage keeps exact products whatever the size of the values:
    columns of ordinary, tiny (products below FP32's range) and huge (products
    above it) values, a mix of both ends, zeros and one-hot vectors give the
    sums of the exact products to 2^-44 of the sum of their magnitudes (FP32
    error terms of 64-element runs are 2^-24 of 2^-24, with 64 roundings);
    an infinity and a NaN come out as in FP64 arithmetic."""
    import torch
    import doci_gb300
    L = doci_gb300.lib()
    g = torch.Generator(device="cuda").manual_seed(n + m)
    base = torch.randn(m, n, device="cuda", generator=g)
    w0 = torch.randn(n, device="cuda", generator=g)
    hot = torch.zeros(n, device="cuda")
    hot[n // 2] = 1.0
    mixed = torch.where(torch.arange(n, device="cuda") % 3 == 0, 1e25, 1e-25).float()
    cases = [(base, w0), (base * 1e-25, w0 * 1e-20), (base * 1e25, w0 * 1e20), (base * mixed, w0 * 1e-15),
             (base * 0, w0), (hot.repeat(m, 1), hot * 3), (hot.repeat(m, 1) * 1e-30, w0 * 1e-30)]
    out = torch.empty(m, dtype=torch.float64, device="cuda")
    for i, (V, w) in enumerate(cases):
        V = V.contiguous()
        assert L.doci_multidot(V.data_ptr(), n, m, w.data_ptr(), n, 1, out.data_ptr(), None) == 0
        prod = V.double() * w.double()
        exact, size = prod.sum(1), prod.abs().sum(1)
        assert bool(((out - exact).abs() <= 2.0 ** -44 * size).all()), i
    for bad in (float("inf"), float("nan")):
        V, w = base.clone(), w0.clone()
        V[m - 1, n - 1] = bad
        assert L.doci_multidot(V.data_ptr(), n, m, w.data_ptr(), n, 1, out.data_ptr(), None) == 0
        exact = (V.double() * w.double()).sum(1)
        assert torch.equal(torch.isnan(out), torch.isnan(exact)) and torch.equal(torch.isinf(out), torch.isinf(exact))


@pytest.mark.parametrize("n,m", [(1, 1), (33, 3), (1023, 4), (1025, 5), (4097, 32), (155649, 17), (319770, 16),
                                 (622593, 2)])
def test_multidot_fp64_grid_edges(n, m):
    """FP64 columns at the edges of the grid (one block, one more than a block's
    four elements per thread, more elements than one wave takes at once): the
    sums to n roundings of the sum of magnitudes."""
    import torch
    import doci_gb300
    g = torch.Generator(device="cuda").manual_seed(n + m)
    V = torch.randn(m, n, device="cuda", generator=g, dtype=torch.float64)
    w = torch.randn(n, device="cuda", generator=g, dtype=torch.float64)
    out = torch.empty(m, dtype=torch.float64, device="cuda")
    assert doci_gb300.lib().doci_multidot(V.data_ptr(), n, m, w.data_ptr(), n, 0, out.data_ptr(), None) == 0
    prod = V * w
    assert bool(((out - prod.sum(1)).abs() <= 2 * n * 2.0 ** -53 * prod.abs().sum(1)).all())


@pytest.mark.parametrize("L,N,max_vec", [(1, 1, 2), (3, 1, 9), (8, 4, 2), (8, 4, 8), (10, 5, 9), (10, 4, 16),
                                         (10, 5, 17), (12, 6, 32)])
def test_fp64_davidson_basis_sizes(L, N, max_vec, synth):
    """FP64 Davidson with bases at the edges of its passes' column counts (8, 16,
    32) on spaces of less than a warp to several blocks: a normalised vector
    whose residual, formed by the oracle, is the reported one, and the energy
    of an eigenvalue.  Residuals below 1e-10 bound the energy's error; the
    oracle's own sums are good to about 1e-12 here."""
    import doci_gb300 as dg
    import oracle
    p = synth(L, N, 300 + L + max_vec)
    o = oracle.Ham(p)
    with dg.Hamiltonian.from_fcidump(p) as h:
        H = np.stack([np.asarray(o.matvec(e)) for e in np.eye(h.D)])
        res, v = h.solve(solver="D", mode="fp64", tol=1e-10, max_its=400, davidson_max_vec=max_vec,
                          davidson_keep=1)
    v = np.asarray(v)
    e = res["energy"]
    assert res["converged"] and abs(np.linalg.norm(v) - 1) < 1e-12
    assert np.linalg.norm(H @ v - (v @ H @ v) * v) < 1e-9
    assert np.abs(np.linalg.eigvalsh(H) - e).min() < 1e-9


@pytest.mark.parametrize("n,m", [(1001, 3), (300_001, 4), (3_000_001, 5), (5_000_003, 9)])
def test_multidot_f32_cancelling_sums(n, m):
    """FP32 vectors whose products nearly cancel: the error of the sums is no more
    than that of FP64 additions of the exact products in the kernel's order (runs
    of 64 or less per thread, then the threads', warps' and blocks' sums: at most 2 sqrt(64)
    roundings at 2^-53 of a thread's sum, and the result's own), where pairs of
    floats in a run would leave 2^-48 of each term."""
    import math
    import torch
    import doci_gb300
    g = torch.Generator(device="cuda").manual_seed(n + m)
    V = torch.randn(m, n, device="cuda", generator=g)
    w = torch.randn(n, device="cuda", generator=g)
    out = torch.empty(m, dtype=torch.float64, device="cuda")
    assert doci_gb300.lib().doci_multidot(V.data_ptr(), n, m, w.data_ptr(), n, 1, out.data_ptr(), None) == 0
    p = (V.double() * w.double()).cpu().numpy()
    for k in range(m):
        exact, size = math.fsum(p[k]), np.abs(p[k]).sum()
        # independent roundings: those of the terms' sums add up as sqrt(n) of sqrt(run) 2^-53 |p|
        bound = 16 * 2.0 ** -53 * np.sqrt(n) * (size / n) + 4 * 2.0 ** -53 * abs(exact)
        assert abs(out[k].item() - exact) <= bound, (k, abs(out[k].item() - exact) / size)
