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
