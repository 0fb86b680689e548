"""GPU sigma / diagonal / addressing parity against the oracle and the
reference's golden fixtures.  Every call goes through the C ABI of
libdoci_gb300.so (doci_gb300._lib is a ctypes binding)."""
import os

import numpy as np
import pytest

import oracle
from conftest import GOLDEN

pytestmark = pytest.mark.gpu

SMALL = ["H2O_STO3G", "N2_STO3G", "H2O_631G", "lili_321g", "synthetic_L14_N7_s1", "synthetic_L10_N5_s3"]
# sigma tolerance: max|y_gpu - y_ref| <= tol * max|y_ref| (FP64 1e-12; FP32 storage/accumulation 2e-6)
TOL64, TOL32 = 1e-12, 2e-6


@pytest.fixture(scope="module")
def dg():
    import doci_gb300
    doci_gb300.lib()
    return doci_gb300


def torch_cuda():
    import torch
    assert torch.cuda.is_available()
    return torch


@pytest.mark.parametrize("name", SMALL)
def test_golden_sigma_diag_bits(name, fcidump, dg):
    z = np.load(os.path.join(GOLDEN, f"sigma_{name}.npz"))
    with dg.Hamiltonian.from_fcidump(fcidump(name)) as h:
        assert h.D == len(z["x"])
        assert np.array_equal(h.diagonal(), z["diag"])  # bit-identical to the reference
        y = h.sigma(z["x"], dg.FP64)
        assert np.abs(y - z["sigma"]).max() <= TOL64 * np.abs(z["sigma"]).max()
        y32 = h.sigma(z["x"].astype(np.float32), dg.FP32)
        assert np.abs(y32 - z["sigma"]).max() <= TOL32 * np.abs(z["sigma"]).max()
        torch = torch_cuda()
        bits = torch.empty(h.D, dtype=torch.int32, device="cuda")
        h.bitstrings_device(0, h.D, bits.data_ptr())
        torch.cuda.synchronize()
        assert np.array_equal(bits.cpu().numpy().view(np.uint32), z["bitstrings"])
        ranks = torch.empty(h.D, dtype=torch.int64, device="cuda")
        h.ranks_device(bits.data_ptr(), h.D, ranks.data_ptr())
        torch.cuda.synchronize()
        assert np.array_equal(ranks.cpu().numpy(), np.arange(h.D))


@pytest.mark.parametrize("kernel", ["auto", "gather", "row1", "rowx", "pair", "tc", "rowff"])
@pytest.mark.parametrize("L,N,seed", [(16, 8, 21), (18, 5, 22), (20, 10, 23), (12, 1, 24), (12, 11, 25),
                                      (7, 0, 26), (6, 6, 27), (32, 2, 28), (32, 30, 29), (24, 12, 30),
                                      (22, 11, 31), (26, 4, 32)])
def test_sigma_vs_oracle(L, N, seed, kernel, synth, dg):
    p = synth(L, N, seed)
    o = oracle.Ham(p)
    with dg.Hamiltonian.from_fcidump(p) as h:
        h.set_sigma_kernel(kernel)
        assert h.D == o.D
        assert np.array_equal(h.diagonal(), o.diag)
        x = np.random.default_rng(seed).standard_normal(h.D)
        yr = o.matvec(x)
        y = h.sigma(x, dg.FP64)
        assert np.abs(y - yr).max() <= TOL64 * np.abs(yr).max()
        y32 = h.sigma(x.astype(np.float32), dg.FP32)
        assert np.abs(y32 - yr).max() <= TOL32 * np.abs(yr).max()


def test_addressing_full_size_properties(synth, dg):
    """L=32, N=16 (D = 601,080,390): unrank -> rank round trip over sampled
    windows, lexical order (strictly increasing as 32-bit reversed strings is
    not the order; use the oracle's rank on samples instead)."""
    torch = torch_cuda()
    p = synth(32, 16, 3)
    with dg.Hamiltonian.from_fcidump(p) as h:
        assert h.D == 601080390
        for first in (0, 123456789, h.D - 4096, 300000000):
            n = min(4096, h.D - first)
            bits = torch.empty(n, dtype=torch.int32, device="cuda")
            h.bitstrings_device(first, n, bits.data_ptr())
            ranks = torch.empty(n, dtype=torch.int64, device="cuda")
            h.ranks_device(bits.data_ptr(), n, ranks.data_ptr())
            torch.cuda.synchronize()
            b = bits.cpu().numpy().view(np.uint32)
            assert np.array_equal(ranks.cpu().numpy(), np.arange(first, first + n))
            for k in range(0, n, 511):
                assert oracle.lib().orc_unrank(first + k, 32, 16) == b[k]
            assert all(bin(int(v)).count("1") == 16 for v in b[:64])


@pytest.mark.parametrize("kernel", ["auto", "gather", "row1", "rowx", "pair", "tc", "rowff"])
def test_sigma_full_size_symmetry_and_linearity(kernel, synth, dg):
    """L=28, N=14 (D = 40,116,600): H is symmetric, sigma is linear, and
    sampled rows agree with the oracle's gather form."""
    torch = torch_cuda()
    p = synth(28, 14, 2)
    o = oracle.Ham(p, keep_diag=False)
    with dg.Hamiltonian.from_fcidump(p) as h:
        h.set_sigma_kernel(kernel)
        D = h.D
        g = torch.Generator(device="cuda").manual_seed(7)
        x = torch.randn(D, dtype=torch.float64, device="cuda", generator=g)
        z = torch.randn(D, dtype=torch.float64, device="cuda", generator=g)
        hx = torch.empty_like(x)
        hz = torch.empty_like(x)
        h.sigma_device(x.data_ptr(), hx.data_ptr(), dg.FP64)
        h.sigma_device(z.data_ptr(), hz.data_ptr(), dg.FP64)
        w = 0.25 * x - 2.0 * z
        hw = torch.empty_like(x)
        h.sigma_device(w.data_ptr(), hw.data_ptr(), dg.FP64)
        torch.cuda.synchronize()
        a, b = float(torch.dot(z, hx)), float(torch.dot(x, hz))
        assert abs(a - b) <= 1e-12 * max(abs(a), 1.0) * 10
        lin = (hw - (0.25 * hx - 2.0 * hz)).abs().max().item()
        assert lin <= 1e-12 * hw.abs().max().item()
        xs = x.cpu().numpy()
        first = np.array([0, 17_000_000, D - 1000], dtype=np.uint64)
        length = np.array([1000, 1000, 1000], dtype=np.uint64)
        rows = np.concatenate([np.arange(f, f + n) for f, n in zip(first, length)]).astype(np.int64)
        dg_rows = h.diagonal()[rows]
        ref = o.gather_rows(xs, first, length, dg_rows)
        got = hx.cpu().numpy()[rows]
        assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("kernel", ["auto", "gather", "row1", "rowx", "pair", "tc"])
def test_sigma_L32_fp32_vs_oracle_samples(kernel, synth, dg):
    """L=32, N=16 (D = 601,080,390), FP32: sampled rank windows across the
    whole space (start, middle, end) against the FP64 oracle gather form."""
    torch = torch_cuda()
    p = synth(32, 16, 3)
    o = oracle.Ham(p, keep_diag=False)
    with dg.Hamiltonian.from_fcidump(p) as h:
        D = h.D
        h.set_sigma_kernel(kernel)
        g = torch.Generator(device="cuda").manual_seed(3)
        x = torch.randn(D, dtype=torch.float32, device="cuda", generator=g)
        y = torch.empty_like(x)
        h.sigma_device(x.data_ptr(), y.data_ptr(), dg.FP32)  # default stream: ordered after randn
        torch.cuda.synchronize()
        first = np.array([0, 12_870, 150_000_000, 300_540_000, 450_000_000, D - 20_000, D - 1000],
                         dtype=np.uint64)
        length = np.full(len(first), 1000, dtype=np.uint64)
        rows = np.concatenate([np.arange(f, f + n) for f, n in zip(first, length)]).astype(np.int64)
        xs = x.double().cpu().numpy()
        ref = o.gather_rows(xs, first, length, h.diagonal()[rows])
        got = y.cpu().numpy()[rows]
        err = np.abs(got - ref)
        bad = np.nonzero(err > 2e-6 * np.abs(ref).max())[0]
        assert bad.size == 0, (kernel, int(rows[bad[0]]), float(got[bad[0]]), float(ref[bad[0]]), int(bad.size))


@pytest.mark.parametrize("kernel", ["auto", "rowx", "gather", "rowff"])
def test_sigma_L32_fp64_vs_oracle_samples(kernel, synth, dg):
    """L=32, N=16 (D = 601,080,390), FP64 (the anchor and verification sigma
    of every mixed solve at this size): sampled rank windows across the whole
    space against the FP64 oracle gather form, 1e-12 of the largest |sigma|."""
    torch = torch_cuda()
    p = synth(32, 16, 3)
    o = oracle.Ham(p, keep_diag=False)
    with dg.Hamiltonian.from_fcidump(p) as h:
        D = h.D
        h.set_sigma_kernel(kernel)
        g = torch.Generator(device="cuda").manual_seed(11)
        x = torch.randn(D, dtype=torch.float64, device="cuda", generator=g)
        y = torch.empty_like(x)
        h.sigma_device(x.data_ptr(), y.data_ptr(), dg.FP64)
        torch.cuda.synchronize()
        first = np.array([0, 12_870, 150_000_000, 300_540_000, 450_000_000, D - 20_000, D - 1000],
                         dtype=np.uint64)
        length = np.full(len(first), 1000, dtype=np.uint64)
        rows = np.concatenate([np.arange(f, f + n) for f, n in zip(first, length)]).astype(np.int64)
        idx = torch.from_numpy(rows).cuda()
        xs = x.cpu().numpy()
        ref = o.gather_rows(xs, first, length, h.diagonal()[rows])
        got = y[idx].cpu().numpy()
        del x, y
        err = np.abs(got - ref)
        bad = np.nonzero(err > 1e-12 * np.abs(ref).max())[0]
        assert bad.size == 0, (kernel, int(rows[bad[0]]), float(got[bad[0]]), float(ref[bad[0]]), int(bad.size))


def test_default_stream_orders_after_caller_work(synth, dg):
    """A NULL stream is CUDA's default stream: a sigma queued right after the
    caller's own kernels on it sees their results (x written by randn)."""
    torch = torch_cuda()
    p = synth(28, 14, 2)
    with dg.Hamiltonian.from_fcidump(p) as h:
        outs = []
        for kernel in ("gather", "row1", "tc"):
            h.set_sigma_kernel(kernel)
            g = torch.Generator(device="cuda").manual_seed(9)
            x = torch.randn(h.D, dtype=torch.float32, device="cuda", generator=g)
            y = torch.empty_like(x)
            h.sigma_device(x.data_ptr(), y.data_ptr(), dg.FP32)
            outs.append(y)
        torch.cuda.synchronize()
        for o in outs[1:]:
            assert (outs[0] - o).abs().max().item() <= 2e-6 * outs[0].abs().max().item()


@pytest.mark.parametrize("kernel", ["auto", "gather", "row1"])
@pytest.mark.parametrize("L,N,seed,nv", [(16, 8, 41, 3), (20, 10, 42, 4), (12, 1, 43, 2), (24, 12, 44, 7),
                                         (18, 17, 45, 4), (26, 4, 46, 5)])
def test_sigma_block_vs_oracle(L, N, seed, nv, kernel, synth, dg):
    """doci_sigma_block: nv column-major vectors with padded leading
    dimensions against the oracle's matvec of each column (FP64 1e-12, FP32
    2e-6 of max|y|), and against doci_sigma column by column."""
    torch = torch_cuda()
    p = synth(L, N, seed)
    o = oracle.Ham(p)
    with dg.Hamiltonian.from_fcidump(p) as h:
        h.set_sigma_kernel(kernel)
        D = h.D
        ldx, ldy = D + 5, D + 3
        rng = np.random.default_rng(seed)
        X = rng.standard_normal((nv, D))
        refs = [o.matvec(X[v]) for v in range(nv)]
        for prec, dt, tol in ((dg.FP64, torch.float64, TOL64), (dg.FP32, torch.float32, TOL32)):
            xb = torch.zeros(nv * ldx, dtype=dt, device="cuda")
            for v in range(nv):
                xb[v * ldx:v * ldx + D] = torch.from_numpy(X[v]).to(dt)
            yb = torch.full((nv * ldy,), 7.0, dtype=dt, device="cuda")
            h.sigma_block_device(xb.data_ptr(), ldx, yb.data_ptr(), ldy, nv, prec)
            y1 = torch.empty(D, dtype=dt, device="cuda")
            torch.cuda.synchronize()
            for v in range(nv):
                y = yb[v * ldy:v * ldy + D].double().cpu().numpy()
                assert np.abs(y - refs[v]).max() <= tol * np.abs(refs[v]).max()
                if v < nv - 1:  # padding between columns untouched
                    assert bool((yb[v * ldy + D:(v + 1) * ldy] == 7.0).all())
                h.sigma_device(xb[v * ldx:].data_ptr(), y1.data_ptr(), prec)
                torch.cuda.synchronize()
                ys = y1.double().cpu().numpy()
                assert np.abs(y - ys).max() <= tol * np.abs(refs[v]).max()
                if kernel in ("gather", "row1"):  # same kernel family: same summation order
                    assert np.array_equal(y, ys)


def test_sigma_plan(synth, dg):
    """doci_sigma_plan reports the path doci_sigma takes: the automatic choice
    resolves to the mma.sync pair form for FP32 (a diag * x pass and the pair
    pass) and to the float-float pair form for FP64 (x conversion with the
    diag * x pass, and the pair pass) once the tiling gives every SM work (or
    to the shape's tuned choice), the gather kernel on small spaces; an explicit
    kind is honoured (the tensor-core pair form: one launch for the rows
    without column elements and one per row-part size of the (N-1)-pair sets,
    11 at L=20, N=10, split 9), FP32-only kinds take the automatic FP64 path,
    and the removed kinds are refused."""
    with dg.Hamiltonian.from_fcidump(synth(20, 10, 51)) as h:
        assert h.sigma_plan(dg.FP32) == (6, 2)
        auto64 = h.sigma_plan(dg.FP64)
        assert auto64 in ((9, 2), (1, 1), (3, 1), (4, 1))  # the float-float pair form, or a tuned choice
        h.set_sigma_kernel("row1")
        assert h.sigma_plan(dg.FP32) == (3, 1)
        h.set_sigma_kernel("pair")
        assert h.sigma_plan(dg.FP32) == (6, 2)
        assert h.sigma_plan(dg.FP64) == auto64  # FP32 only
        h.set_sigma_kernel("tc")
        assert h.sigma_plan(dg.FP32) == (8, 11)
        assert h.sigma_plan(dg.FP64) == auto64
        h.set_sigma_kernel("rowff")
        assert h.sigma_plan(dg.FP64) == (9, 2)
        assert h.sigma_plan(dg.FP32) == (6, 2)  # FP64 only
        for bad in (2, 5, 7, 10, -1):
            with pytest.raises(dg.DociError):
                h.set_sigma_kernel(bad)
    with dg.Hamiltonian.from_fcidump(synth(12, 6, 52)) as h:
        assert h.sigma_plan(dg.FP32) == (1, 1)
        assert h.sigma_plan(dg.FP64) == (1, 1)


@pytest.mark.parametrize("prec_name", ["FP64", "FP32"])
def test_sigma_host_pinned_and_pageable(prec_name, synth, dg):
    """doci_sigma_host on pinned host buffers (copied by kernels through
    their device mapping), on pageable ones (cudaMemcpyAsync), and on an
    offset inside a pinned buffer: all equal doci_sigma on device buffers."""
    torch = torch_cuda()
    import ctypes as C
    prec = getattr(dg, prec_name)
    tdt = torch.float64 if prec == dg.FP64 else torch.float32
    with dg.Hamiltonian.from_fcidump(synth(18, 9, 61)) as h:
        h.set_sigma_kernel("row1")  # deterministic: results compare bit for bit
        D = h.D
        x = torch.randn(D + 7, dtype=tdt, generator=torch.Generator().manual_seed(3))
        xd = x[:D].cuda()
        yd = torch.empty_like(xd)
        h.sigma_device(xd.data_ptr(), yd.data_ptr(), prec)
        torch.cuda.synchronize()
        ref = yd.cpu()
        lib = dg.lib()
        for pinned, off in ((True, 0), (True, 3), (False, 0)):
            xs = x.pin_memory() if pinned else x.clone()
            ys = torch.full((D + 7,), float("nan"), dtype=tdt)
            ys = ys.pin_memory() if pinned else ys
            src = xs[off:off + D] if off else xs[:D]
            if off:  # same values at an offset inside the buffer
                src.copy_(x[:D])
            st = lib.doci_sigma_host(h.handle, C.c_void_p(src.data_ptr()), C.c_void_p(ys[off:].data_ptr()), prec)
            assert st == 0
            assert torch.equal(ys[off:off + D], ref), (pinned, off)


@pytest.mark.parametrize("prec_name,kernel", [("FP32", "pair"), ("FP64", "rowff")])
@pytest.mark.parametrize("L,N,seed,off,pinned", [(22, 11, 31, 0, True), (24, 12, 30, 3, True), (20, 7, 33, 1, True),
                                                 (22, 11, 34, 0, False)])
def test_sigma_host_pair_overlapped_copies(prec_name, kernel, L, N, seed, off, pinned, synth, dg):
    """doci_sigma_host on the pair forms (FP32 kind 6, FP64-accurate kind 9)
    uploads x in pieces on a copy stream while the unit groups whose rows
    have all arrived run (each piece's diagonal pass before the first group
    reaching it) and downloads a pinned y piece by piece as no later group
    reaches it: the result matches the oracle within the precision's
    tolerance, for buffers at an offset and for pageable ones, and a second
    call on the same handle (reused stream, events, staging) agrees with the
    first."""
    torch = torch_cuda()
    import ctypes as C
    prec = getattr(dg, prec_name)
    tdt, tol = (torch.float32, TOL32) if prec == dg.FP32 else (torch.float64, TOL64)
    p = synth(L, N, seed)
    o = oracle.Ham(p)
    with dg.Hamiltonian.from_fcidump(p) as h:
        h.set_sigma_kernel(kernel)
        assert h.sigma_plan(prec)[0] == (6 if prec == dg.FP32 else 9)
        D = h.D
        x = np.random.default_rng(seed).standard_normal(D)
        yr = o.matvec(x)
        xs = torch.zeros(D + 8, dtype=tdt)
        ys = torch.full((D + 8,), float("nan"), dtype=tdt)
        if pinned:
            xs, ys = xs.pin_memory(), ys.pin_memory()
        xs[off:off + D] = torch.from_numpy(x).to(tdt)
        lib = dg.lib()
        outs = []
        for _ in range(2):
            st = lib.doci_sigma_host(h.handle, C.c_void_p(xs[off:].data_ptr()), C.c_void_p(ys[off:].data_ptr()), prec)
            assert st == 0
            outs.append(ys[off:off + D].numpy().astype(np.float64).copy())
        for y in outs:
            assert np.abs(y - yr).max() <= tol * np.abs(yr).max()
        assert np.abs(outs[0] - outs[1]).max() <= tol * np.abs(yr).max()


def test_autotune_keeps_parity(synth, dg):
    """doci_ham_autotune picks a path that fits, the plan reports it, sigma on
    the tuned path still matches the oracle, and a second handle of the same
    shape uses the same choice; block sigmas after tuning match too."""
    torch = torch_cuda()
    p = synth(20, 10, 71)
    o = oracle.Ham(p)
    with dg.Hamiltonian.from_fcidump(p) as h, dg.Hamiltonian.from_fcidump(synth(20, 10, 72)) as h2:
        for prec, tol in ((dg.FP32, TOL32), (dg.FP64, TOL64)):
            kind = h.autotune(prec, 1)
            assert kind in (1, 3, 4, 6)
            assert h.sigma_plan(prec)[0] == kind and h2.sigma_plan(prec)[0] == kind
            x = np.random.default_rng(7).standard_normal(h.D)
            yr = o.matvec(x)
            y = h.sigma(x.astype(np.float32) if prec == dg.FP32 else x, prec)
            assert np.abs(y - yr).max() <= tol * np.abs(yr).max()
            method = h.autotune(prec, 3)
            assert method in (1, 2, 3)
            tdt = torch.float64 if prec == dg.FP64 else torch.float32
            X = torch.from_numpy(np.random.default_rng(8).standard_normal((3, h.D))).to(tdt).cuda()
            Y = torch.empty_like(X)
            h.sigma_block_device(X.data_ptr(), h.D, Y.data_ptr(), h.D, 3, prec)
            torch.cuda.synchronize()
            for v in range(3):
                ref = o.matvec(X[v].double().cpu().numpy())
                assert np.abs(Y[v].double().cpu().numpy() - ref).max() <= tol * np.abs(ref).max()


@pytest.mark.parametrize("L,N,seed,off", [
    (10, 1, 81, 0), (10, 5, 82, 1), (11, 10, 83, 2), (13, 13, 84, 3), (32, 2, 85, 1),  # 8 column orbitals
    (22, 8, 86, 3), (23, 9, 87, 1), (24, 20, 88, 0),  # 10
    (28, 6, 89, 1), (26, 19, 90, 3),  # 12
])
def test_sigma_pair_warp_edges(L, N, seed, off, synth, dg):
    """The warp-per-unit pair form on each of its tilings (8, 10 and 12 column
    orbitals), at the smallest and nearly full spaces, odd lengths and buffers
    off 16-byte alignment, with y full of NaN before the call: the oracle's
    matvec within the FP32 sigma tolerance, nothing written around y."""
    torch = torch_cuda()
    p = synth(L, N, seed)
    o = oracle.Ham(p)
    with dg.Hamiltonian.from_fcidump(p) as h:
        h.set_sigma_kernel("pair")
        assert h.sigma_plan(dg.FP32)[0] == 6
        D = h.D
        x = np.random.default_rng(seed).standard_normal(D).astype(np.float32)
        xs = torch.zeros(D + 8, dtype=torch.float32, device="cuda")
        xs[off:off + D] = torch.from_numpy(x)
        ys = torch.full((D + 8,), float("nan"), dtype=torch.float32, device="cuda")
        h.sigma_device(xs[off:].data_ptr(), ys[off:].data_ptr(), dg.FP32)
        torch.cuda.synchronize()
        yr = o.matvec(x.astype(np.float64))
        y = ys.double().cpu().numpy()
        assert np.abs(y[off:off + D] - yr).max() <= TOL32 * np.abs(yr).max()
        assert np.isnan(y[:off]).all() and np.isnan(y[off + D:]).all()


@pytest.mark.parametrize("L,N,seed", [
    (10, 1, 91), (10, 5, 92), (11, 10, 93), (13, 13, 94), (32, 2, 95), (32, 30, 96),  # 8 column orbitals
    (22, 8, 97), (24, 20, 98),  # 10
    (28, 6, 99), (26, 19, 100),  # 12
])
def test_sigma_fp64_warp_edges(L, N, seed, synth, dg):
    """The FP64-accurate pair form on each of its tilings, with values over
    many orders of magnitude: random vectors, one-hot, all equal, falling off
    over 2^-60, and small and large overall scales, each against the oracle's
    matvec of the same vector within 1e-12 of its largest element."""
    torch = torch_cuda()
    p = synth(L, N, seed)
    o = oracle.Ham(p)
    rng = np.random.default_rng(seed)
    with dg.Hamiltonian.from_fcidump(p) as h:
        h.set_sigma_kernel("rowff")
        assert h.sigma_plan(dg.FP64) == (9, 2)
        D = h.D
        base = rng.standard_normal(D)
        hot = np.zeros(D)
        hot[D // 2] = -3.0
        vecs = [base, hot, np.ones(D), np.full(D, 1 / 3), base * np.exp2(-60 * rng.random(D)), base * 1e-20,
                base * 1e25, np.where(rng.random(D) < 0.5, 1.0, -1.0)]
        y = torch.empty(D, dtype=torch.float64, device="cuda")
        for i, x in enumerate(vecs):
            xd = torch.from_numpy(x).cuda()
            y.fill_(float("nan"))
            h.sigma_device(xd.data_ptr(), y.data_ptr(), dg.FP64)
            torch.cuda.synchronize()
            ref = o.matvec(x)
            assert np.abs(y.cpu().numpy() - ref).max() <= TOL64 * np.abs(ref).max(), i


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("prec_name,kernel", [("FP32", "pair"), ("FP64", "rowff")])
@pytest.mark.parametrize("L,N,seed", [(12, 6, 101), (22, 8, 102)])
def test_sigma_pair_warp_nonfinite(L, N, seed, prec_name, kernel, bad, synth, dg):
    """An infinity or a NaN in x reaches the same elements of sigma (its own and
    its neighbours') as in the gather kernel, and no others."""
    torch = torch_cuda()
    prec = getattr(dg, prec_name)
    tdt = torch.float64 if prec == dg.FP64 else torch.float32
    with dg.Hamiltonian.from_fcidump(synth(L, N, seed)) as h:
        x = torch.randn(h.D, dtype=tdt, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))
        x[h.D // 3] = bad
        out = []
        for k in ("gather", kernel):
            h.set_sigma_kernel(k)
            y = torch.empty_like(x)
            h.sigma_device(x.data_ptr(), y.data_ptr(), prec)
            torch.cuda.synchronize()
            out.append(torch.isfinite(y))
        assert torch.equal(out[0], out[1]) and int((~out[0]).sum()) == N * (L - N) + 1


@pytest.mark.parametrize("L,N,seed,nv", [(18, 9, 111, 2), (20, 13, 112, 3), (22, 8, 113, 5), (23, 17, 114, 1),
                                         (28, 6, 115, 2), (32, 4, 116, 3)])
def test_sigma_block_reproducible(L, N, seed, nv, synth, dg):
    """The automatic block sigma (the pair form with contributions stored apart
    on these sizes: 8, 10 and 12 column orbitals, many and few pairs) gives the
    oracle's matvec of each column and the same bits when called again."""
    torch = torch_cuda()
    p = synth(L, N, seed)
    o = oracle.Ham(p)
    with dg.Hamiltonian.from_fcidump(p) as h:
        D = h.D
        X = np.random.default_rng(seed).standard_normal((nv, D))
        refs = [o.matvec(x) for x in X]
        for prec, dt, tol in ((dg.FP64, torch.float64, TOL64), (dg.FP32, torch.float32, TOL32)):
            xb = torch.from_numpy(X).to(dt).cuda()
            outs = []
            for _ in range(2):
                y = torch.full((nv, D + 1), float("nan"), dtype=dt, device="cuda")
                h.sigma_block_device(xb.data_ptr(), D, y.data_ptr(), D + 1, nv, prec)
                torch.cuda.synchronize()
                outs.append(y[:, :D].clone())
                assert bool(torch.isnan(y[:, D]).all())
            assert torch.equal(outs[0], outs[1])
            for v in range(nv):
                assert np.abs(outs[0][v].double().cpu().numpy() - refs[v]).max() <= tol * np.abs(refs[v]).max()


@pytest.mark.parametrize("L,N,seed,nv", [(1, 1, 121, 1), (2, 1, 122, 2), (3, 1, 123, 4), (7, 6, 124, 3), (9, 4, 125, 5),
                                         (13, 5, 126, 2), (32, 1, 127, 3), (32, 31, 128, 4), (32, 3, 129, 2),
                                         (19, 9, 130, 1), (20, 7, 131, 4)])
def test_sigma_neighbour_table(L, N, seed, nv, synth, dg):
    """The gather kernel from the neighbour table (small spaces, the automatic
    choice there), on spaces of one determinant up to nearly the largest with
    a table (92,378 determinants of 90 hops): the oracle's matvec, single and block calls bit for bit alike, y
    written nowhere else."""
    torch = torch_cuda()
    p = synth(L, N, seed)
    o = oracle.Ham(p)
    with dg.Hamiltonian.from_fcidump(p) as h:
        D = h.D
        X = np.random.default_rng(seed).standard_normal((nv, D))
        for prec, dt, tol in ((dg.FP64, torch.float64, TOL64), (dg.FP32, torch.float32, TOL32)):
            assert h.sigma_plan(prec) == (1, 1)
            xb = torch.from_numpy(X).to(dt).cuda()
            yb = torch.full((nv, D + 3), 7.0, dtype=dt, device="cuda")
            h.sigma_block_device(xb.data_ptr(), D, yb.data_ptr(), D + 3, nv, prec)
            y1 = torch.full((D + 3,), 7.0, dtype=dt, device="cuda")
            for v in range(nv):
                h.sigma_device(xb[v].data_ptr(), y1.data_ptr(), prec)
                torch.cuda.synchronize()
                ref = o.matvec(X[v])
                assert torch.equal(y1[:D], yb[v, :D]) and bool((yb[v, D:] == 7.0).all() and (y1[D:] == 7.0).all())
                assert np.abs(y1[:D].double().cpu().numpy() - ref).max() <= tol * max(np.abs(ref).max(), 1e-300)


def pair_integrals(h1, K):
    """Integrals with the pair hops K (symmetric) and no Coulomb part: the
    diagonal is sum_i 2 h_i - sum_{i,j} K_ij over the pairs."""
    L = len(h1)
    eri = np.zeros((L, L, L, L))
    i, j = np.nonzero(~np.eye(L, dtype=bool))
    for a, b, c, d in ((i, j, i, j), (i, j, j, i)):
        eri[a, b, c, d] = K[i, j]
    return np.diag(np.asarray(h1, dtype=np.float64)), eri


@pytest.mark.parametrize("L,N", [(27, 3), (32, 2), (19, 3)])
def test_fp64_pair_form_constant_hops(L, N, dg):
    """A pure pairing Hamiltonian (constant K) on constant vectors with 17 to 31
    open slots, whose digits all add up with one sign: within 2^-45 of the sum
    of the terms' magnitudes.  (What is cut is below 2^-51, a set's product is
    rounded to 2^-48, and the own rows' pairs of floats to 2^-47 per addition.)"""
    torch = torch_cuda()
    rng = np.random.default_rng(L)
    for k in range(8):
        c = rng.uniform(0.5, 1)
        K = c * (1 - np.eye(L))
        with dg.Hamiltonian.from_integrals(L, N, 0.0, *pair_integrals(np.linspace(-1, 1, L), K)) as h:
            h.set_sigma_kernel("rowff")
            assert h.sigma_plan(dg.FP64)[0] == 9
            dx = h.diagonal().astype(np.longdouble)
            y = torch.empty(h.D, dtype=torch.float64, device="cuda")
            for v in rng.uniform(0.5, 1, 12):
                x = torch.full((h.D,), v, dtype=torch.float64, device="cuda")
                h.sigma_device(x.data_ptr(), y.data_ptr(), dg.FP64)
                torch.cuda.synchronize()
                hops = N * (L - N) * np.longdouble(c) * np.longdouble(v)
                err = np.abs(y.cpu().numpy() - (dx * v + hops))
                assert (err <= 2.0 ** -45 * (np.abs(dx * v) + hops)).all(), (k, v, float((err / hops).max()))


def exact_sigma(h, L, K, X):
    """sigma of the vectors X in long double, with the handle's diagonal, and
    the sum of its terms' magnitudes, for small spaces."""
    torch = torch_cuda()
    bits = torch.empty(h.D, dtype=torch.int32, device="cuda")
    h.bitstrings_device(0, h.D, bits.data_ptr())
    bits = bits.cpu().numpy().astype(np.int64) & 0xffffffff
    at = {int(b): r for r, b in enumerate(bits)}
    y = h.diagonal().astype(np.longdouble) * X
    mag = np.abs(y)
    for r, b in enumerate(int(v) for v in bits):
        for i in range(L):
            for a in range(L):
                if b >> i & 1 and not b >> a & 1:
                    t = np.longdouble(K[i, a]) * X[:, at[b ^ (1 << i) ^ (1 << a)]]
                    y[:, r] += t
                    mag[:, r] += np.abs(t)
    return y, mag


def graded_hops(L, how, f, rng):
    """K between 1/2 and 1, graded by f: "core" K_ij s_i s_j with s falling from 1
    to f over the orbitals, "small" with every other orbital's row at f, "fragments" two halves
    with f between them."""
    K = rng.uniform(0.5, 1, (L, L))
    K = np.triu(K, 1) + np.triu(K, 1).T
    if how == "core":
        s = f ** (np.arange(L) / (L - 1))
        return K * s[:, None] * s[None, :]
    if how == "small":
        s = np.where(np.arange(L) % 2, f, 1.0)
        return K * np.minimum(s[:, None], s[None, :])
    half = np.arange(L) < L // 2
    return np.where(half[:, None] == half[None, :], K, f * K)


@pytest.mark.parametrize("how,f", [("core", 0.5), ("core", 1e-2), ("core", 1e-5), ("small", 1e-2), ("small", 1e-4),
                                   ("small", 1e-10), ("fragments", 1e-1), ("fragments", 1e-6)])
def test_fp64_pair_form_graded_hops(how, f, dg):
    """Every component of the FP64-accurate pair form, also one that only small
    elements of K reach (one-hot vectors), to the float pairs' accuracy: seven
    open slots at 2^-47 each, 2^-44 of the sum of the terms' magnitudes."""
    torch = torch_cuda()
    L, N = 12, 6
    rng = np.random.default_rng(12)
    K = graded_hops(L, how, f, rng)
    with dg.Hamiltonian.from_integrals(L, N, 0.0, *pair_integrals(np.linspace(-1, 1, L), K)) as h:
        h.set_sigma_kernel("rowff")
        assert h.sigma_plan(dg.FP64)[0] == 9
        X = np.concatenate([np.eye(h.D)[[0, h.D // 3, h.D - 1]], rng.standard_normal((2, h.D))])
        ref, mag = exact_sigma(h, L, K, X)
        y = torch.empty(h.D, dtype=torch.float64, device="cuda")
        for v, x in enumerate(X):
            xd = torch.from_numpy(x).cuda()
            h.sigma_device(xd.data_ptr(), y.data_ptr(), dg.FP64)
            torch.cuda.synchronize()
            assert (np.abs(y.cpu().numpy() - ref[v]) <= 2.0 ** -44 * mag[v]).all(), v


@pytest.mark.parametrize("how,f", [("core", 0.5), ("small", 1e-8)])
def test_fp64_graded_hops_automatic(how, f, dg):
    """The same on a space without a neighbour table, through the automatic
    single and block sigmas: on one-hot vectors every element of sigma is one product, as
    the FP64 row pass forms it."""
    torch = torch_cuda()
    L, N = 20, 10
    K = graded_hops(L, how, f, np.random.default_rng(20))
    with dg.Hamiltonian.from_integrals(L, N, 0.0, *pair_integrals(np.linspace(-1, 1, L), K)) as h:
        D = h.D
        x = torch.zeros((3, D), dtype=torch.float64, device="cuda")
        x[torch.arange(3), torch.tensor([0, D // 2, D - 1])] = 1.0
        out = []
        for kind in ("rowx", "auto", "block"):
            h.set_sigma_kernel("auto" if kind == "block" else kind)
            y = torch.full((3, D), float("nan"), dtype=torch.float64, device="cuda")
            if kind == "block":
                h.sigma_block_device(x.data_ptr(), D, y.data_ptr(), D, 3, dg.FP64)
            else:
                for v in range(3):
                    h.sigma_device(x[v].data_ptr(), y[v].data_ptr(), dg.FP64)
            torch.cuda.synchronize()
            out.append(y)
        for y in out[1:]:
            assert bool(((y - out[0]).abs() <= 2.0 ** -46 * out[0].abs()).all())


@pytest.mark.parametrize("L,N,seed", [(21, 12, 141), (22, 14, 142)])
def test_sigma_block_reproducible_after_tuning(L, N, seed, synth, dg):
    """Block sigmas of one vector and of four and one repeat bit for bit on an FP64
    shape that was tuned (where the fastest single sigma adds with atomics), and
    agree with the oracle."""
    torch = torch_cuda()
    p = synth(L, N, seed)
    o = oracle.Ham(p)
    with dg.Hamiltonian.from_fcidump(p) as h:
        h.autotune(dg.FP64, 1)
        D = h.D
        X = np.random.default_rng(seed).standard_normal((5, D))
        xb = torch.from_numpy(X).cuda()
        refs = [o.matvec(x) for x in X]
        for nv in (1, 5):
            outs = []
            for _ in range(4):
                y = torch.empty((nv, D), dtype=torch.float64, device="cuda")
                h.sigma_block_device(xb.data_ptr(), D, y.data_ptr(), D, nv, dg.FP64)
                torch.cuda.synchronize()
                outs.append(y)
            assert all(torch.equal(outs[0], y) for y in outs[1:])
            for v in range(nv):
                assert np.abs(outs[0][v].cpu().numpy() - refs[v]).max() <= TOL64 * np.abs(refs[v]).max()


@pytest.mark.parametrize("prec_name,nv", [("FP32", 1), ("FP32", 4), ("FP32", 6)])
def test_sigma_block_captured_without_allocations(prec_name, nv, synth, dg):
    """A captured FP32 block sigma on a space whose automatic form takes scratch
    holds no allocation, so its graph can be instantiated more than once; the
    graph gives the oracle's matvec."""
    import ctypes as C
    torch = torch_cuda()
    rt = C.CDLL("libcudart.so.13")
    prec = getattr(dg, prec_name)
    p = synth(20, 10, 151)
    o = oracle.Ham(p)

    def ok(st):
        assert st == 0, st

    with dg.Hamiltonian.from_fcidump(p) as h:
        D = h.D
        X = np.random.default_rng(9).standard_normal((nv, D)).astype(np.float32)
        x = torch.from_numpy(X).cuda()
        y = torch.zeros_like(x)
        torch.cuda.synchronize()
        st = C.c_void_p(torch.cuda.Stream().cuda_stream)
        graph, execs, n = C.c_void_p(), [C.c_void_p(), C.c_void_p()], C.c_size_t()
        ok(rt.cudaStreamBeginCapture(st, 2))  # relaxed
        h.sigma_block_device(x.data_ptr(), D, y.data_ptr(), D, nv, prec, stream=st.value)
        ok(rt.cudaStreamEndCapture(st, C.byref(graph)))
        ok(rt.cudaGraphGetNodes(graph, None, C.byref(n)))
        nodes, kind = (C.c_void_p * n.value)(), C.c_int()
        ok(rt.cudaGraphGetNodes(graph, nodes, C.byref(n)))
        for node in nodes:
            ok(rt.cudaGraphNodeGetType(C.c_void_p(node), C.byref(kind)))
            assert kind.value not in (10, 11)  # cudaGraphNodeTypeMemAlloc, cudaGraphNodeTypeMemFree
        for e in execs:
            ok(rt.cudaGraphInstantiate(C.byref(e), graph, C.c_ulonglong(0)))
        for e in execs:
            y.zero_()
            torch.cuda.synchronize()
            ok(rt.cudaGraphLaunch(e, st))
            torch.cuda.synchronize()
            for v in range(nv):
                ref = o.matvec(X[v].astype(np.float64))
                assert np.abs(y[v].cpu().numpy() - ref).max() <= TOL32 * np.abs(ref).max()
        for e in execs:
            ok(rt.cudaGraphExecDestroy(e))
        ok(rt.cudaGraphDestroy(graph))


def test_sigma_block_scratch_is_given_back(synth, dg):
    """The block sigma's scratch (14 vectors of 40.1M elements here) is the
    device's again when the handle is destroyed, all but 256 MiB."""
    torch = torch_cuda()
    L, N, nv = 28, 14, 2
    h = dg.Hamiltonian.from_fcidump(synth(L, N, 152))
    x = torch.randn((nv, h.D), dtype=torch.float32, device="cuda")
    y = torch.empty_like(x)
    h.sigma_block_device(x.data_ptr(), h.D, y.data_ptr(), h.D, nv, dg.FP32)
    torch.cuda.synchronize()
    held = torch.cuda.mem_get_info()[0]
    h.close()
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] - held >= 14 * x.shape[1] * 4 - (256 << 20)


@pytest.mark.parametrize("L,N,seed", [(20, 11, 161), (20, 12, 162), (21, 14, 163), (22, 14, 164), (22, 15, 165), (26, 20, 166)])
def test_sigma_fp64_open_slots(L, N, seed, synth, dg):
    """The FP64-accurate pair form on both sides of the step from eight open slots per
    set (float pairs) to nine (digits), on spaces without a neighbour table: the oracle's matvec."""
    torch = torch_cuda()
    p = synth(L, N, seed)
    o = oracle.Ham(p)
    with dg.Hamiltonian.from_fcidump(p) as h:
        h.set_sigma_kernel("rowff")  # (the automatic choice too, unless the shape was tuned in this process)
        assert h.sigma_plan(dg.FP64)[0] == 9
        x = np.random.default_rng(seed).standard_normal(h.D)
        xd, y = torch.from_numpy(x).cuda(), torch.full((h.D,), float("nan"), dtype=torch.float64, device="cuda")
        h.sigma_device(xd.data_ptr(), y.data_ptr(), dg.FP64)
        torch.cuda.synchronize()
        ref = o.matvec(x)
        assert np.abs(y.cpu().numpy() - ref).max() <= TOL64 * np.abs(ref).max()


@pytest.mark.parametrize("ratio", [1.5, 8.0, 17.9, 18.6, 64.0])
def test_fp64_hops_at_the_digits_limit(ratio, dg):
    """Elements of K up to 18 times smaller than the power of two above the
    largest go through the digits, smaller ones through float pairs: on one-hot
    vectors each product is good to 2^-45 either way (in the digits at 18: what is
    cut is 4 x 2^20 x 2^-77 of x k > 2^-9.2, K's rounding 2^-49.8 of it, the pair's 2^-48)."""
    torch = torch_cuda()
    L, N = 20, 10
    rng = np.random.default_rng(21)
    K = np.where(rng.random((L, L)) < 0.5, rng.uniform(0.9, 0.999, (L, L)), rng.uniform(1.0, 1.03, (L, L)) / ratio)
    K = np.triu(K, 1) + np.triu(K, 1).T
    with dg.Hamiltonian.from_integrals(L, N, 0.0, *pair_integrals(np.linspace(-1, 1, L), K)) as h:
        D = h.D
        x = torch.zeros(D, dtype=torch.float64, device="cuda")
        ref, y = torch.empty_like(x), torch.empty_like(x)
        for at in rng.integers(0, D, 6):
            x.zero_()
            x[int(at)] = float(rng.standard_normal())
            for kind, out in (("rowx", ref), ("rowff", y)):
                h.set_sigma_kernel(kind)
                h.sigma_device(x.data_ptr(), out.data_ptr(), dg.FP64)
            torch.cuda.synchronize()
            assert bool(((y - ref).abs() <= 2.0 ** -45 * ref.abs()).all())
