"""The tensor-core sigma's bounded device waits (sigma_tc.cu).

In a child process whose wait limit is 0 (DOCI_TC_SPIN_LIMIT=0: every
mbarrier wait of the kernel gives up at once, as a wait on a barrier that
nothing completes would after its limit), doci_sigma_host must return
DOCI_ERR_DEVICE_TIMEOUT: the kernel sets its error word, drains its copies in
flight, frees its tensor memory and returns.  The context stays usable: a
sigma by another kernel in the same process afterwards matches the oracle.
No GPU fault, trap or endless wait is involved."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes as C, sys
import numpy as np
sys.path.insert(0, {root!r})
import doci_gb300 as dg, oracle
p = {path!r}
o = oracle.Ham(p)
with dg.Hamiltonian.from_fcidump(p) as h:
    h.set_sigma_kernel("tc")
    assert h.sigma_plan(dg.FP32)[0] == 8, h.sigma_plan(dg.FP32)
    x = np.random.default_rng(1).standard_normal(h.D).astype(np.float32)
    y = np.empty_like(x)
    st = dg.lib().doci_sigma_host(h.handle, x.ctypes.data_as(C.c_void_p), y.ctypes.data_as(C.c_void_p), dg.FP32)
    print("status", st)
    h.set_sigma_kernel("row1")
    y2 = h.sigma(x, dg.FP32)
    ref = o.matvec(x.astype(np.float64))
    print("after", float(np.abs(y2 - ref).max() / np.abs(ref).max()))
"""


def test_wait_limit_reports_timeout(synth):
    p = synth(20, 10, 71)
    env = dict(os.environ, DOCI_TC_SPIN_LIMIT="0")
    r = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT, path=p)], capture_output=True, text=True,
                       env=env, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    lines = dict(ln.split(" ", 1) for ln in r.stdout.splitlines() if ln.startswith(("status", "after")))
    assert int(lines["status"]) == 12  # DOCI_ERR_DEVICE_TIMEOUT
    assert float(lines["after"]) <= 2e-6


WARP_CHILD = r"""
import ctypes as C, sys
import numpy as np, torch
sys.path.insert(0, {root!r})
import doci_gb300 as dg, oracle
p = {path!r}
o = oracle.Ham(p)
with dg.Hamiltonian.from_fcidump(p) as h:
    for name, prec in (("pair", dg.FP32), ("rowff", dg.FP64)):
        h.set_sigma_kernel(name)
        assert h.sigma_plan(prec)[0] == (6 if prec == dg.FP32 else 9)
        x = np.random.default_rng(1).standard_normal(h.D).astype(np.float32 if prec == dg.FP32 else np.float64)
        y = np.empty_like(x)
        for _ in range(3):
            print("status", dg.lib().doci_sigma_host(h.handle, x.ctypes.data_as(C.c_void_p),
                                                     y.ctypes.data_as(C.c_void_p), prec))
        h.set_sigma_kernel("auto")
        X = torch.from_numpy(np.stack([x, x])).cuda()
        Y = torch.empty_like(X)
        h.sigma_block_device(X.data_ptr(), h.D, Y.data_ptr(), h.D, 2, prec)
        torch.cuda.synchronize()
        h.set_sigma_kernel("gather")
        st = dg.lib().doci_sigma_host(h.handle, x.ctypes.data_as(C.c_void_p), y.ctypes.data_as(C.c_void_p), prec)
        print("block", st)
        y2 = h.sigma(x, prec)
        ref = o.matvec(x.astype(np.float64))
        print("after", float(np.abs(y2 - ref).max() / np.abs(ref).max()))
"""


# one tile in the only slot; one to three tiles a slot; slots with many units
@pytest.mark.parametrize("L,N", [(10, 1), (12, 4), (22, 11)])
def test_warp_wait_limit_reports_timeout(L, N, synth):
    """The same for the warp-per-unit pair forms (kinds 6 and 9, and their
    reproducible forms in the block sigma on the space without a neighbour
    table): a scattering warp whose wait runs out leaves the slot's last MMAs
    to the issuing warp, which waits for them before the tensor memory goes."""
    p = synth(L, N, 72)
    env = dict(os.environ, DOCI_TC_SPIN_LIMIT="0")
    r = subprocess.run([sys.executable, "-c", WARP_CHILD.format(root=ROOT, path=p)], capture_output=True, text=True,
                       env=env, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    got = [ln.split() for ln in r.stdout.splitlines() if ln.startswith(("status", "block", "after"))]
    assert [int(v) for k, v in got if k == "status"] == [12] * 6  # DOCI_ERR_DEVICE_TIMEOUT
    assert [int(v) for k, v in got if k == "block"] == [12 if (L, N) == (22, 11) else 0] * 2
    assert all(float(v) <= 2e-6 for k, v in got if k == "after")


SOLVE_CHILD = r"""
import ctypes as C, sys
import numpy as np
sys.path.insert(0, {root!r})
import doci_gb300 as dg
small, p = {small!r}, {path!r}
with dg.Hamiltonian.from_fcidump(p) as h, dg.Hamiltonian.from_fcidump(small) as hs:
    for mode in ("fp64", "mixed"):
        try:
            dg.solve_roots(h, nroots=2, max_vec=6, max_its=2, mode=mode)
        except dg.DociError as e:
            print("roots", e)
        st, res = dg.batch_solve([hs, h], nroots=2, max_vec=6, max_its=2, mode=mode)
        print("batch", st, [r["status"] for r in res])
    for nvec in (1, 2):
        try:
            h.autotune(dg.FP32, nvec)
            print("tune ok")
        except dg.DociError as e:
            print("tune", e)
    # nothing is left for a later call that ran no such kernel
    h.set_sigma_kernel("gather")
    x = np.ones(h.D)
    print("clean", dg.lib().doci_sigma_host(h.handle, x.ctypes.data_as(C.c_void_p),
                                            np.empty_like(x).ctypes.data_as(C.c_void_p), dg.FP64))
if len(sys.argv) > 1:  # the reference's entry points print the error and exit
    L = dg.lib()
    dat = C.c_void_p()
    L.fill_doci_data(p.encode(), C.byref(dat))
    D = L.doci_get_basis_size(dat)
    vec = np.zeros(D)
    vec[0] = 1.0
    e = C.c_double()
    L.sparse_eigensolve(vec.ctypes.data_as(C.POINTER(C.c_double)), D, C.byref(e), C.cast(L.doci_matvec, C.c_void_p),
                        L.doci_get_diagonal(dat), None, 1e-8, 2, sys.argv[1].encode(), 2, 4, dat)
    print("returned")
"""


@pytest.mark.parametrize("solver", [None, "D", "CG"])
def test_wait_limit_reaches_the_solvers(solver, synth):
    """With a wait limit of 0 the solves that run the warp-per-unit kernels (a
    space large enough for the batch engine to take them) report
    DOCI_ERR_DEVICE_TIMEOUT, a problem beside them that does not stays fine,
    and no error is left for a later call."""
    p, small = synth(25, 12, 73), synth(10, 5, 74)
    env = dict(os.environ, DOCI_TC_SPIN_LIMIT="0")
    code = SOLVE_CHILD.format(root=ROOT, path=p, small=small)
    r = subprocess.run([sys.executable, "-u", "-c", code] + ([solver] if solver else []), capture_output=True, text=True,
                       env=env, timeout=300)
    out = r.stdout.splitlines()
    assert sum(ln.startswith("roots") and "DOCI_ERR_DEVICE_TIMEOUT" in ln for ln in out) == 2, r.stdout + r.stderr
    assert out.count("batch 12 [0, 12]") == 2, r.stdout
    assert any(ln.startswith("tune") and "DOCI_ERR_DEVICE_TIMEOUT" in ln for ln in out)
    assert "clean 0" in out
    if solver is None:
        assert r.returncode == 0, r.stderr
    else:
        assert r.returncode != 0 and "returned" not in out
        assert "device wait timed out" in r.stderr + r.stdout


UNALIGNED_CHILD = r"""
import ctypes as C, sys
import numpy as np, torch
sys.path.insert(0, {root!r})
import doci_gb300 as dg, oracle
p = {path!r}
o = oracle.Ham(p)
with dg.Hamiltonian.from_fcidump(p) as h:
    h.set_sigma_kernel("tc")
    x = np.random.default_rng(1).standard_normal(h.D).astype(np.float32)
    xs = torch.zeros(h.D + 1, dtype=torch.float32, device="cuda")
    xs[1:] = torch.from_numpy(x)
    y = torch.empty(h.D, dtype=torch.float32, device="cuda")
    h.sigma_device(xs[1:].data_ptr(), y.data_ptr(), dg.FP32)
    torch.cuda.synchronize()
    ref = o.matvec(x.astype(np.float64))
    print("err", float(np.abs(y.cpu().numpy() - ref).max() / np.abs(ref).max()))
    h.set_sigma_kernel("gather")
    print("status", dg.lib().doci_sigma_host(h.handle, x.ctypes.data_as(C.c_void_p),
                                             np.empty_like(x).ctypes.data_as(C.c_void_p), dg.FP32))
"""


def test_unaligned_tc_runs_kind_6(synth):
    """Kind 8 on an x that is not 16-byte aligned runs what kind 6 runs: right with
    the ordinary wait limit, and a timeout with none (the kernel of kind 6 has
    device waits; the one it took the place of has not)."""
    p = synth(20, 10, 75)
    for limit in (None, "0"):
        env = dict(os.environ, **({"DOCI_TC_SPIN_LIMIT": limit} if limit else {}))
        r = subprocess.run([sys.executable, "-c", UNALIGNED_CHILD.format(root=ROOT, path=p)], capture_output=True,
                           text=True, env=env, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
        got = dict(ln.split() for ln in r.stdout.splitlines() if ln.startswith(("err", "status")))
        if limit:
            assert int(got["status"]) == 12
        else:
            assert int(got["status"]) == 0 and float(got["err"]) <= 2e-6
