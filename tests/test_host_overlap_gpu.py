"""doci_sigma_host with its copies overlapped with the sigma (host_plan.h), which
large spaces take, on small ones.

In a child process DOCI_HOST_OVERLAP_MIN_D=1 makes every handle take that
path, and DOCI_TC_SPIN_LIMIT=0 shows that it was taken: the kernels of the other
path (copy, sigma, copy) have device waits, which then run out and are
reported, those of the overlapped one have none."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes as C, sys
import numpy as np, torch
sys.path.insert(0, {root!r})
import doci_gb300 as dg, oracle
from test_sigma_gpu import pair_integrals
L, N, seed, off, graded = {L}, {N}, {seed}, {off}, {graded}
rng = np.random.default_rng(seed)
lib = dg.lib()
for prec, tdt in ((dg.FP32, torch.float32), (dg.FP64, torch.float64)):
    if graded:  # a K that the FP64 form's digits cannot hold
        K = np.where((np.arange(L) % 2)[:, None] * (np.arange(L) % 2)[None, :], 1e-3, 1.0) * rng.uniform(0.5, 1, (L, L))
        K = np.triu(K, 1) + np.triu(K, 1).T
        h = dg.Hamiltonian.from_integrals(L, N, 0.0, *pair_integrals(np.linspace(-1, 1, L), K))
        if N * (L - N) < 200:
            h.set_sigma_kernel("pair" if prec == dg.FP32 else "rowff")
    else:
        h = dg.Hamiltonian.from_fcidump({path!r})
        h.set_sigma_kernel("pair" if prec == dg.FP32 else "rowff")
    D = h.D
    x = rng.standard_normal(D)
    for pinned in (True, False):
        xs = torch.zeros(D + 8, dtype=tdt)
        ys = torch.full((D + 8,), float("nan"), dtype=tdt)
        if pinned:
            xs, ys = xs.pin_memory(), ys.pin_memory()
        xs[off:off + D] = torch.from_numpy(x).to(tdt)
        for rep in range(3):
            ys.fill_(float("nan"))
            st = lib.doci_sigma_host(h.handle, C.c_void_p(xs[off:].data_ptr()), C.c_void_p(ys[off:].data_ptr()), prec)
            y = ys[off:off + D].double().numpy()
            clean = bool(torch.isnan(ys[:off]).all() and torch.isnan(ys[off + D:]).all())
            kind = h.sigma_plan(prec)[0]
            h.set_sigma_kernel("gather")
            ref = h.sigma(xs[off:off + D].double().numpy(), dg.FP64)
            h.set_sigma_kernel("pair" if prec == dg.FP32 else "rowff")
            err = float(np.abs(y - ref).max() / np.abs(ref).max()) if st == 0 else -1.0
            print("call", 32 if prec == dg.FP32 else 64, int(pinned), st, kind, err, int(clean))
    h.close()
"""


@pytest.mark.parametrize("L,N,seed,off,graded", [(22, 11, 31, 0, False), (24, 12, 30, 3, False), (20, 7, 33, 1, False),
                                                 (13, 5, 35, 0, False), (22, 11, 36, 1, True), (13, 4, 37, 0, True)])
def test_overlapped_copies(L, N, seed, off, graded, synth):
    """FP32 between pinned buffers, and FP64 on a K that the float-pair kernel
    takes (into pinned and pageable y), go through the overlapped path: right
    against the FP64 gather kernel (which the oracle checks elsewhere) three times on
    one handle, with nothing written around y.  The others report the
    timeout of the kernels they run."""
    env = dict(os.environ, DOCI_HOST_OVERLAP_MIN_D="1", DOCI_TC_SPIN_LIMIT="0",
               PYTHONPATH=os.path.join(ROOT, "tests") + os.pathsep + os.environ.get("PYTHONPATH", ""))
    code = CHILD.format(root=ROOT, path=synth(L, N, seed), L=L, N=N, seed=seed, off=off, graded=graded)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, env=env, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    calls = [ln.split()[1:] for ln in r.stdout.splitlines() if ln.startswith("call")]
    assert len(calls) == 12
    for bits, pinned, st, kind, err, clean in calls:
        assert int(kind) == (6 if bits == "32" else 9) and clean == "1"
        if (bits == "32" and pinned == "1") or (bits == "64" and graded):
            assert st == "0" and 0 <= float(err) <= (2e-6 if bits == "32" else 1e-12)
        else:
            assert st == "12"
