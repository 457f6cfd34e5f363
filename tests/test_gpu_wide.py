"""One-thread-per-quartet kernels of the larger Cartesian classes (wide.cuh),
which a J/K class launch takes from 3 x 128 quartets per SM.

Their results are compared with igpu_jk_device_static, whose general
eight-image path runs the team kernels on the same quartet list, within the
J/K contract (1e-12 of the maxima; sums of some 1e4 products per element
round to about 1e-14), and on a sample of the bra pairs with the oracle.  An
18-atom s,s,s,p,p,d system puts every wide class above the line; subsets, erf,
missing exchange, several density counts and pairs without primitives take
their branches."""
import numpy as np
import pytest

import integral_b200 as ib
import oracle_py as O
from integral_b200 import systems as S

pytestmark = pytest.mark.gpu

WIDE = {(2, 1, 2, 0), (2, 1, 1, 1), (2, 1, 2, 1), (2, 2, 1, 0), (2, 2, 2, 0)}
WIDE32 = WIDE | {(2, 2, 1, 1)}


def rel(a, b):
    return float((a - b).abs().max() / b.abs().max())


def build(dc, D, thr, want_k=True, precision=0, bras=None):
    import torch

    J, K = torch.zeros_like(D), torch.zeros_like(D)
    dc.jk_device(D.data_ptr(), D.shape[0], J.data_ptr(), K.data_ptr(), thr, want_exchange=want_k, precision=precision,
                 bras=bras)
    return J, K


@pytest.fixture(scope="module")
def system():
    import torch

    s = S.jk_system(natom=18, side=13.1, ndens=5)
    dc = ib.Basis(s["shells"]).direct_contractor()
    return dc, torch.tensor(s["dens"], dtype=torch.float64, device="cuda"), s["threshold"]


@pytest.mark.parametrize("ndens, want_k, omega", [(1, True, 0.0), (2, False, 0.0), (5, True, 0.3)])
def test_wide_kernels_match_the_team_kernels(system, ndens, want_k, omega):
    import torch

    dc, D, thr = system
    D = D[:ndens].contiguous()
    dc.plan.set_erf_omega(omega)
    try:
        J, K = build(dc, D, thr, want_k)
        ran = {(r["la"], r["lb"], r["lc"], r["ld"]) for r in dc.plan.profile() if r["team"] == 1}
        J0, K0 = torch.zeros_like(D), torch.zeros_like(D)
        dc.jk_device_static(D.data_ptr(), ndens, J0.data_ptr(), K0.data_ptr(), thr, want_exchange=want_k)
        torch.cuda.synchronize()
    finally:
        dc.plan.set_erf_omega(0.0)
    assert WIDE <= ran
    assert rel(J, J0) < 1e-12
    if want_k:
        assert rel(K, K0) < 1e-12


def test_wide_kernels_on_bra_subsets(system):
    """Two interleaved shares of the bra pairs add up to the whole build."""
    dc, D, thr = system
    D = D[:1].contiguous()
    J, K = build(dc, D, thr)
    n = len(dc.bra_pairs())
    parts = [build(dc, D, thr, bras=np.arange(k, n, 2)) for k in range(2)]
    assert rel(parts[0][0] + parts[1][0], J) < 1e-12
    assert rel(parts[0][1] + parts[1][1], K) < 1e-12


def test_wide_kernels_in_fp32(system):
    """Every quartet below 1e3 in FP32: errors of FP32 rounding (24 bits, each
    block element within some 1e-6 of the largest), no more."""
    dc, D, thr = system
    D = D[:4].contiguous()
    J, K = build(dc, D, thr)
    cutoff, _ = dc.mixed_cutoffs()
    dc.set_mixed_cutoff(1e3)
    try:
        J32, K32 = build(dc, D, thr, precision=1)
        prof = dc.plan.profile()
    finally:
        dc.set_mixed_cutoff(cutoff)
    assert WIDE32 <= {(r["la"], r["lb"], r["lc"], r["ld"]) for r in prof if r["team"] == 1 and r["fp32"] and r["quartets"]}
    assert rel(J32, J) < 1e-5 and rel(K32, K) < 1e-5


def test_wide_kernels_match_the_oracle(system):
    """A sample of the bra pairs (the launches keep their lists, so the wide
    kernels run), quartet list and values."""
    dc, D, thr = system
    n = len(dc.bra_pairs())
    bras = np.arange(7, n, 61)
    J, K = build(dc, D[:2].contiguous(), thr, bras=bras)
    st = dc.last_stats()
    assert WIDE <= {(r["la"], r["lb"], r["lc"], r["ld"]) for r in dc.plan.profile() if r["team"] == 1 and r["quartets"]}
    shells = S.jk_system(natom=18, side=13.1, ndens=5)["shells"]
    Jo, Ko, cnt, hsh = O.OracleBasis(shells).direct_jk(D[:2].cpu().numpy(), thr, bras=bras, nthreads=8)
    assert st["quartets"] == cnt and st["quartet_hash"] == hsh
    for a, b in ((J, Jo), (K, Ko)):
        assert float(np.max(np.abs(a.cpu().numpy() - b))) < 1e-12 * float(np.max(np.abs(b)))


@pytest.fixture(scope="module")
def spread_system():
    """18 atoms in a 60-bohr cube: every wide class has enough quartets at
    threshold zero, which keeps every bound, and near half of its pairs of
    shells have no primitives left.  The device memory that the plan gets held
    NaN before, so that a value read without having been written shows."""
    import torch

    x = torch.full((1 << 28,), float("nan"), dtype=torch.float64, device="cuda")
    del x
    torch.cuda.empty_cache()
    s = S.jk_system(natom=18, side=60.0, ndens=1)
    dc = ib.Basis(s["shells"]).direct_contractor()
    return dc, torch.tensor(s["dens"], dtype=torch.float64, device="cuda")


def test_wide_kernels_on_pairs_without_primitives(spread_system):
    import torch

    dc, D = spread_system
    J, K = build(dc, D, 0.0)
    ran = {(r["la"], r["lb"], r["lc"], r["ld"]) for r in dc.plan.profile() if r["team"] == 1}
    J0, K0 = torch.zeros_like(D), torch.zeros_like(D)
    dc.jk_device_static(D.data_ptr(), 1, J0.data_ptr(), K0.data_ptr(), 0.0)
    torch.cuda.synchronize()
    assert WIDE <= ran
    assert bool(torch.isfinite(J0).all()) and bool(torch.isfinite(K0).all())
    assert rel(J, J0) < 1e-12 and rel(K, K0) < 1e-12


def test_wide_kernels_in_fp32_on_pairs_without_primitives(spread_system):
    dc, D = spread_system
    J, K = build(dc, D, 0.0)
    cutoff, _ = dc.mixed_cutoffs()
    dc.set_mixed_cutoff(1e3)
    try:
        J32, K32 = build(dc, D, 0.0, precision=1)
        prof = dc.plan.profile()
    finally:
        dc.set_mixed_cutoff(cutoff)
    assert WIDE32 <= {(r["la"], r["lb"], r["lc"], r["ld"]) for r in prof if r["team"] == 1 and r["fp32"] and r["quartets"]}
    assert rel(J32, J) < 1e-5 and rel(K32, K) < 1e-5
