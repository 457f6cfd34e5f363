"""Branches of the J/K launches that the other parity tests do not set apart.

General densities of an FP64 build run on their symmetric and antisymmetric
parts up to 32 of them (64 matrices) and on the general eight-image sums
beyond; jk_device_static always runs the latter.  One-thread launches of few
quartets share each quartet among up to 16 lanes, by primitive pairs of the
bra: molecules of one to a few atoms and contractions of 1, 3 and 5 primitives
take every lane count, against the oracle."""
import numpy as np
import pytest

import integral_b200 as ib
import oracle_py as O
from integral_b200 import systems as S

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(abs(a - b).max() / abs(b).max())


@pytest.mark.parametrize("spherical", [False, True, None], ids=["cart", "sph", "both"])
@pytest.mark.parametrize("ndens, want_k", [(1, True), (3, False), (32, True), (33, True)])
def test_general_densities(spherical, ndens, want_k):
    import torch

    shells = S.jk_system(natom=2, side=3.0, ndens=1)["shells"]
    for k, s in enumerate(shells):
        s["spherical"] = k % 2 == 0 if spherical is None else spherical
    dc = ib.Basis(shells).direct_contractor()
    n = dc.nao()
    D = torch.tensor(np.random.default_rng(3).normal(size=(ndens, n, n)), device="cuda")
    J, K, J0, K0 = (torch.zeros_like(D) for _ in range(4))
    dc.jk_device(D.data_ptr(), ndens, J.data_ptr(), K.data_ptr(), 1e-13, want_exchange=want_k)
    q = dc.last_stats()["quartets"]
    dc.jk_device_static(D.data_ptr(), ndens, J0.data_ptr(), K0.data_ptr(), 1e-13, want_exchange=want_k)
    torch.cuda.synchronize()
    assert q > 0 and rel(J, J0) < 1e-12
    if want_k:
        assert rel(K, K0) < 1e-12


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_general_density_without_finite_parts(value):
    """One element that the symmetric and antisymmetric parts cannot hold, between
    two atoms 80 bohr apart: the general sums keep it out of J and out of three
    quarters of K, the parts would bring it into half of K."""
    import torch

    rng = np.random.default_rng(5)
    shells = S.build_shells(rng, np.array([[0.0, 0.0, 0.0], [0.0, 0.0, 80.0]]), "sssppd", 3, 0.1, 2.5, 0.2, 1.0)
    dc = ib.Basis(shells).direct_contractor()
    n = dc.nao()
    D = rng.normal(size=(1, n, n))
    D[0, 1, n // 2 + 4] = value
    ob = O.OracleBasis(shells)
    Jo, Ko, _, _ = ob.direct_jk(D, 1e-13)
    Dt = D.transpose(0, 2, 1)
    with np.errstate(invalid="ignore"):
        Kp = sum(ob.direct_jk(0.5 * p, 1e-13)[1] for p in (D + Dt, D - Dt))
    assert np.isfinite(Jo).all() and np.isfinite(Ko).sum() == 3 * n * n // 4
    assert np.isfinite(Kp).sum() == n * n // 2
    D = torch.tensor(D, device="cuda")
    J, K, J0, K0 = (torch.zeros_like(D) for _ in range(4))
    dc.jk_device(D.data_ptr(), 1, J.data_ptr(), K.data_ptr(), 1e-13)
    dc.jk_device_static(D.data_ptr(), 1, J0.data_ptr(), K0.data_ptr(), 1e-13)
    torch.cuda.synchronize()
    for a, b in ((J, Jo), (J0, Jo), (K, Ko), (K0, Ko)):
        a, ok = a.cpu().numpy(), np.isfinite(b)
        assert np.array_equal(np.isfinite(a), ok)
        assert rel(a[ok], b[ok]) < 1e-12


@pytest.mark.parametrize("natom", [1, 2, 4])
@pytest.mark.parametrize("nprim", [1, 3, 5])
def test_shared_quartets_of_small_launches(natom, nprim):
    rng = np.random.default_rng(10 * natom + nprim)
    centers = S.place_atoms(rng, natom, 4.0, 1.5)
    shells = S.build_shells(rng, centers, "ssp", nprim, 0.2, 2.5, 0.2, 1.0)
    D = S.densities(rng, S.nao_of(shells), 2, 2)
    dc = ib.Basis(shells).direct_contractor()
    J, K = dc.jk(D, 1e-12)
    st = dc.last_stats()
    Jo, Ko, cnt, hsh = O.OracleBasis(shells).direct_jk(D, 1e-12)
    assert st["quartets"] == cnt and st["quartet_hash"] == hsh
    assert rel(J, Jo) < 1e-12 and rel(K, Ko) < 1e-12
    gpu, ref = ib.Basis(shells).eri(), O.OracleBasis(shells).eri()
    assert float(np.max(np.abs(gpu - ref))) < 1e-13 * max(1.0, float(np.max(np.abs(ref))))


@pytest.mark.parametrize("natom", [3, 8])
def test_launch_records_add_up(natom):
    """The class launches of a small molecule overlap; their records divide the
    run's device time (moments without a launch in flight, and the events'
    resolution of 0.5 us a launch, aside)."""
    import torch

    s = S.jk_system(natom=natom, side=5.0 * natom ** (1 / 3), ndens=1)
    dc = ib.Basis(s["shells"]).direct_contractor()
    D = torch.tensor(s["dens"], device="cuda")
    J, K = torch.zeros_like(D), torch.zeros_like(D)
    for _ in range(3):
        dc.jk_device(D.data_ptr(), 1, J.data_ptr(), K.data_ptr(), s["threshold"])
    span, prof = dc.last_stats()["kernel_ms"], dc.plan.profile()
    total = sum(r["ms"] for r in prof)
    assert len(prof) > 10 and all(r["ms"] >= 0.0 for r in prof)
    assert 0.5 * span <= total <= span + 1e-3 * len(prof), (total, span)
