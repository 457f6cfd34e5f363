"""Builds on a device that is nearly full.  What a call takes for speed alone,
scratch for overlapped launches, ket copies and the parts of general densities,
it does without where there is no room; it fails only when the scratch of its
largest launch cannot be had.  The device is filled from torch up to a stated
rest; the kernels are loaded before."""
import contextlib

import numpy as np
import pytest

import integral_b200 as ib
from integral_b200 import systems as S

pytestmark = pytest.mark.gpu

MB = 1 << 20


@contextlib.contextmanager
def little_memory(rest):
    """Leaves `rest` bytes of the device, and less than 32 MB by rounding."""
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    spare = torch.empty(rest, dtype=torch.uint8, device="cuda")
    held, size = [], 1 << 34
    while size >= 32 * MB:
        try:
            held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        except torch.cuda.OutOfMemoryError:
            size //= 2
    del spare
    torch.cuda.empty_cache()
    try:
        yield
    finally:
        held.clear()
        torch.cuda.empty_cache()


def rel(a, b):
    return float(abs(a - b).max() / abs(b).max())


def test_overlapped_launches_without_room():
    """Gradient over spherical f shells of 5 atoms: some 0.7 GB of scratch on
    eight streams, run in 256 MB."""
    rng = np.random.default_rng(4)
    shells = S.build_shells(rng, S.place_atoms(rng, 5, 7.0, 1.5), "ssppdf", 3, 0.12, 2.5, 0.2, 1.0, spherical=True)
    D = S.densities(rng, S.nao_of(shells), 8, 1)[0]

    def gradient():
        gc = ib.Basis(shells).direct_grad_contractor()
        d = gc.density([ib.GradDensityTerm(0.5, D, D)], [ib.GradDensityTerm(-0.25, D, D)])
        return gc.contract(d, threshold=1e-11)

    want = gradient()
    with little_memory(256 * MB):
        got = gradient()
    assert rel(got, want) < 1e-12


@pytest.mark.parametrize("rest", [200, 500])
def test_general_densities_without_room(rest):
    """32 general densities of 330 functions, 28 MB as a stack: 139 MB of parts
    and their sums and 0.7 GB for the running sums of 64 matrices, beside some
    140 MB of every build; run in 200 MB, which ends with the parts, and in
    500 MB, which ends with the running sums."""
    import torch

    s = S.jk_system(natom=22, side=30.0, ndens=1)
    D = torch.tensor(np.random.default_rng(3).normal(size=(32, 330, 330)), device="cuda")
    J, K, J0, K0 = (torch.zeros_like(D) for _ in range(4))
    bras = np.arange(0, len(s["shells"]) * (len(s["shells"]) + 1) // 2, 64)

    def build(J, K, ndens):
        dc = ib.Basis(s["shells"]).direct_contractor()
        dc.jk_device(D.data_ptr(), ndens, J.data_ptr(), K.data_ptr(), 1e-9, bras=bras)

    build(J0, K0, 32)
    # the general sums' kernels too: a NaN keeps a density on them
    D[0, 0, 1] = float("nan")
    build(J, K, 1)
    D[0, 0, 1] = D[0, 1, 0]
    torch.cuda.synchronize()
    build(J0.zero_(), K0.zero_(), 32)
    J.zero_(), K.zero_()
    with little_memory(rest * MB):
        build(J, K, 32)
    assert rel(J, J0) < 1e-12 and rel(K, K0) < 1e-12
