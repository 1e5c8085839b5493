"""Density kernels: shared and direct occupations, ragged grids and strides; renormalisation of even and odd grids."""

from types import SimpleNamespace

import numpy as np
import pytest
import torch

from isogriddft_gb300 import _lib, density
from isogriddft_gb300.device import ptr, stream_ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,eps", [(torch.float32, 2.0**-24), (torch.float64, 2.0**-53)])
@pytest.mark.parametrize("n,pad", [(1, 0), (1000, 0), (1021, 3), (262145, 0), (400000, 1)])
@pytest.mark.parametrize("nb", [0, 1, 17, 64, 65])
def test_density_against_fp64(n, pad, nb, dtype, eps):
    g = torch.Generator(device="cuda").manual_seed(n + nb)
    psi = torch.randn(nb, n + pad, generator=g, device="cuda", dtype=dtype)
    occ = torch.rand(nb, generator=g, device="cuda", dtype=torch.float64)
    w = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    start = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    for accumulate in (0, 1):
        rho = start.clone()
        integral = torch.full((1,), 7.0, device="cuda", dtype=torch.float64)
        code = _lib.IGD_F32 if dtype == torch.float32 else _lib.IGD_F64
        _lib.check(_lib.call("igd_density", code, n, nb, n + pad, ptr(psi) if nb else None, ptr(occ) if nb else None,
                             ptr(w), ptr(rho), ptr(integral), accumulate, stream_ptr()))
        terms = occ[:, None] * psi[:, :n].double() ** 2
        want = terms.sum(0) + accumulate * start
        # the occupation, its product with psi, the fused square and sum round once each per orbital
        assert bool(((rho - want).abs() <= (nb + 4) * eps * terms.sum(0) + 2.0**-52 * want).all())
        total = (rho * w).sum()
        assert abs(float(integral - total)) <= n * 2.0**-52 * float(total) + 1e-300


@pytest.mark.parametrize("n", [1, 2, 999, 100000, 2097153])
def test_renormalisation(n):
    for shift in (0, 1):  # pairs need 16-byte data
        rho = torch.rand(n + 1, device="cuda", dtype=torch.float64)[shift:shift + n]
        before = rho.clone()
        integral = torch.tensor([0.37], device="cuda", dtype=torch.float64)
        flags = torch.zeros(1, device="cuda", dtype=torch.int32)
        call = lambda: _lib.check(_lib.call("igd_density_renormalize", n, ptr(rho), ptr(integral), 2.5, ptr(flags),  # noqa: E731
                                            stream_ptr()))
        call()
        assert torch.equal(rho, before * (2.5 / 0.37)) and int(flags) == 0
        for bad in (0.0, -1.0, float("nan")):
            integral.fill_(bad)
            flags.zero_()
            kept = rho.clone()
            call()
            assert torch.equal(rho, kept) and int(flags) == 4


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("nb,count", [(0, 0), (3, 3), (5, 2), (2, 5), (64, 64), (65, 65), (70, 64)])
def test_occupations_by_value_and_from_memory_agree(nb, count, dtype):
    n = 4099
    dg = SimpleNamespace(n=n, device=torch.device("cuda", 0),
                         cell_volumes=torch.rand(n, device="cuda", dtype=torch.float64))
    psi = torch.randn(nb, n, device="cuda", dtype=dtype) if nb else None
    occ = np.random.default_rng(nb).random(2 * count)[::2]  # a strided array
    used = min(nb, count)
    dev_occ = torch.as_tensor(np.ascontiguousarray(occ), device="cuda")
    want = torch.zeros(n, device="cuda", dtype=torch.float64)
    code = _lib.IGD_F32 if dtype == torch.float32 and nb else _lib.IGD_F64
    _lib.check(_lib.call("igd_density", code, n, used, n, ptr(psi) if used else None, ptr(dev_occ) if used else None,
                         ptr(dg.cell_volumes), ptr(want), None, 0, stream_ptr()))
    integral = torch.empty(1, device="cuda", dtype=torch.float64)
    assert torch.equal(density.build_density_device(dg, psi, occ, integral=integral), want)
    assert torch.equal(density.build_density_device(dg, psi, list(occ)), want)
    twice = density.build_density_device(dg, psi, occ, out=want.clone(), accumulate=True)
    assert torch.equal(twice, want + want)
    if used:
        scaled = density.renormalize_device(dg, want.clone(), 2.0, integral)
        assert torch.equal(scaled, want * (2.0 / integral.item()))
    else:
        with pytest.raises(ValueError, match="positive density integral"):
            density.renormalize_device(dg, want, 2.0, integral)
