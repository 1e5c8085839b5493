"""The linear-tile H.Psi kernels (FP64, and FP32 rows of any length and alignment) against the oracle."""

import numpy as np
import pytest

import oracle.kinetic as OK

pytestmark = pytest.mark.gpu


def _geom(shape):
    from isogriddft_gb300.config import H2_BENCHMARK_CASE
    from isogriddft_gb300.grid import assemble_monitor_geometry, build_monitor_grid_spec_for_case, monitor_box_axes

    spec = build_monitor_grid_spec_for_case(H2_BENCHMARK_CASE, shape=shape, box_half_extents=(5.0, 6.0, 7.0))
    lx, ly, lz, box = monitor_box_axes(spec)
    X = box.copy()
    X[..., 0] += 0.25 * np.sin(box[..., 2] * 0.45) * np.exp(-np.sum(box**2, axis=-1) / 25)
    X[..., 1] += 0.2 * np.sin(box[..., 0] * 0.5) * np.exp(-np.sum(box**2, axis=-1) / 20)
    return assemble_monitor_geometry(H2_BENCHMARK_CASE, spec, lx, ly, lz, X)


def _rel(a, b):
    return float(np.max(np.abs(a - b)) / np.max(np.abs(b)))


# the smallest grid; tiles of two and three rows; marches of 3 to 5 planes; rows at the limits of
# two (204) and three (205, 256) points per thread; more CTAs than planes and several segments
@pytest.mark.parametrize("shape", [(3, 3, 3), (3, 7, 5), (4, 4, 9), (5, 6, 205), (4, 9, 251), (3, 5, 256),
                                   (6, 7, 204), (23, 13, 81), (61, 8, 33), (9, 70, 17)])
@pytest.mark.parametrize("closure", ["trial_fix", "production"])
def test_linear_tile_kernels_against_the_oracle(shape, closure):
    """Orbital counts 1 to 6 (whole and partial groups), strided and unaligned blocks, with and
    without v_eff; tolerances as for the other kernels (FP64 1e-12, FP32 2e-5 of the maximum)."""

    import torch

    from isogriddft_gb300 import _lib, device
    from isogriddft_gb300.device import ptr, stream_ptr

    geom = _geom(shape)
    dg = device.device_grid(geom)
    n = dg.n
    rng = np.random.default_rng(11)
    psi = rng.normal(size=(6,) + shape)
    veff = rng.normal(size=shape)
    ref = OK.hpsi_block(psi, geom, veff, closure).reshape(6, n)
    ref0 = OK.hpsi_block(psi, geom, np.zeros(shape), closure).reshape(6, n)  # the kinetic part
    cl = _lib.IGD_CLOSURE_PRODUCTION if closure == "production" else _lib.IGD_CLOSURE_TRIAL_FIX
    _lib.check(_lib.call("igd_hpsi_select", 3), "igd_hpsi_select")
    try:
        for dt, tol in ((torch.float64, 1e-12), (torch.float32, 2e-5)):
            code = _lib.IGD_F64 if dt == torch.float64 else _lib.IGD_F32
            co = dg.coeffs("fp64" if dt == torch.float64 else "fp32")
            v = torch.as_tensor(veff.reshape(-1), device="cuda", dtype=dt)
            for nb, pad, shift in ((1, 0, 0), (2, 0, 0), (3, 5, 0), (4, 0, 1), (5, 1, 3), (6, 0, 0)):
                st = n + pad
                buf = torch.full((nb * st + shift,), float("nan"), device="cuda", dtype=dt)
                out = torch.full_like(buf, float("nan"))
                for o in range(nb):
                    buf[shift + o * st: shift + o * st + n] = torch.as_tensor(psi[o].reshape(-1), dtype=dt)
                for vp, ks, want in ((ptr(v), -0.5, ref), (None, 1.0, -2.0 * ref0), (None, 0.3, -0.6 * ref0)):
                    out.fill_(float("nan"))
                    _lib.check(_lib.call("igd_hpsi_agrid", code, cl, *shape, ptr(co), vp,
                                         ptr(buf) + shift * buf.element_size(), ptr(out) + shift * out.element_size(),
                                         nb, st, ks, 1.0, stream_ptr()), "igd_hpsi_agrid")
                    # the same bits as the cp.async kernel, which sums in the same order
                    gen = torch.full_like(out, float("nan"))
                    _lib.check(_lib.call("igd_hpsi_select", 2), "igd_hpsi_select")
                    _lib.check(_lib.call("igd_hpsi_agrid", code, cl, *shape, ptr(co), vp,
                                         ptr(buf) + shift * buf.element_size(), ptr(gen) + shift * gen.element_size(),
                                         nb, st, ks, 1.0, stream_ptr()), "igd_hpsi_agrid")
                    _lib.check(_lib.call("igd_hpsi_select", 3), "igd_hpsi_select")
                    assert torch.equal(torch.nan_to_num(out, nan=1e30), torch.nan_to_num(gen, nan=1e30))
                    host = out.double().cpu().numpy()
                    for o in range(nb):
                        got = host[shift + o * st: shift + o * st + n]
                        assert _rel(got, want[o]) < tol, (dt, nb, pad, shift, ks, _rel(got, want[o]))
                        assert np.isnan(host[shift + o * st + n: shift + (o + 1) * st]).all()  # padding untouched
    finally:
        _lib.call("igd_hpsi_select", 0)


@pytest.mark.parametrize("nz,linear", [(128, False), (132, True), (160, True), (164, False)])
def test_production_blocks_of_long_rows(nz, linear):
    """Rows of 129 to 160 points take the linear tiles, their neighbours the TMA kernels: the default
    route equals the forced kernel to the bit and the tiled kernel to FP32 rounding."""

    import torch

    from isogriddft_gb300 import _lib, device, ops

    geom = _geom((9, 11, nz))
    dg = device.device_grid(geom)
    g = torch.Generator(device="cuda").manual_seed(nz)
    for nb in (2, 5):
        psi = torch.randn(nb, dg.n, generator=g, device="cuda")
        v = torch.randn(dg.n, generator=g, device="cuda")
        got = {}
        for path in (0, 1, 3):
            _lib.call("igd_hpsi_select", path)
            try:
                got[path] = ops.hpsi_device(dg, psi, closure="production", veff=v).clone()
            finally:
                _lib.call("igd_hpsi_select", 0)
        if linear:
            assert torch.equal(got[0], got[3])
        scale = float(got[1].abs().max())
        assert float((got[0] - got[1]).abs().max()) <= 2e-5 * scale
        assert float((got[3] - got[1]).abs().max()) <= 2e-5 * scale
