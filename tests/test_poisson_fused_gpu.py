"""The fused BiCGSTAB of the Poisson solve in every form that it takes, against the unfused one."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _grid(shape):
    from isogriddft_gb300.config import H2_BENCHMARK_CASE
    from isogriddft_gb300.device import device_grid
    from isogriddft_gb300.grid import build_monitor_grid_for_case, build_two_peak_element_parameters

    geom = build_monitor_grid_for_case(H2_BENCHMARK_CASE, shape=shape, box_half_extents=(8.0, 8.0, 10.0),
                                       element_parameters=build_two_peak_element_parameters(("H",)), device=True)
    return geom, device_grid(geom)


def _solve(shape, c64, c32, f, precision, path=0, u=None, rtol=1e-10, maxit=3000):
    """igd_poisson_solve, or igd_poisson_solve_from with u: return code, solution, info."""

    import torch

    from isogriddft_gb300 import _lib
    from isogriddft_gb300.device import ptr, stream_ptr

    n = int(np.prod(shape))
    prec = _lib.IGD_PREC_FP64 if precision == "fp64" else _lib.IGD_PREC_MIXED
    wsb = int(_lib.call("igd_poisson_workspace_bytes", prec, n))
    ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
    out = torch.empty(n, dtype=torch.float64, device="cuda") if u is None else u.clone()
    info = np.zeros(6)
    _lib.check(_lib.call("igd_poisson_select", path), "igd_poisson_select")
    try:
        code = _lib.call("igd_poisson_solve" if u is None else "igd_poisson_solve_from", _lib.IGD_GRID_MONITOR, prec,
                         *shape, ptr(c64), ptr(c32), ptr(f), ptr(out), rtol, maxit, ptr(ws), wsb, info.ctypes.data,
                         stream_ptr())
    finally:
        _lib.call("igd_poisson_select", 0)
    return code, out, info


@pytest.mark.parametrize("shape", [(11, 13, 15), (12, 14, 16)])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_nonfinite_right_hand_side_is_a_breakdown(shape, bad):
    """A right-hand side with a NaN or an infinity inside is refused with the unfused iteration's return code."""

    import torch

    from isogriddft_gb300 import _lib

    geom, dg = _grid(shape)
    f = torch.randn(shape, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    f[4, 5, 6] = bad
    for path in (1, 0):
        code, _, info = _solve(shape, dg.coeffs("fp64"), None, f.reshape(-1), "fp64", path)
        assert code == _lib.IGD_ERR_BREAKDOWN and info[0] == 0 and info[2] == _lib.IGD_ERR_BREAKDOWN, (path, code, info)


@pytest.mark.parametrize("shape", [(11, 13, 15), (7, 9, 211)])
def test_ragged_mixed_solve_sums_dots_in_fp64(shape):
    """Rows that are no multiple of four points: the FP32 iteration forms the products of its dot products in FP64, so
    an operator of 1e24 times the size (t.t beyond FP32's range) gives the same solution, scaled."""

    import torch

    from isogriddft_gb300 import _lib

    geom, dg = _grid(shape)
    n = int(np.prod(shape))
    f = torch.randn(n, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(4))
    c64, c32 = dg.coeffs("fp64").reshape(7, n), dg.coeffs("fp32").reshape(7, n)
    scale = 2.0**80
    s64, s32 = c64.clone(), c32.clone()
    s64[6] *= scale
    s32[6] *= scale
    sols = [_solve(shape, a, b, f, "mixed") for a, b in ((c64, c32), (s64, s32))]
    for code, _, info in sols:
        assert code == _lib.IGD_OK and info[1] <= 1e-10, (code, info)
    # two solutions with relative residuals of 1e-10 each
    u, v = sols[0][1], sols[1][1] * scale
    assert float((u - v).norm() / u.norm()) < 1e-7


def test_large_grid_with_a_workspace_aligned_to_a_double():
    """More points than 32-bit offsets reach and vectors without 16-byte alignment: neither fused operator takes the
    grid, so the unfused iteration does."""

    import torch

    from isogriddft_gb300 import _lib
    from isogriddft_gb300.device import ptr, stream_ptr

    shape = (800, 800, 248)
    n = int(np.prod(shape))
    assert 28 * n >= 1 << 32
    c64 = torch.zeros((7, n), dtype=torch.float64, device="cuda")
    for i in (0, 1, 2, 6):
        c64[i] = 1.0
    c32 = c64.float()
    f = torch.zeros(n, dtype=torch.float64, device="cuda")
    f[(400 * 800 + 400) * 248 + 124] = 1.0  # an interior point
    u = torch.empty_like(f)
    wsb = int(_lib.call("igd_poisson_workspace_bytes", _lib.IGD_PREC_MIXED, n))
    buf = torch.empty(wsb + 16, dtype=torch.uint8, device="cuda")
    info = np.zeros(6)
    code = _lib.call("igd_poisson_solve", _lib.IGD_GRID_MONITOR, _lib.IGD_PREC_MIXED, *shape, ptr(c64), ptr(c32),
                     ptr(f), ptr(u), 1e-2, 1, ptr(buf) + 8, wsb, info.ctypes.data, stream_ptr())
    assert code == _lib.IGD_OK and info[0] == 1 and 0.0 < info[1] < 1.0, (code, info)


# E = 2, odd rows (E = 1), rows of 205 to 256 points of either parity, the smallest grid; from_u: a warm start
@pytest.mark.parametrize("shape", [(20, 18, 26), (21, 22, 23), (9, 11, 205), (8, 10, 256), (3, 3, 3)])
@pytest.mark.parametrize("from_u", [False, True])
def test_fused_fp64_iteration_matches_unfused(shape, from_u):
    """FP64: both iterations meet the stopping rule and give the same solution."""

    import torch

    from isogriddft_gb300 import _lib

    geom, dg = _grid(shape)
    n = int(np.prod(shape))
    g = torch.Generator("cuda").manual_seed(5)
    f = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
    u0 = None
    if from_u:
        u0 = torch.zeros(shape, dtype=torch.float64, device="cuda")
        u0[1:-1, 1:-1, 1:-1] = torch.randn([m - 2 for m in shape], dtype=torch.float64, device="cuda", generator=g)
        u0 = u0.reshape(-1)
    sols = [_solve(shape, dg.coeffs("fp64"), None, f, "fp64", path, u0, rtol=1e-11) for path in (0, 1)]
    for code, u, info in sols:
        assert code == _lib.IGD_OK and info[1] <= 2e-11, (code, info)  # the recomputed residual, not the recursion's
        q = u.reshape(shape)
        for face in (q[0], q[-1], q[:, 0], q[:, -1], q[:, :, 0], q[:, :, -1]):
            assert not face.any()
    a, b = (s[1] for s in sols)
    assert float((a - b).norm() / b.norm()) < 1e-8


# rows of 205 to 256 points: no multiple of four, and of eight with at least 50 thousand points (both linear tiles)
@pytest.mark.parametrize("shape", [(9, 11, 211), (16, 16, 208)])
def test_fused_mixed_iteration_on_long_rows(shape):
    """Mixed precision on rows that the linear-tile operator takes with three points per thread."""

    import torch

    from isogriddft_gb300 import _lib

    geom, dg = _grid(shape)
    f = torch.randn(int(np.prod(shape)), dtype=torch.float64, device="cuda",
                    generator=torch.Generator("cuda").manual_seed(6))
    sols = [_solve(shape, dg.coeffs("fp64"), dg.coeffs("fp32"), f, "mixed", path) for path in (0, 1)]
    for code, _, info in sols:
        assert code == _lib.IGD_OK and info[1] <= 1e-10, (code, info)
    a, b = (s[1] for s in sols)
    assert float((a - b).norm() / b.norm()) < 1e-7
