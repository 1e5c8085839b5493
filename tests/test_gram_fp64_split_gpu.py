"""The FP64 Gram by exact splitting against extended-precision sums, and the FP64 rotation's column tiles."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gram(A, B, w, path, sa, sb, n, accumulate=None):
    import torch

    from isogriddft_gb300 import _lib
    from isogriddft_gb300.device import ptr, stream_ptr

    a, b = A.shape[0], B.shape[0]
    out = torch.zeros((a, b), dtype=torch.float64, device="cuda") if accumulate is None else accumulate
    wsb = int(_lib.call("igd_block_gram_workspace_bytes", n, a, b))
    ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
    _lib.check(_lib.call("igd_gram_select", path), "igd_gram_select")
    try:
        _lib.check(_lib.call("igd_block_gram", _lib.IGD_F64, n, a, ptr(A), sa, b, ptr(B), sb, ptr(w), ptr(out),
                             int(accumulate is not None), ptr(ws), wsb, stream_ptr()), "igd_block_gram")
        assert path != 4 or _lib.call("igd_gram_last_path") == 4
    finally:
        _lib.call("igd_gram_select", 0)
    return out.cpu().numpy()


def _rows(k, n, pad, kind, seed):
    """(k, n) view of a padded block: normal, or decaying over the grid with rows of scales 1 to 1e-9."""

    import torch

    g = torch.Generator(device="cuda").manual_seed(seed)
    full = torch.randn((k, n + pad), dtype=torch.float64, device="cuda", generator=g)
    if kind == "decay":
        r = torch.linspace(0, 12, n + pad, dtype=torch.float64, device="cuda")
        full *= torch.exp(-2.5 * r) * 10.0 ** torch.linspace(0, -9, k, dtype=torch.float64, device="cuda")[:, None]
    return full[:, :n]


# n: below one window of a CTA, ragged windows, several CTAs; a, b: edges of the 16-row and 24-column tiles
@pytest.mark.parametrize("n,a,b,pad", [(33, 1, 1, 0), (1031, 16, 24, 0), (4133, 17, 25, 3), (9000, 21, 21, 1),
                                       (20011, 5, 49, 0), (1500, 64, 33, 0)])
@pytest.mark.parametrize("kind", ["normal", "decay"])
def test_split_gram_against_extended_precision(n, a, b, pad, kind):
    """Bound: one rounding of w b per point and one of the result (2^-52 of sum |a w b|), and the bits below 2^-61 of
    each row's largest value (2^-59 with the powers of two around it)."""

    import torch

    A, B = _rows(a, n, pad, kind, 1), _rows(b, n, pad, kind, 2)
    w = torch.rand(n, dtype=torch.float64, device="cuda") + 1e-3
    for BB, ww in ((B, w), (B, None), (A, w)):
        got = _gram(A, BB, ww, 4, n + pad, n + pad, n)
        x, y = A.cpu().numpy().astype(np.longdouble), BB.cpu().numpy()
        wy = (y * w.cpu().numpy() if ww is not None else y).astype(np.longdouble)
        exact_wy = y.astype(np.longdouble) * (w.cpu().numpy().astype(np.longdouble) if ww is not None else 1)
        want = np.array([[np.sum(p * q) for q in exact_wy] for p in x])
        ax, aw = np.abs(x), np.abs(wy)
        bound = 2.0**-52 * (ax @ aw.T) + 2.0**-59 * (ax.max(1)[:, None] * aw.sum(1)[None] + ax.sum(1)[:, None] * aw.max(1)[None])
        assert np.all(np.abs(got - want) <= bound), float(np.max(np.abs(got - want) / bound))
        if BB is A:
            assert np.array_equal(got, got.T)
    seed = torch.full((a, b), 0.25, dtype=torch.float64, device="cuda")
    twice = _gram(A, B, w, 4, n + pad, n + pad, n, accumulate=seed.clone())
    assert np.array_equal(twice, 0.25 + _gram(A, B, w, 4, n + pad, n + pad, n))


def test_split_gram_special_values():
    """Zero and subnormal rows, infinities and NaN, values near both ends of the exponent range: as the plain kernel."""

    import torch

    n = 2000
    A = _rows(6, n, 0, "normal", 5).clone()
    A[1] = 0.0
    A[2] *= 5e-324 / 1e-2
    A[3, 17] = float("inf")
    A[4, 3] = float("nan")
    A[5] *= 1e300
    B = _rows(5, n, 0, "normal", 6).clone()
    B[1] *= 1e-300
    B[2, 5] = float("-inf")
    w = torch.rand(n, dtype=torch.float64, device="cuda")
    got, plain = _gram(A, B, w, 4, n, n, n), _gram(A, B, w, 3, n, n, n)
    assert np.array_equal(np.isnan(got), np.isnan(plain)) and np.array_equal(np.isinf(got), np.isinf(plain))
    # finite outputs against extended precision: the bound of the test above and one subnormal unit (the plain kernel
    # itself rounds each of 2000 subnormal products)
    fine = np.isfinite(plain)
    x, y = A.cpu().numpy().astype(np.longdouble), B.cpu().numpy().astype(np.longdouble) * w.cpu().numpy()
    with np.errstate(all="ignore"):
        want = np.array([[np.sum(p * q) for q in y] for p in x])
        ax, aw = np.abs(x), np.abs(y)
        bound = 2.0**-52 * (ax @ aw.T) + 2.0**-59 * (ax.max(1)[:, None] * aw.sum(1)[None]
                                                     + ax.sum(1)[:, None] * aw.max(1)[None]) + np.longdouble(2.0**-1074)
        assert np.all((np.abs(got - want) <= bound)[fine])
    z = torch.zeros((3, n), dtype=torch.float64, device="cuda")
    assert np.array_equal(_gram(z, z, w, 4, n, n, n), np.zeros((3, 3)))


@pytest.mark.parametrize("c", [1, 2, 3, 7, 19, 20, 21, 34, 41])
def test_fp64_rotation_column_tiles(c):
    """Every column count takes equal tiles of at most 20 columns; each output is the same sequence of FMAs."""

    import torch

    from isogriddft_gb300 import _lib
    from isogriddft_gb300.device import ptr, stream_ptr

    n, a, b = 5003, 13, 6
    A, B = _rows(a, n, 2, "normal", 7), _rows(b, n, 2, "normal", 8)
    C = torch.randn((a + b, c), dtype=torch.float64, device="cuda")
    out = torch.full((c, n + 1), float("nan"), dtype=torch.float64, device="cuda")
    _lib.check(_lib.call("igd_block_rotate", _lib.IGD_F64, n, a, ptr(A), n + 2, ptr(C), b, ptr(B), n + 2,
                         ptr(C) + 8 * a * c, c, ptr(out), n + 1, 0, stream_ptr()), "igd_block_rotate")
    want = C[:a].T @ A + C[a:].T @ B
    bound = 20 * 2.0**-53 * (C[:a].abs().T @ A.abs() + C[a:].abs().T @ B.abs())
    assert bool(((out[:, :n] - want).abs() <= bound).all()) and bool(torch.isnan(out[:, n]).all())
