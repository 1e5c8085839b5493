"""The FP64 Gram by splitting where its fixed-point rows would lose digits, and the limits of its workspace."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gram(A, B, w, path, ws=None, wsb=None, out=None):
    """igd_block_gram on FP64 rows: return code, result, the kernel that ran."""

    import torch

    from isogriddft_gb300 import _lib
    from isogriddft_gb300.device import ptr, stream_ptr

    a, n = A.shape
    b = B.shape[0]
    if ws is None:
        wsb = int(_lib.call("igd_block_gram_workspace_bytes", n, a, b))
        ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
    acc = out is not None
    out = out if acc else torch.zeros((a, b), dtype=torch.float64, device="cuda")
    _lib.check(_lib.call("igd_gram_select", path), "igd_gram_select")
    try:
        code = _lib.call("igd_block_gram", _lib.IGD_F64, n, a, ptr(A), A.stride(0), b, ptr(B), B.stride(0), ptr(w),
                         ptr(out), int(acc), ptr(ws), wsb, stream_ptr())
        last = _lib.call("igd_gram_last_path")
    finally:
        _lib.call("igd_gram_select", 0)
    return code, out.cpu().numpy(), last


def test_split_gram_above_nine_million_points():
    """More windows than int32 level sums of one launch hold: taken in pieces, against the plain kernel."""

    import torch

    n = 9_500_001
    g = torch.Generator("cuda").manual_seed(8)
    A = torch.randn((3, n), dtype=torch.float64, device="cuda", generator=g)
    B = torch.randn((2, n), dtype=torch.float64, device="cuda", generator=g)
    w = torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
    (_, got, last), (_, plain, _) = _gram(A, B, w, 4), _gram(A, B, w, 3)
    scale = (A.abs() * w) @ B.abs().T
    assert last == 4 and np.all(np.abs(got - plain) <= 2.0**-44 * scale.cpu().numpy())
    _, more, _ = _gram(A, B, w, 4, out=torch.full((3, 2), 1.0, dtype=torch.float64, device="cuda"))
    assert np.all(np.abs(more - 1.0 - got) <= 2.0**-50 * np.abs(got) + 2.0**-50)
    # rows that do not overlap: zero in every piece, by either route
    A[0, n // 2:] = 0.0
    B[0, :n // 2] = 0.0
    (_, got, _), (_, plain, _) = _gram(A, B, w, 4), _gram(A, B, w, 3)
    scale = (A.abs() * w) @ B.abs().T
    assert got[0, 0] == 0.0 and np.all(np.abs(got - plain) <= 2.0**-44 * scale.cpu().numpy())


def test_self_gram_with_an_overflowing_product():
    """w x of one row overflows while x is finite: outputs of that row and column as the plain kernel gives them."""

    import torch

    n, a = 4000, 19
    g = torch.Generator("cuda").manual_seed(1)
    X = torch.randn((a, n), dtype=torch.float64, device="cuda", generator=g)
    w = torch.rand(n, dtype=torch.float64, device="cuda", generator=g) + 1e-3
    p = 777
    w[p] = 1e150
    X[:, p] = 1e-200
    X[7, p] = 1e200
    (_, got, last), (_, plain, _) = _gram(X, X, w, 4), _gram(X, X, w, 3)
    assert last == 4
    assert np.array_equal(np.isnan(got), np.isnan(plain)) and np.array_equal(np.isinf(got), np.isinf(plain))
    fine = np.isfinite(plain)
    assert fine[7].sum() == a - 1 and not fine[:, 7].any()  # (i, 7) multiplies the infinity, (7, j) does not
    assert np.all(np.abs(got[fine] - plain[fine]) <= 1e-12 * np.abs(plain[fine]) + 1e-9)


@pytest.mark.parametrize("path", [0, 4])
def test_workspace_alignment_and_size(path):
    """A workspace aligned to a double, and one of the plain kernels' size, are taken as ever; one that is smaller is
    refused."""

    import torch

    from isogriddft_gb300 import _lib

    n, a, b = 1 << 18, 12, 9
    g = torch.Generator("cuda").manual_seed(7)
    A = torch.randn((a, n), dtype=torch.float64, device="cuda", generator=g)
    B = torch.randn((b, n), dtype=torch.float64, device="cuda", generator=g)
    w = torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
    want = ((A * w) @ B.T).cpu().numpy()
    blocks = max(min(-(-n // 256), 608), min(-(-n // 16384), 4096))
    plain = 8 * blocks * a * b  # one FP64 partial per block and output
    full = int(_lib.call("igd_block_gram_workspace_bytes", n, a, b))
    assert full <= 1.1 * plain
    buf = torch.full((full // 8 + 4,), float("nan"), dtype=torch.float64, device="cuda")
    for ws, size in ((buf[1:], full), (buf, plain), (buf[1:], plain), (buf, full)):
        code, got, _ = _gram(A, B, w, path, ws, size)
        assert code == 0 and np.all(np.abs(got - want) <= 1e-9)
    assert bool(torch.isnan(buf[-3:]).all())
    assert _gram(A, B, w, path, buf, plain - 8)[0] == _lib.IGD_ERR_ARG


def _wide(kind, n):
    """Rows A (5, n) and B (4, n), whose products are far below max|a| max|b| at every point."""

    import torch

    r = torch.linspace(0.0, 60.0, n, dtype=torch.float64, device="cuda")
    g = torch.Generator("cuda").manual_seed(2)
    A = torch.randn((5, n), dtype=torch.float64, device="cuda", generator=g)
    B = torch.randn((4, n), dtype=torch.float64, device="cuda", generator=g)
    if kind == "opposite":  # localised at opposite ends
        A *= torch.exp(-r)
        B *= torch.exp(r - 60.0)
    elif kind == "spike":  # one value of A far above the rest, where B is zero
        A[:, 5] = 1e8
        B[:, 5] = 0.0
    elif kind == "weight":  # one weight far above the rest, where A is zero
        A[:, 9] = 0.0
        B[:, 9] = 1e9
    elif kind == "disjoint":
        A[:, n // 2:] = 0.0
        B[:, :n // 2] = 0.0
    elif kind == "zero":
        A[1] = 0.0
        B[2] = 0.0
    return A, B


# one window, several, and the size from which the automatic choice is the splitting kernel
@pytest.mark.parametrize("n", [50, 5003, 1 << 18])
@pytest.mark.parametrize("kind", ["normal", "opposite", "spike", "weight", "disjoint", "zero"])
def test_split_gram_keeps_the_plain_accuracy(n, kind):
    """Every output to the plain kernels' bound, relative to sum |a w b|: 2^-53 for each of at most 64 products of a
    thread, their sums, the tree over 256 threads and the sum over at most 608 blocks (10 steps): 2^-45 in all."""

    import torch

    A, B = _wide(kind, n)
    w = torch.rand(n, dtype=torch.float64, device="cuda") + 1e-3
    for X, Y, ww in ((A, B, w), (A, B, None), (A, A, w)):
        for path in (4, 0):
            code, got, last = _gram(X, Y, ww, path)
            assert code == 0 and (path == 0 or last == 4)
            x, y = X.cpu().numpy().astype(np.longdouble), Y.cpu().numpy().astype(np.longdouble)
            y = y * (ww.cpu().numpy() if ww is not None else 1)
            want, scale = x @ y.T, np.abs(x) @ np.abs(y).T
            assert np.all(np.abs(got - want) <= 2.0**-45 * scale), (
                last, float(np.max(np.abs(got - want) / (scale + (scale == 0)))))
            # added to a non-zero result, outputs of every route once
            _, twice, _ = _gram(X, Y, ww, path, out=torch.full(got.shape, 0.5, dtype=torch.float64, device="cuda"))
            assert np.array_equal(twice, 0.5 + got)
