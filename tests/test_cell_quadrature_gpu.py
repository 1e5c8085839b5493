"""Cell quadrature of the corrected moments against NumPy least squares, cell by cell."""

import numpy as np
import pytest
import torch

from isogriddft_gb300 import _lib
from isogriddft_gb300.device import ptr, stream_ptr

pytestmark = pytest.mark.gpu


def _basis(p):
    u, v, t = p[..., 0], p[..., 1], p[..., 2]
    return np.stack([np.ones_like(u), u, v, t, u * u, v * v, t * t, u * v, u * t, v * t], -1)


def _moments(w, d):
    r2 = (d * d).sum(-1)
    q = [3 * d[:, a] * d[:, b] - (r2 if a == b else 0) for a, b in ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))]
    return np.array([w.sum(), *(w[:, None] * d).sum(0), *[(w * x).sum() for x in q]])


def _oracle(P, J, R, cell, dvol, mode, centre):
    i, j, k = cell
    near = np.s_[i - 1:i + 3, j - 1:j + 3, k - 1:k + 3]
    box = np.s_[i:i + 2, j:j + 2, k:k + 2]
    c = P[box].reshape(-1, 3).mean(0)
    L = np.abs(P[i + 1, j + 1, k + 1] - P[i, j, k]).max()
    coef = np.linalg.lstsq(_basis((P[near].reshape(-1, 3) - c) / L), R[near].reshape(-1), rcond=None)[0]
    s = np.array([0.25, 0.75])
    W = np.stack([1 - s, s], -1)
    tri = lambda F: np.einsum("ai,bj,ck,ijk...->abc...", W, W, W, F[box]).reshape(8, *F.shape[3:])  # noqa: E731
    p, jac, rt = tri(P), tri(J), tri(R)
    rq = _basis((p - c) / L) @ coef
    if mode == 0:
        return _moments(rq * jac * dvol, p - centre)
    delta = (rq - rt) * jac * dvol
    if mode == 2:
        return _moments(delta, p - centre)
    a = np.abs(delta)
    return np.array([a.sum(), *(a[:, None] * p).sum(0), 0, 0, 0, 0, 0, 0])


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("shape,stretch", [((4, 4, 4), 0.0), ((5, 6, 7), 0.3), ((9, 8, 7), 0.9)])
def test_against_numpy(shape, stretch, mode):
    rng = np.random.default_rng(sum(shape) + mode)
    g = np.stack(np.meshgrid(*[np.arange(n) * h for n, h in zip(shape, (0.3, 0.25, 0.4))], indexing="ij"), -1)
    P = g + stretch * 0.1 * rng.standard_normal(g.shape) - 0.5
    J, R = rng.random(shape) + 0.5, rng.standard_normal(shape)
    cells = np.stack(np.meshgrid(*[np.arange(1, n - 2) for n in shape], indexing="ij"), -1).reshape(-1, 3)
    dvol, centre = 0.01, np.array([0.2, -0.1, 0.3])
    f = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    x, y, z, jac, rho = (f(P[..., 0]), f(P[..., 1]), f(P[..., 2]), f(J), f(R))
    idx = f(cells.astype(np.int32))
    out = torch.zeros(10, device="cuda", dtype=torch.float64)
    fail = torch.zeros(1, device="cuda", dtype=torch.int32)
    _lib.check(_lib.call("igd_multipole_cell_quadrature", *shape, ptr(x), ptr(y), ptr(z), ptr(jac), ptr(rho), ptr(idx),
                         len(cells), dvol, mode, *centre, ptr(out), ptr(fail), stream_ptr()))
    each = np.array([_oracle(P, J, R, c, dvol, mode, centre) for c in cells])
    # normal equations of the scaled basis (condition below 1e6) in FP64, against an orthogonal solve
    bound = 1e-9 * np.abs(each).max(0) * len(cells) + 1e-12
    assert int(fail) == 0
    assert np.all(np.abs(out.cpu().numpy() - each.sum(0)) <= bound)


def test_coincident_nodes_are_flagged():
    n = (4, 4, 4)
    zero = torch.zeros(n, device="cuda", dtype=torch.float64)
    idx = torch.ones(3, device="cuda", dtype=torch.int32)
    out = torch.zeros(10, device="cuda", dtype=torch.float64)
    fail = torch.zeros(1, device="cuda", dtype=torch.int32)
    _lib.check(_lib.call("igd_multipole_cell_quadrature", *n, ptr(zero), ptr(zero), ptr(zero), ptr(zero), ptr(zero),
                         ptr(idx), 1, 1.0, 0, 0.0, 0.0, 0.0, ptr(out), ptr(fail), stream_ptr()))
    assert int(fail) == 1 and not out.any()
