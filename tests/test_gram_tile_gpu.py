"""Plain tiled Gram: tile edges, ragged rows, weights at the ends of the FP32 range, sums in FP64."""

import pytest
import torch

from isogriddft_gb300 import _lib
from isogriddft_gb300.device import ptr, stream_ptr

pytestmark = pytest.mark.gpu


def _gram(A, B, w):
    a, n = A.shape
    b = B.shape[0]
    out = torch.empty(a, b, device="cuda", dtype=torch.float64)
    size = int(_lib.call("igd_block_gram_workspace_bytes", n, a, b))
    ws = torch.empty(size, dtype=torch.uint8, device="cuda")
    code = _lib.IGD_F32 if A.dtype == torch.float32 else _lib.IGD_F64
    try:
        _lib.check(_lib.call("igd_gram_select", 3))
        _lib.check(_lib.call("igd_block_gram", code, n, a, ptr(A), A.stride(0), b, ptr(B), B.stride(0),
                             ptr(w) if w is not None else None, ptr(out), 0, ptr(ws), size, stream_ptr()))
        assert _lib.call("igd_gram_last_path") == 3
    finally:
        _lib.call("igd_gram_select", 0)
    return out


@pytest.mark.parametrize("dtype,eps", [(torch.float32, 2.0**-24), (torch.float64, 2.0**-53)])
@pytest.mark.parametrize("n", [1, 33, 257, 16385, 100003])
@pytest.mark.parametrize("a,b", [(1, 1), (4, 4), (5, 3), (21, 8), (9, 70)])
def test_against_fp64(n, a, b, dtype, eps):
    g = torch.Generator(device="cuda").manual_seed(n + a + b)
    A = torch.randn(a, n + 1, generator=g, device="cuda", dtype=dtype)[:, 1:]
    B = torch.randn(b, n + 1, generator=g, device="cuda", dtype=dtype)[:, 1:]
    w = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) + 0.5
    for weight in (w, None):
        W = w if weight is not None else torch.ones_like(w)
        want = (A.double() * W) @ B.double().T
        # at most 64 terms of a thread are summed in the operands' type, the rest in FP64
        bound = 70 * eps * ((A.double().abs() * W) @ B.double().abs().T) + 1e-300
        assert bool(((_gram(A, B, weight) - want).abs() <= bound).all())


def test_weights_round_to_nearest_fp32():
    tie = 1.0 + 2.0**-24
    values = [0.0, -0.0, 1.0, -3.7, tie, 1.0 + 3 * 2.0**-24, tie + 2.0**-52, 2.0**-126, 2.0**-127, 2.0**-149, 2.0**-151,
              (2 - 2.0**-24) * 2.0**127, 3.4e38, -3.4e38, 1e-40, 5e-324, 1.0 / 3.0, -1.0 / 3.0]
    w = torch.tensor(values, dtype=torch.float64, device="cuda")
    A = torch.ones(1, 1, device="cuda")
    for k in range(len(values)):
        got = _gram(A, A, w[k:k + 1].clone())
        assert float(got) == float(w[k:k + 1].float()), values[k]
    for bad in (float("inf"), float("-inf"), float("nan"), 1e39):
        got, want = float(_gram(A, A, torch.tensor([bad], dtype=torch.float64, device="cuda"))), float(torch.tensor(bad))
        assert got == want or (got != got and want != want)
