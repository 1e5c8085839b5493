"""Tensor-core FP32 Gram with rows padded to eight: column halves of unequal width, weight tails, few stages."""

import pytest
import torch

from isogriddft_gb300 import _lib
from isogriddft_gb300.device import ptr, stream_ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 127, 4098, 70_003])
@pytest.mark.parametrize("a,b", [(47, 47), (40, 41), (17, 24), (23, 9), (64, 49), (3, 33), (8, 8), (1, 64), (50, 7)])
def test_row_padding_and_weight_tails(n, a, b):
    g = torch.Generator(device="cuda").manual_seed(97 * n + 64 * a + b)
    ld = (n + 3) // 4 * 4 + 4
    A = torch.randn(a, ld, generator=g, device="cuda")
    B = torch.randn(b, ld, generator=g, device="cuda")
    w = torch.rand(n + 4, generator=g, device="cuda", dtype=torch.float64) + 0.5
    for M in (A, B):
        M[:, n:] = float("nan")  # never read
    w[n:] = float("nan")
    out = torch.empty(a, b, device="cuda", dtype=torch.float64)
    size = int(_lib.call("igd_block_gram_workspace_bytes", n, a, b))
    ws = torch.empty(size, dtype=torch.uint8, device="cuda")
    try:
        _lib.check(_lib.call("igd_gram_select", 1))
        for weight in (w, None):
            _lib.check(_lib.call("igd_block_gram", _lib.IGD_F32, n, a, ptr(A), ld, b, ptr(B), ld,
                                 ptr(weight) if weight is not None else None, ptr(out), 0, ptr(ws), size,
                                 stream_ptr()))
            assert _lib.call("igd_gram_last_path") == 1
            wd = w[:n] if weight is not None else torch.ones_like(w[:n])
            ref = (A[:, :n].double() * wd) @ B[:, :n].double().T
            # the split keeps 2^-21 of a product, FP32 weights 2^-24, the accumulator's window sums 2^-20 of theirs
            bound = 2.0**-19 * (A[:, :n].double().abs() * wd) @ B[:, :n].double().abs().T
            assert bool(((out - ref).abs() <= bound).all())
    finally:
        _lib.call("igd_gram_select", 0)
    assert _lib.error_flags(clear=True, stream=stream_ptr()) == 0
