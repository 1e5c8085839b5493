"""FP32 block rotation: every width of the pipelined and the register kernels, at tile edges and ragged rows."""

import pytest
import torch

from isogriddft_gb300 import _lib

pytestmark = pytest.mark.gpu

EDGE = 1 << 19  # grids of this size and larger take the shared-memory pipeline when their rows are 16-byte aligned


def _rotate(A, C1, B, C2, out, accumulate):
    b = 0 if B is None else B.shape[0]
    _lib.check(_lib.call("igd_block_rotate", 0, A.shape[1], A.shape[0], A.data_ptr(), A.stride(0), C1.data_ptr(), b,
                         B.data_ptr() if b else None, B.stride(0) if b else 0, C2.data_ptr() if b else None,
                         out.shape[0], out.data_ptr(), out.stride(0), accumulate,
                         torch.cuda.current_stream().cuda_stream))


@pytest.mark.parametrize("n", [1, 255, 100001, EDGE - 1, EDGE, EDGE + 1, EDGE + 1027])
@pytest.mark.parametrize("a,b,c", [(1, 0, 1), (7, 1, 4), (8, 3, 5), (9, 0, 9), (16, 5, 13), (21, 1, 17), (13, 4, 24),
                                   (32, 15, 25), (17, 16, 32), (35, 15, 33), (20, 0, 48), (12, 4, 49), (5, 2, 70),
                                   (180, 20, 33)])
def test_fp32_rotation_against_fp64(n, a, b, c):
    g = torch.Generator(device="cuda").manual_seed(n + 100 * a + b + c)
    rnd = lambda *s, **k: torch.randn(*s, generator=g, device="cuda", **k)
    pad = -n % 4
    for aligned in (True, False):
        # rows of a larger buffer: aligned rows, or rows that start one value later
        A = rnd(a, n + pad + 4)[:, 0 if aligned else 1:][:, :n]
        B = rnd(b, n + pad + 4)[:, 0 if aligned else 1:][:, :n] if b else None
        C1 = rnd(a, c, dtype=torch.float64)
        C2 = rnd(max(b, 1), c, dtype=torch.float64)
        for accumulate in (0, 1):
            buf = rnd(c + 1, n + pad + 4)
            out = buf[:c, :n] if aligned else buf[:c, 1:n + 1]
            before = buf.clone()
            want = out.double() * accumulate + C1.T @ A.double()
            scale = out.double().abs() * accumulate + C1.T.abs() @ A.double().abs()
            if b:
                want += C2.T @ B.double()
                scale += C2.T.abs() @ B.double().abs()
            _rotate(A, C1, B, C2, out, accumulate)
            # every product and sum rounds once to FP32, and so does every coefficient
            bound = (a + b + 3) * 2.0**-24 * scale + 1e-30
            assert bool(((out.double() - want).abs() <= bound).all())
            out.copy_(before[:c, :n] if aligned else before[:c, 1:n + 1])
            assert torch.equal(buf, before), "values outside the rotated rows changed"


def test_pipeline_and_register_kernels_agree_to_the_bit():
    n, a, b, c = EDGE + 4, 19, 6, 30
    big = torch.randn(a + b, n + 4, device="cuda")
    C1 = torch.randn(a, c, device="cuda", dtype=torch.float64)
    C2 = torch.randn(b, c, device="cuda", dtype=torch.float64)
    got = []
    for shift in (0, 1):
        rows = torch.empty(a + b, n + 4, device="cuda")
        X = rows[:, shift:shift + n]
        X.copy_(big[:, :n])
        out = torch.empty(c, n, device="cuda")
        _rotate(X[:a], C1, X[a:], C2, out, 0)
        got.append(out)
    assert torch.equal(got[0].view(torch.int32), got[1].view(torch.int32))


@pytest.mark.parametrize("c,most", [(4, 12800), (16, 3200), (17, 1600), (33, 1600)])
def test_coefficients_beyond_shared_memory_are_refused(c, most):
    out = torch.empty(c, 8, device="cuda")
    for a in (most, most + 1):
        args = (torch.zeros(a, 8, device="cuda"), torch.zeros(a, c, device="cuda", dtype=torch.float64), None, None, out)
        if a == most:
            _rotate(*args, 0)
            assert not out.any()
        else:
            with pytest.raises(Exception):
                _rotate(*args, 0)


@pytest.mark.parametrize("a,b,c", [(512, 0, 12), (300, 170, 13), (1536, 0, 4)])
def test_many_rows_to_few_columns(a, b, c):
    """Coefficients that leave one CTA of the pipeline on an SM."""
    n = EDGE + 4
    g = torch.Generator(device="cuda").manual_seed(a + b + c)
    rnd = lambda *s, **k: torch.randn(*s, generator=g, device="cuda", **k)
    A, C1, C2 = rnd(a, n), rnd(a, c, dtype=torch.float64), rnd(max(b, 1), c, dtype=torch.float64)
    B = rnd(b, n) if b else None
    out = rnd(c, n)
    _rotate(A, C1, B, C2, out, 0)
    bound = torch.zeros(c, n, device="cuda", dtype=torch.float64)
    want = torch.zeros_like(bound)
    for X, C in ((A, C1), (B, C2)):
        for r in range(0, X.shape[0] if X is not None else 0, 64):
            want += C[r:r + 64].T @ X[r:r + 64].double()
            bound += C[r:r + 64].T.abs() @ X[r:r + 64].double().abs()
    assert bool(((out.double() - want).abs() <= (a + b + 3) * 2.0**-24 * bound).all())
