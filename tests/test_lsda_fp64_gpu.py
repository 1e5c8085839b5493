"""The FP64 LSDA kernel (piecewise polynomials, seeded roots) against 45-digit values of the published forms."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _exact(u, d, functional):
    """(eps, v_up, v_down) from the closed forms in multiprecision, potentials by their rs and zeta derivatives."""

    import importlib.util
    import os

    mp = pytest.importorskip("mpmath")
    path = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "make_lsda_tables.py")
    spec = importlib.util.spec_from_file_location("make_lsda_tables", path)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    gp, gf, ga = mod.channels()["VWN" if functional == "lda,vwn" else "PW"]
    third = mp.mpf(1) / 3
    fden, fpp = 2 * mp.mpf(2) ** third - 2, mp.mpf(4) / (9 * (mp.mpf(2) ** third - 1))
    cx = (6 / mp.pi) ** third
    out = []
    for uu, dd in zip(u, d):
        uu, dd = mp.mpf(float(uu)), mp.mpf(float(dd))
        r = uu + dd
        if r < mp.mpf(1e-15):
            out.append((0.0, 0.0, 0.0))
            continue
        x, z = mp.sqrt((3 / (4 * mp.pi * r)) ** third), (uu - dd) / r

        def f(s):
            return ((1 + s) * mp.cbrt(1 + s) + (1 - s) * mp.cbrt(1 - s) - 2) / fden

        df = mp.mpf(4) / 3 * (mp.cbrt(1 + z) - mp.cbrt(1 - z)) / fden
        G = [g(x) for g in (gp, gf, ga)]
        H = [x * mp.diff(g, x) / 6 for g in (gp, gf, ga)]  # rs dG/drs / 3
        mix = lambda v: v[0] + v[2] * f(z) * (1 - z**4) / fpp + (v[1] - v[0]) * f(z) * z**4  # noqa: E731
        ec, sl = mix(G), mix(H)
        dz = G[2] * (df * (1 - z**4) - 4 * z**3 * f(z)) / fpp + (G[1] - G[0]) * (df * z**4 + 4 * z**3 * f(z))
        ex = -mp.mpf(3) / 4 * cx * (uu * mp.cbrt(uu) + dd * mp.cbrt(dd)) / r
        out.append((ex + ec, -cx * mp.cbrt(uu) + ec - sl + (1 - z) * dz, -cx * mp.cbrt(dd) + ec - sl - (1 + z) * dz))
    return np.array([[float(v) for v in row] for row in out])


@pytest.mark.parametrize("functional", ["lda,vwn", "lda,pw92"])
def test_lsda_fp64_against_multiprecision(functional):
    """Densities from below the 1e-15 cut-off to beyond the tables (2^15), polarised and not, at table edges, tiny
    and subnormal minority spins.  Bound: 40 units of 2^-53 of the point's largest term (about 30 roundings of
    terms no larger than the exchange and correlation energies enter each output)."""

    import torch

    from isogriddft_gb300.xc import lsda_device

    rng = np.random.default_rng(3)
    total = np.concatenate([10.0 ** rng.uniform(-16, 6, 60), [1e-15, 9.99e-16, 0.0, 2.0**15, 32767.9, 62579.0, 1e3],
                            (0.6203504908994 / np.array([0.25, 0.5, 1.0, 1.125, 2.0, 64.0]) ** 2) ** 3])
    frac = np.concatenate([rng.uniform(0, 1, total.size - 24), np.full(8, 0.5), np.zeros(4), np.ones(4),
                           np.full(4, 1e-40), np.full(4, 1e-300)])
    u, d = total * frac, total * (1.0 - frac)
    u[-1], d[-2] = 3e-310, 5e-324
    tu, td = (torch.as_tensor(a, device="cuda") for a in (u, d))
    got = lsda_device(tu, td, functional=functional)
    want = _exact(u, d, functional)
    scale = np.abs(want).max(axis=1)
    for k, name in enumerate(("eps", "v_up", "v_down")):
        g = got[name].cpu().numpy()
        off = np.abs(g - want[:, k]) / np.where(scale > 0, scale, 1.0)
        assert off.max() < 40 * 2.0**-53, (name, int(off.argmax()), off.max(), u[off.argmax()], d[off.argmax()])
    assert np.array_equal(got["edens"].cpu().numpy(), (u + d) * got["eps"].cpu().numpy())


def test_lsda_fp64_flags_and_sizes():
    """Negative within roundoff counts as zero, beyond it and non-finite values raise; 1 to 70001 points."""

    import torch

    from isogriddft_gb300.xc import lsda_device

    one = lambda v: torch.tensor([v, 0.3], dtype=torch.float64, device="cuda")  # noqa: E731
    a, b = lsda_device(one(-0.9e-14), one(0.2)), lsda_device(one(0.0), one(0.2))
    assert all(torch.equal(a[k], b[k]) for k in ("eps", "v_up", "v_down", "edens"))
    with pytest.raises(ValueError, match="non-negative"):
        lsda_device(one(-1.1e-14), one(0.2))
    for v in (float("nan"), float("inf"), float("-inf")):
        with pytest.raises(ValueError, match="finite"):
            lsda_device(one(v), one(0.2))
    rng = np.random.default_rng(0)
    big = torch.as_tensor(rng.random(70001) ** 4, device="cuda")
    full = lsda_device(big, big.flip(0))
    for n in (1, 2, 255, 257, 40001):
        part = lsda_device(big[:n].clone(), big.flip(0)[:n].clone())
        assert torch.equal(part["v_up"], full["v_up"][:n])
