"""The yield screen's short cuts (csrc/des_rheology.cuh: yield_screen3_f,
csrc/des_common.cuh: screen_terms_any), restated in numpy: an element that the
norm bounds pass also passes with the eigenvalues, the FP32 material terms lie
within the stated 2^-17 of the FP64 ones, and with that allowance the screen's
yes and no are those of the exact terms (the rest is left undecided).
The restatements use IEEE FP32 operations; a tolerance of 2^-17 is the
kernel's own, derived beside it.
"""
import numpy as np
import pytest

from test_yield_screen import F, _rotations, _voigt, f32_of, jacobi3f

ERR = F(2.0 ** -17)


def screen(af, cf, tf, mf, d, err):
    """yield_screen3_f with mag = |mf|, dev_err = 0: (answer, passed by the bounds)."""
    nf = np.sqrt(d[:, 0] ** 2 + d[:, 1] ** 2 + d[:, 2] ** 2 + F(2) * (d[:, 3] ** 2 + d[:, 4] ** 2 + d[:, 5] ** 2))
    tol = F(2.0 ** -12) * nf + F(2.0 ** -19) * (np.abs(mf) + nf) + F(2.0 ** -100)
    fs_min = (F(1) + af) * tol + F(2.0 ** -19) * np.abs(cf)
    ft_max = -(tol + F(2.0 ** -19) * np.abs(tf))
    e2 = F(2) * err + F(2.0 ** -20) if err > 0 else F(0)
    dt = e2 * (np.abs(tf) + np.abs(ft_max))
    R = F(float.fromhex("0x1.004p0")) * nf + F(2.0 ** -70)
    hi, lo = mf + R, mf - R
    ds = e2 * (np.abs(lo) + np.abs(hi) * af + np.abs(cf) + fs_min)
    quick = (lo - hi * af + cf > fs_min + ds) & (hi - tf < ft_max - dt)
    w = jacobi3f(d)
    p0, p2 = mf + w[:, 0], mf + w[:, 2]
    fs, ft = p0 - p2 * af + cf, p2 - tf
    if err == 0:
        return np.where((fs > fs_min) & (ft < ft_max), 1, 0), quick
    ds = e2 * (np.abs(p0) + np.abs(p2) * af + np.abs(cf) + fs_min)
    yes = (fs > fs_min + ds) & (ft < ft_max - dt)
    no = (fs < fs_min - ds) | (ft > ft_max + dt)
    return np.where(quick | yes, 1, np.where(no, 0, -1)), quick


def materials(rng, n):
    """Cohesions and angles within a factor 16, and the softening's place between them."""
    c0, f0 = 10 ** rng.uniform(5, 8, n), rng.uniform(1, 60, n)
    c1, f1 = c0 / rng.uniform(1, 16, n), f0 / rng.uniform(1, 16, n)
    swap = rng.uniform(size=n) < 0.3
    c0, c1 = np.where(swap, c1, c0), np.where(swap, c0, c1)
    l1 = 10 ** rng.uniform(-2, 0, n)
    pls = l1 * rng.uniform(1e-9, 1, n) ** rng.choice((1, 4), n)
    q = pls / l1
    c, phi = c0 + q * (c1 - c0), np.radians(f0 + q * (f1 - f0))
    anphi = (1 + np.sin(phi)) / (1 - np.sin(phi))
    exact = anphi, 2 * c * np.sqrt(anphi), np.minimum(1e9, c / np.tan(phi))
    qf = f32_of(pls) / f32_of(l1)
    cf = f32_of(c0) + qf * (f32_of(c1) - f32_of(c0))
    rad = (f32_of(f0) + qf * (f32_of(f1) - f32_of(f0))) * F(0.017453292519943295)
    sp = np.sin(rad)
    af = (F(1) + sp) / (F(1) - sp)
    return exact, (af, F(2) * cf * np.sqrt(af), np.minimum(F(1e9), cf / np.tan(rad)))


def test_fp32_terms_lie_within_their_allowance():
    exact, approx = materials(np.random.default_rng(0), 400_000)
    for x, a in zip(exact, approx):
        x = f32_of(x).astype(np.float64)
        assert np.max(np.abs(a.astype(np.float64) - x) / x) < 2.0 ** -17


@pytest.mark.parametrize("place", ["surface", "cutoff", "anywhere"])
def test_screen_with_an_allowance_agrees_with_the_exact_terms(place):
    rng = np.random.default_rng(1)
    n = 120_000
    (anphi, amc, ten), (af, cf, tf) = materials(rng, n)
    p2 = -10 ** rng.uniform(4, 9, n)
    rel = rng.choice((-1, 1), n) * 10 ** rng.uniform(-9, -1, n)
    if place == "cutoff":
        p2 = ten * (1 + rel)
        p0 = p2 - rng.uniform(0, 1, n) * amc
    elif place == "surface":
        p0 = (p2 * anphi - amc) * (1 + rel)
    else:
        p0 = p2 - np.abs(p2) * 10 ** rng.uniform(-12, 1, n)
    p1 = p0 + rng.choice((0.0, 1.0, 0.3), n) * (p2 - p0)
    s = _voigt(_rotations(rng, n), np.stack([p0, p1, p2], axis=1))
    m = (s[:, 0] + s[:, 1] + s[:, 2]) / 3
    d = np.concatenate([s[:, :3] - m[:, None], s[:, 3:]], axis=1)
    d, mf = f32_of(d), f32_of(m)
    want, quick = screen(f32_of(anphi), f32_of(amc), f32_of(ten), mf, d, F(0))
    assert np.all(want[quick] == 1)   # the bounds pass nothing that the eigenvalues do not
    got, _ = screen(af, cf, tf, mf, d, ERR)
    sure = got >= 0
    assert np.all(got[sure] == want[sure])
    assert sure.mean() > (0.95 if place == "anywhere" else 0.3)
