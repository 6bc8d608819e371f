"""The EPA's two stop tests in one FP32 comparison (narrow.cu epa_stops), restated in numpy float32 and
checked against the reference's double tests (gpu_fine_contact_detection.cu:437-439)."""
import numpy as np

f32 = np.float32


def epa_stops(x, p):
    """(answer, decided): where `decided` is False the kernel runs the reference's tests."""
    hi = x * f32(1.00001)
    tol = x * f32(2.384185791015625e-7)
    ranged = (x > f32(1e-30)) & (x < f32(1e37))
    yes, no = p < hi - tol, p > hi + tol
    return yes, ranged & (yes | no)


def reference(x, p):
    xd, pd = x.astype(np.float64), p.astype(np.float64)
    return (x > p) | ((xd * 1.00001 > pd) & (xd * 0.99999 < pd))


def test_epa_stops_decides_almost_always():
    # the undecided band is 4.8e-7 of x wide: p within a factor of two of x lies in it once in some millions
    rng = np.random.default_rng(1)
    x = rng.uniform(0.5, 1.0, 200_000).astype(f32)
    got, decided = epa_stops(x, (x * rng.uniform(0.5, 2.0, x.size)).astype(f32))
    assert decided.mean() > 0.999 and got.any() and not got.all()
    # and a p within 2e-5 of x, as near the end of a search, 97 times in 100
    near = (x.astype(np.float64) * (1 + rng.normal(scale=2e-5, size=x.size))).astype(f32)
    assert epa_stops(x, near)[1].mean() > 0.97


def test_epa_stops_is_the_references_double_test():
    rng = np.random.default_rng(0)
    x = (rng.uniform(0.5, 1.0, 400_000) * 2.0 ** rng.integers(-110, 120, 400_000)).astype(f32)
    near = [x, x * f32(1.00001), x * f32(0.99999)]
    cases = [(x, (x * rng.uniform(0.5, 2.0, x.size)).astype(f32))]
    for base in near:  # ulp by ulp around the bounds
        for k in range(-12, 13):
            cases.append((x, (base.view(np.int32) + k).view(f32)))
    odd = np.array([0.0, -0.0, 1e-38, -1.0, 1.0, np.inf, -np.inf, np.nan, 3e20, 1e30], f32)
    cases.append(tuple(a.ravel() for a in np.meshgrid(odd, odd)))
    with np.errstate(all="ignore"):
        for a, b in cases:
            got, decided = epa_stops(a, b)
            assert np.array_equal(got[decided], reference(a, b)[decided])
