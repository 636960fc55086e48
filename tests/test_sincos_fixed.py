"""The GPU's fixed-point sine and cosine phase, compiled for the host: wherever it does not
decline it has to give the accurate phase's doubles, and it has to decline rarely."""
import numpy as np
import pytest

RANGES = {
    "angles": lambda r, n: r.uniform(-10.0, 10.0, n),
    "small": lambda r, n: r.uniform(-1.0, 1.0, n) * np.pi / 4,
    "tiny": lambda r, n: np.exp(r.uniform(np.log(2.0 ** -27), np.log(1e-2), n)) * r.choice([-1.0, 1.0], n),
    "large": lambda r, n: r.uniform(-65536.0, 65536.0, n),
    "steps": lambda r, n: r.integers(1, 2 ** 23, n) * (np.pi / 512),
    "half steps": lambda r, n: (r.integers(0, 2 ** 22, n) + 0.5) * (np.pi / 512),
    "near steps": lambda r, n: r.integers(1, 2 ** 16, n) * (np.pi / 512) + r.uniform(-1.0, 1.0, n) * 1e-7,
    "quadrants": lambda r, n: np.nextafter(r.integers(1, 2 ** 15, n) * (np.pi / 2), r.choice([-1e9, 1e9], n)),
}


@pytest.mark.parametrize("name", sorted(RANGES))
def test_fixed_phase_is_the_accurate_phase(oracle_lib, name):
    x = RANGES[name](np.random.default_rng(len(name)), 300_000)
    x = x[(np.abs(x) >= 2.0 ** -27) & (np.abs(x) < 65536.0)]
    got, ok = oracle_lib.sincos_phase(x, 3)
    want, _ = oracle_lib.sincos_phase(x, 0)
    ok = ok.astype(bool)
    for k in (0, 2):
        assert np.array_equal(got[ok, k].view(np.int64), want[ok, k].view(np.int64)), x[ok][got[ok, k] != want[ok, k]][:5]
    if name in ("angles", "small", "tiny", "large"):
        assert (~ok).mean() < 2.0 ** -13


@pytest.mark.parametrize("x", [2.0 ** -27, np.nextafter(2.0 ** -27, 1.0), np.pi / 1024, np.nextafter(np.pi / 1024, 1.0),
                               np.pi / 512, np.pi / 4, np.pi / 2, np.pi, 22.0, 355.0, 65535.99999999999])
def test_fixed_phase_at_the_edges(oracle_lib, x):
    for v in (x, -x):
        got, ok = oracle_lib.sincos_phase(np.array([v]), 3)
        want, _ = oracle_lib.sincos_phase(np.array([v]), 0)
        if ok[0]:
            assert got[0, 0] == want[0, 0] and got[0, 2] == want[0, 2]
