"""The FP32 build's density terms, which are evaluated and summed in FP64: particles whose neighbours lie where
rho - rho0 cancels, against extended precision. There the stored FP32 value resolves 1e-11 kg/m^3, so a
square root of less than FP64's accuracy shows."""
import math

import numpy as np
import pytest

from splishsplash_for_cuda_b200.dfsph import DFSPHCUDA
from splishsplash_for_cuda_b200.scene import Configuration, Scene

pytestmark = pytest.mark.gpu


def _w(q):
    """W / k in the precision of q."""
    return np.where(q <= 0.5, 1 + 6 * q * q * (q - 1), np.where(q < 1, 2 * (1 - q) ** 3, 0))


def _clusters(r, seed):
    """Centres far apart, each with 4 to 40 neighbours at distances around the one that gives rho0."""
    rng = np.random.default_rng(seed)
    H = float(np.float32(4 * r))
    mass = float(np.float32(0.8 * (2 * r) ** 3 * 1000.0))
    k = 8 / (math.pi * H ** 3)
    x, centre = [], []
    for c in range(512):
        n = 4 + c % 37
        o = rng.normal(size=(n, 3))
        o /= np.linalg.norm(o, axis=1)[:, None]
        o *= rng.uniform(0.9, 1.1, (n, 1))
        lo, hi = 0.0, 1.0
        for _ in range(200):
            s = 0.5 * (lo + hi)
            lo, hi = (s, hi) if mass * k * (1 + _w(s * np.linalg.norm(o, axis=1)).sum()) > 1000.0 else (lo, s)
        at = (np.array([c % 8, c // 8 % 8, c // 64]) + 1.0) * 3 * H + rng.uniform(0, 0.2 * H, 3)
        centre.append(len(x))
        x += [at, *(at + s * H * o)]
    return np.array(x).astype(np.float32), np.array(centre), H, mass


@pytest.mark.parametrize("r", [0.01, 0.025])
def test_terms_where_the_deviation_cancels(r):
    x, centre, H, mass = _clusters(r, seed=int(1000 * r))
    d = DFSPHCUDA(Scene(config=Configuration(particleRadius=r), fluid=x, boundary=np.zeros((0, 3), np.float32)),
                  grid_box=(0, 0, 0) + (27 * H,) * 3)
    d.neighbors_search()
    d.divergence_solve(0, 1e9)
    got = d.field("density", np.float64) - 1000.0
    ends = np.append(centre[1:], len(x))
    L = np.longdouble
    pi = L("3.14159265358979323846264338327950288")
    for c, e in zip(centre, ends):
        n = e - c - 1
        o = x[c] - x[c + 1:e]  # in FP32, as the device forms them
        q = np.sqrt((o.astype(L) ** 2).sum(1)) / L(H)
        exact = L(mass) * (L(8) / (pi * L(H) ** 3)) * (1 + _w(q).sum()) - L(1000)
        assert abs(exact) < 0.01  # the cancellation is there
        # FP32 storage; n + 1 additions and the read-back at 1000 (half an ulp is 2^-44); terms of 20 ulp
        bound = abs(exact) * 2.0 ** -24 + (n + 2) * 2.0 ** -44 + 20 * 2.0 ** -53 * 750
        assert abs(got[c] - exact) <= bound, (n, float(exact), float(got[c] - exact), float(bound))
