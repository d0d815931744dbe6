"""The event generator against its definition in FP64 numpy (Philox4x32-10 at
counter (candidate, draw), the candidate steps of the source file): the same
candidates accepted, in the same order, at one event, around the 1024
candidates of a block and over several passes, for every region kind, with
masking and additive regions, counting detected events and emissions.

Tolerance: the responses are the FP64 values rounded to float (relative 6e-8);
numpy's sine, cosine, tangent and logarithm differ from the device's by a few
units of FP64, which moves a rounding in rare cases: 2e-7 of the largest
coordinate.  Which candidates are accepted is exact."""
import math

import numpy as np
import pytest

from jpet_strip import capi

pytestmark = pytest.mark.gpu

R, L, SZ, SDL = 450.0, 1000.0, 10.0, 42.0
E, B, P = capi.REGION_ELLIPSE, capi.REGION_RECTANGLE, capi.REGION_POINT
REGIONS = {
    "ellipses": [(E, 30.0, -20.0, 5.0, 90.0, 30.0, 3.0), (E, 0.0, 0.0, 300.0, 250.0, 0.0, 1.0),
                 (E, -50.0, 10.0, 400.0, 380.0, 75.0, 0.5)],
    "mixed": [(P, 10.0, 5.0, 0.0, 0.0, 0.0, 4000.0), (B, 0.0, 0.0, 60.0, 40.0, 0.0, 1.0),
              (P, 10.0, 5.0, 0.0, 0.0, 0.0, 2000.0), (E, 20.0, 0.0, 150.0, 100.0, 10.0, 0.3)],
    "wide": [(B, 100.0, 0.0, 480.0, 440.0, 0.0, 1.0)],
}


def _philox(i, draw, seed):
    mask = np.uint64(0xFFFFFFFF)
    x = [i & mask, i >> np.uint64(32), np.full_like(i, draw), np.zeros_like(i)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        a, b = x[0] * np.uint64(0xD2511F53), x[2] * np.uint64(0xCD9E8D57)
        x = [(b >> np.uint64(32)) ^ x[1] ^ np.uint64(k0), b & mask,
             (a >> np.uint64(32)) ^ x[3] ^ np.uint64(k1), a & mask]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return x


def _u53(a, b):
    return ((a >> np.uint64(5)).astype(np.float64) * 67108864.0 +
            (b >> np.uint64(6)).astype(np.float64)) / 9007199254740992.0


def _reference(regions, n, seed, detected, additive):
    m = 4 * n + 4096
    i = np.arange(m, dtype=np.uint64)
    r = [_philox(i, d, seed) for d in range(4)]
    w = np.array([q[6] * {E: math.pi * q[3] * q[4], B: 4 * q[3] * q[4], P: 1.0}[q[0]]
                  for q in regions])
    k = np.minimum(np.searchsorted(np.cumsum(w) / w.sum(), _u53(r[0][0], r[0][1])),
                   len(regions) - 1)
    u1, u2 = _u53(r[0][2], r[0][3]), _u53(r[1][0], r[1][1])
    x, y = np.empty(m), np.empty(m)
    for j, (kind, cx, cy, a, b, ang, _) in enumerate(regions):
        s = k == j
        sn, cs = math.sin(math.radians(ang)), math.cos(math.radians(ang))
        if kind == E:
            ex = a * np.sqrt(u1[s]) * np.cos(2 * math.pi * u2[s])
            ey = b * np.sqrt(u1[s]) * np.sin(2 * math.pi * u2[s])
            x[s], y[s] = cs * ex - sn * ey + cx, sn * ex + cs * ey + cy
        elif kind == B:
            x[s], y[s] = cx + a * (2 * u1[s] - 1), cy + b * (2 * u2[s] - 1)
        else:
            x[s], y[s] = cx, cy
    emitted = np.ones(m, bool)
    if not additive:
        for j, (kind, cx, cy, a, b, ang, _) in enumerate(regions):
            dx, dy = x - cx, y - cy
            if kind == E:
                sn, cs = math.sin(math.radians(ang)), math.cos(math.radians(ang))
                inside = ((cs * dx + sn * dy) / a) ** 2 + ((cs * dy - sn * dx) / b) ** 2 <= 1
            elif kind == B:
                inside = (np.abs(dx) <= a) & (np.abs(dy) <= b)
            else:
                inside = (dx == 0) & (dy == 0)
            emitted &= ~((k > j) & inside)
    phi_max = math.atan(L / (2 * R)) if detected else math.pi / 2
    t = np.tan(phi_max * (2 * _u53(r[1][2], r[1][3]) - 1))
    zu, zd, dl = x + (R - y) * t, x - (R + y) * t, -2 * y * np.sqrt(t * t + 1)
    ok = emitted & (np.abs(zu) < L / 2) & (np.abs(zd) < L / 2)
    if not detected:
        ok &= np.cumsum(emitted) <= n
    m0 = np.sqrt(-2 * np.log(1 - _u53(r[2][0], r[2][1])))
    m1 = np.sqrt(-2 * np.log(1 - _u53(r[3][0], r[3][1])))
    a0, a1 = 2 * math.pi * _u53(r[2][2], r[2][3]), 2 * math.pi * _u53(r[3][2], r[3][3])
    ev = np.stack([zu + SZ * m0 * np.cos(a0), zd + SZ * m0 * np.sin(a0),
                   dl + SDL * m1 * np.cos(a1)], 1)[ok]
    return ev[:n]


@pytest.mark.parametrize("additive", [False, True])
@pytest.mark.parametrize("detected", [True, False])
@pytest.mark.parametrize("regions", REGIONS)
def test_accepted_candidates_are_the_fp64_definition(regions, detected, additive):
    for n, seed in ((1, 3), (400, 5), (1024, (7 << 32) + 11), (30011, 13)):
        got = capi.generate(REGIONS[regions], n, R, L, SZ, SDL, seed, detected=detected,
                            additive=additive)
        want = _reference(REGIONS[regions], n, seed, detected, additive)
        assert got.shape == want.shape, (n, got.shape, want.shape)
        assert np.max(np.abs(got - want), initial=0.0) <= 2e-7 * np.max(np.abs(want), initial=1.0)
