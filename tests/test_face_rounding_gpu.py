"""Rounding of the faces' mass flux. Quotients that share a divisor are products
with one reciprocal and a correction (face.cuh: quotient), which is to cost no
accuracy against dividing: the density's residual with AUSM+ is compared with
extended precision (x87 long double, 11 bits more), and its error must not exceed
that of the same formulas in FP64 with divisions.

The error is a 2-norm over some ten thousand cells. Against the FP64 evaluation
below it is 0.97 of that without species and 1.00 with nine, with divisions as
with corrected products, and 1.02 and 1.19 with products alone; the bound lies
between."""
import numpy as np
import pytest

import ostc

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(np.finfo(np.longdouble).nmant < 63, reason="no extended precision")]


def density_residual(case, bv, sv, dt):
    """dq of the density: MUSCL (minmod) and AUSM+ over the three directions, in type dt"""
    b = case.blocks[0]
    g, n = b.ngg, (b.mz, b.my, b.mx)
    bv, sv = bv.astype(dt), sv.astype(dt)
    jac = b.arrays["jac"].astype(dt)
    met = np.moveaxis(b.arrays["metric"].view(ostc.METRIC_DTYPE).reshape(bv.shape[1:])["m"], -1, 0).astype(dt)
    ns = sv.shape[0]
    if ns:
        t = {k: np.asarray(v).astype(dt) for k, v in case.mech.tables.items() if v.dtype == np.float64}
        R = dt(ostc.R_U) / t["mw"]

    def sound2(w):  # gamma p / rho
        if not ns:
            return dt(1.4) * (w[4] / w[0])
        Rm = np.tensordot(R, w[5:], 1)
        T = w[4] / w[0] / Rm
        cp = 0
        for l in range(ns):
            lo, hi = t["low_temp_coeff"][l], t["high_temp_coeff"][l]
            tt = np.maximum(T, t["t_low"][l])
            k = [np.where(tt < t["t_mid"][l], lo[c], hi[c]) for c in range(5)]
            cp = cp + w[5 + l] * R[l] * (k[0] + tt * (k[1] + tt * (k[2] + tt * (k[3] + tt * k[4]))))
        return cp / (cp - Rm) * (w[4] / w[0])

    def minmod(a, c):
        return np.where((a < 0) != (c < 0), dt(0), np.where(np.abs(a) < np.abs(c), a, c))

    v = np.concatenate([bv[:5], sv])
    out = np.zeros(n, dt)
    for face in range(3):
        ax = 2 - face

        def at(a, m):  # the faces' cells: faces -1/2 .. n - 1/2 along ax, offset m
            ix = [slice(g, g + n[x]) for x in range(3)]
            ix[ax] = slice(g - 1 + m, g + n[ax] + m)
            return a[(Ellipsis,) + tuple(ix)]

        d0, d1, d2 = at(v, 0) - at(v, -1), at(v, 1) - at(v, 0), at(v, 2) - at(v, 1)
        l, r = at(v, 0) + dt(0.5) * minmod(d0, d1), at(v, 1) - dt(0.5) * minmod(d1, d2)
        k = met[3 * face:3 * face + 3]
        k = dt(0.5) * (at(jac, 0) * at(k, 0) + at(jac, 1) * at(k, 1))
        gk = np.sqrt((k * k).sum(0))
        c = dt(0.5) * (np.sqrt(sound2(l)) + np.sqrt(sound2(r)))
        mh = 0
        for s, w in ((1, l), (-1, r)):
            m = s * ((k * w[1:4]).sum(0) / gk / c)
            sub = dt(0.25) * (m + 1) * (m + 1) + dt(0.125) * (m * m - 1) * (m * m - 1)
            mh = mh + s * np.where(np.abs(m) > 1, dt(0.5) * (m + np.abs(m)), sub)
        F = c * (l[0] * (dt(0.5) * (mh + np.abs(mh))) + r[0] * (dt(0.5) * (mh - np.abs(mh)))) * gk
        hi, lo = [slice(None)] * 3, [slice(None)] * 3
        hi[ax], lo[ax] = slice(1, None), slice(0, -1)
        out -= F[tuple(hi)] - F[tuple(lo)]
    return out


def noisy(ns):
    """a workload with 1 % noise on its velocities, pressure and temperature, and a little of every species"""
    c = ostc.case_mixing_layer(31, 37, 11) if ns else ostc.case_vortex(41, 33, 10, reconstruction=2, inviscid_scheme=3)
    bv, sv = c.blocks[0].arrays["bv"], c.blocks[0].arrays["sv"]
    rng = np.random.default_rng(1)
    bv[1:4] += 0.01 * np.abs(bv[1:4]).max() * (2 * rng.random(bv[1:4].shape) - 1)
    ft, fp = 1 + 0.01 * (2 * rng.random((2,) + bv.shape[1:]) - 1)
    bv[5] *= ft
    bv[4] *= fp
    bv[0] *= fp / ft
    if ns:
        imw = 1.0 / c.mech.tables["mw"]
        before = np.tensordot(imw, sv, 1)
        sv += 2e-4 * rng.random(sv.shape)
        sv /= sv.sum(0)
        bv[0] *= before / np.tensordot(imw, sv, 1)
    return c


@pytest.mark.parametrize("ns", [0, 9])
def test_mass_flux_is_as_accurate_as_with_divisions(ns):
    case = noisy(ns)
    s, blocks = case.solver()
    s.initialize()
    s.compute_rhs()
    bv, sv = blocks[0].download("bv"), blocks[0].download("sv") if ns else np.zeros((0,) + case.blocks[0].arrays["bv"].shape[1:])
    true = density_residual(case, bv, sv, np.longdouble)
    got, plain = (np.linalg.norm((a - true).astype(np.float64).ravel())
                  for a in (blocks[0].download("dq")[0].astype(np.longdouble), density_residual(case, bv, sv, np.float64)))
    assert got <= 1.01 * plain, got / plain
    s.close()
