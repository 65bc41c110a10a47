"""The face kernels' two forms of the Roe flux: pairs of floats for the dissipation where the jump is
small, FP64 elsewhere (csrc/dg_roe_ff.cuh)."""
import ctypes as C

import numpy as np
import pytest

from conftest import push_affine_geometry

GAM = 1.4


def _pair(pkg, qm, qp, nrm, gam=GAM):
    f = pkg.lib().dg_roe_pair_flux
    dp = C.POINTER(C.c_double)
    f.restype, f.argtypes = C.c_int, [C.c_double, C.c_int, dp, dp, dp, C.POINTER(C.c_int), dp]
    a = [np.ascontiguousarray(v, dtype=np.float64) for v in (qm, qp, nrm)]
    n = len(a[0])
    taken, out = np.zeros(n, dtype=np.int32), np.zeros((n, 4))
    rc = f(gam, n, *[v.ctypes.data_as(dp) for v in a], taken.ctypes.data_as(C.POINTER(C.c_int)), out.ctypes.data_as(dp))
    assert rc == 0
    return taken.astype(bool), out


def _long(qm, qp, nrm, gam=GAM):
    """Twice the Roe flux (src/euler_rhs.h:120-220) and its scale in extended precision."""
    L = np.longdouble
    q, p, n = (np.asarray(v, dtype=L) for v in (qm, qp, nrm))
    g1 = L(gam - 1.0)
    nx, ny = n[:, 0], n[:, 1]

    def side(s):
        m, t = nx * s[:, 1] + ny * s[:, 2], nx * s[:, 2] - ny * s[:, 1]
        u, v = m / s[:, 0], t / s[:, 0]
        return m, t, u, v, g1 * (s[:, 3] - (m * u + t * v) / 2)
    mL, tL, uL, vL, pL = side(q)
    mR, tR, uR, vR, pR = side(p)
    sL, sR = np.sqrt(q[:, 0]), np.sqrt(p[:, 0])
    rho, w = sL * sR, sL + sR
    u, v = (sL * uL + sR * uR) / w, (sL * vL + sR * vR) / w
    H = ((q[:, 3] + pL) / sL + (p[:, 3] + pR) / sR) / w
    c2 = g1 * (H - (u * u + v * v) / 2)
    c = np.sqrt(c2)
    a, b = (pR - pL) / c2 / 2, rho * (uR - uL) / c / 2
    w1, w4 = abs(u - c) * (a - b), abs(u + c) * (a + b)
    w2, w3 = abs(u) * ((p[:, 0] - q[:, 0]) - 2 * a), abs(u) * rho * (vR - vL)
    d = (w1 + w2 + w4, w1 * (u - c) + w2 * u + w4 * (u + c), (w1 + w2 + w4) * v + w3,
         w1 * (H - u * c) + w4 * (H + u * c) + w2 * (u * u + v * v) + w3 * v)
    g = (mL + mR - d[0], mL * uL + pL + mR * uR + pR - d[1], tL * uL + tR * uR - d[2],
         uL * (q[:, 3] + pL) + uR * (p[:, 3] + pR) - d[3])
    s = abs(u) + abs(v) + c
    scale = np.stack([rho * s, rho * s * s, rho * s * s, rho * s * H], 1)
    return np.stack([g[0], nx * g[1] - ny * g[2], ny * g[1] + nx * g[2], g[3]], 1), scale


def _states(rng, n, jump, R=1.0, S=1.0, mach=0.8):
    """Pairs of states with relative jumps up to `jump`, density scale R, pressure scale S."""
    rho, p, th, ph = (rng.uniform(a, b, n) for a, b in ((0.5, 2), (0.5, 2), (0, 2 * np.pi), (0, 2 * np.pi)))
    sp = rng.uniform(0, mach, n) * np.sqrt(GAM * p / rho)
    u, v = sp * np.cos(th), sp * np.sin(th)
    u[::5], v[::7] = 0.0, 0.0
    a = np.sqrt(S / R)
    qm = np.stack([R * rho, R * a * rho * u, R * a * rho * v, S * (p / (GAM - 1) + 0.5 * rho * (u * u + v * v))], 1)
    e = rng.uniform(-1, 1, (n, 4)) * jump
    ms = 0.7 * np.sqrt(qm[:, 0] * qm[:, 3])
    qp = qm + e * np.stack([qm[:, 0], ms, ms, qm[:, 3]], 1)
    return qm, qp, np.stack([np.cos(ph), np.sin(ph)], 1)


@pytest.mark.parametrize("jump", [0.0, 1e-14, 1e-6, 1e-3, 3.9e-3])
@pytest.mark.parametrize("R,S", [(1.0, 1.0), (1.2, 1e5), (1e3, 1e-6)])
def test_small_jump_flux_is_fp64_accurate(pkg, jump, R, S):
    """Every component within 16 units of 2^-53 of the flux's scale: a dozen FP64 roundings of the
    central flux, and a dissipation of at most 2^-8 of that scale known to about 2^-43 (ten pair
    operations of 2^-46 each), 2^-51 together."""
    qm, qp, nrm = _states(np.random.default_rng(7), 4000, jump, R, S)
    taken, f = _pair(pkg, qm, qp, nrm)
    # at 3.9e-3 the jump of some pairs, relative to the smaller side, is beyond the rule's 2^-8
    assert taken.all() if jump <= 1e-3 else taken.mean() > 0.9
    want, scale = _long(qm, qp, nrm)
    assert float((abs(f - want) / scale)[taken].max()) < 16 * 2.0 ** -53


def test_small_jump_rule_refuses_the_rest(pkg):
    """Strong jumps, high Mach numbers, non-finite or non-physical states and extreme scales take
    the general form."""
    rng = np.random.default_rng(3)
    qm, _, nrm = _states(rng, 64, 0.0)
    assert _pair(pkg, qm, qm, nrm)[0].all()
    for k in (0, 1, 2, 3):
        for bad in (np.nan, np.inf, -np.inf, 1e300):
            for side in (0, 1):
                s = [qm.copy(), qm.copy()]
                s[side][:, k] = bad
                assert not _pair(pkg, s[0], s[1], nrm)[0].any()
    for k in (0, 3):
        for bad in (0.0, -1.0, 5e-324):
            q = qm.copy()
            q[:, k] = bad
            assert not _pair(pkg, q, q, nrm)[0].any()
    for f in (2.0 ** -40, 2.0 ** 40):  # a scaled gas: the rule keeps to 2^-30 .. 2^30
        assert not _pair(pkg, qm * f, qm * f, nrm)[0].any()
    q = qm.copy()
    q[:, 0] *= 1.01
    assert not _pair(pkg, qm, q, nrm)[0].any()
    q = qm.copy()
    q[:, 1] = 3.0 * np.sqrt(qm[:, 0] * qm[:, 3])
    assert not _pair(pkg, q, q, nrm)[0].any()


@pytest.mark.gpu
@pytest.mark.parametrize("jump", [0.0, 1e-6, 1e-3, 6e-3, 0.3])
@pytest.mark.parametrize("N", [1, 3, 6])
def test_rhs_across_the_rule_matches_oracle(pkg, orc, oops, omesh, N, jump):
    """One right-hand side of states whose jumps lie below, around and above the rule's line, both
    forms in one warp among them (1e-13, as the other right-hand-side tests)."""
    m = omesh.naca_ogrid(33, 7, farfield="characteristic")
    s = pkg.Solver(pkg.Mesh.from_tables(m), pkg.config(N=N, cfl=0.5)).init()
    o = orc.Oracle(m, oops.operators(N), orc.freestream(0.4, 0.0), kind="port")
    o.init(0.5)
    push_affine_geometry(o, s.get("geo").reshape(-1, 16))
    q = o.get("q")
    rng = np.random.default_rng(N)
    q = q * (1.0 + 0.01 * np.sin(np.arange(q.size) // (2 * (N + 1) * (N + 2))))  # cell to cell
    W = q * (1.0 + jump * rng.uniform(-0.5, 0.5, q.size))
    o.set("workingQ", W)
    assert orc.rel_l2(s.rhs(W), o.rhs(0)) < 1e-13
