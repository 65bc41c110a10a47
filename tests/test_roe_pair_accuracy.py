"""The face kernels' two forms of the Roe flux (csrc/dg_roe_ff.cuh) against extended precision: the pair form's
error, component by component, is no larger than the general FP64 form's, whatever gamma, Mach number and jump
the rule accepts."""
import ctypes as C

import numpy as np
import pytest

from test_roe_pair import _long, _pair

dp = C.POINTER(C.c_double)


def _states(rng, n, jump, gam, mach):
    """Pairs of states with jumps up to `jump` of rho, E and the momentum's measure in the rule."""
    rho, p, th, ph = (rng.uniform(a, b, n) for a, b in ((0.5, 2), (0.5, 2), (0, 2 * np.pi), (0, 2 * np.pi)))
    sp = rng.uniform(0, mach, n) * np.sqrt(gam * p / rho)
    u, v = sp * np.cos(th), sp * np.sin(th)
    u[::5], v[::7] = 0.0, 0.0
    qm = np.stack([rho, rho * u, rho * v, p / (gam - 1) + 0.5 * rho * (u * u + v * v)], 1)
    ms = 0.7 * np.sqrt(min(1.0, 2.5 * (gam - 1)) * qm[:, 0] * qm[:, 3])
    qp = qm + rng.uniform(-1, 1, (n, 4)) * jump * np.stack([qm[:, 0], ms, ms, qm[:, 3]], 1)
    return qm, qp, np.stack([np.cos(ph), np.sin(ph)], 1)


@pytest.mark.parametrize("jump", [1e-3, 3.9e-3])
@pytest.mark.parametrize("gam", [1.001, 1.1, 1.4, 5.0 / 3.0])
def test_pair_bound_at_every_gamma(pkg, gam, jump):
    """16 units of 2^-53 of the flux's scale, the bound of the gamma = 1.4 test, for whatever the rule accepts:
    the jumps here are relative to sqrt(rho E), so that the rule has to refuse most of them as gamma nears 1."""
    rng = np.random.default_rng(11)
    qm, qp, nrm = _states(rng, 20000, jump, gam, 1.9)
    ms = 0.7 * np.sqrt(qm[:, 0] * qm[:, 3])
    qp[::2, 1:3] = (qm[:, 1:3] + rng.uniform(-1, 1, (len(qm), 2)) * jump * ms[:, None])[::2]
    taken, f = _pair(pkg, qm, qp, nrm, gam)
    assert taken.mean() > 0.3
    want, scale = _long(qm, qp, nrm, gam)
    assert float((abs(f - want) / scale)[taken].max()) < 16 * 2.0 ** -53


@pytest.mark.gpu
@pytest.mark.parametrize("mach", [0.1, 0.8, 1.9])
@pytest.mark.parametrize("jump", [1e-8, 1e-3, 3.9e-3])
@pytest.mark.parametrize("gam", [1.001, 1.1, 1.4, 5.0 / 3.0])
def test_pair_error_on_the_device_is_no_larger(pkg, gam, jump, mach):
    """Root mean square over the pairs that the rule takes, of each component's error relative to the flux's
    scale, both forms as the device computes them."""
    qm, qp, nrm = (np.ascontiguousarray(a) for a in _states(np.random.default_rng(5), 30000, jump, gam, mach))
    taken = _pair(pkg, qm, qp, nrm, gam)[0]
    assert taken.mean() > 0.3
    g = pkg.lib().dg_roe_flux_nodes
    g.restype, g.argtypes = C.c_int, [C.c_double, C.c_int, C.c_int, dp, dp, dp, dp]
    want, scale = _long(qm, qp, nrm, gam)
    rms, peak = [], []
    for form in (0, 1):
        f = np.zeros((len(qm), 4))
        assert g(gam, form, len(qm), *[a.ctypes.data_as(dp) for a in (qm, qp, nrm, f)]) == 0
        e = (abs(f - want) / scale)[taken].astype(np.float64)
        rms.append(np.sqrt((e * e).mean(axis=0)))
        peak.append(float(e.max()))
    assert (rms[1] <= rms[0]).all(), (rms[0] * 2 ** 53, rms[1] * 2 ** 53)
    assert peak[1] < 16 * 2.0 ** -53
