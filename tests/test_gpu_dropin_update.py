"""The drop-in's update_Q (src/update_Q.h) on values over the whole range of doubles: its quotients by 6
and 3 must be the correctly rounded ones, signs of zero, subnormals and non-finite values included."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,N", [(1, 3), (37, 3), (4001, 4)])
def test_update_q_bit_exact(pkg, K, N):
    o = importlib.import_module(pkg.__name__ + ".op2")
    n = K * 2 * (N + 1) * (N + 2)
    rng = np.random.default_rng(K)
    bits = rng.integers(0, 1 << 63, (3, n), dtype=np.int64) ^ (rng.integers(0, 2, (3, n), dtype=np.int64) << 63)
    k = bits.view(np.float64).copy()  # any exponent, with infinities and NaN among them
    k[:, ::3] = rng.standard_normal((3, n))[:, ::3] * 10.0 ** rng.integers(-6, 7, (3, n))[:, ::3]
    special = [0.0, -0.0, 5e-324, -5e-324, 2.0 ** -1022, 2.0 ** -1023, 1.7976931348623157e308, np.inf, -np.inf, np.nan,
               3.0, 6.0, 1.0, -1.0, 2.0 ** 53 - 1, 1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52]
    k[:, 1:1 + len(special)] = special
    q0 = rng.standard_normal(n)
    q0[1:1 + len(special)] = -0.0
    dt = np.array([1.0])
    o.op_init(0)
    cells = o.op_decl_set(K, "cells")
    dim = 2 * (N + 1) * (N + 2)
    d = [o.op_decl_dat(cells, dim, "double", v, s) for v, s in ((q0, "q"), (k[0], "rk1"), (k[1], "rk2"), (k[2], "rk3"),
                                                               (q0, "workingQ"))]
    acc = (o.OP_RW, o.OP_READ, o.OP_READ, o.OP_READ, o.OP_WRITE)
    o.op_par_loop_update_Q("update_Q", cells, o.op_arg_gbl(dt, 1, "double", o.OP_READ),
                           *[o.op_arg_dat(x, -1, None, dim, "double", a) for x, a in zip(d, acc)])
    out = np.empty(n)
    o.op_fetch_data(d[0], out)
    o.op_exit()
    with np.errstate(all="ignore"):
        want = q0 + dt[0] * (k[0] / 6.0 + k[1] / 6.0 + 2.0 * k[2] / 3.0)
    ok = (out.view(np.int64) == want.view(np.int64)) | (np.isnan(out) & np.isnan(want))
    assert ok.all()
