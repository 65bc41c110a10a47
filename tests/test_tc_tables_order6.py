"""The tensor-core tables with all 48 slots (no GPU needed).  At order 6 the contraction takes three k-steps, for
which no bound by the number of slots keeps the level sums exact: the operator's own digits do, so they are
checked here from the exported tables, independently of the library's own check."""
from fractions import Fraction

import numpy as np
import pytest


def tables(pkg, N):
    lib = pkg.lib()
    dims = np.zeros(4, np.int32)
    assert lib.dg_tc_operator_digits48(N, dims.ctypes.data, None, None, None) == 0
    NUe, NUo, NRe, NRo = (int(x) for x in dims)
    S = np.zeros(NRe * NUe + NRo * NUo)
    fexp = np.zeros(64, np.int32)
    dig = np.zeros(2 * 7 * 48 * 32, np.int32)
    assert lib.dg_tc_operator_digits48(N, dims.ctypes.data, S.ctypes.data, fexp.ctypes.data, dig.ctypes.data) == 0
    return (NUe, NUo, NRe, NRo), S, fexp.reshape(2, 32), dig.reshape(2, 7, 48, 32)


@pytest.mark.parametrize("N", [3, 4, 5, 6])
def test_digits_rebuild_the_operator(pkg, N):
    (NUe, NUo, NRe, NRo), S, fexp, dig = tables(pkg, N)
    assert np.abs(dig).max() <= 255 and max(NUe, NUo) <= 48 and (N < 6) == (max(NUe, NUo) <= 32)
    for p, (K, R, base) in enumerate([(NUe, NRe, 0), (NUo, NRo, NRe * NUe)]):
        B = S[base:base + R * K].reshape(R, K)
        assert not dig[p, :, K:, :].any() and not dig[p, :, :, R:].any()  # padding is zero
        for n in range(R):
            F = int(fexp[p, n]) - 1023
            assert 2.0 ** F <= np.abs(B[n]).max() < 2.0 ** (F + 1)
            for k in range(K):
                d = [int(dig[p, s, k, n]) for s in range(7)]
                exact = Fraction(float(B[n, k])) * Fraction(2) ** (55 - F)
                trunc = int(abs(exact)) * (1 if exact >= 0 else -1)  # toward zero
                assert sum(x * 256 ** (6 - s) for s, x in enumerate(d)) == trunc, (p, n, k)


@pytest.mark.parametrize("N", [3, 4, 5, 6])
def test_level_sums_and_their_joins_stay_exact(pkg, N):
    """Level L sums the products of input digit j and operator digit s with j + s = L.  With input digits up to 255:
    every level below 2^24 (exact in FP32), and the joins 256 lev0 + lev1 and 256 lev3 + lev4 below 2^31 (32-bit
    integers on the device)."""
    (NUe, NUo, NRe, NRo), _, _, dig = tables(pkg, N)
    for p, R in enumerate([NRe, NRo]):
        per_s = np.abs(dig[p].astype(np.int64)).sum(axis=1)  # [s][row]
        lev = 255 * np.cumsum(per_s, axis=0)                 # [L][row]: s = 0..L
        assert lev[:, :R].max() < 2 ** 24
        assert (256 * lev[0] + lev[1]).max() < 2 ** 31 and (256 * lev[3] + lev[4]).max() < 2 ** 31
        if N == 6:
            assert 7 * 48 * 255 ** 2 > 2 ** 24  # by the number of slots alone it would not be


def test_orders_of_the_tables(pkg):
    """48 slots for the orders whose even/odd blocks run on the tensor cores; order 6 does not fit 32."""
    dims = np.zeros(4, np.int32)
    ok = [pkg.lib().dg_tc_operator_digits48(N, dims.ctypes.data, None, None, None) == 0 for N in range(0, 8)]
    assert ok == [False, False, False, True, True, True, True, False]
    assert pkg.lib().dg_tc_operator_digits(6, dims.ctypes.data, None, None, None) != 0
