"""op_timers around OP2 loops: the loops run in stream order without waiting, so the clock itself has to wait
for them, or an application that reads it around loops (src/airfoil.cpp) times their launches only."""
import ctypes as C
import importlib
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_op_timers_cover_the_loops_before_them(pkg):
    o = importlib.import_module(pkg.__name__ + ".op2")
    K, N, loops = 100000, 3, 200  # ~0.2 ms a loop, far more than its launch
    dim = 2 * (N + 1) * (N + 2)
    o.op_init(0)
    cells = o.op_decl_set(K, "cells")
    d = [o.op_decl_dat(cells, dim, "double", np.ones(K * dim), s) for s in ("q", "rk1", "rk2", "rk3", "workingQ")]
    dt = np.array([1e-3])
    args = [o.op_arg_gbl(dt, 1, "double", o.OP_READ)] + [
        o.op_arg_dat(x, -1, None, dim, "double", a)
        for x, a in zip(d, (o.OP_RW, o.OP_READ, o.OP_READ, o.OP_READ, o.OP_WRITE))]
    lib = pkg.lib()
    lib.op_timers.restype, lib.op_timers.argtypes = None, [C.POINTER(C.c_double)] * 2

    def clock():
        c, w = C.c_double(), C.c_double()
        lib.op_timers(C.byref(c), C.byref(w))
        return w.value
    o.op_par_loop_update_Q("update_Q", cells, *args)
    lib.op2_gb300_sync()
    t0, a = time.perf_counter(), clock()
    for _ in range(loops):
        o.op_par_loop_update_Q("update_Q", cells, *args)
    b = clock()
    lib.op2_gb300_sync()
    all_of_it = time.perf_counter() - t0
    o.op_exit()
    assert b - a > 0.8 * all_of_it, (b - a, all_of_it)
