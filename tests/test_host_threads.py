"""The reduced system's analysis and its threads: where no thread can be
started it runs on the caller's, and where they can their number is bounded
by the cores, not by the grid.  The order, and with it every bit of a
solution, does not depend on them."""
import ctypes as C
import os
import threading

import numpy as np
import pytest

from helpers import LY, synthetic
from test_host import _reduced_S, lib  # noqa: F401 (the library fixture)


def selftest(lib, n_bus, n_gen):
    w = synthetic._planar("planar", 11, n_bus, n_gen, 0.55, 1, 1.0, "random")
    PA = LY.ProblemArrays(w.ps)
    P = PA.as_ctypes()
    S = _reduced_S(w.ps, np.random.default_rng(n_bus))
    rhs = np.random.default_rng(1).normal(size=S.shape[0])
    x, out = np.zeros_like(rhs), np.zeros(12)
    rp, ci, sv = S.indptr.astype(np.int32), S.indices.astype(np.int32), S.data.astype(np.float64)
    lib.gp_reduced_selftest.argtypes = [C.c_void_p] * 7

    def run():
        rc = lib.gp_reduced_selftest(C.addressof(P), rp.ctypes.data, ci.ctypes.data, sv.ctypes.data, rhs.ctypes.data,
                                     x.ctypes.data, out.ctypes.data)
        return rc, x.copy()
    run.keep = PA   # P points into it
    return run


def test_analysis_where_no_thread_starts(lib):  # noqa: F811
    """A default stack larger than the address space: every thread creation
    of the process fails (EAGAIN), as at a container's process limit."""
    run = selftest(lib, 1999, 150)
    rc, x0 = run()
    assert rc == 0
    c = C.CDLL(None)
    if not hasattr(c, "pthread_setattr_default_np"):
        pytest.skip("no way to set the default stack")
    c.pthread_attr_setstacksize.argtypes = [C.c_void_p, C.c_size_t]
    attr, was = (C.c_char * 128)(), (C.c_char * 128)()
    assert c.pthread_getattr_default_np(was) == 0
    assert c.pthread_attr_init(attr) == 0
    assert c.pthread_attr_setstacksize(attr, 1 << 56) == 0 and c.pthread_setattr_default_np(attr) == 0
    try:
        with pytest.raises(RuntimeError):
            threading.Thread(target=lambda: None).start()
        rc, x1 = run()
    finally:
        assert c.pthread_setattr_default_np(was) == 0
    assert rc == 0 and np.array_equal(x0, x1)


def test_analysis_threads_bounded_by_cores(lib):  # noqa: F811
    run = selftest(lib, 30000, 2000)

    def threads():
        with open("/proc/self/status") as f:
            return int(next(line for line in f if line.startswith("Threads")).split()[1])
    peak, stop = [0], threading.Event()

    def watch():
        while not stop.is_set():
            peak[0] = max(peak[0], threads())
    t = threading.Thread(target=watch)
    t.start()
    base = threads()
    try:
        rc, _ = run()
    finally:
        stop.set()
        t.join()
    # (two a core at once; a joined one may still be listed for a moment)
    assert rc == 0 and peak[0] - base <= 3 * os.cpu_count()
