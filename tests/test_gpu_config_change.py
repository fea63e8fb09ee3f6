"""Changing a context's form: raising the precision of a case whose FP64 tiles are
wider than the mixed forms take, and set_config and case_add that run out of
memory at any of their allocations (cfdl_fail_alloc: the allocation is not
made, nothing faults)."""
import ctypes as C

import numpy as np
import pytest

import cfdl

pytestmark = pytest.mark.gpu

OOM = 2
STATE = ("u", "v", "w", "p", "u0", "v0", "w0", "gu", "gv", "gw", "gp", "mip", "mip0")
FIELDS = ("u", "v", "w", "p", "mip")
WIDE = 86        # 636056 cells: above the 622592 from which FP64 flow tiles take more rows per thread


@pytest.mark.parametrize("precision", [1, 2, 3])
def test_precision_raised(need_gpu, precision):
    """FP64 steps first, so that the wide tiles have been in use, then the
    same state and steps as a solver created in the form: the same bits."""
    s = cfdl.Setup(cfdl.Zone(WIDE, jitter=0.1, seed=1))
    cfg = cfdl.steady(mu=0.01, precision=precision)
    a, b = cfdl.Solver(s, cfg), cfdl.Solver(s, cfdl.steady())
    start = {f: b.get(f) for f in STATE}
    b.step(2, 0)
    b.set_config(cfg)
    for f, v in start.items():
        b.set(f, v)
    for g in (a, b):
        g.step(2, 0)
    for f in FIELDS:
        assert np.array_equal(a.get(f), b.get(f)), f


def _pair():
    setups = [cfdl.Setup(cfdl.Zone(n, jitter=0.1, seed=n)) for n in (WIDE, 9)]
    return [cfdl.Batch(setups, [cfdl.steady()] * 2) for _ in range(2)]


def _same(a, b):
    for c in a.ids():
        for f in FIELDS:
            assert np.array_equal(a.case_get(c, f), b.case_get(c, f)), (c, f)


def _until_it_succeeds(call, after, order=range(400)):
    """call() with its n-th allocation failing, n in `order`; after(tries so far)
    follows each failure.  Returns the failures."""
    L = cfdl.lib()
    for failed, n in enumerate(order):
        L.cfdl_fail_alloc(C.c_int(n))
        status = call()
        L.cfdl_fail_alloc(C.c_int(-1))
        if status == 0:
            return failed
        assert status == OOM, (n, status)
        after(failed)
    raise AssertionError("never succeeded")


def test_set_config_out_of_memory(need_gpu):
    """Whatever fails, the old form stands and goes on as if it had not been
    asked for; the call that succeeds gives the new one."""
    a, b = _pair()
    for g in (a, b):
        g.step(1, 0)
    cfg = cfdl.steady(mu=0.02, precision=3)

    def after(n):
        if n in (0, 3, 7):
            for g in (a, b):
                g.step(1, 0)
            _same(a, b)

    L = cfdl.lib()
    # a case keeps its three arrays once it has them: each of the first case's
    # fails, then the second's first and each of them, then the lists
    failed = _until_it_succeeds(lambda: L.cfdl_set_config(b._h, C.byref(cfg)), after, [0, 1, 2, 3] * 2 + [50])
    assert failed == 8
    a.set_config(cfg)
    for g in (a, b):
        g.step(2, 0)
    _same(a, b)


def test_case_add_out_of_memory(need_gpu):
    a, b = _pair()
    extra = cfdl.Setup(cfdl.Zone(5, jitter=0.1, seed=3))
    mesh, cfg, cid = extra.mesh(1.0), cfdl.steady(), C.c_int()
    L = cfdl.lib()

    def after(n):
        assert L.cfdl_case_count(b._h) == 2
        if n % 20 == 0:
            for g in (a, b):
                g.step(1, 0)
            _same(a, b)

    failed = _until_it_succeeds(lambda: L.cfdl_case_add(b._h, C.byref(mesh), C.byref(cfg), C.byref(cid)), after)
    assert failed > 40
    assert L.cfdl_case_count(b._h) == 3
    b.remove(cid.value)
    for g in (a, b):
        g.step(2, 0)
    _same(a, b)


@pytest.mark.parametrize("precision", [0, 1])
def test_hierarchy_out_of_memory(need_gpu, precision):
    """The multigrid hierarchy is built by the first solve: one that runs out of
    memory there leaves none half built for the next."""
    s = cfdl.Setup(cfdl.Zone(24, jitter=0.1, seed=2))
    a, b = (cfdl.Solver(s, cfdl.steady(precision=precision)) for _ in range(2))
    L = cfdl.lib()
    failed = _until_it_succeeds(lambda: L.cfdl_step(b._h, 1, 0, None), lambda n: None)
    assert failed > 30
    a.step(1, 0)
    for g in (a, b):
        g.step(1, 0)
    for f in FIELDS:
        assert np.array_equal(a.get(f), b.get(f)), f


@pytest.mark.parametrize("precision", [1, 2, 3])
def test_case_added_without_multigrid(need_gpu, precision):
    """The 16-bit offsets come with the multigrid set-up: a case added after the
    preconditioner was changed has none, so its context goes without them."""
    s, t = (cfdl.Setup(cfdl.Zone(n, jitter=0.1, seed=n)) for n in (12, 7))
    jac = cfdl.steady(precision=precision, precond=0)
    a = cfdl.Batch([s], [cfdl.steady(precision=precision)])
    b = cfdl.Batch([s, t], [jac, jac])
    start = {f: a.case_get(0, f) for f in STATE}
    a.step(1, 0)
    assert a.index_bytes() == 2
    a.set_config(jac)
    assert a.add(t, jac) == 1
    for f, v in start.items():
        a.case_set(0, f, v)
    for g in (a, b):
        g.step(2, 0)
    _same(a, b)
