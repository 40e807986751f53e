"""The serving loop (fmmlib3d_b200.serving): requests in a mix equal requests alone.

Requests of both kernels, several sizes, iprec values and geometries are
submitted together to a server with four slots (their kernels overlap on the
GPU), then one at a time; every result must be bitwise identical, and equal
to the plain C-ABI call.  A budget smaller than any request forces one
request at a time.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _requests(count, seed):
    from fmmlib3d_b200.serving import Request
    rng = np.random.default_rng(seed)
    out = []
    for i in range(count):
        n = int(10 ** rng.uniform(3, 4.5))
        src = rng.random((n, 3)) if i % 2 else rng.normal(size=(n, 3)) * 0.2
        q = rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n)
        helm = i % 3 == 0
        out.append(Request("helmholtz" if helm else "laplace", src, q, iprec=int(rng.integers(0, 3)),
                           zk=float(rng.uniform(1, 20)) if helm else 0.0, tag=i))
    return out


def test_results_equal_alone_and_in_the_mix():
    from fmmlib3d_b200.serving import FMMServer, run_stream
    import fmmlib3d_b200 as F
    reqs = _requests(12, 3)
    srv = FMMServer(slots=4)
    try:
        stats, mixed = run_stream(srv, reqs, float("inf"))
    finally:
        srv.close()
    assert stats["max_ier"] == 0 and srv.max_running > 1
    srv1 = FMMServer(slots=1)
    try:
        alone = [srv1.submit(r).result() for r in reqs]
    finally:
        srv1.close()
    for r, a, b in zip(reqs, mixed, alone):
        assert a.tag == b.tag == r.tag
        assert np.array_equal(a.pot, b.pot) and np.array_equal(a.fld, b.fld)
        if r.kernel == "laplace":
            ier, pot, fld, _, _ = F.lfmm3dparttarg(r.iprec, r.source, 1, r.charge, 0, None, None, 1, 1)
        else:
            ier, pot, fld, _, _ = F.hfmm3dparttarg(r.iprec, r.zk, r.source, 1, r.charge, 0, None, None, 1, 1)
        assert ier == 0 and np.array_equal(a.pot, pot) and np.array_equal(a.fld, fld)


def test_budget_limits_concurrency():
    from fmmlib3d_b200.serving import FMMServer, run_stream
    reqs = _requests(6, 4)
    srv = FMMServer(slots=4, hbm_budget_bytes=1)
    try:
        stats, _ = run_stream(srv, reqs, float("inf"))
    finally:
        srv.close()
    assert stats["max_ier"] == 0 and srv.max_running == 1


def test_precision_per_request():
    """A server in the mixed form (and requests that override it) gives every request the bits of a
    single call in that request's form; the process-wide setting is left as it was."""
    from fmmlib3d_b200.serving import FMMServer, run_stream
    import fmmlib3d_b200 as F
    reqs = _requests(10, 5)
    for i, r in enumerate(reqs):
        if r.kernel == "laplace" and i % 4 == 1:
            r.precision = 0
    srv = FMMServer(slots=4, precision=1)
    try:
        stats, res = run_stream(srv, reqs, float("inf"))
    finally:
        srv.close()
    assert stats["max_ier"] == 0
    for r, a in zip(reqs, res):
        form = 1 if r.precision is None else r.precision
        if r.kernel == "laplace":
            F.set_precision(form)
            try:
                ier, pot, fld, _, _ = F.lfmm3dparttarg(r.iprec, r.source, 1, r.charge, 0, None, None, 1, 1)
            finally:
                F.set_precision(0)
        else:
            ier, pot, fld, _, _ = F.hfmm3dparttarg(r.iprec, r.zk, r.source, 1, r.charge, 0, None, None, 1, 1)
        assert ier == 0 and np.array_equal(a.pot, pot) and np.array_equal(a.fld, fld), (r.tag, r.kernel, r.iprec)
    with pytest.raises(ValueError):
        F.set_precision_thread(2)


def test_repeated_geometries_run_on_resident_plans():
    """Laplace requests naming a repeated geometry run on a plan kept on the device: after the
    first request of each geometry no tree is rebuilt (plan hits), every result carries the bits of
    a plain call, and a plan budget smaller than two plans evicts the least recently used one and
    still gives the same bits."""
    from fmmlib3d_b200.serving import FMMServer, Request, run_stream
    import fmmlib3d_b200 as F
    rng = np.random.default_rng(9)
    geoms = [(rng.random((20000, 3)), 1), (rng.normal(size=(8000, 3)) * 0.3, 0), (rng.random((3000, 3)), 2)]
    reqs = []
    for i in range(18):
        g = i % 3
        src, iprec = geoms[g]
        q = rng.uniform(-1, 1, len(src)) + 1j * rng.uniform(-1, 1, len(src))
        reqs.append(Request("laplace", src, q, iprec=iprec, tag=i, geometry=g))
    want = []
    for r in reqs:
        ier, pot, fld, _, _ = F.lfmm3dparttarg(r.iprec, r.source, 1, r.charge, 0, None, None, 1, 1)
        assert ier == 0
        want.append((pot, fld))
    for plan_bytes in (None, 1):
        srv = FMMServer(slots=4, plan_bytes=plan_bytes)
        try:
            stats, res = run_stream(srv, reqs, float("inf"))
            st = srv.stats()
        finally:
            srv.close()
        assert stats["max_ier"] == 0
        for r, a, (pot, fld) in zip(reqs, res, want):
            assert a.tag == r.tag
            assert np.array_equal(a.pot, pot) and np.array_equal(a.fld, fld)
        if plan_bytes is None:
            assert st["plans_built"] == 3 and st["plan_hits"] == 15 and st["plans_evicted"] == 0
        else:
            assert st["plans_evicted"] >= 1


def _pool(attr):
    """An attribute of the device's default memory pool (the pool the library allocates from), in bytes."""
    from cuda.bindings import driver as drv
    assert drv.cuInit(0)[0] == drv.CUresult.CUDA_SUCCESS
    err, pool = drv.cuDeviceGetDefaultMemPool(0)
    assert err == drv.CUresult.CUDA_SUCCESS
    a = getattr(drv.CUmemPool_attribute, "CU_MEMPOOL_ATTR_USED_MEM_" + attr)
    err, v = drv.cuMemPoolGetAttribute(pool, a)
    assert err == drv.CUresult.CUDA_SUCCESS
    if attr == "HIGH":   # and back to the current use
        assert drv.cuMemPoolSetAttribute(pool, a, drv.cuuint64_t(0))[0] == drv.CUresult.CUDA_SUCCESS
    return int(v)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("shape,n,iprec", [("sphere", 10000, 1), ("cube", 100000, 1), ("plummer", 100000, 2),
                                           ("sphere", 1000000, 0), ("cube", 20000, 3)])
def test_admission_covers_what_plans_hold_and_calls_take(shape, n, iprec, precision):
    """The library's count of a plan's memory is what the pool has handed out for it, plan_bytes
    covers it and the server's own buffers, and the projection of a request covers the peak of its
    call.  The pool rounds each of a plan's fewer than 100 allocations up, by less than 512 bytes."""
    import torch
    import fmmlib3d_b200 as F
    from fmmlib3d_b200.serving import Request, plan_bytes, projected_bytes
    rng = np.random.default_rng(n + iprec)
    src = rng.random((n, 3)) if shape == "cube" else rng.normal(size=(n, 3))
    if shape != "cube":
        src /= np.linalg.norm(src, axis=1)[:, None]
    if shape == "plummer":
        src *= (0.1 / np.sqrt(np.maximum(rng.random(n), 1e-9) ** (-2 / 3) - 1)).clip(0, 1)[:, None]
    d_src = torch.from_numpy(src).cuda()
    q = torch.ones((n, 2), dtype=torch.float64, device="cuda")
    pot, fld = torch.empty((n, 2), dtype=torch.float64, device="cuda"), torch.empty((n, 6), dtype=torch.float64,
                                                                                    device="cuda")
    torch.cuda.synchronize()
    F.set_precision(precision)
    try:
        F.LaplacePlan(iprec, d_src, 1, 0, 1, 1).close()    # the order's tables
        torch.cuda.synchronize()
        before = _pool("CURRENT")
        plan = F.LaplacePlan(iprec, d_src, 1, 0, 1, 1)
        torch.cuda.synchronize()
        held, info = _pool("CURRENT") - before, plan.info()
        plan.close()
        torch.cuda.synchronize()
        _pool("HIGH")
        base = _pool("HIGH")
        assert F.lfmm3dparttarg_device(iprec, d_src, q, None, None, pot, fld) == 0
        torch.cuda.synchronize()
        peak = _pool("HIGH") - base
    finally:
        F.set_precision(0)
    arrays = n * (24 + 16 + 64)
    assert info["bytes"] <= held < info["bytes"] + 100 * 512
    assert plan_bytes(info) >= held + arrays - 100 * 512
    assert projected_bytes(Request("laplace", src, None, iprec=iprec)) >= peak + arrays
