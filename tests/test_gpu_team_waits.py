"""Limits of the persistent kernels' waits: a CTA that has come to a system waits
for those of its team that are still in another one, however long that takes; a
wait within a system ends with a timeout, and the next solve is right."""
import numpy as np
import pytest

import wgpu_solver_backend_b200 as wsb
from test_gpu_stream import ring_system
from test_gpu_team_csr import csr_system
from wgpu_solver_backend_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.fixture()
def own_ctx():
    c = wsb.GpuContext.create("auto", 0)  # the limit cannot reach other tests
    yield c
    c.set_wait_limit(0)


def endless_chain(nbr, seed):
    """A chain whose right-hand side has a NaN: no residual passes the test."""
    rp, ci, v, bs, b = ring_system(nbr, (1,), seed)
    b[5] = np.nan
    return rp, ci, v, bs, b


# Block rows, 70 a part. On 148 SMs the widest system (BSR6: two parts a CTA) and
# the endless one of one part start together; of the next two, which share the
# device, the second has the CTA of the endless one in its team. That one runs
# for a hundred times the limit.
@pytest.mark.parametrize("layout, wide, then", [("BSR6", 20510, (13930, 6650)), ("CSR", 10290, (7000, 3360))])
def test_teams_wait_for_a_long_system(own_ctx, layout, wide, then):
    systems = [ring_system(wide, (1,), 1), endless_chain(70, 2)] + [ring_system(n, (1,), n) for n in then]
    kw = dict(max_iter=30000, rel_tol=1e-6)
    mats = [wsb.Matrix.create(own_ctx, *s[:4], layout=getattr(wsb, "LAYOUT_" + layout)) for s in systems]
    alone = [m.solve(s[4], raise_on_error=False, **kw) for m, s in zip(mats, systems)]
    assert [r["rc"] for _, r in alone] == [0, _lib.NOT_CONVERGED, 0, 0]
    own_ctx.set_wait_limit(2000000)  # about 1 ms
    batch = wsb.Batch(own_ctx)
    ids = [batch.add(m, s[4], **kw) for m, s in zip(mats, systems)]
    batch.solve()
    for i, m, (x, r) in zip(ids, mats, alone):
        xb, rb = batch.result(i, m.n)
        assert (rb["rc"], rb["iterations"]) == (r["rc"], r["iterations"])
        assert np.array_equal(xb.view(np.uint32), x.view(np.uint32))


# Limits from far below an exchange to about as long as one with the load before
# it: whichever waits run out, a system that ends as converged has its bits.
@pytest.mark.parametrize("limit", [100, 1000, 3000, 10000, 30000, 100000])
def test_what_converges_under_a_short_limit_is_right(own_ctx, limit):
    systems = [ring_system(n, (1, 7), n) for n in (10290, 70, 7000, 3360, 281, 141, 9000, 21000)]
    kw = dict(max_iter=3000, rel_tol=1e-6)
    mats = [wsb.Matrix.create(own_ctx, *s[:4]) for s in systems]
    alone = [m.solve(s[4], **kw) for m, s in zip(mats, systems)]
    own_ctx.set_wait_limit(limit)
    batch = wsb.Batch(own_ctx)
    ids = [batch.add(m, s[4], **kw) for m, s in zip(mats, systems)]
    try:
        batch.solve()
    except wsb.WsbError:
        pass
    for i, m, (x, r) in zip(ids, mats, alone):
        xb, rb = batch.result(i, m.n)
        assert rb["rc"] in (0, _lib.TIMEOUT)
        if rb["rc"] == 0:
            assert rb["iterations"] == r["iterations"] and np.array_equal(xb.view(np.uint32), x.view(np.uint32))


# Two workgroups, many, and more than one tree of partials.
@pytest.mark.parametrize("n", [300, 4001, 70001])
def test_reference_arithmetic_honours_the_limit(own_ctx, n):
    rp, ci, v, bs, b = csr_system(n, 1, 6, n)
    m = wsb.Matrix.create(own_ctx, rp, ci, v, bs, layout=wsb.LAYOUT_CSR)
    kw = dict(max_iter=500, rel_tol=1e-5, precision=wsb.PREC_REFERENCE_F32, raise_on_error=False)
    x_ok, r_ok = m.solve(b, **kw)
    assert r_ok["rc"] == 0
    own_ctx.set_wait_limit(1)
    x0 = np.full(n, 3.0, np.float32)
    x, r = m.solve(b, x0=x0, **kw)
    assert r["rc"] == _lib.TIMEOUT and np.array_equal(x, x0)
    own_ctx.set_wait_limit(0)
    x, r = m.solve(b, **kw)
    assert r["iterations"] == r_ok["iterations"] and np.array_equal(x.view(np.uint32), x_ok.view(np.uint32))
