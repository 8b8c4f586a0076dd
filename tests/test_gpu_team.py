"""Systems that one cooperative launch iterates (k_team): sizes at the edges of
its warp tiles and CTAs, long block rows, and operands outside the range of its
short divisions."""
import numpy as np
import pytest

import oracle
import wgpu_solver_backend_b200 as wsb

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - np.asarray(b, np.float64)) / np.linalg.norm(b))


def block_system(nbr, extra, seed):
    """A symmetric positive definite BSR6 system of nbr block rows: a chain plus
    `extra` random couplings a block row (rows of very different lengths)."""
    rng = np.random.default_rng(seed)
    pairs = {(i, i + 1) for i in range(nbr - 1)}
    for i in range(nbr):
        for j in rng.integers(0, nbr, extra):
            if i != j:
                pairs.add((min(i, int(j)), max(i, int(j))))
    blocks = {(i, i): 1e-3 * np.eye(6) for i in range(nbr)}
    for i, j in pairs:
        g = rng.standard_normal((6, 6))
        s = g @ g.T / 6 + 0.1 * np.eye(6)
        blocks[i, i] = blocks[i, i] + s
        blocks[j, j] = blocks[j, j] + s
        blocks[i, j] = -s
        blocks[j, i] = -s.T
    rows = [[] for _ in range(nbr)]
    for i, j in blocks:
        rows[i].append(j)
    rp, ci, v = [0], [], []
    for i in range(nbr):
        cols = sorted(rows[i])
        for a in range(6):
            for j in cols:
                ci.extend(range(6 * j, 6 * j + 6))
                v.extend(blocks[i, j][a])
            rp.append(len(ci))
    b = rng.uniform(-1, 1, 6 * nbr).astype(np.float32)
    return (np.array(rp, np.uint32), np.array(ci, np.uint32), np.array(v, np.float32),
            np.arange(0, 6 * nbr + 1, 6, dtype=np.uint32), b)


def check(ctx, rp, ci, v, bs, b, x0=None):
    """Same iterations as the FP64-dot oracle, x within the 1e-6 of the fused
    path's bar against it (their FP64 sums differ in grouping only)."""
    n = len(rp) - 1
    m = wsb.Matrix.create(ctx, rp, ci, v, bs, layout=wsb.LAYOUT_BSR6)
    x, r = m.solve(b, x0=x0, max_iter=4000, rel_tol=1e-6, history_capacity=4000)
    lu = wsb.build_lu_blocks_from_csr_block_starts_6(n, rp, ci, v, bs)
    start = np.zeros(n, np.float32) if x0 is None else x0
    f64 = oracle.pcg_f64dot(rp, ci, v, lu, bs, b, start, 4000, 1e-6, 0.0)
    assert r["iterations"] == f64["iterations"]
    assert rel(x, f64["x"]) < 1e-6
    np.testing.assert_allclose(r["history"], f64["history"], rtol=1e-6)
    return m, x, r


# Block rows: one; a warp tile less one, exactly, plus one; a CTA (70) less
# one, exactly, plus one; several CTAs with a ragged last one.
@pytest.mark.parametrize("nbr", [1, 4, 5, 6, 69, 70, 71, 281])
def test_edges_of_tiles_and_teams(ctx, nbr):
    check(ctx, *block_system(nbr, 1, nbr))


def test_long_block_rows(ctx):
    # About 24 blocks a row, some rows over 30: several groups of eight columns.
    check(ctx, *block_system(90, 12, 5))


def test_start_vector_and_steps_of_a_batch(ctx):
    rp, ci, v, bs, b = block_system(150, 2, 9)
    x0 = np.random.default_rng(1).standard_normal(len(b)).astype(np.float32)
    m, x, r = check(ctx, rp, ci, v, bs, b, x0=x0)
    # In the server the solve is cut into launches of a few iterations.
    srv = wsb.Server(ctx, iters_per_step=3)
    try:
        rid = srv.submit(rp, ci, v, bs, b, x0=x0, max_iter=4000, rel_tol=1e-6)
        xs, rs = srv.wait(rid, 60.0)
    finally:
        srv.close()
    assert rs["iterations"] == r["iterations"] and np.array_equal(xs.view(np.uint32), x.view(np.uint32))


@pytest.mark.parametrize("scale", [2.0**-70, 2.0**70])
def test_divisions_outside_the_short_range(ctx, scale):
    # Scaling b by a power of two scales every FP32 and FP64 value of the
    # recurrence exactly, but takes the block solves' quotients (and the FP64
    # scalars) out of the range of the short divisions.
    rp, ci, v, bs, b = block_system(75, 2, 3)
    m = wsb.Matrix.create(ctx, rp, ci, v, bs)
    x, r = m.solve(b, max_iter=4000, rel_tol=1e-5)
    xs, rs = m.solve((b * np.float32(scale)).astype(np.float32), max_iter=4000, rel_tol=1e-5)
    assert rs["iterations"] == r["iterations"]
    assert np.array_equal((xs / np.float32(scale)).view(np.uint32), x.view(np.uint32))


def test_zero_entries_of_the_residual(ctx):
    # b is zero outside one block: the first residuals are zero almost everywhere.
    rp, ci, v, bs, b = block_system(200, 1, 4)
    b[12:] = 0.0
    check(ctx, rp, ci, v, bs, b)


# Block rows (70 a part): 120 parts exactly, plus one row; the most with one
# part a CTA (148 SMs); one more (two parts a CTA, an odd count: 149); a ragged
# last warp tile; two parts on all SMs.
@pytest.mark.parametrize("nbr", [8400, 8401, 10360, 10361, 13318, 20720])
def test_one_and_two_parts_a_cta(ctx, nbr):
    check(ctx, *block_system(nbr, 0, nbr))


def test_more_teams_than_the_device_holds(ctx):
    # Two parts a CTA, and systems that wait for idle CTAs: the same bits as
    # alone (one part a CTA, but for the first).
    systems = [block_system(nbr, 1, nbr) for nbr in (10500, 8401, 3000, 1, 71, 140, 141, 6000, 8500, 500, 69, 2000, 281)]
    mats = [wsb.Matrix.create(ctx, rp, ci, v, bs, layout=wsb.LAYOUT_BSR6) for rp, ci, v, bs, _ in systems]
    batch = wsb.Batch(ctx)
    ids = [batch.add(m, s[4], max_iter=4000, rel_tol=1e-6) for m, s in zip(mats, systems)]
    batch.solve()
    for i, m, s in zip(ids, mats, systems):
        x, r = m.solve(s[4], max_iter=4000, rel_tol=1e-6)
        xb, rb = batch.result(i, m.n)
        assert rb["iterations"] == r["iterations"]
        assert np.array_equal(xb.view(np.uint32), x.view(np.uint32))


# One CTA, one part a CTA, two parts a CTA; cut into steps by a server.
@pytest.mark.parametrize("nbr, layout", [(1, "BSR6"), (71, "BSR6"), (2000, "BSR6"), (10361, "BSR6"), (71, "CSR"),
                                         (2000, "CSR")])
def test_single_reduction(ctx, nbr, layout):
    rp, ci, v, bs, b = block_system(nbr, 1, nbr)
    n = len(rp) - 1
    x0 = np.random.default_rng(1).standard_normal(n).astype(np.float32)
    kw = dict(max_iter=4000, rel_tol=1e-6, algorithm=wsb.ALG_SINGLE_REDUCTION)
    m = wsb.Matrix.create(ctx, rp, ci, v, bs, layout=getattr(wsb, "LAYOUT_" + layout))
    x, r = m.solve(b, x0=x0, history_capacity=4000, **kw)
    lu = wsb.build_lu_blocks_from_csr_block_starts_6(n, rp, ci, v, bs)
    f64 = oracle.pcg_single_reduction_f64dot(rp, ci, v, lu, bs, b, x0, 4000, 1e-6, 0.0)
    assert r["iterations"] == f64["iterations"]
    assert rel(x, f64["x"]) < 1e-6
    np.testing.assert_allclose(r["history"], f64["history"], rtol=1e-6)
    if layout == "BSR6":
        srv = wsb.Server(ctx, iters_per_step=3)
        try:
            xs, rs = srv.wait(srv.submit(rp, ci, v, bs, b, x0=x0, **kw), 60.0)
        finally:
            srv.close()
        assert rs["iterations"] == r["iterations"]
        assert np.array_equal(xs.view(np.uint32), x.view(np.uint32))
