"""CSR systems that one cooperative launch iterates (k_team): edges of its warp
tiles and CTAs, blocks of 1 to 6 rows, long and unsorted rows, and more columns
outside a CTA's rows than its plan has room for."""
import numpy as np
import pytest

import oracle
import wgpu_solver_backend_b200 as wsb

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - np.asarray(b, np.float64)) / np.linalg.norm(b))


def csr_system(n, couplings, longest_block, seed, shuffle=False, hub=0):
    """A diagonally dominant symmetric CSR system of n rows: a chain and
    `couplings` random neighbours a row, blocks of 1 to longest_block rows.
    shuffle: the entries of a row in any order. hub: row 0 is coupled to this
    many rows."""
    rng = np.random.default_rng(seed)
    i = np.concatenate([np.arange(n - 1), np.repeat(np.arange(n), couplings), np.zeros(hub, int)])
    j = np.concatenate([np.arange(1, n), rng.integers(0, n, couplings * n), rng.integers(0, n, hub)])
    i, j = np.minimum(i, j), np.maximum(i, j)
    pair = np.unique((i * n + j)[i != j])
    i, j = pair // n, pair % n
    w = -rng.uniform(0.1, 1.0, len(i))
    diag = 0.02 - np.bincount(i, w, n) - np.bincount(j, w, n)
    r = np.concatenate([np.arange(n), i, j])
    c = np.concatenate([np.arange(n), j, i])
    v = np.concatenate([diag, w, w])
    order = np.lexsort((rng.random(len(c)) if shuffle else c, r))
    rp = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))])
    cuts = [0]
    while cuts[-1] < n:
        cuts.append(min(n, cuts[-1] + int(rng.integers(1, longest_block + 1))))
    b = rng.uniform(-1, 1, n).astype(np.float32)
    return rp.astype(np.uint32), c[order].astype(np.uint32), v[order].astype(np.float32), np.array(cuts, np.uint32), b


def check(ctx, rp, ci, v, bs, b, x0=None, **kw):
    """Same iterations as the FP64-dot oracle, x within the 1e-6 of the fused
    path's bar against it (their FP64 sums differ in grouping only)."""
    n = len(rp) - 1
    m = wsb.Matrix.create(ctx, rp, ci, v, bs, layout=wsb.LAYOUT_CSR)
    x, r = m.solve(b, x0=x0, max_iter=4000, rel_tol=1e-6, history_capacity=4000)
    lu = wsb.build_lu_blocks_from_csr_block_starts_6(n, rp, ci, v, bs)
    start = np.zeros(n, np.float32) if x0 is None else x0
    f64 = oracle.pcg_f64dot(rp, ci, v, lu, bs, b, start, 4000, 1e-6, 0.0)
    assert r["iterations"] == f64["iterations"]
    assert rel(x, f64["x"]) < 1e-6
    np.testing.assert_allclose(r["history"], f64["history"], rtol=1e-6)
    return m, x, r


# Rows: one; a warp tile of single rows less one, exactly, plus one; a CTA of
# them (448) less one, exactly, plus one; blocks of up to 6 rows, several CTAs.
@pytest.mark.parametrize("n, longest", [(1, 1), (31, 1), (32, 1), (33, 1), (447, 1), (448, 1), (449, 1), (5, 6),
                                        (33, 6), (449, 6), (4001, 6), (20011, 3)])
def test_edges_of_tiles_and_teams(ctx, n, longest):
    s = csr_system(n, 1, longest, n)
    check(ctx, *s, x0=np.random.default_rng(n).standard_normal(n).astype(np.float32))


def test_unsorted_rows_and_a_long_one(ctx):
    check(ctx, *csr_system(3000, 2, 6, 5, shuffle=True, hub=700))


# Columns outside a CTA's 448 rows, all different nearly: within the plan's
# 4,096, about as many, too many (the loop kernels).
@pytest.mark.parametrize("couplings", [3, 5, 9])
def test_columns_outside_a_part(ctx, couplings):
    check(ctx, *csr_system(30000, couplings, 6, couplings))


def test_divisions_outside_the_short_range(ctx):
    rp, ci, v, bs, b = csr_system(700, 2, 6, 7)
    m = wsb.Matrix.create(ctx, rp, ci, v, bs, layout=wsb.LAYOUT_CSR)
    x, r = m.solve(b, max_iter=4000, rel_tol=1e-5)
    for scale in (2.0**-70, 2.0**70):
        xs, rs = m.solve((b * np.float32(scale)).astype(np.float32), max_iter=4000, rel_tol=1e-5)
        assert rs["iterations"] == r["iterations"]
        assert np.array_equal((xs / np.float32(scale)).view(np.uint32), x.view(np.uint32))


def test_batch_and_server_with_both_layouts(ctx):
    # Both kernels of a step, waiting teams, steps of a few iterations, a system
    # of the loop kernels: the bits of each solved alone.
    lattice = wsb.lattice_generate(7, seed=1)
    systems = [csr_system(n, 2, 6, n) for n in (20000, 300, 9000, 1, 30000, 2000)] + [csr_system(30000, 9, 6, 9)]
    systems.append(tuple(lattice[k] for k in ("row_ptr", "col_idx", "values", "block_starts", "b")))
    kw = dict(max_iter=4000, rel_tol=1e-6)
    mats = [wsb.Matrix.create(ctx, *s[:4]) for s in systems]
    alone = [m.solve(s[4], **kw) for m, s in zip(mats, systems)]
    batch = wsb.Batch(ctx)
    ids = [batch.add(m, s[4], **kw) for m, s in zip(mats, systems)]
    batch.solve()
    srv = wsb.Server(ctx, iters_per_step=3)
    try:
        rids = [srv.submit(*s, **kw) for s in systems]
        served = [srv.wait(r, 60.0) for r in rids]
    finally:
        srv.close()
    for i, m in enumerate(mats):
        for x, r in (batch.result(ids[i], m.n), served[i]):
            assert r["iterations"] == alone[i][1]["iterations"], i
            assert np.array_equal(x.view(np.uint32), alone[i][0].view(np.uint32)), i
