"""Systems that k_stream iterates (larger than the device's shared memory), in
both recurrences, at the edges of its tiles and CTAs."""
import numpy as np
import pytest

import oracle
import wgpu_solver_backend_b200 as wsb
from wgpu_solver_backend_b200 import _lib

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - np.asarray(b, np.float64)) / np.linalg.norm(b))


def ring_system(nbr, offsets, seed):
    """A BSR6 system of nbr block rows, each coupled to the ones `offsets` away
    (without wrapping around), as row pointers, columns, values, starts, b."""
    rng = np.random.default_rng(seed)
    i = np.concatenate([np.arange(nbr - o) for o in offsets if o < nbr] or [np.zeros(0, int)])
    j = np.concatenate([np.arange(o, nbr) for o in offsets if o < nbr] or [np.zeros(0, int)])
    g = rng.standard_normal((len(i), 6, 6))
    s = g @ g.transpose(0, 2, 1) / 6 + 0.1 * np.eye(6)
    s = 0.5 * (s + s.transpose(0, 2, 1))
    d = np.zeros((nbr, 6, 6)) + 0.3 * np.eye(6)
    np.add.at(d, i, s)
    np.add.at(d, j, s)
    br = np.concatenate([np.arange(nbr), i, j])
    bc = np.concatenate([np.arange(nbr), j, i])
    v = np.concatenate([d, -s, -s])
    order = np.lexsort((bc, br))
    br, bc, v = br[order], bc[order], v[order]
    per = np.bincount(br, minlength=nbr)
    start = np.concatenate([[0], np.cumsum(per)])
    rp = np.concatenate([[0], np.cumsum(np.repeat(6 * per, 6))])
    ci = np.empty(36 * len(br), np.uint32)
    val = np.empty(36 * len(br), np.float32)
    pos = rp[6 * br] + 6 * (np.arange(len(br)) - start[br])
    for a in range(6):
        for c in range(6):
            at = pos + a * 6 * per[br] + c
            ci[at] = 6 * bc + c
            val[at] = v[:, a, c]
    b = rng.uniform(-1, 1, 6 * nbr).astype(np.float32)
    return rp.astype(np.uint32), ci, val, np.arange(0, 6 * nbr + 1, 6, dtype=np.uint32), b


# Block rows: the fewest; 80 a CTA less one, exactly (16 warps with one product
# tile each), plus one; the same with 100 and 160; several update tiles a warp, an odd
# count.
@pytest.mark.parametrize("nbr", [10361, 11839, 11840, 11841, 13321, 14799, 14800, 14801, 19241, 23679, 23680, 23681, 75777])
def test_single_reduction(ctx, nbr):
    rp, ci, v, bs, b = ring_system(nbr, (1, 3, 170), nbr)
    n = len(rp) - 1
    m = wsb.Matrix.create(ctx, rp, ci, v, bs, layout=wsb.LAYOUT_BSR6)
    x, r = m.solve(b, max_iter=2000, rel_tol=1e-6, algorithm=wsb.ALG_SINGLE_REDUCTION, history_capacity=2000)
    lu = wsb.build_lu_blocks_from_csr_block_starts_6(n, rp, ci, v, bs)
    f64 = oracle.pcg_single_reduction_f64dot(rp, ci, v, lu, bs, b, np.zeros(n, np.float32), 2000, 1e-6, 0.0)
    assert r["iterations"] == f64["iterations"]
    assert rel(x, f64["x"]) < 1e-6  # FP64 sums grouped differently, all else equal


# More block rows than k_team's CTAs hold (148 x 70): odd and even counts, with
# rows that end in the middle of tiles.
@pytest.mark.parametrize("nbr", [10361, 12346, 13321, 19241, 19999, 75777])
def test_classic_beyond_shared_memory(ctx, nbr):
    rp, ci, v, bs, b = ring_system(nbr, (1, 7, 101), nbr)
    n = len(rp) - 1
    x0 = np.random.default_rng(2).standard_normal(n).astype(np.float32)
    m = wsb.Matrix.create(ctx, rp, ci, v, bs, layout=wsb.LAYOUT_BSR6)
    x, r = m.solve(b, x0=x0, max_iter=2000, rel_tol=1e-6, history_capacity=2000)
    lu = wsb.build_lu_blocks_from_csr_block_starts_6(n, rp, ci, v, bs)
    f64 = oracle.pcg_f64dot(rp, ci, v, lu, bs, b, x0, 2000, 1e-6, 0.0)
    assert r["iterations"] == f64["iterations"]
    assert rel(x, f64["x"]) < 1e-6
    np.testing.assert_allclose(r["history"], f64["history"], rtol=1e-6)


def test_paths_together_and_cut_into_steps(ctx):
    """A batch and a server with systems of all three paths (k_team, k_stream,
    loop kernels): the bits of each solved alone."""
    small = wsb.lattice_generate(6, seed=1)
    large = ring_system(10500, (1, 7, 101), 3)
    larger = ring_system(19500, (1, 7, 101), 3)
    long_rows = ring_system(12000, (1, 2, 3, 4, 5, 6), 4)  # 13 blocks a row: too long for k_stream
    systems = [(small["row_ptr"], small["col_idx"], small["values"], small["block_starts"], small["b"]), large, larger, long_rows]
    kw = dict(max_iter=3000, rel_tol=1e-6)
    mats = [wsb.Matrix.create(ctx, *s[:4]) for s in systems]
    alone = [m.solve(s[4], **kw) for m, s in zip(mats, systems)]
    bt = wsb.Batch(ctx)
    ids = [bt.add(m, s[4], **kw) for m, s in zip(mats, systems)]
    bt.solve()
    srv = wsb.Server(ctx, iters_per_step=3)
    try:
        rids = [srv.submit(*s, **kw) for s in systems]
        served = [srv.wait(r, 60.0) for r in rids]
    finally:
        srv.close()
    for i, m in enumerate(mats):
        for x, r in (bt.result(ids[i], m.n), served[i]):
            assert r["iterations"] == alone[i][1]["iterations"], i
            assert np.array_equal(x.view(np.uint32), alone[i][0].view(np.uint32)), i


@pytest.mark.parametrize("nbr", [10400, 19400])
def test_wait_limit_and_recovery(nbr):
    c = wsb.GpuContext.create("auto", 0)
    try:
        rp, ci, v, bs, b = ring_system(nbr, (1, 7, 101), 5)
        m = wsb.Matrix.create(c, rp, ci, v, bs)
        x_ok, r_ok = m.solve(b, max_iter=2000, rel_tol=1e-6)
        c.set_wait_limit(1)
        x0 = np.full(len(b), 3.0, np.float32)
        x, r = m.solve(b, x0=x0, max_iter=2000, rel_tol=1e-6, raise_on_error=False)
        assert r["rc"] == _lib.TIMEOUT and np.array_equal(x, x0)
        c.set_wait_limit(0)
        x2, r2 = m.solve(b, max_iter=2000, rel_tol=1e-6)
        assert r2["iterations"] == r_ok["iterations"] and np.array_equal(x2, x_ok)
    finally:
        c.set_wait_limit(0)


@pytest.mark.parametrize("nbr", [10400, 19400])
def test_zero_rhs_and_iteration_limit(ctx, nbr):
    rp, ci, v, bs, b = ring_system(nbr, (1, 7, 101), 6)
    m = wsb.Matrix.create(ctx, rp, ci, v, bs)
    x0 = np.full(len(b), 2.0, np.float32)
    x, r = m.solve(np.zeros_like(b), x0=x0, max_iter=10, rel_tol=1e-6)
    assert r["iterations"] == 0 and np.array_equal(x, x0)
    x, r = m.solve(b, x0=x0, max_iter=3, rel_tol=1e-12, raise_on_error=False)
    assert r["rc"] == _lib.NOT_CONVERGED and r["iterations"] == 3 and np.array_equal(x, x0)
