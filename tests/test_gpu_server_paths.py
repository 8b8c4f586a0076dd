"""A server whose requests take different paths: systems of the loop kernels
that retire while others of theirs go on, beside a refined system of a
persistent kernel (whose sweeps upload the descriptors again); and budgets
without room for what the persistent kernels need besides."""
import numpy as np
import pytest

import wgpu_solver_backend_b200 as wsb
from wgpu_solver_backend_b200 import _lib

pytestmark = pytest.mark.gpu


def chain_system(n, shift, seed, hub=0):
    """A chain of n rows (the smaller `shift`, the more iterations) in CSR with
    blocks of 1 to 6 rows; row 0 is also (weakly) coupled to `hub` rows. Above 66,304 rows
    (148 SMs x 14 warps x 32), or with a row above 1,210 nonzeros, only the loop
    kernels take it."""
    rng = np.random.default_rng(seed)
    i = np.concatenate([np.arange(n - 1), np.zeros(hub, int)])
    j = np.concatenate([np.arange(1, n), np.arange(2, 2 + hub)])
    w = rng.uniform(0.5, 1.0, len(i)) * np.where(np.arange(len(i)) < n - 1, 1.0, 1e-5)
    diag = shift + np.bincount(i, w, n) + np.bincount(j, w, n)
    rows = np.concatenate([np.arange(n), i, j])
    cols = np.concatenate([np.arange(n), j, i])
    vals = np.concatenate([diag, -w, -w]).astype(np.float32)
    order = np.lexsort((cols, rows))
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.uint32)
    cuts = [0]
    while cuts[-1] < n:
        cuts.append(min(n, cuts[-1] + int(rng.integers(1, 7))))
    b = rng.uniform(-1, 1, n).astype(np.float32)
    return rp, cols[order].astype(np.uint32), vals[order], np.array(cuts, np.uint32), b


def test_retired_loop_systems_beside_a_refined_one(ctx):
    s = wsb.lattice_generate(12, 7, 2.0)
    refined = (s["row_ptr"], s["col_idx"], s["values"], s["block_starts"], s["b"])
    plain = dict(max_iter=20000, rel_tol=1e-6)
    sweeps = dict(max_iter=60000, rel_tol=0.0, precision=wsb.PREC_MIXED_F64_IR, target_relres=1e-10, inner_rel_tol=1e-2)
    # The small one has a few of the lists' tiles and stops well before the large.
    requests = [(chain_system(80000, 2e-5, 1), plain), (chain_system(70000, 2e-5, 2), plain),
                (chain_system(1500, 2e-4, 3, hub=1400), plain), (refined, sweeps)]
    alone = []
    for system, kw in requests:
        m = wsb.Matrix.create(ctx, *system[:4])
        alone.append(m.solve(system[4], **kw))
    assert alone[3][1]["refine_sweeps"] >= 3
    assert alone[2][1]["iterations"] < alone[1][1]["iterations"] / 2
    srv = wsb.Server(ctx, iters_per_step=4)
    try:
        rids = [srv.submit(*system, **kw) for system, kw in requests]
        served = [srv.wait(r, 120.0) for r in rids]
    finally:
        srv.close()
    for (x, r), (xa, ra) in zip(served, alone):
        assert r["rc"] == 0 and r["iterations"] == ra["iterations"]
        assert np.array_equal(x.view(np.uint32), xa.view(np.uint32))


# A system of the loop kernels, and one that k_team would take.
@pytest.mark.parametrize("n", [80000, 4000])
def test_budget_of_the_loop_kernels_memory(ctx, n):
    """A budget of what a system needs in the loop kernels (matrix, factors,
    vectors, partials) admits it, whatever the other kernels would need."""
    rp, ci, v, bs, b = chain_system(n, 1e-2, n)
    nnz, nb, pad, tiles = len(v), len(bs) - 1, 64, n // 16 + 64
    matrix = 8 * nnz + 4 * (n + 1) + 8 * pad + 8 * tiles
    factors = 144 * nb + 4 * (nb + 1) + 16 * tiles + 1024
    vectors = 24 * (n + pad) + 24 * tiles + 8 * 4096
    kw = dict(max_iter=5000, rel_tol=1e-6)
    xa, ra = wsb.Matrix.create(ctx, rp, ci, v, bs).solve(b, **kw)
    for budget, rc in ((matrix + factors + vectors, 0), (matrix + factors + vectors - 1, _lib.OUT_OF_MEMORY)):
        srv = wsb.Server(ctx, memory_budget_bytes=budget)
        try:
            x, r = srv.wait(srv.submit(rp, ci, v, bs, b, **kw), 60.0)
        finally:
            srv.close()
        assert r["rc"] == rc
        if rc == 0:  # (FP64 sums may be grouped in another way)
            assert r["iterations"] == ra["iterations"]
            assert np.linalg.norm(x.astype(np.float64) - xa) < 1e-6 * np.linalg.norm(xa)
