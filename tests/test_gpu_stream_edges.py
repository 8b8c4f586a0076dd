"""Systems that k_stream takes for certain (the number of launches says so), at
the edges of its tiles and CTAs on 148 SMs and at its limits: 8 blocks a block
row, 36 blocks in five consecutive ones."""
import numpy as np
import pytest

import oracle
import wgpu_solver_backend_b200 as wsb

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - np.asarray(b, np.float64)) / np.linalg.norm(b))


def coupled_system(nbr, extra, seed):
    """A BSR6 system of nbr block rows, each coupled to those 1, 3 and 170 away
    (7 blocks a block row, fewer at the ends), and the pairs `extra`."""
    rng = np.random.default_rng(seed)
    i = np.concatenate([np.arange(nbr - o) for o in (1, 3, 170)] + [np.array(extra, int).reshape(-1, 2)[:, 0]])
    j = np.concatenate([np.arange(o, nbr) for o in (1, 3, 170)] + [np.array(extra, int).reshape(-1, 2)[:, 1]])
    g = rng.standard_normal((len(i), 6, 6))
    s = g @ g.transpose(0, 2, 1) / 6 + 0.1 * np.eye(6)
    s = 0.5 * (s + s.transpose(0, 2, 1))
    d = np.zeros((nbr, 6, 6)) + 0.3 * np.eye(6)
    np.add.at(d, i, s)
    np.add.at(d, j, s)
    br, bc = np.concatenate([np.arange(nbr), i, j]), np.concatenate([np.arange(nbr), j, i])
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
    return per, (rp.astype(np.uint32), ci, val, np.arange(0, 6 * nbr + 1, 6, dtype=np.uint32), b)


def check(ctx, system, streamed, single_reduction=False):
    """Same iterations as the FP64-dot oracle, x within the 1e-6 of the fused
    path's bar against it (their FP64 sums differ in grouping only)."""
    rp, ci, v, bs, b = system
    n = len(rp) - 1
    x0 = np.random.default_rng(2).standard_normal(n).astype(np.float32)
    m = wsb.Matrix.create(ctx, rp, ci, v, bs, layout=wsb.LAYOUT_BSR6)
    x, r = m.solve(b, x0=x0, max_iter=2000, rel_tol=1e-6, history_capacity=2000,
                   algorithm=wsb.ALG_SINGLE_REDUCTION if single_reduction else wsb.ALG_CLASSIC)
    # k_stream: two kernels that start the system and one; k_team: one; the loop
    # kernels: two or three an iteration.
    assert (r["kernel_launches"] == 3) == streamed and r["kernel_launches"] >= 3
    lu = wsb.build_lu_blocks_from_csr_block_starts_6(n, rp, ci, v, bs)
    solve = oracle.pcg_single_reduction_f64dot if single_reduction else oracle.pcg_f64dot
    f64 = solve(rp, ci, v, lu, bs, b, x0, 2000, 1e-6, 0.0)
    assert r["iterations"] == f64["iterations"]
    assert rel(x, f64["x"]) < 1e-6
    np.testing.assert_allclose(r["history"], f64["history"], rtol=1e-6)


# Block rows: one more than k_team holds; 160 and 240 a CTA (two and three product
# tiles a warp) less one, exactly, plus one; 448 and 512 a CTA (one update tile a
# warp, 28 and 32 block rows), exactly, plus one.
@pytest.mark.parametrize("nbr, single_reduction", [
    (19241, True), (19242, False), (23679, False), (23680, False), (23681, False), (35519, True), (35520, True),
    (35521, True), (35519, False), (35520, False), (35521, False), (66304, True), (66305, True), (75776, False),
    (75777, False)])
def test_edges_of_tiles(ctx, nbr, single_reduction):
    check(ctx, coupled_system(nbr, [], nbr)[1], True, single_reduction)


def pairs_of_every_fifth(nbr):
    """Every fifth block row coupled to one a thousand away: 8 blocks."""
    k = np.arange(0, nbr - 1000, 5)
    k = k[(k // 1000) % 2 == 0]
    return [(int(q), int(q) + 1000) for q in k]


@pytest.mark.parametrize("single_reduction", [False, True])
def test_full_product_tiles(ctx, single_reduction):
    per, system = coupled_system(18003, pairs_of_every_fifth(18003), 1)
    assert per.max() == 8 and np.convolve(per, np.ones(5, int), "valid").max() == 36
    check(ctx, system, True, single_reduction)


# A block row of 9 blocks where five have 33; 37 blocks in five.
@pytest.mark.parametrize("longest, most", [(9, 36), (8, 37)])
def test_beyond_a_product_tile(ctx, longest, most):
    if longest == 9:
        extra = [(501, 19953), (601, 19953), (701, 19953)]
    else:
        extra = pairs_of_every_fifth(20003) + [(501, 1502)]
    per, system = coupled_system(20003, extra, 2)
    assert (per.max(), np.convolve(per, np.ones(5, int), "valid").max()) == (longest, most)
    check(ctx, system, False)
