"""Solves in the reference's arithmetic that one cooperative launch iterates
(k_ref_pcg): edges of its workgroups of 256 rows, blocks across them, more
columns than a CTA lists, and the sizes beyond which the passes run one by one.
Bits as the oracle's (x is only written by a solve that converges)."""
import numpy as np
import pytest

import oracle
import wgpu_solver_backend_b200 as wsb
from test_gpu_team_csr import csr_system

pytestmark = pytest.mark.gpu


def check(ctx, rp, ci, v, bs, b, max_iter=60, x0=None):
    n = len(rp) - 1
    lu = wsb.build_lu_blocks_from_csr_block_starts_6(n, rp, ci, v, bs)
    start = np.zeros(n, np.float32) if x0 is None else x0
    ref = oracle.pcg_ref_f32(rp, ci, v, lu, bs, b, start, max_iter, 1e-6, 0.0)
    m = wsb.Matrix.create(ctx, rp, ci, v, bs, layout=wsb.LAYOUT_CSR)
    x, r = m.solve(b, x0=x0, max_iter=max_iter, rel_tol=1e-6, precision=wsb.PREC_REFERENCE_F32, raise_on_error=False,
                   history_capacity=max(max_iter, 1))
    assert (r["rc"], r["iterations"]) == (ref["status"], ref["iterations"])
    assert np.array_equal(x.view(np.uint32), np.asarray(ref["x"], np.float32).view(np.uint32))
    assert np.array_equal(np.asarray(r["history"]), np.asarray(ref["history"], np.float64))


# Rows: one; a workgroup less one, exactly, plus one, plus the five rows beside
# it; several; more partials than one tree takes (65,536 rows), less one and
# plus one; the last size on 148 SMs with two CTAs each, and one more.
@pytest.mark.parametrize("n, longest", [(1, 1), (5, 6), (255, 6), (256, 1), (257, 6), (261, 6), (262, 4), (4001, 6),
                                        (65535, 6), (65537, 3), (75776, 6), (75777, 6)])
def test_edges_of_workgroups(ctx, n, longest):
    check(ctx, *csr_system(n, 1, longest, n), x0=np.random.default_rng(n).standard_normal(n).astype(np.float32))


# Blocks longer than six rows across workgroups; unsorted rows; columns nearly
# all different (more than a CTA lists); a row too long for shared memory.
@pytest.mark.parametrize("n, couplings, longest, hub", [(1500, 2, 9, 0), (3000, 2, 6, 100), (20000, 6, 6, 0),
                                                        (3000, 1, 6, 900)])
def test_blocks_columns_and_long_rows(ctx, n, couplings, longest, hub):
    check(ctx, *csr_system(n, couplings, longest, n, shuffle=True, hub=hub))


def test_limits_and_zero_rhs(ctx):
    s = csr_system(700, 2, 6, 1)
    for max_iter in (0, 1, 3):
        check(ctx, *s, max_iter=max_iter)
    check(ctx, *s[:4], np.zeros_like(s[4]), x0=np.full(700, 2.0, np.float32))
