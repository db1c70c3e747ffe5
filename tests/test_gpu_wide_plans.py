"""GPU: windowed plans with many annotation bins and with many super-bins, whose
phase-1 CTAs are chosen from the lists, against the FP64 oracle.

Tolerance: weights and sketch enter as 28-bit values of their column's maximum
(or a-priori bound), which holds LD scores to the stated 1e-6."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu
TOL = 1e-6


# K = 97 has no divisor near the best number per CTA; 97 bins x 700 windows are
# 67,900 super-bins, more than CTAs fit along grid.y at one each.
@pytest.mark.parametrize("n,W,size,check", [(300, 4, 90, [0, 3]), (130, 700, 2, [0, 350, 699])])
def test_many_bins(oracle, n, W, size, check):
    from summit_b200 import bedfile
    from summit_b200.session import GwSession, WinPlan, window_seed

    K, B, m = 97, 3, W * size
    rng = np.random.default_rng(W)
    g = rng.binomial(2, rng.uniform(0.1, 0.5, (m, 1)), (m, n)).astype(np.int8)
    g[rng.random((m, n)) < 0.02] = -9
    rows = bedfile.pack_bed_rows(g)
    annot = (rng.random((m, K)) < 0.5).astype(float)
    annot[:, 0] = 1.0
    ws = np.arange(0, m + 1, size, dtype=np.int64)
    sess = GwSession(rows, n)
    out = []
    for shape in (0, 8):
        plan = WinPlan(sess, annot, ws, B, 250, 5)
        plan.set_tiling(shape)
        plan.execute()
        out.append(plan.results()["meansq_accum"])
        plan.close()
    np.testing.assert_array_equal(out[0], out[1])
    for w in check:
        a, e = int(ws[w]), int(ws[w + 1])
        ref = oracle.gw_ldscore(rows, n, annot[a:e], nvecs=B, step=250, seed=window_seed(5, w),
                                snp0=a)
        assert rel_err(out[0][a:e], ref["meansq_accum"]) < TOL, f"window {w}"
    sess.close()
