"""GPU: the launch forms that the estimate's kernels choose by size, each at the
sizes where its split can go wrong, against the FP64 oracle.

Tolerance: weights and sketch enter as 28-bit values of their column's maximum
(or, windowed, of its a-priori bound), which holds LD scores to the stated 1e-6."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu
TOL = 1e-6


def _rows(n, m, seed):
    """Packed rows of independent hard calls with 2 % missing."""
    from summit_b200 import bedfile

    rng = np.random.default_rng(seed)
    g = rng.binomial(2, rng.uniform(0.1, 0.5, (m, 1)), (m, n)).astype(np.int8)
    g[rng.random((m, n)) < 0.02] = -9
    return bedfile.pack_bed_rows(g)


# (N, M, K, B): lists of 2,304 and 5,000 members share their K-steps among CTAs
# (the second with an uneven last part, two column groups and an empty bin);
# 110,000 samples give sketch columns whose cluster slices do not fit the cache,
# 30,001 ones that do; 1,100 members take the cluster form of the weight digits.
@pytest.mark.parametrize("n,m,K,B", [(130, 2304, 1, 3), (257, 5000, 3, 70), (110000, 40, 1, 2),
                                     (30001, 60, 2, 3), (300, 1100, 1, 130)])
def test_genome_wide_forms(oracle, n, m, K, B):
    from summit_b200.session import GwSession

    rows = _rows(n, m, seed=n + m)
    annot = np.ones((m, K))
    annot[::3, 1:] = 0.0
    annot[:, 2:] = 0.0
    sess = GwSession(rows, n)
    plan = sess.plan(annot, B, 500, 11)
    plan.execute()
    first = plan.results()
    plan.execute()
    got = plan.results()
    np.testing.assert_array_equal(first["ldscore"], got["ldscore"])
    ref = oracle.gw_ldscore(rows, n, annot, nvecs=B, step=500, seed=11)
    assert rel_err(got["meansq_accum"], ref["meansq_accum"]) < TOL
    plan.close()
    sess.close()


# Windowed lists: 9,000 equal members push a column's digit shift past 14 (the
# 64-bit rounding), 300 keep it inside; 66 and 7 probes leave a second column
# group and a chunk of 8 probes partly filled.
@pytest.mark.parametrize("n,sizes,B", [(140, [9000], 7), (200, [300, 1, 700], 66),
                                       (129, [128, 129, 60], 8)])
def test_windowed_forms(oracle, n, sizes, B):
    from summit_b200.session import GwSession, WinPlan, window_seed

    ws = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    m = int(ws[-1])
    rows = _rows(n, m, seed=m)
    annot = np.ones((m, 2))
    annot[::2, 1] = 0.0
    sess = GwSession(rows, n)
    plan = WinPlan(sess, annot, ws, B, 250, 5)
    plan.execute()
    got = plan.results()["meansq_accum"]
    for w, (a, e) in enumerate(zip(ws[:-1], ws[1:])):
        ref = oracle.gw_ldscore(rows, n, annot[a:e], nvecs=B, step=250, seed=window_seed(5, w),
                                snp0=int(a))
        assert rel_err(got[a:e], ref["meansq_accum"]) < TOL, f"window {w}"
    plan.close()
    sess.close()


# One instance per basis count and per range of fixed effects; several
# annotation chunks, SNP parts of uneven length, a last sample tile of 44.
@pytest.mark.parametrize("Q,R,K,m", [(1, 0, 20, 70), (2, 2, 6, 33), (3, 5, 3, 200), (4, 4, 2, 31),
                                     (5, 0, 1, 64), (6, 16, 2, 40)])
def test_component_diagonal_forms(oracle, Q, R, K, m):
    from oracle import generalized_oracle as go
    from summit_b200 import generalized_gxe as gg
    from summit_b200.session import GwSession

    n = 300
    rng = np.random.default_rng(Q * 100 + R)
    rows = _rows(n, m, seed=Q)
    X = oracle.standardize(rows, n, 0, m)[0]
    sess = GwSession(rows, n)
    basis = np.asfortranarray(rng.normal(size=(n, Q)))
    fixed = np.asfortranarray(np.linalg.qr(rng.normal(size=(n, max(R, 1))))[0][:, :R])
    annot = rng.random((m, K))
    annot[::4, 0] = 0.0
    coef = np.ascontiguousarray(rng.normal(size=(m, Q, R))) if R else None
    got = rng.normal(size=(K * Q * (Q + 1) // 2, n))
    want = got.copy()
    gg._component_diagonal(sess, 0, m, annot, basis, fixed, coef, got)
    go.component_diagonal(X, 0, m, annot, basis, fixed, coef, want)
    assert rel_err(got, want) < 1e-12   # FP64 sums of at most 200 terms
    sess.close()


# Unordered tile pairs: one tile; a ragged last tile; runs of several tiles per
# CTA (many pairs); one-sided and empty partner intervals, which the two orders of
# a pair see differently; K over one pass of 8, at 4 and at 1; a sub-range.
@pytest.mark.parametrize("n,m,K,reach,row0", [(300, 100, 1, 30, 0), (200, 700, 3, 260, 0),
                                              (40, 6000, 2, 5999, 0), (257, 500, 9, 200, 37),
                                              (130, 400, 4, 400, 0), (30000, 520, 2, 300, 0)])
def test_window_ld_pairs(oracle, n, m, K, reach, row0):
    from oracle.oracle import windowed_ld_exact
    from summit_b200.session import GwSession

    rng = np.random.default_rng(m)
    rows = _rows(n, m, seed=K)
    X = oracle.standardize(rows, n, 0, m)[0]
    mm = m - row0
    j = np.arange(mm)
    lo, hi = np.maximum(0, j - reach), np.minimum(mm, j + reach + 1)
    odd = rng.random(mm) < 0.3
    lo[odd] = j[odd]                 # these look only to the right
    hi[::7] = lo[::7]                # and these have no partner
    annot = rng.random((mm, K))
    sess = GwSession(rows, n)
    got = sess.window_ld(lo + row0, hi + row0, annot, corr_dim=n - 1.0, row0=row0)
    again = sess.window_ld(lo + row0, hi + row0, annot, corr_dim=n - 1.0, row0=row0)
    np.testing.assert_array_equal(got, again)
    ref = windowed_ld_exact(X[:, row0:], annot, lo, hi, restandardize=True, corr_dim=n - 1.0)
    assert rel_err(got, ref) < 1e-11   # integer Gram sums, FP64 after them
    sess.close()


# The launch shapes chosen from a plan's sizes (several windows per phase-1 CTA
# with a partial last group; bins shared out evenly among phase-2 CTAs) leave every
# bit as one super-bin and one bin per CTA give it.
@pytest.mark.parametrize("n,m,W,K,B", [(300, 1200, 9, 6, 10), (1500, 2600, 70, 5, 20), (140, 500, 2, 3, 50)])
def test_launch_shapes(n, m, W, K, B):
    from summit_b200.session import GwSession, WinPlan

    rng = np.random.default_rng(m)
    rows = _rows(n, m, seed=m)
    annot = (rng.random((m, K)) < 0.3).astype(float)
    annot[:, 0] = 1.0
    cuts = np.sort(rng.choice(np.arange(1, m), W - 1, replace=False))
    ws = np.concatenate([[0], cuts, [m]]).astype(np.int64)
    sess = GwSession(rows, n)
    out = []
    for shape in (None, 1):
        plan = WinPlan(sess, annot, ws, B, 250, 5)
        if shape:
            plan.set_tiling(shape)
            plan.set_p2_bins(shape)
        plan.execute()
        out.append(plan.results()["ldscore"])
        plan.close()
    np.testing.assert_array_equal(out[0], out[1])
    sess.close()


# GxE source member lists made on the device: several columns of different density
# (one empty), more than one pass of 1,024 SNPs, a list of exactly one K-step, both
# annotation forms, against the same products of a dense standardized block, whose
# weights the host forms.
@pytest.mark.parametrize("m,start,K,is_sqrt", [(2500, 0, 3, False), (1100, 13, 4, True), (64, 0, 1, False)])
def test_gxe_member_lists(m, start, K, is_sqrt):
    from oracle.gxe_oracle import design
    from summit_b200 import bedfile, gxeldcore
    from summit_b200.session import GwSession

    n, T, B = 260, 2, 5
    rng = np.random.default_rng(m + K)
    g = rng.binomial(2, 0.3, (m, n)).astype(np.int8)
    g[rng.random((m, n)) < 0.02] = -9
    sess = GwSession(bedfile.pack_bed_rows(g), n)
    mean, sdinv = (sess.stats()[key] for key in ("mean", "sdinv"))
    X = np.where(g < 0, 0.0, (g - mean[:, None]) * sdinv[:, None]).T
    d = design(n, T, seed=1)
    k = gxeldcore.MultiEnvironmentKernel(d["environments"], d["feature_basis"],
                                         d["power_indices"], d["power_offsets"], d["ranks"],
                                         d["gram_values"], d["gram_offsets"], d["e2_gram_values"],
                                         d["common_basis"], d["directions"], 1, K, 2)
    L = m - start
    ann = rng.random((L, K)) * (rng.random((L, K)) < np.linspace(1.0, 0.05, K))
    if K > 1:
        ann[:, 1] = 0.0
    z = rng.choice([-1.0, 1.0], (L, B))
    sx, sw = rng.random((L, T)) + 0.5, rng.random((L, T)) + 0.5
    out = []
    for block in (sess.block(start, m), np.asfortranarray(X[:, start:])):
        target = np.zeros((n, T * 2 * K * B), order="F")
        assert k.source_block(target, block, z, ann, sx, sw, 0, annotation_is_sqrt=is_sqrt) == 0
        out.append(target)
    assert rel_err(out[0], out[1]) < TOL
    sess.close()


# The per-block calls' sketch crosses PCIe in pieces of whole columns: 300,007
# samples make a column longer than a piece, 60,001 ones several pieces of four
# columns with a last partial one; a second block merges into the first's.
@pytest.mark.parametrize("n,m,K,B", [(300007, 24, 1, 3), (60001, 30, 2, 5)])
def test_block_call_pieces(oracle, tmp_path, n, m, K, B):
    from summit_b200 import bedfile, gwldcore

    rows = _rows(n, m, seed=n)
    prefix = bedfile.write_plink(tmp_path / "p", packed=rows, n=n)
    annot = np.ones((m, K))
    annot[::3, 1:] = 0.0
    step = m // 2
    xz = np.full((n, K * B), np.nan, order="F")   # (the first block overwrites)
    init, inv, meansq = np.zeros(K, dtype=np.uint8), np.empty(m), np.zeros((m, K))
    for a in range(0, m, step):
        e = min(m, a + step)
        gwldcore.phase1_compute_Xz_bed_chunk(
            prefix, prefix + ".fam", a, e, annot_blk=annot[a:e], inv_right=inv[a:e], v_start=0,
            v_count=B, kmax_hint=e - a, seed=9, Xz2d_chunk=xz, bin_init_mask=init, inv_out=inv[a:e],
            impute_mode="mean")
    for a in range(0, m, step):
        e = min(m, a + step)
        gwldcore.phase2_accum_XtXz_bed(prefix, prefix + ".fam", a, e, inv_left=inv[a:e], tile_nvecs=B,
                                       Xz2d=xz, meansq_accum=meansq, N_denom=n, impute_mode="mean")
    ref = oracle.gw_ldscore(rows, n, annot, nvecs=B, step=step, seed=9)
    assert rel_err(meansq, ref["meansq_accum"]) < TOL


# One-call estimates take their buffers from a pool: what an earlier call of
# another size left in them, or the pool having been emptied, changes no bit.
def test_one_call_buffers_are_reused():
    from summit_b200 import _lib, gwldcore

    def run(n, m):
        r = gwldcore.gw_ldscore(_rows(n, m, seed=n), n, np.ones((m, 2)), 6, 100, 3)
        return np.array(r["ldscore"])

    first = run(300, 200)
    run(1500, 700)
    np.testing.assert_array_equal(run(300, 200), first)
    _lib.load().lds_clear_device_cache()
    np.testing.assert_array_equal(run(300, 200), first)


# (n_in, n_out, n): the forward with several row tiles per CTA (with and without a
# last partial one, and at the widest layers, where shared memory holds fewer
# groups), the weight gradient with several 64-row chunks per split.  Loss and
# gradient in norm, at the network's own tolerance: BF16 operands against an oracle
# that rounds as the kernels do.
@pytest.mark.parametrize("n_in,n_out,n", [(5, 2, 148 * 32 + 1), (128, 64, 19000), (33, 17, 38912)])
def test_network_forms(n_in, n_out, n):
    import torch

    from oracle import mlp_oracle as mo
    from summit_b200.surrogate import Surrogate

    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, n_in)).astype(np.float32)
    t = rng.normal(size=(n, n_out)).astype(np.float32)
    p = mo.init_params(n_in, n_out, 3)
    p += rng.normal(0, 0.02, p.size).astype(np.float32)
    net = Surrogate(n_in, n_out, params=p)
    xt, tt = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    x64, t64, p64 = x.astype(np.float64), t.astype(np.float64), p.astype(np.float64)
    # a row's result does not depend on the launch: pieces of one tile per CTA agree
    parts = torch.cat([net.forward(xt[i:i + 4736]) for i in range(0, n, 4736)])
    assert torch.equal(net.forward(xt), parts)
    loss, g = net.loss_grad(xt, tt)
    want_loss, want_g = mo.loss_grad(p64, x64, t64, n_in, n_out)
    assert abs(loss - want_loss) <= 1e-4 * want_loss
    g = g.cpu().numpy().astype(np.float64)
    L = mo.layout(n_in, n_out)
    for k in ["W1", "b1", "W2", "b2", "W3", "b3", "W4", "b4"]:
        off, m = L[k]
        err = np.linalg.norm(g[off:off + m] - want_g[off:off + m])
        assert err <= 2e-3 * max(np.linalg.norm(want_g[off:off + m]), 1e-30), k
