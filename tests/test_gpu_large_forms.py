"""GPU: forms that only larger launches take: exact windowed LD over a chip full of
CTAs and over several batches of partial sums, and GxE source products whose
super-bins share decoded tiles over several K-steps, against FP64."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


def _genotypes(n, m, seed):
    rng = np.random.default_rng(seed)
    g = rng.binomial(2, rng.uniform(0.1, 0.5, (m, 1)), (m, n)).astype(np.int8)
    g[rng.random((m, n), dtype=np.float32) < 0.02] = -9
    return g


# 496 tile pairs of 157 K-steps each: 256 CTAs, more than the chip holds at once, so
# that every stage's producers and consumers run beside busy neighbours; 6,000 SNPs x
# 150 columns: units of 150 KB, 1,128 tile pairs, two batches of at most 512 MB.
# The sums have at most 6,000 terms: 6,000 x 2^-53 = 7e-13, and the Gram sums are exact.
@pytest.mark.parametrize("n,m,K", [(20000, 3900, 2), (40, 6000, 150)])
def test_window_ld_full_launches(oracle, n, m, K):
    from oracle.oracle import windowed_ld_exact
    from summit_b200 import bedfile
    from summit_b200.session import GwSession

    rng = np.random.default_rng(m)
    rows = bedfile.pack_bed_rows(_genotypes(n, m, m))
    j = np.arange(m)
    lo, hi = np.zeros(m, dtype=np.int64), np.full(m, m)
    odd = rng.random(m) < 0.2
    lo[odd] = j[odd]                  # these look only to the right
    hi[::7] = j[::7] + 1              # and these only to the left, or at themselves
    annot = rng.random((m, K))
    sess = GwSession(rows, n)
    got = sess.window_ld(lo, hi, annot, corr_dim=n - 1.0)
    for _ in range(3):
        np.testing.assert_array_equal(sess.window_ld(lo, hi, annot, corr_dim=n - 1.0), got)
    sess.close()
    X = oracle.standardize(rows, n, 0, m)[0]
    assert rel_err(got, windowed_ld_exact(X, annot, lo, hi, restandardize=True, corr_dim=n - 1.0)) < 1e-11


# One annotation bin: 2 T super-bins with one member list, as many to a CTA as 256
# digit columns hold.  B = 20: three of four, then the last alone; B = 32: pairs;
# B = 5: all six.  1,100 and 700 members are 18 and 11 K-steps, 4,500 are shared among
# CTAs as well.  Against the same products of a dense block, whose weights the host
# forms; tolerance: 28-bit weights and sketch.
@pytest.mark.parametrize("m,T,B", [(1100, 2, 20), (700, 3, 32), (1100, 3, 5), (4500, 2, 20)])
def test_gxe_shared_tiles(m, T, B):
    from oracle.gxe_oracle import design
    from summit_b200 import bedfile, gxeldcore
    from summit_b200.session import GwSession

    n = 260
    rng = np.random.default_rng(m + B)
    g = _genotypes(n, m, m)
    sess = GwSession(bedfile.pack_bed_rows(g), n)
    mean, sdinv = (sess.stats()[key] for key in ("mean", "sdinv"))
    X = np.where(g < 0, 0.0, (g - mean[:, None]) * sdinv[:, None]).T
    d = design(n, T, seed=1)
    k = gxeldcore.MultiEnvironmentKernel(d["environments"], d["feature_basis"],
                                         d["power_indices"], d["power_offsets"], d["ranks"],
                                         d["gram_values"], d["gram_offsets"], d["e2_gram_values"],
                                         d["common_basis"], d["directions"], 1, 1, 2)
    ann = rng.random((m, 1)) * (rng.random((m, 1)) < 0.97)
    z = rng.choice([-1.0, 1.0], (m, B))
    sx, sw = rng.random((m, T)) + 0.5, rng.random((m, T)) + 0.5
    out = []
    for block in (sess.block(0, m), np.asfortranarray(X)):
        target = np.zeros((n, T * 2 * B), order="F")
        assert k.source_block(target, block, z, ann, sx, sw, 0) == 0
        out.append(target)
    for c in range(T * 2 * B):   # (column by column: a wrong one among many shows)
        assert rel_err(out[0][:, c], out[1][:, c]) < 1e-6
    sess.close()


# The directed numerator's split over variants and entries (chunks of 64 variants; ten
# chunks of 90; two blocks of variants, whose sums add up), against the sum over the
# scores that the same call returns: FP64 sums of at most 900 terms.
@pytest.mark.parametrize("K,Q,m,width", [(2, 2, 130, 130), (60, 2, 900, 900), (97, 1, 700, 500)])
def test_directed_numerator_forms(K, Q, m, width):
    from conftest import rel_err
    from summit_b200 import bedfile, generalized_gxe as gg
    from summit_b200.session import GwSession

    n, B = 64, 2
    rng = np.random.default_rng(K)
    sess = GwSession(bedfile.pack_bed_rows(rng.binomial(2, 0.4, (m, n)).astype(np.int8)), n)
    pairs = gg.pair_order(Q)
    term_off, term_f1, term_f2 = [0], [], []
    for tp in pairs:
        for sp in pairs:
            for tl, tr in gg._orientations(tp):
                for sl, sr in gg._orientations(sp):
                    term_f1.append(tr * Q + sl)
                    term_f2.append(tl * Q + sr)
            term_off.append(len(term_f1))
    to, f1, f2 = (np.asarray(x, np.int32) for x in (term_off, term_f1, term_f2))
    annot = rng.uniform(0.0, 1.0, size=(m, K))
    rhs = np.asfortranarray(rng.normal(size=(n, K * B * Q * Q)))
    P = len(pairs)
    directional, directed = gg._pass2_scores(sess, rhs, K, B, Q * Q, P, to, f1, f2, float(n - 1),
                                             annot, width)
    want = np.einsum("vk,vpc->kpc", annot, directional.reshape(m, P, K * P)).reshape(K * P, K * P)
    assert rel_err(directed.reshape(K * P, K * P), want) < 1e-12
    sess.close()
