"""The exchange symmetry in the stored form (exchange matrix kept on the device): rows and contraction over
index pairs against the full rows, at n = 2 (one antisymmetric pair), odd n, a full 64-row FP64 tile, and
n = 65 (the smallest tensor-core case), one and several chunks.  Cholesky vectors that are not symmetric keep
the full rows.  Tolerances: FP64 sums of at most n^2 + L terms in another order (1e-12 of the largest
element); int8 slices 1e-9, the digit remainder of S = 5 with k = n^2.

The int8 plans' residue products (n(n+1)/2 pairs as rows and contraction, tiles of 256 x 256, k-steps of 32)
against the FP64 plan at n <= 64, where every other step is FP64: sizes on both sides of a tile and of a k-step
(n = 22, 23: 253, 276 pairs; n = 63, 64: 2016 = 63 k-steps, 2080), an odd and a single tile of points, and
vectors whose squares vanish in FP64.  Tolerance 1e-10: 2^-43.5 sqrt(k) per entry is 4e-12, and sums over
points amplify an entry's error by less than ten here."""
import numpy as np
import pytest
import torch

from phf_pcc_b200 import api, synth

pytestmark = pytest.mark.gpu


def _plan(p, B=None, **kw):
    g = p.grid
    return api.Plan(h=p.h, B=p.B if B is None else B, ref=p.Qfull, ngrid=list(g.ngrid), nci=g.nci, cmplxconj=g.CmplxConj,
                    ncisp=g.ncisp, nocc=p.N, r1=g.R1, r2=g.R2, rpg=g.Rpg, weightsp=g.weightsp, weightpg=g.weightpg,
                    roota=g.roota, rootb=g.rootb, rooty=g.rooty, qj=g.J, sp=g.SP, jk_form="eri", **kw)


def _sums(p, **kw):
    with _plan(p, **kw) as plan:
        return [x.cpu().numpy() for x in plan.eval_device(torch.from_numpy(p.C).cuda())]


@pytest.mark.parametrize("n,N,prec,gradient,ws", [
    (2, 1, "fp64", "reference", 0), (5, 3, "fp64", "exact", 0), (17, 9, "fp64", "reference", 1 << 20),
    (64, 20, "fp64", "reference", 0), (65, 21, "ozaki_i8", "exact", 0), (70, 35, "ozaki_i8", "reference", 256 << 20)])
def test_stored_pairs_match_full_rows(n, N, prec, gradient, ws):
    p = synth.make_problem(n, N, 3 * n, ngrid=(6, 4), seed=n, pg="C2v")
    kw = dict(precision=prec, gradient=gradient, workspace_bytes=ws)
    tol = 1e-12 if prec == "fp64" else 1e-9
    for x, y in zip(_sums(p, **kw), _sums(p, exchange_symmetry=False, **kw)):
        assert np.abs(x - y).max() <= tol * max(1.0, np.abs(y).max())


def test_vectors_that_are_not_symmetric_keep_the_full_rows():
    p = synth.make_problem(6, 3, 12, ngrid=(6, 4), seed=4)
    B = p.B + np.random.default_rng(0).normal(scale=0.02, size=p.B.shape)
    for x, y in zip(_sums(p, B=B), _sums(p, B=B, exchange_symmetry=False)):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("n,N,ngrid,pg,scale,gradient", [
    (2, 1, (6, 1), "None", 1.0, "reference"), (3, 2, (6, 3), "None", 1.0, "exact"), (22, 7, (6, 4), "None", 1.0, "reference"),
    (23, 9, (14, 5), "C2v", 1.0, "reference"), (40, 32, (6, 2), "C2v", 1.0, "exact"), (63, 11, (6, 1), "None", 1.0, "reference"),
    (64, 32, (6, 6), "None", 1.0, "reference"), (12, 5, (6, 3), "None", 1e-80, "reference")])
def test_residue_products_match_fp64(n, N, ngrid, pg, scale, gradient):
    p = synth.make_problem(n, N, 4 * n + 1, ngrid=ngrid, seed=n, pg=pg)
    if scale != 1.0:
        p.h[:] = 0.0
        p.B[:] *= scale
    got, ref = _sums(p, precision="ozaki_i8", gradient=gradient), _sums(p, precision="fp64", gradient=gradient)
    assert np.abs(got[0][:, 1] - ref[0][:, 1]).max() <= 1e-12 * np.abs(ref[0][:, 1]).max()
    for x, y in ((got[0][:, 0], ref[0][:, 0]), (got[1], ref[1])):
        assert np.isfinite(x).all() and np.abs(x - y).max() <= 1e-10 * np.abs(y).max()
