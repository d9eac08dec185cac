"""Cholesky vectors that are symmetric to rounding: X^T B X of symmetric vectors with an orthogonal X, as a change of
basis leaves them.  Up to 2 sqrt(n) units in the last place of a vector's largest element the pair forms of the
exchange run on (B + B^T) / 2: the results are bitwise those of a plan given that mean, and agree with the full
rows of the vectors as given.  A larger difference keeps the full rows, bitwise.

Tolerance against the full rows, in units of the largest element: FP64 1e-12 (sums in another order; the mean moves
an element by at most sqrt(n) ulp), residues of a stored plan 1e-10 against FP64 full rows."""
import numpy as np
import pytest
import torch

from phf_pcc_b200 import api, synth

pytestmark = pytest.mark.gpu


def _sums(p, B, **kw):
    g = p.grid
    with api.Plan(h=p.h, B=B, ref=p.Qfull, ngrid=list(g.ngrid), nci=g.nci, cmplxconj=g.CmplxConj, ncisp=g.ncisp,
                  nocc=p.N, r1=g.R1, r2=g.R2, rpg=g.Rpg, weightsp=g.weightsp, weightpg=g.weightpg, roota=g.roota,
                  rootb=g.rootb, rooty=g.rooty, qj=g.J, sp=g.SP, **kw) as plan:
        return [x.cpu().numpy() for x in plan.eval_device(torch.from_numpy(p.C).cuda())]


def _case(n, N):
    p = synth.make_problem(n, N, 3 * n + 1, ngrid=(6, 4), seed=n, pg="C2v")
    X = np.linalg.qr(np.random.default_rng(n).normal(size=(n, n)))[0]
    B = np.stack([X.T @ b @ X for b in p.B])
    assert not np.array_equal(B, B.transpose(0, 2, 1))
    return p, B, 0.5 * B + 0.5 * B.transpose(0, 2, 1)


@pytest.mark.parametrize("n,N,form,prec,slices,tol", [
    (20, 9, "eri", "fp64", 0, 1e-12), (37, 11, "eri", "ozaki_i8", 0, 1e-10), (66, 13, "eri", "ozaki_i8", 0, 1e-10),
    (66, 13, "eri", "ozaki_i8", 5, 1e-9), (66, 13, "streamed", "ozaki_i8", 0, 1e-9)])
def test_rounding_differences_keep_the_pair_form(n, N, form, prec, slices, tol):
    p, B, mean = _case(n, N)
    kw = dict(jk_form=form, precision=prec, slices=slices)
    got, same = _sums(p, B, **kw), _sums(p, mean, **kw)
    full = _sums(p, B, jk_form="eri", precision="fp64", exchange_symmetry=False)
    for x, y, z in zip(got, same, full):
        np.testing.assert_array_equal(x, y)
        assert np.abs(x - z).max() <= tol * np.abs(z).max()


def test_a_larger_difference_keeps_the_full_rows():
    n = 21
    p, _, _ = _case(n, 8)
    ulp = 2.0 ** -52 * np.abs(p.B[3]).max()
    for units, pairs in ((0.9 * 2 * n ** 0.5, True), (1.1 * 2 * n ** 0.5, False)):
        B = p.B.copy()
        B[3, 2, 5] = 0.0  # (no rounding of its own in the difference below)
        B[3, 5, 2] = units * ulp
        full = _sums(p, B, precision="fp64", exchange_symmetry=False)
        mean = _sums(p, 0.5 * B + 0.5 * B.transpose(0, 2, 1), precision="fp64")
        for x, y, z in zip(_sums(p, B, precision="fp64"), full, mean):
            np.testing.assert_array_equal(x, z if pairs else y)
