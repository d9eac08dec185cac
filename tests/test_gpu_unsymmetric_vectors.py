"""Cholesky vectors that are not symmetric in the streamed tensor-core forms (n > 64): the Coulomb term over pairs
l <= j reads one triangle of each vector, so such plans run the full rows.  Against the stored FP64 form with
the full rows, in units of the largest element: int8 1e-9, BF16x3 and TF32 1e-4 (1e-6 of an entry, summed)."""
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


@pytest.mark.parametrize("prec,slices,symmetry,tol", [
    ("ozaki_i8", 0, "auto", 1e-9), ("ozaki_i8", 0, True, 1e-9), ("ozaki_i8", 5, "auto", 1e-9),
    ("bf16x3", 0, "auto", 1e-4), ("tf32", 0, "auto", 1e-4), ("fp64", 0, True, 1e-11)])
def test_streamed_form_with_vectors_that_are_not_symmetric(prec, slices, symmetry, tol):
    p = synth.make_problem(65, 9, 70, ngrid=(6, 3), seed=5)
    B = p.B + np.random.default_rng(1).normal(scale=0.02, size=p.B.shape)
    got = _sums(p, B, jk_form="streamed", precision=prec, slices=slices, exchange_symmetry=symmetry)
    ref = _sums(p, B, jk_form="eri", precision="fp64", exchange_symmetry=False)
    for x, y in zip(got, ref):
        assert np.abs(x - y).max() <= tol * np.abs(y).max(), np.abs(x - y).max() / np.abs(y).max()
