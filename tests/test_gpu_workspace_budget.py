"""Residue-form plans keep to workspace_bytes: what a plan takes beyond one with a single point per chunk is at most the
requested budget, with 5 % for what the per-point estimate leaves out (exponents, partial sums of the accumulation).
And the parts of a chunk whose residue products exceed one GiB (more than 2624 points at n = 64), the last part
shorter, match the FP64 plan (1e-10 of the largest element, as for one part)."""
import numpy as np
import pytest
import torch

from phf_pcc_b200 import api, synth

pytestmark = pytest.mark.gpu


def _plan(p, **kw):
    g = p.grid
    return api.Plan(h=p.h, B=p.B, ref=p.Qfull, ngrid=list(g.ngrid), nci=g.nci, cmplxconj=g.CmplxConj, ncisp=g.ncisp,
                    nocc=p.N, r1=g.R1, r2=g.R2, rpg=g.Rpg, weightsp=g.weightsp, weightpg=g.weightpg, roota=g.roota,
                    rootb=g.rootb, rooty=g.rooty, qj=g.J, sp=g.SP, **kw)


@pytest.mark.parametrize("n,form,mib", [(20, "eri", 64), (40, "eri", 100), (64, "eri", 400), (70, "eri", 80),
                                        (70, "streamed", 120), (101, "eri", 500), (130, "streamed", 600)])
def test_reported_workspace_stays_within_the_budget(n, form, mib):
    p = synth.make_problem(n, n // 3, 3 * n, ngrid=(50, 16), seed=n)
    size = []
    for ws in (1, mib << 20):
        with _plan(p, precision="ozaki_i8", jk_form=form, workspace_bytes=ws) as plan:
            size.append(plan.workspace_bytes)
            chunk = plan.chunk
    assert chunk > 16
    assert size[1] - size[0] <= 1.05 * (mib << 20), (chunk, size)


@pytest.mark.parametrize("n,N,form,panel", [(64, 8, "eri", 0), (66, 5, "streamed", 33)])
def test_parts_of_a_chunk_match_fp64(n, N, form, panel):
    p = synth.make_problem(n, N, 40, ngrid=(50, 18), seed=n, pg="C2v")
    C = torch.from_numpy(p.C).cuda()
    out = []
    for prec in ("ozaki_i8", "fp64"):
        with _plan(p, precision=prec, jk_form=form, exchange_panel=panel, workspace_bytes=12 << 30) as plan:
            assert plan.chunk == 3600
            out.append([x.cpu().numpy() for x in plan.eval_device(C)])
    for x, y in zip(*out):
        assert np.abs(x - y).max() <= 1e-10 * np.abs(y).max()
