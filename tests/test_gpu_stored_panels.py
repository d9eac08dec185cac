"""A stored symmetric plan forms its exchange rows in panels of the Gram block: where the whole block would not fit
beside the rows (n = 128: 2.1 GB beside 1.1 in FP64, 1.5 as residues) the plan is made all the same and agrees with the
one made with memory to spare (1e-12 of the largest element, FP64 sums over other chunks) and with the streamed
form's full rows (FP64 1e-12, residues 1e-10)."""
import numpy as np
import pytest
import torch

from phf_pcc_b200 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,gib,tol", [("fp64", 2.7, 1e-12), ("ozaki_i8", 3.2, 1e-10)])
def test_stored_rows_fit_beside_one_panel(prec, gib, tol):
    p = synth.make_problem(128, 4, 10, ngrid=(6, 2), seed=3)
    g = p.grid

    def sums(**kw):
        with api.Plan(h=p.h, B=p.B, ref=p.Qfull, ngrid=list(g.ngrid), nci=g.nci, cmplxconj=g.CmplxConj, ncisp=g.ncisp,
                      nocc=p.N, r1=g.R1, r2=g.R2, rpg=g.Rpg, weightsp=g.weightsp, weightpg=g.weightpg, roota=g.roota,
                      rootb=g.rootb, rooty=g.rooty, qj=g.J, sp=g.SP, **kw) as plan:
            return [x.cpu().numpy() for x in plan.eval_device(torch.from_numpy(p.C).cuda())]

    want = sums(jk_form="streamed", precision="fp64", exchange_symmetry=False)
    free = sums(jk_form="eri", precision=prec)
    api.release_memory()
    torch.cuda.empty_cache()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - int(gib * 2 ** 30), dtype=torch.uint8, device="cuda")
    tight = sums(jk_form="eri", precision=prec, workspace_bytes=1 << 20)
    del hold
    torch.cuda.empty_cache()
    for x, y, z in zip(tight, free, want):
        assert np.abs(x - y).max() <= 1e-12 * np.abs(y).max()  # (other chunks of points)
        assert np.abs(x - z).max() <= tol * np.abs(z).max()
