"""The weighted accumulation over grid points where its groups of 32 points and of four loads end early: 6, 30, 42
and 98 points, one chunk against chunks of a few points, with the ket side (exact gradient) and several spin
components.  Both sum the same terms in FP64 with compensation; the chunks only change the grouping, so they agree
to a few roundings of the largest element (64 eps)."""
import numpy as np
import pytest

from phf_pcc_b200 import api, synth
from tests.test_gpu_batch import _kwargs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ngrid,J", [((6, 1), 0), ((6, 5), 0), ((6, 7), 1), ((14, 7), 0)])
@pytest.mark.parametrize("exact", [False, True])
def test_chunks_agree(ngrid, J, exact):
    import torch

    p = synth.make_problem(7, 6, 21, ngrid=ngrid, seed=5, J=0 if exact else J)  # exact mode has one component
    C = torch.from_numpy(p.C).cuda()
    outs = []
    for ws in (0, 1):  # the default, and as few points a chunk as the plan allows
        with api.Plan(ref=np.eye(p.M), h=p.h, B=p.B, precision="fp64", workspace_bytes=ws,
                      gradient="exact" if exact else "reference", **_kwargs(p)) as plan:
            outs.append([t.clone() for t in plan.eval_device(C)])
            chunk = plan.chunk
    assert chunk < ngrid[0] * ngrid[1] or ngrid == (6, 1)
    for a, b in zip(*outs):
        scale = a.abs().max().item()
        assert (a - b).abs().max().item() <= 64 * 2.0 ** -52 * scale
