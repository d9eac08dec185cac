"""Device memory that one-shot calls keep for the next one goes back to others: to an allocation of a plan and of
torch that would fail without it, to the chunk size of a streamed plan (a share of the free memory), and with
release_memory to other processes.  A BuildSC call over 112 points at M = 32 leaves two to four GiB; the rest of the
device is held by a torch buffer."""
import numpy as np
import pytest
import torch

from phf_pcc_b200 import api, synth
from tests.test_gpu_buildsc_rounding import _gpu, _problem

pytestmark = pytest.mark.gpu
GIB = 1 << 30


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.fixture
def kept():
    """A function that runs the one-shot call and returns the bytes it leaves; the device's memory given back after."""
    torch.cuda.empty_cache()
    api.release_memory()
    vec, a = _problem(16, 2, (14, 8), 1)
    one_shot = lambda: _gpu(vec, a, 32)
    one_shot()  # loads the kernels
    api.release_memory()

    def run():
        before = _free()
        one_shot()
        return before - _free()

    yield run
    torch.cuda.empty_cache()
    api.release_memory()


def _plan(p, **kw):
    g = p.grid
    return api.Plan(h=p.h, B=p.B, ref=p.Qfull, ngrid=list(g.ngrid), nci=g.nci, cmplxconj=g.CmplxConj, ncisp=g.ncisp,
                    nocc=p.N, r1=g.R1, r2=g.R2, rpg=g.Rpg, weightsp=g.weightsp, weightpg=g.weightpg, roota=g.roota,
                    rootb=g.rootb, rooty=g.rooty, qj=g.J, sp=g.SP, **kw)


def test_release_memory_returns_what_is_kept(kept):
    size = kept()
    assert size > GIB
    before = _free()
    api.release_memory()
    assert _free() - before > 0.9 * size


def test_allocations_of_the_process_get_the_kept_memory(kept):
    p = synth.make_problem(64, 32, 100, ngrid=(50, 16), seed=1)
    assert kept() > 2 * GIB
    hold = torch.empty(_free() - 400 * 2 ** 20, dtype=torch.uint8, device="cuda")
    more = torch.empty(600 * 2 ** 20, dtype=torch.uint8, device="cuda")
    with _plan(p, workspace_bytes=GIB) as plan:  # about a GiB
        assert plan.workspace_bytes > 0.7 * GIB
        assert np.isfinite(plan.eval_device(torch.from_numpy(p.C).cuda())[0].cpu().numpy()).all()
    del hold, more


def test_streamed_chunk_does_not_depend_on_the_kept_memory(kept):
    p = synth.make_problem(128, 8, 8, ngrid=(50, 16), seed=1, pg="C2v")
    hold = torch.empty(_free() - 24 * GIB, dtype=torch.uint8, device="cuda")
    chunks = []
    for keep in (False, True):
        if keep:
            assert kept() > 2 * GIB
        with _plan(p, jk_form="streamed", precision="fp64") as plan:
            chunks.append(plan.chunk)
    assert abs(chunks[0] - chunks[1]) <= 64, chunks  # a block of ny npg points
    del hold
