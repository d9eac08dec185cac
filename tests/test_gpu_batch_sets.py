"""phf_eval_batch when sets of plans and buffers alternate: a set is launched directly the first time, captured when
it comes again and replayed after that.  Every call gives bitwise what the plans give one by one, also with the
inputs of a captured set overwritten in place."""
import numpy as np
import pytest

from phf_pcc_b200 import api, synth
from tests.test_gpu_batch import _kwargs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 3, 18])
def test_alternating_sets_match_one_by_one(count):
    import torch

    probs = [synth.make_problem(4 + i % 5, 4, 12, ngrid=(6, 2), seed=60 + i) for i in range(count)]
    plans = [api.Plan(ref=np.eye(p.M), h=p.h, B=p.B, precision="fp64", **_kwargs(p)) for p in probs]
    try:
        Cs = [torch.from_numpy(p.C).cuda() for p in probs]
        C2 = [torch.conj(C).resolve_conj().contiguous() for C in Cs]
        ref = [[t.clone() for t in pl.eval_device(C)] for pl, C in zip(plans, Cs)]
        ref2 = [[t.clone() for t in pl.eval_device(C)] for pl, C in zip(plans, C2)]

        def check(outs, want):
            assert all(torch.equal(a, b) for o, r in zip(outs, want) for a, b in zip(o, r))

        a = api.eval_batch(plans, Cs)
        check(a, ref)
        b = api.eval_batch(plans, C2)
        check(b, ref2)
        for _ in range(3):  # direct, captured, replayed
            for o in a:
                for t in o:
                    t.zero_()
            check(api.eval_batch(plans, Cs, a), ref)
        for C, D in zip(Cs, C2):
            C.copy_(D)
        check(api.eval_batch(plans, Cs, a), ref2)
    finally:
        for pl in plans:
            pl.close()
