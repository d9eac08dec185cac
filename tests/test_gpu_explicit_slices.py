"""Int8 plans with explicit ``slices``: the digit products, which the default (``slices`` = 0) replaces by residues where
the exchange symmetry runs.  Stored and streamed forms with the symmetry (symmetric and antisymmetric halves sliced
apart, the exchange GEMM's two Gamma modes) and with the full rows, the fused density slicing (n <= 64), the int8
density and F X products (n > 64) with several sub-batches of points, the wide and the narrow issue, the tuner.
Every test asserts that the plan did not run what the default runs.

Tolerances as for the int8 forms elsewhere: five slices and more 1e-9 of the largest element, one product against the
same product in another order or issue bitwise, another chunking 1e-12."""
import numpy as np
import pytest
import torch

from oracle import phf_oracle as orc
from oracle import phf_oracle_c as corc
from phf_pcc_b200 import _lib, api, synth
from phf_pcc_b200.autograd import energy_and_gradient

pytestmark = pytest.mark.gpu


class _setting:
    """A comparison switch of the library set for a while."""

    def __init__(self, name, value):
        self.f, self.value = getattr(_lib.load(), name), value

    def __enter__(self):
        self.was = self.f(self.value)

    def __exit__(self, *exc):
        self.f(self.was)


def _plan(p, ref=None, **kw):
    g = p.grid
    return api.Plan(h=p.h, B=p.B, ref=p.Qfull if ref is None else ref, ngrid=list(g.ngrid), nci=g.nci, cmplxconj=g.CmplxConj,
                    ncisp=g.ncisp, nocc=p.N, r1=g.R1, r2=g.R2, rpg=g.Rpg, weightsp=g.weightsp, weightpg=g.weightpg,
                    roota=g.roota, rootb=g.rootb, rooty=g.rooty, qj=g.J, sp=g.SP, **kw)


def _sums(p, **kw):
    with _plan(p, **kw) as plan:
        return [x.cpu().numpy() for x in plan.eval_device(torch.from_numpy(p.C).cuda())]


def _launches(f):
    n0 = _lib.load().phf_kernel_launches()
    out = f()
    return out, _lib.load().phf_kernel_launches() - n0


def _close(a, b, tol):
    for x, y in zip(a, b):
        assert np.isfinite(x).all()
        assert np.abs(x - y).max() <= tol * max(1.0, np.abs(y).max()), np.abs(x - y).max()


def _differ(a, b):
    assert any(not np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("n,N,form,slices,panel", [
    (65, 21, "eri", 5, 0), (70, 35, "eri", 6, 0), (65, 6, "streamed", 5, 5), (73, 9, "streamed", 5, 1),
    (96, 10, "streamed", 7, 0), (60, 21, "eri", 5, 0), (64, 40, "eri", 5, 0), (72, 10, "eri", 5, 0), (40, 7, "streamed", 5, 3)])
def test_slices_match_fp64_and_full_rows(n, N, form, slices, panel):
    p = synth.make_problem(n, N, 50, ngrid=(6, 3), seed=n + panel, pg="C2v")
    kw = dict(jk_form=form, precision="ozaki_i8", exchange_panel=panel)
    got, ref = _sums(p, slices=slices, **kw), _sums(p, jk_form="eri", precision="fp64")
    _close(got, ref, 1e-9)
    full = _sums(p, slices=slices, exchange_symmetry=False, **kw)
    _close(got, full, 1e-9)
    if n > 64:
        _differ(got, full)  # pairs, not full rows
    if n > 64 or form == "eri":
        _differ(got, _sums(p, **kw))  # slices, not residues


@pytest.mark.parametrize("form", ["eri", "streamed"])
def test_chunks_of_the_symmetric_slices_match_one_chunk(form):
    p = synth.make_problem(70, 7, 30, ngrid=(6, 3), seed=4, pg="C2v")  # 72 points in blocks of 12
    kw = dict(jk_form=form, precision="ozaki_i8", slices=5)
    one = _sums(p, **kw)
    with _plan(p, workspace_bytes=80 << 20, **kw) as plan:
        assert plan.chunk < 72 and 72 % plan.chunk != 0, plan.chunk
        many = [x.cpu().numpy() for x in plan.eval_device(torch.from_numpy(p.C).cuda())]
    _close(many, one, 1e-12)


@pytest.mark.parametrize("n,N,L,form,cap,slices", [(65, 6, 40, "eri", 2, 5), (96, 10, 50, "streamed", 7, 5),
                                                   (72, 11, 40, "eri", 5, 5), (130, 20, 60, "streamed", 5, 0)])
def test_fock_product_in_sub_batches(n, N, L, form, cap, slices):
    p = synth.make_problem(n, N, L, ngrid=(6, 3), seed=n, pg="C2v" if n < 128 else "None")
    Ref, Z = p.ref_and_z()
    Z = Z + 0.05 * np.random.default_rng(n).normal(size=Z.shape)
    ora = corc.buildhsg(HOne=orc.mo_transform_1(p.hone_ao(), Ref), HTwo=None, Ref=Ref, Z=Z, Bs=p.B, **p.grid_kwargs())
    out, launches = {}, {}
    for on in (0, 1, cap):
        with _setting("phf_int8_fock_product", on):
            with _plan(p, ref=Ref, precision="ozaki_i8", jk_form=form, slices=slices) as plan:
                assert plan.chunk > cap and plan.chunk % cap != 0 or cap == 2
                out[on], launches[on] = _launches(lambda: plan.buildhsg(Z, check_hermitian=False))
    _close(out[cap], out[0], 1e-9)
    _close(out[cap], ora, 1e-9)
    for x, y in zip(out[cap], out[1]):
        np.testing.assert_array_equal(x, y)  # the same products, a part of the points at a time
    _differ(out[1], out[0])
    assert launches[cap] > launches[1] and launches[1] != launches[0], launches


def test_exact_gradient_with_int8_fock_product():
    p = synth.make_problem(70, 7, 30, ngrid=(6, 3), seed=70, pg="C2v")
    C = torch.from_numpy(p.C).cuda()
    rng = np.random.default_rng(5)
    d = rng.normal(size=C.shape) + 1j * rng.normal(size=C.shape)
    d = torch.from_numpy(d / np.linalg.norm(d)).cuda()
    out = {}
    for on in (0, 1):
        with _setting("phf_int8_fock_product", on):
            with _plan(p, ref=np.eye(p.M), precision="ozaki_i8", slices=5, gradient="exact") as plan:
                E, G = energy_and_gradient(C, plan)
                out[on] = (E.item(), G.cpu().numpy())
                if on:
                    ep, em = (energy_and_gradient(C + s * 1e-5 * d, plan)[0].item() for s in (1, -1))
                    an = torch.real(torch.sum(torch.conj(2.0 * G) * d)).item()
                    # 1e-5: energies at 1e-12, amplified by the differences over 2e-5
                    assert abs((ep - em) / 2e-5 - an) <= 1e-5 * max(1.0, abs(an))
    assert abs(out[1][0] - out[0][0]) <= 1e-9 * max(1.0, abs(out[0][0]))
    _close([out[1][1]], [out[0][1]], 1e-9)
    _differ([out[1][1]], [out[0][1]])


@pytest.mark.parametrize("n,form", [(40, "eri"), (40, "streamed"), (66, "eri"), (66, "streamed")])
def test_wide_and_narrow_issue_agree_bitwise(n, form):
    p = synth.make_problem(n, 10, 60, ngrid=(6, 3), seed=9, pg="C2v")
    out = []
    for on in (0, 1):
        with _setting("phf_int8_wide_mma", on):
            out.append(_sums(p, jk_form=form, precision="ozaki_i8", slices=5))
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)
    if form == "eri" or n > 64:
        _differ(out[0], _sums(p, jk_form=form, precision="ozaki_i8"))


@pytest.mark.parametrize("n,form", [(24, "eri"), (66, "eri"), (66, "streamed")])
def test_tuned_slices_are_bitwise_equal_to_untuned(n, form):
    p = synth.make_problem(n, n // 2, 60, ngrid=(14, 4), seed=31, pg="C2v")
    kw = dict(jk_form=form, precision="ozaki_i8", slices=5, exchange_panel=5)
    before = _lib.load().phf_tuned_shapes()
    plain, tuned = _sums(p, **kw), _sums(p, autotune=True, **kw)
    assert _lib.load().phf_tuned_shapes() > before
    for x, y in zip(plain, tuned):
        np.testing.assert_array_equal(x, y)
