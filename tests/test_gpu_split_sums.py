"""Small FP64 products whose sum over k is split over groups of a block: sizes where the groups get unequal or no
k-tiles and the last k-tile and the output tile are partial (k = 34, 36, 46, 66 in tiles of 16), against the C oracle,
with the parity tests' tolerance for this problem size."""
import numpy as np
import pytest

from oracle import phf_oracle as orc
from phf_pcc_b200 import api, synth
from tests.test_gpu_batch import _kwargs
from tests.test_gpu_parity import _close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,N,L", [(17, 8, 35), (18, 14, 97), (23, 4, 81), (33, 18, 50)])
def test_split_sums_match_the_oracle(n, N, L):
    from oracle import phf_oracle_c as corc

    p = synth.make_problem(n, N, L, ngrid=(6, 3), seed=n)
    Ref, Z = p.ref_and_z()
    rng = np.random.default_rng(n)
    Z = 0.05 * (rng.normal(size=Z.shape) + 1j * rng.normal(size=Z.shape))
    out = api.buildhsg_chol(p.h, p.B, Ref, Z, check_hermitian=False, **_kwargs(p))
    Bt = np.transpose(orc.chol_spin_orbital(p.B, Ref), (1, 2, 0))
    H1 = orc.mo_transform_1(p.hone_ao(), Ref)
    ref = corc.buildhsg(H1, None, Ref, Z, Bt=Bt, **p.grid_kwargs())
    for x, y, key in zip(out, ref, ("Hmat", "Smat", "Gradmat", "Rdmmat")):
        assert _close(x, y), key
