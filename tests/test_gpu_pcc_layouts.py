"""The elementwise and short-sum products of the projected-CC grid kernel at sizes whose index spaces are odd in
some dimensions (pairs of elements along a transposed dimension end in a half pair) and whose GEMMs end in partial
32 x 64 tiles, against the oracle: 7 and 9 occupied orbitals, several grid chunks and one.  Tolerance as for the
other sizes: 1e-10 of the largest element of each output (FP64 on both sides, terms in another order)."""
import pytest

from oracle import phf_pcc as pcc
from tests.test_gpu_pcc import _compare, _gpu, _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,N,ngrid,workspace", [(8, 7, (14, 6), 0), (9, 9, (6, 6), 0), (8, 7, (6, 4), 1 << 25)])
def test_odd_index_spaces_match_oracle(n, N, ngrid, workspace):
    p = _problem(n, N, ngrid, seed=n + N, J=1)
    _compare(_gpu(p, workspace=workspace), pcc.pbarhbarolap(**p))
