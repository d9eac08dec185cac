"""phf_overlap_inverse at the sizes where its padded kernels change: every row count around a multiple of four up
to 33 (one warp per matrix), the edges of the register form, matrix counts that leave the last CTA part empty, and
all-NaN or all-zero pivot columns late in the elimination.  Against numpy; error bound n cond eps as for the other
sizes."""
import numpy as np
import pytest

from phf_pcc_b200 import _lib
from tests.test_gpu_inverse import _cases, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 8, 9, 12, 13, 16, 17, 20, 21, 24, 25, 28, 29, 31, 35, 36, 63, 66, 99])
def test_every_padding_matches_numpy(n):
    S = _cases(n, np.random.default_rng(n))
    st, inv, det, logdet = _run(S)
    assert st == _lib.PHF_OK
    for b in range(S.shape[0]):
        cond = np.linalg.cond(S[b])
        assert np.abs(inv[b] @ S[b] - np.eye(n)).max() <= 64 * n * cond * 2.0 ** -52, b
        sign, lad = np.linalg.slogdet(S[b])
        assert abs(det[b] - sign * np.exp(lad)) <= 64 * n * cond * 2.0 ** -52 * np.exp(lad), b
        assert abs(logdet[b].real - lad) <= 64 * n * cond * 2.0 ** -52, b


@pytest.mark.parametrize("n", [6, 30, 50, 90])
def test_singular_in_the_last_step(n):
    rng = np.random.default_rng(n)
    S = rng.integers(-3, 4, size=(3, n, n)).astype(complex)
    S[1] = np.triu(S[1]) + 8.0 * np.eye(n)
    S[1][n - 1, n - 1] = 0.0  # every earlier pivot is fine, the last is exactly zero
    S[0] += 9.0 * np.eye(n)
    S[2] += 9.0 * np.eye(n)
    st, inv, det, logdet = _run(S)
    assert st == _lib.PHF_ERR_SINGULAR
    assert np.all(inv[1] == 0) and det[1] == 0 and np.isneginf(logdet[1].real)
    for b in (0, 2):
        assert np.abs(inv[b] @ S[b] - np.eye(n)).max() <= 64 * n * np.linalg.cond(S[b]) * 2.0 ** -52
