"""Rounding error of BuildSC's t2 against extended precision.

Near a singular rotated overlap the transition density goes as 1 / sigma, a point's contributions to t2 as its fourth
power, and they cancel.  Over sixteen problems the error must not exceed, as a geometric mean, that of the
reference's sequence point by point in FP64 (the numpy oracle).  Also whole tiles and remainders of the kernels over
M^4 elements (M = 32 and 34 spin orbitals) and two chunks of 36 points (M = 34; a block takes eight at a
time), against the oracle (1e-11 of the largest element)."""
import numpy as np
import pytest

from oracle.phf_buildsc import buildsc as oracle, buildsc_vec
from phf_pcc_b200 import api, synth
from phf_pcc_b200.grid import make_grid

pytestmark = pytest.mark.gpu
LD = np.clongdouble


def _problem(n, N, grid, seed):
    g = make_grid(n, ngrid=grid, pg="None")
    rng = np.random.default_rng(seed)
    M = 2 * n
    U = synth.random_unitary(M, rng)
    cz = lambda *s: rng.normal(size=s) + 1j * rng.normal(size=s)
    mo = lambda R: np.asfortranarray(U.conj().T @ R @ U)
    vec = (complex(cz(1)[0]), np.asfortranarray(0.3 * cz(M, M)), np.asfortranarray(0.1 * cz(M, M, M, M)))
    one = np.ones(1, complex)
    return vec, dict(nocc=N, ngrid=list(g.ngrid), qj=g.J, r1=mo(g.R1), r2=mo(g.R2), rpg=mo(g.Rpg), roota=g.roota,
                     rootb=g.rootb, rooty=g.rooty, weightsp=g.weightsp, weightpg=g.weightpg, fsp=one, fpg=one)


def _gpu(vec, a, M):
    return api.buildsc(*vec, a["nocc"], a["ngrid"], a["qj"], a["r1"], a["r2"], a["rpg"], np.eye(M, dtype=complex)[None],
                       a["roota"], a["rootb"], a["rooty"], a["weightsp"], a["weightpg"], a["fsp"], a["fpg"], [1.0])


def _det(S):
    S, det = S.copy(), LD(1)
    for q in range(len(S)):
        p = q + int(np.argmax(np.abs(S[q:, q])))
        if p != q:
            S[[q, p]] = S[[p, q]]
            det = -det
        det *= S[q, q]
        for r in range(q + 1, len(S)):
            S[r, q:] -= S[q, q:] * (S[r, q] / S[q, q])
    return det


def _extended(vec, a):
    c0, c1, c2 = vec
    N, e = a["nocc"], np.einsum
    t2, ov = 0, LD(0)
    for i in range(a["ngrid"][0]):
        for j in range(a["ngrid"][1]):
            R = a["r1"][i].astype(LD) @ a["r2"][j].astype(LD) @ a["rpg"][0].astype(LD)
            X = np.linalg.inv(R[:N, :N].astype(complex)).astype(LD)
            for _ in range(5):  # Newton: the FP64 inverse to extended precision
                X = X + X @ (np.eye(N) - R[:N, :N] @ X)
            Y = np.zeros_like(R)
            Y[:, :N] = R[:, :N] @ X
            t = e("pqrx,lx->pqrl", c2.astype(LD), R.conj())
            t = e("pqxl,kx->pqkl", t, R.conj())
            t = e("xjkl,ix->ijkl", e("pxkl,jx->pjkl", t, R), R)
            s = _det(R[:N, :N]) * a["weightsp"][i, j] * a["weightpg"][0, 0, 0]
            t2 = t2 + s * buildsc_vec(LD(c0), R @ c1.astype(LD) @ R.conj().T, t, Y)[2]
            ov += s
    return t2 / ov


def test_error_not_above_the_sequence_point_by_point():
    ratios = []
    for n, N in ((4, 2), (4, 4), (5, 3), (5, 5)):
        for seed in range(1, 5):
            vec, a = _problem(n, N, (6, 6), seed)
            ref = _extended(vec, a)
            err = lambda t2: float(np.abs(np.asarray(t2) - ref).max())
            ratios.append(err(_gpu(vec, a, 2 * n)[2]) / err(oracle(*vec, **a)[2]))
    assert np.exp(np.mean(np.log(ratios))) <= 1.0, ratios


@pytest.mark.parametrize("n,N,grid", [(16, 8, (6, 1)), (17, 3, (6, 12)), (3, 6, (6, 2)), (2, 1, (6, 1))])
def test_tiles_and_chunks_match_oracle(n, N, grid):
    vec, a = _problem(n, N, grid, n)
    points = [w for w in range(grid[0] * grid[1]) if grid[1] == 1 or w % 7 == 0]  # the others weigh nothing
    keep = np.zeros(grid[0] * grid[1])
    keep[points] = 1.0
    a["weightsp"] = np.asfortranarray(a["weightsp"] * keep.reshape(grid))
    got = _gpu(vec, a, 2 * n)
    for x, y in zip(got, oracle(*vec, **a, point_list=points)):
        x, y = np.asarray(x), np.asarray(y)
        assert np.abs(x - y).max() <= 1e-11 * max(1.0, float(np.abs(y).max()))
    t2 = np.asarray(got[2])
    np.testing.assert_array_equal(t2, -t2.transpose(1, 0, 2, 3))
    np.testing.assert_array_equal(t2, -t2.transpose(0, 1, 3, 2))
