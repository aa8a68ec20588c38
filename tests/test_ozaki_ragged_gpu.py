"""The Ozaki split on sizes that are no multiple of its tiles: residue planes whose
padding rows are never converted, column tiles cut evenly in multiples of 32.
Bar: the repository's 1e-13 relative Frobenius error against Dot2; the integer
product is exact."""
import numpy as np
import pytest
import torch

import oracle
import skgemm
from tests._cases import gaussian

pytestmark = pytest.mark.gpu


def dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).to("cuda")


@pytest.mark.parametrize("precision", [skgemm.PREC_OZAKI_I8, skgemm.PREC_OZAKI_BF16])
@pytest.mark.parametrize("M,N,K", [(1, 1, 130), (17, 33, 1000), (64, 257, 900), (129, 96, 2000),
                                   (257, 264, 3000), (333, 333, 2500), (500, 520, 1500)])
def test_gemm_syrk(cuda, M, N, K, precision):
    A, B = gaussian((M, K), M + K), gaussian((K, N), N + 3 * K)
    a = dev(oracle.pack(A, 16))
    d = torch.full((M, N), np.nan, dtype=torch.float64, device="cuda")
    skgemm.dgemm_packed_dev(M, N, K, a, dev(oracle.pack(np.ascontiguousarray(B.T), 32)), d, N,
                            precision=precision)
    c = torch.zeros(M, M, dtype=torch.float64, device="cuda")
    skgemm.dsyrk_packed_dev(K, M, a, c, M, precision=precision)
    skgemm.stream_status()
    assert oracle.rel_frobenius(d.cpu().numpy(), oracle.dot2_matmul(A, B)) <= 1e-13
    iu = np.triu_indices(M)
    want = oracle.dot2_matmul(A, np.ascontiguousarray(A.T))
    assert oracle.rel_frobenius(c.cpu().numpy().T[iu], want[iu]) <= 1e-13


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (130, 257, 300), (300, 264, 1000), (513, 700, 129)])
def test_integer_product(cuda, M, N, K):
    rng = np.random.default_rng(M + N + K)
    A = rng.integers(-128, 128, (M, K), dtype=np.int8)
    B = rng.integers(-128, 128, (N, K), dtype=np.int8)
    C = torch.zeros(M, N, dtype=torch.int32, device="cuda")
    skgemm.igemm_s8_dev(M, N, K, dev(A), K, dev(B), K, C, N)
    skgemm.stream_status()
    assert np.array_equal(C.cpu().numpy(), A.astype(np.int32) @ B.astype(np.int32).T)


@pytest.mark.parametrize("Nd,nb", [(10016, 48), (9616, 336), (4112, 1040)])
def test_rotation(cuda, Nd, nb):
    psi, Q = gaussian((Nd, nb), Nd + nb), gaussian((nb, nb), nb)
    d = torch.full((Nd * nb,), np.nan, dtype=torch.float64, device="cuda")
    skgemm.drot_band_dev(Nd, nb, dev(oracle.band_pack(psi).ravel()), dev(Q), d,
                         precision=skgemm.PREC_OZAKI_I8)
    skgemm.stream_status()
    want = oracle.band_pack(oracle.dot2_matmul(psi, Q)).ravel()
    assert oracle.rel_frobenius(d.cpu().numpy(), want) <= 1e-13
