"""Stream-K tiles cut into many parts: the fix-up shared by the CTAs that end in
a tile (five parts or more) and the owner's own (fewer), on the three tile shapes
that the sizes choose, every output layout and the grouped launch. One 64 x 64 tile over the whole
machine, parts of one iteration, uneven splits and tiles that end on a range
boundary. Bar: the repository's 1e-13 relative Frobenius error against Dot2."""
import numpy as np
import pytest
import torch

import oracle
import skgemm
from tests._cases import gaussian

pytestmark = pytest.mark.gpu


def dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).to("cuda")


@pytest.mark.parametrize("M,N,K", [(1, 1, 4736), (32, 32, 10000), (64, 64, 300), (64, 64, 4736),
                                   (65, 40, 1185), (128, 128, 2368), (128, 128, 13824),
                                   (200, 136, 3000), (500, 300, 900), (1000, 1000, 200),
                                   (33, 31, 17), (96, 70, 20000), (257, 129, 1000)])
def test_gemm_parts(cuda, M, N, K):
    A, B = gaussian((M, K), M + K), gaussian((K, N), N + 3 * K)
    a, b = dev(oracle.pack(A, 16)), dev(oracle.pack(np.ascontiguousarray(B.T), 32))
    out = []
    for _ in range(2):
        d = torch.full((M, N), np.nan, dtype=torch.float64, device="cuda")
        skgemm.dgemm_packed_dev(M, N, K, a, b, d, N, 1.5, 0.25)
        skgemm.stream_status()
        out.append(d.cpu().numpy())
    assert np.array_equal(out[0], out[1])
    assert oracle.rel_frobenius(out[0], oracle.dot2_matmul(A, B, 1.5, 0.25)) <= 1e-13


@pytest.mark.parametrize("M,K", [(16, 5000), (64, 777), (100, 4736), (130, 12000), (512, 600),
                                 (31, 40), (70, 9000), (33, 16)])
def test_syrk_parts(cuda, M, K):
    A, C = gaussian((M, K), M * 7 + K), gaussian((M, M), M)
    c = dev(C.T)  # column-major
    skgemm.dsyrk_packed_dev(K, M, dev(oracle.pack(A, 16)), c, M, 0.5, -2.0)
    skgemm.stream_status()
    got = c.cpu().numpy().T
    iu = np.triu_indices(M)
    want = 0.5 * oracle.dot2_matmul(A, np.ascontiguousarray(A.T)) - 2.0 * C
    assert oracle.rel_frobenius(got[iu], want[iu]) <= 1e-13
    il = np.tril_indices(M, -1)
    assert np.array_equal(got[il], C[il])


@pytest.mark.parametrize("Nd,nb", [(64, 64), (16, 512), (128, 1024), (208, 336), (4096, 32),
                                   (1008, 96), (16, 16)])
def test_rotation_parts(cuda, Nd, nb):
    psi, Q = gaussian((Nd, nb), Nd + nb), gaussian((nb, nb), nb)
    want = oracle.band_pack(oracle.dot2_matmul(psi, Q)).ravel()
    got = []
    for fn, x in ((skgemm.drot_dev, oracle.grid_pack(psi)), (skgemm.drot_band_dev,
                                                             oracle.band_pack(psi))):
        d = torch.full((Nd * nb,), np.nan, dtype=torch.float64, device="cuda")
        fn(Nd, nb, dev(x.ravel()), dev(Q), d)
        skgemm.stream_status()
        got.append(d.cpu().numpy())
        assert oracle.rel_frobenius(got[-1], want) <= 1e-13
    assert np.array_equal(got[0], got[1])


@pytest.mark.parametrize("tile", [64, 128])
def test_grouped_parts(cuda, tile):
    shapes = [(16, 9000), (130, 5000), (64, 20000), (200, 40)]
    items, keep = [], []
    for i, (nb, K) in enumerate(shapes):
        A, B = gaussian((nb, K), i), gaussian((K, nb), 10 + i)
        a, b = dev(oracle.pack(A, 16)), dev(oracle.pack(np.ascontiguousarray(B.T), 32))
        s = torch.zeros(nb, nb, dtype=torch.float64, device="cuda")
        h = torch.full((nb, nb), np.nan, dtype=torch.float64, device="cuda")
        items += [skgemm.batch_item(skgemm.OP_SYRK_PACKED, nb, nb, K, a, None, s, nb),
                  skgemm.batch_item(skgemm.OP_GEMM_PACKED, nb, nb, K, a, b, h, nb)]
        keep.append((A, B, a, b, s, h))
    plan = skgemm.Plan(items, tile=tile, tune=False)
    for _ in range(2):
        plan.run()
    plan.status()
    for A, B, _, _, s, h in keep:
        iu = np.triu_indices(A.shape[0])
        assert oracle.rel_frobenius(h.cpu().numpy(), oracle.dot2_matmul(A, B)) <= 1e-13
        want = oracle.dot2_matmul(A, np.ascontiguousarray(A.T))
        assert oracle.rel_frobenius(s.cpu().numpy().T[iu], want[iu]) <= 1e-13
    plan.close()
