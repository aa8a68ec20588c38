"""The H Psi producer on device (skgemm_stencil_ext_dev, skgemm_halo_periodic_dev):
bit for bit against the oracle (itself equal to the reference's SVE kernels,
tests/test_stencil_cpu.py), and feeding Hs = Psi^T (H Psi) through the GEMM."""
import numpy as np
import pytest
import torch

import oracle
import skgemm
from tests.test_stencil_cpu import C0, CX, F, extended_case

pytestmark = pytest.mark.gpu


def dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).to("cuda")


@pytest.mark.parametrize("ni,nj,nk,nb", [(12, 10, 8, 48), (13, 7, 9, 40), (16, 16, 16, 32),
                                         (33, 5, 20, 17), (48, 48, 48, 64)])
@pytest.mark.parametrize("T", [32, 16])
def test_stencil_equals_oracle(cuda, ni, nj, nk, nb, T):
    _, A, ext = extended_case(ni, nj, nk, nb, 7 * ni + nb)
    K = ni * nj * nk
    CY = [0.0] + [c * 0.75 for c in CX[1:]]
    CZ = [0.0] + [c * 1.25 for c in CX[1:]]
    out = torch.full(((nb + T - 1) // T * K * T,), np.nan, dtype=torch.float64, device="cuda")
    skgemm.stencil_ext_dev(ni, nj, nk, nb, dev(ext), dev(A), CX, CY, CZ, C0, out, T)
    skgemm.stream_status()
    want = oracle.stencil_ext(ext, A, ni, nj, nk, nb, CX, CY, CZ, C0, T, threads=oracle.nthreads())
    got = out.cpu().numpy()
    lanes = np.arange(got.size) % T + (np.arange(got.size) // (K * T)) * T
    assert np.array_equal(got[lanes < nb], want[lanes < nb])
    assert np.isnan(got[lanes >= nb]).all()  # padding lanes untouched


@pytest.mark.parametrize("ni,nj,nk,nb", [
    (1, 1, 1, 1),          # one point, one band
    (15, 7, 2, 7),         # below one tile, fewer planes than a queue
    (17, 9, 13, 9),        # one past the tile and the slab on every axis
    (16, 8, 40, 8),        # one tile: its planes shared out over CTAs
    (31, 25, 14, 23),      # odd rows of A, shares across tile boundaries
    (33, 17, 11, 200),     # more tiles than CTAs: whole waves and shares
])
def test_stencil_tiles_and_shares(cuda, ni, nj, nk, nb):
    """Tile and slab edges and the split of planes over CTAs; equal bits."""
    _, A, ext = extended_case(ni, nj, nk, nb, 3 * ni + nb)
    K, T = ni * nj * nk, 32
    out = torch.full(((nb + T - 1) // T * K * T,), np.nan, dtype=torch.float64, device="cuda")
    skgemm.stencil_ext_dev(ni, nj, nk, nb, dev(ext), dev(A), CX, CX, CX, C0, out, T)
    skgemm.stream_status()
    want = oracle.stencil_ext(ext, A, ni, nj, nk, nb, CX, CX, CX, C0, T, threads=oracle.nthreads())
    got = out.cpu().numpy()
    lanes = np.arange(got.size) % T + (np.arange(got.size) // (K * T)) * T
    assert np.array_equal(got[lanes < nb], want[lanes < nb])
    assert np.isnan(got[lanes >= nb]).all()


def test_halo_periodic_equals_oracle(cuda):
    ni, nj, nk, nb = 24, 20, 16, 40
    rng = np.random.default_rng(11)
    local = rng.standard_normal((nb + 15) // 16 * ni * nj * nk * 16)
    ext = torch.full((oracle.ext_size(ni, nj, nk, nb),), np.nan, dtype=torch.float64, device="cuda")
    skgemm.halo_periodic_dev(ni, nj, nk, nb, dev(local), ext)
    skgemm.stream_status()
    assert np.array_equal(ext.cpu().numpy(), oracle.halo_periodic(local, ni, nj, nk, nb))


@pytest.mark.parametrize("ni,nj,nk,nb,FDn", [
    (1, 1, 1, 1, 1),     # one point, every row a wrap
    (6, 7, 6, 17, 6),    # halo as wide as the domain
    (47, 3, 5, 16, 3),  # a row of 53 points: under one round of loads
    (48, 6, 6, 16, 6),   # 60 points: one round exactly
    (49, 6, 7, 33, 6),   # one point over
    (130, 2, 3, 8, 2),   # three rounds
    (5, 4, 3, 40, 0),    # no halo: a copy
])
def test_halo_rows(cuda, ni, nj, nk, nb, FDn):
    """Row lengths around the loads a warp has in flight, and a row count that is
    no multiple of the warps in a block."""
    rng = np.random.default_rng(ni + nb)
    local = rng.standard_normal((nb + 15) // 16 * ni * nj * nk * 16)
    ext = torch.full((oracle.ext_size(ni, nj, nk, nb, FDn),), np.nan, dtype=torch.float64,
                     device="cuda")
    skgemm.halo_periodic_dev(ni, nj, nk, nb, dev(local), ext, FDn)
    skgemm.stream_status()
    assert np.array_equal(ext.cpu().numpy(), oracle.halo_periodic(local, ni, nj, nk, nb, FDn))


def test_stencil_feeds_hs(cuda):
    """Psi (band-packed) -> periodic halo -> H Psi (32-band-packed) -> Hs =
    Psi^T H Psi with the GEMM, all on the device; against Dot2 of the oracle's
    H Psi."""
    ni = nj = nk = 24
    nb = 96
    K = ni * nj * nk
    rng = np.random.default_rng(5)
    psi = rng.standard_normal((K, nb)) / np.sqrt(K)
    A = rng.uniform(-1, 1, K)
    band = oracle.band_pack(psi).ravel()
    ext = torch.empty(oracle.ext_size(ni, nj, nk, nb), dtype=torch.float64, device="cuda")
    skgemm.halo_periodic_dev(ni, nj, nk, nb, dev(band), ext)
    hpsi = torch.zeros(K * nb, dtype=torch.float64, device="cuda")
    skgemm.stencil_ext_dev(ni, nj, nk, nb, ext, dev(A), CX, CX, CX, C0, hpsi, 32)
    Hs = torch.zeros(nb * nb, dtype=torch.float64, device="cuda")
    skgemm.dgemm_packed_dev(nb, nb, K, dev(band), hpsi, Hs, nb)
    skgemm.stream_status()
    h32 = oracle.stencil_ext(oracle.halo_periodic(band, ni, nj, nk, nb), A, ni, nj, nk, nb,
                             CX, CX, CX, C0, 32)
    hdense = oracle.unpack(h32.reshape(-1, K, 32), nb).T  # (K, nb)
    assert np.array_equal(hpsi.cpu().numpy(), h32)
    ref = oracle.dot2_matmul(np.ascontiguousarray(psi.T), hdense)
    assert oracle.rel_frobenius(Hs.cpu().numpy().reshape(nb, nb), ref) <= 1e-13


def test_stencil_rejects_other_radius(cuda):
    x = torch.zeros(16 * 32 ** 3, dtype=torch.float64, device="cuda")
    with pytest.raises(skgemm.SkgemmError) as e:
        skgemm.stencil_ext_dev(8, 8, 8, 16, x, x, CX[:5], CX[:5], CX[:5], C0, x, 32, FDn=4)
    assert e.value.code == skgemm.ERR_UNSUPPORTED
