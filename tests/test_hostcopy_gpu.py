"""The blocking host calls on pageable memory, whose copies run through pinned
slots on several threads: the same bits as from pinned memory (copied directly),
for sizes below the threshold, with rows longer and shorter than a slot, and for
downloads; and after the slots were given back."""
import numpy as np
import pytest
import torch

import skgemm

pytestmark = pytest.mark.gpu


def pinned(x):
    t = torch.empty(x.size, dtype=torch.float64, pin_memory=True)
    t.numpy()[:] = x.ravel()
    return t.numpy()


def both(rng, *sizes):
    a = [rng.standard_normal(n) for n in sizes]
    return a, [pinned(x) for x in a]


@pytest.mark.parametrize("M,N,K", [(32, 32, 500), (48, 64, 40000), (16, 32, 150001),
                                   (200, 264, 9000)])
def test_gemm_syrk(cuda, M, N, K):
    rng = np.random.default_rng(M + K)
    pa, pp = both(rng, -(-M // 16) * 16 * K, -(-N // 32) * 32 * K)
    out = []
    for a, b in (pa, pp):
        d, c = np.zeros(M * N), np.arange(M * M, dtype=np.float64)
        skgemm.gemm.compute_packed(M, N, K, a, b, d, 1.5, 0.25)
        skgemm.sme_syrk.compute(K, M, a, c, 0.5, 2.0)
        out.append((d, c))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    assert np.abs(out[0][0]).max() > 0


@pytest.mark.parametrize("Nd,nb", [(512, 64), (16384, 48), (4112, 272)])
@pytest.mark.parametrize("precision", [None, skgemm.PREC_OZAKI_I8])
def test_rotation(cuda, Nd, nb, precision):
    pa, pp = both(np.random.default_rng(Nd), Nd * nb, nb * nb)
    out = []
    for a, q in (pa, pp):
        # The output is pageable once and pinned once.
        d = np.full(Nd * nb, np.nan) if a is pa[0] else pinned(np.full(Nd * nb, np.nan))
        skgemm.sme_gemm_trp_3d.compute(Nd, nb, a, q, d, precision=precision)
        out.append(d)
    assert np.array_equal(out[0], out[1]) and not np.isnan(out[0]).any()


@pytest.mark.parametrize("Nd,nb", [(40, 8), (70001, 40), (4096, 513)])
def test_converters(cuda, Nd, nb):
    skgemm.stream_release()  # the slots are allocated again
    R = Nd // 16 * 16
    src = np.random.default_rng(nb).standard_normal((nb, Nd))
    packed = np.zeros(R * nb)
    skgemm.sme_pack.pack_c16(Nd, nb, src.ravel(), packed)
    want = src[:, :R].reshape(nb, R // 16, 16).transpose(1, 0, 2)
    assert np.array_equal(packed.reshape(R // 16, nb, 16), want)
    back = np.full((nb, Nd), 7.0)
    skgemm.sme_pack.unpack_c16(Nd, nb, packed, back.reshape(-1))
    assert np.array_equal(back[:, :R], src[:, :R]) and (back[:, R:] == 7.0).all()
