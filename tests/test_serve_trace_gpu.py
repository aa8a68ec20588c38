"""A split-path serving trace of some hundred requests of very different sizes, so that
short requests' first calls on new shapes run beside long ones on the other
stream: every request completes, with the bits of the direct calls on its inputs.
And the products' column tiles narrower than 256 where there are more than two."""
import numpy as np
import pytest
import torch

import oracle
import skgemm

pytestmark = pytest.mark.gpu
OZAKI = skgemm.PREC_OZAKI_I8


def mixed_trace(n, seed):
    """Grid points 1e4 .. 4e4 and states 32 .. 512 (log-uniform, as the serving bench);
    every tenth request is a long one."""
    rng = np.random.default_rng(seed)
    out = []
    for i in range(n):
        ng = 16 * int(np.exp(rng.uniform(np.log(625), np.log(2500))))
        nb = 16 * int(np.exp(rng.uniform(np.log(2), np.log(33))))
        if i % 10 == 9:
            ng, nb = 16 * int(rng.integers(5000, 9000)), 16 * int(rng.integers(40, 60))
        out.append((i * 0.002, ng, nb, 104729 * seed + i))
    return out


def direct(ng, nb, k):
    s = torch.cuda.Stream()
    psi, hpsi, q = (torch.from_numpy(k[x]).cuda() for x in ("Psi_in", "HPsi_in", "Q"))
    S, Hs, P = (torch.zeros(n, dtype=torch.float64, device="cuda") for n in (nb * nb, nb * nb, ng * nb))
    torch.cuda.synchronize()
    skgemm.dsubspace_packed_dev(ng, nb, psi, hpsi, S, Hs, precision=OZAKI, stream=s)
    skgemm.drot_band_dev(ng, nb, psi, q, P, precision=OZAKI, stream=s)
    skgemm.stream_status(s)
    skgemm.stream_release(s)
    return S.cpu().numpy(), Hs.cpu().numpy(), P.cpu().numpy()


@pytest.mark.parametrize("streams", [2, 3])
def test_mixed_trace_completes_with_the_direct_calls_bits(cuda, streams):
    trace = mixed_trace(300, seed=streams)
    checked = [i for i, t in enumerate(trace) if i % 10 < 9][::12]
    keep = {}
    for i in checked:
        _, ng, nb, _ = trace[i]
        nb32 = (nb + 31) // 32 * 32
        keep[i] = {"S": np.zeros(nb * nb), "Hs": np.zeros(nb * nb), "Psi": np.zeros(ng * nb),
                   "Psi_in": np.zeros(ng * nb), "HPsi_in": np.zeros(ng * nb32),
                   "Q": np.zeros(nb * nb)}
    rows, o = skgemm.serve(trace, precision=OZAKI, hbm_budget=60e9, realtime=True, keep=keep,
                           ozaki_streams=streams)
    assert len(rows) == len(trace) and o.makespan_s > 0
    for i in checked:
        _, ng, nb, _ = trace[i]
        S, Hs, P = direct(ng, nb, keep[i])
        up = np.triu_indices(nb)
        got = keep[i]["S"].reshape(nb, nb)[up[1], up[0]]
        assert np.array_equal(got, S.reshape(nb, nb)[up[1], up[0]]), (i, ng, nb)
        assert np.array_equal(keep[i]["Hs"], Hs) and np.array_equal(keep[i]["Psi"], P), (i, ng, nb)


@pytest.mark.parametrize("nb", [32, 96, 528, 592, 784, 1040, 1296, 1555])
def test_pair_products_of_narrow_column_tiles(cuda, nb):
    """Widths 32, 96, 192 and 224 in up to seven column tiles, on a stream of their own."""
    K = 1500
    rng = np.random.default_rng(nb)
    X, Y = rng.standard_normal((K, nb)), rng.standard_normal((K, nb))
    s = torch.cuda.Stream()
    a = torch.from_numpy(oracle.pack(np.ascontiguousarray(X.T), 16).ravel()).cuda()
    b = torch.from_numpy(oracle.pack(np.ascontiguousarray(Y.T), 32).ravel()).cuda()
    S, Hs = (torch.zeros(nb * nb, dtype=torch.float64, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    skgemm.dsubspace_packed_dev(K, nb, a, b, S, Hs, precision=OZAKI, stream=s)
    skgemm.stream_status(s)
    up = np.triu_indices(nb)
    got = S.cpu().numpy().reshape(nb, nb)[up[1], up[0]]
    assert oracle.rel_frobenius(got, (X.T @ X)[up]) <= 1e-13
    assert oracle.rel_frobenius(Hs.cpu().numpy().reshape(nb, nb), X.T @ Y) <= 1e-13
