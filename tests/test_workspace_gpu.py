"""A stream's Stream-K workspace is allocated by its first native call and serves every
later shape on that stream: no call on a warm stream allocates or frees."""
import pytest
import torch

import skgemm

pytestmark = pytest.mark.gpu


def test_later_shapes_allocate_nothing(cuda):
    s = torch.cuda.Stream()
    shapes = [(32, 10000), (96, 10000), (128, 40000), (256, 20000), (512, 20000), (130, 500),
              (512, 110000)]
    ops = [(torch.zeros((nb + 15) // 16 * 16 * nd, dtype=torch.float64, device="cuda"),
            torch.zeros((nb + 31) // 32 * 32 * nd, dtype=torch.float64, device="cuda"),
            torch.zeros(nb * nb, dtype=torch.float64, device="cuda")) for nb, nd in shapes]
    t = torch.cuda.Stream()  # the kernels' code is loaded before anything is measured
    for (nb, nd), (a, b, d) in zip(shapes, ops):
        skgemm.dsyrk_packed_dev(nd, nb, a, d, stream=t)
        skgemm.dgemm_packed_dev(nb, nb, nd, a, b, d, stream=t)
    torch.cuda.synchronize()
    skgemm.stream_release(t)
    (nb, nd), (a, b, d) = shapes[0], ops[0]
    skgemm.dsyrk_packed_dev(nd, nb, a, d, stream=s)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    for (nb, nd), (a, b, d) in zip(shapes, ops):
        skgemm.dsyrk_packed_dev(nd, nb, a, d, stream=s)
        skgemm.dgemm_packed_dev(nb, nb, nd, a, b, d, stream=s)
        torch.cuda.synchronize()
        assert torch.cuda.mem_get_info()[0] == free, (nb, nd)
    skgemm.stream_status(s)
    skgemm.stream_release(s)
