"""What the serving engine says it holds beside the requests is what it holds."""
import pytest
import torch

import skgemm

pytestmark = pytest.mark.gpu


def test_native_scratch_counts_both_slots_of_a_cta(cuda):
    """The launches follow one another on partial tiles of two 128 x 128 slots per SM."""
    _, o = skgemm.serve([(0.0, 1600, 64, 1)], precision=skgemm.PREC_NATIVE, hbm_budget=2e9,
                        realtime=False)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert 2 * sms * 128 * 128 * 8 <= o.scratch_bytes <= 58e6
    assert o.scratch_bytes + o.peak_admitted_bytes <= 2e9


@pytest.mark.parametrize("ng,nb", [(20000, 256), (6400, 1040), (40000, 528)])
def test_split_path_scratch_is_reserved_for_every_smaller_request(cuda, ng, nb):
    """The scratch reserved for the largest request holds whatever mix of smaller ones
    comes with it: nothing is allocated later."""
    def held(extra):
        trace = [(0.0, ng, nb, 1)] + [(0.0, g, b, 2) for g, b in extra]
        _, o = skgemm.serve(trace, precision=skgemm.PREC_OZAKI_I8, hbm_budget=40e9,
                            realtime=False)
        return o.scratch_bytes
    smaller = [(16 * g, b) for g in (10, 100, ng // 16) for b in range(32, nb, 48)]
    assert held(smaller) == held([])
