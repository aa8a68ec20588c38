"""What the serving engine says it holds beside the requests is what it holds."""
import pytest
import torch

import skgemm

pytestmark = pytest.mark.gpu


def test_native_scratch_counts_both_slots_of_a_cta(cuda):
    """Three launches' partial tiles: two 128 x 128 slots per SM each."""
    _, o = skgemm.serve([(0.0, 1600, 64, 1)], precision=skgemm.PREC_NATIVE, hbm_budget=2e9,
                        realtime=False)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert o.scratch_bytes >= 3 * 2 * sms * 128 * 128 * 8
    assert o.scratch_bytes + o.peak_admitted_bytes <= 2e9
