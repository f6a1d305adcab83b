"""Tuning and timing a batch that has never stepped. Its groups have more than
16 tiles for every SM, so that the stage kernels hand their tiles out by the
counter among the group's error words, which must then start at zero."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def new_batch(vt):
    import torch
    # what the batch's allocations find in memory is not zero
    junk = [torch.full((1 << 21,), 0x5B, dtype=torch.uint8, device="cuda") for _ in range(64)]
    torch.cuda.synchronize()
    del junk
    torch.cuda.empty_cache()
    pbs = [vt.Problem(vt.make_params(280, 272, p=1, integration_order=4, perturb_grid=0.1), vt.vortex(epsilon=eps))
           for eps in (0.2, 0.4)]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert sum(pb.K for pb in pbs) // 64 > 16 * 2 * sms
    return vt.Batch(pbs), pbs


@pytest.mark.parametrize("what", ["autotune", "time_groups"])
def test_a_new_batch_is_tuned_and_timed(vt, what):
    b, pbs = new_batch(vt)
    dts = [1e-3, 8e-4]
    b.set_dt(dts)
    mapping = 1
    if what == "autotune":
        ((blocks, mapping),) = b.autotune(trials=1)
        assert 1 <= blocks <= 32
    else:
        (ms,) = b.time_groups(2)
        assert ms > 0
    for i, pb in enumerate(pbs):
        np.testing.assert_array_equal(b.download(i), pb.array("U0"))
    b.rk4(2)
    for i, pb in enumerate(pbs):
        s = vt.Solver(pb)
        s.stage_mapping = mapping
        s.rk4(dts[i], 2)
        np.testing.assert_array_equal(b.download(i), s.download())
        s.close()
    b.close()


def test_error_words_of_a_new_batch(vt):
    """The calls that only time the kernels leave no failure behind: the next
    step reports its own."""
    b, pbs = new_batch(vt)
    b.set_dt([1e-3, 1e-3])
    b.time_groups(1)
    U = pbs[1].array("U0")
    U[5, :, 0] = -1.0
    b.upload(1, U)
    with pytest.raises(vt.NonPhysicalState) as e:
        b.rk4(1)
    assert e.value.instance == 1 and e.value.step == 0 and e.value.stage == 0
    info, inst = vt.vt_error_info(), ctypes.c_int(-2)
    assert vt.lib().vt_batch_last_error(b._h, ctypes.byref(inst), ctypes.byref(info)) == 0
    assert inst.value == 1
    b.close()
