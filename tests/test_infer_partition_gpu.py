"""Inference on an SM partition: the fp32 kernel splits its reductions over CTA pairs at most, the bf16 layers take the
persistent kernel instead of clusters (a partition may have no room for one), and the pass computes what it computes on the
whole device.

Bounds: fp32 sums in another order through 54 layers, 2e-5 in the 2-norm; in bf16 another order of the fp32 sums moves a
value to its neighbour here and there, which the layers behind it carry on: 1e-2 (the error of the pass against float64 is
4e-3)."""
import ctypes as C

import numpy as np
import pytest

from oracle import resnet_oracle as O
from sirius_b200 import _runtime, ops  # noqa: F401  (_runtime registers the partition's entry points)
from sirius_b200._lib import call
from sirius_b200.step import ResNetStep

pytestmark = pytest.mark.gpu
ARCH, IMG = "resnet50", 64
FULL = (C.c_uint64 * 3)(2 ** 64 - 1, 2 ** 64 - 1, 2 ** 64 - 1)


def _mask_of(n_sms):
    bits = (1 << n_sms) - 1
    return (C.c_uint64 * 3)(bits & (2 ** 64 - 1), (bits >> 64) & (2 ** 64 - 1), (bits >> 128) & (2 ** 64 - 1))


@pytest.mark.parametrize("batch", [1, 5])
@pytest.mark.parametrize("dtype,bound", [("f32", 2e-5), ("bf16", 1e-2)])
def test_forward_infer_on_a_partition(batch, dtype, bound):
    sms, n = (C.c_int * 32)(), C.c_int()
    call("srt_smp_partition_levels", 0, sms, 32, C.byref(n))
    levels = list(sms[:n.value])
    (images, labels), = O.make_batches(batch, 1, IMG)
    step = ResNetStep(layers=O.LAYERS[ARCH], max_batch=batch, image=IMG, dtype=dtype)
    step.load_state_dict(O.state_arrays(O.build_model(ARCH, 0)))
    step.upload_batch(images, labels)

    def logits():
        step.forward_infer(batch)
        return step.logits(batch).astype(np.float64)

    whole = logits()
    try:
        step.follow_sm_mask(True)
        for allowed in (levels[1], levels[-1]):
            call("srt_set_sm_mask", _mask_of(allowed))
            part = logits()
            assert step.current_sms() == allowed
            assert np.linalg.norm(part - whole) <= bound * np.linalg.norm(whole), allowed
        step.follow_sm_mask(False)
        assert (logits() == whole).all()
        assert ops.tc_status() == 0
        step.close()
    finally:
        call("srt_set_sm_mask", FULL)
