"""An inference pass is queued whole, without the host waiting for any of it: beside a training process, a queue that runs
dry between two convolutions gives the device away for a time slice."""
import pytest
import torch

from oracle import resnet_oracle as O
from sirius_b200 import ops
from sirius_b200._lib import SrtError
from sirius_b200.step import ResNetStep

pytestmark = pytest.mark.gpu
ARCH, B, IMG = "resnet50", 2, 64


@pytest.mark.parametrize("dtype", ["bf16", "f32"])
def test_forward_infer_returns_before_the_stream_reaches_it(dtype):
    step = ResNetStep(layers=O.LAYERS[ARCH], max_batch=B, image=IMG, dtype=dtype)
    step.load_state_dict(O.state_arrays(O.build_model(ARCH, 0)))
    (images, labels), = O.make_batches(B, 1, IMG)
    step.upload_batch(images, labels)
    for _ in range(2):
        step.forward_infer(B)
    want = step.logits(B)
    done = torch.cuda.Event()
    with torch.cuda.stream(torch.cuda.ExternalStream(step.stream)):
        torch.cuda._sleep(1_000_000_000)           # half a second of device time in front of the pass
        done.record()
    step.forward_infer(B)
    assert not done.query()                         # the whole pass is queued while the device is still in front of it
    assert (step.logits(B) == want).all()
    # the kill flag still ends a pass between units
    step.request_abort(True)
    with pytest.raises(SrtError, match="aborted"):
        step.forward_infer(B)
    step.request_abort(False)
    step.forward_infer(B)
    assert (step.logits(B) == want).all()
    assert ops.tc_status() == 0
    step.close()
