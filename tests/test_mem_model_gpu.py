"""The memory line that the TrainAdjuster uses by default, against the device memory that the executors take. The adjuster
divides what inference needs by the slope: half the slope frees half of the memory asked for, twice the slope twice."""
import ctypes as C
import gc

import pytest
import torch

from sirius_b200 import mem_model
from sirius_b200._lib import call

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", ["resnet152", "swin_b", "gpt2", "qwen"])
def test_measured_table_is_what_the_executor_takes(model):
    gc.collect()
    torch.cuda.empty_cache()
    got = mem_model.measure((model,))[model]
    base, slope = C.c_double(), C.c_double()
    call("srt_adjuster_model_mem_param_measured", model.encode(), C.byref(base), C.byref(slope))
    # 10 %: far below what a forgotten change of layout moves it by, above the 2 MB granules of the device and the pages
    # of the kernels loaded meanwhile (both below 2 % of the smallest executor)
    for batch, mb in zip(got["batches"], got["device_mb"]):
        assert abs(base.value + slope.value * batch - mb) <= 0.1 * mb, (got, base.value, slope.value)
    assert abs(slope.value - got["slope_mb"]) <= 0.1 * got["slope_mb"], (got, slope.value)
