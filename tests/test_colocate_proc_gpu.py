"""A colocated run that fails leaves nothing behind: the trainer it launched has ended, the pool and the channel are gone, and
the next run in the same process works."""
import ctypes as C
import os

import pytest
import torch

from sirius_b200 import _lib, colocate_proc
from sirius_b200.server import Controller

pytestmark = pytest.mark.gpu


def test_a_run_after_a_failed_run(monkeypatch):
    pytest.importorskip("torchvision")
    for name in [n for n in os.environ if n.startswith(("COLTRAIN_", "SIRIUS_B200_COMM", "SIRIUS_B200_DIST"))]:
        monkeypatch.delenv(name)                       # what other tests left for trainers of their own
    monkeypatch.setenv("SIRIUS_PORT", "0")             # set by the run; the old value comes back afterwards
    pids = []
    real_pid, real_wait = Controller.set_train_pid, Controller.wait_colocate_adjust_done
    monkeypatch.setattr(Controller, "set_train_pid", lambda self, pid: (pids.append(pid), real_pid(self, pid)))

    def lost(self, device, cid, timeout_ms=-1):
        real_wait(self, device, cid, timeout_ms)       # the trainer has answered: nothing of the handover is in flight
        raise RuntimeError("the server loses its request")

    monkeypatch.setattr(Controller, "wait_colocate_adjust_done", lost)
    with pytest.raises(RuntimeError, match="loses its request"):
        colocate_proc.run(duration_s=2.0, rate=20.0)
    assert len(pids) == 1 and not colocate_proc._CHILDREN
    with pytest.raises(ProcessLookupError):
        os.kill(pids[0], 0)
    with pytest.raises(_lib.SrtError):
        _lib.call("srt_pool_default", 0, C.byref(C.c_void_p()))
    monkeypatch.setattr(Controller, "wait_colocate_adjust_done", real_wait)
    out = colocate_proc.run(duration_s=2.0, rate=20.0)
    assert out["trainer_exit_status"] == 0 and out["final_loss_finite"] and out["requests"] > 0
    assert out["handovers"] == out["requests"]
    torch.cuda.synchronize()
