"""L1 adjusts that no killed batch answers: one that arrives while the optimizer runs (the trainer looks again when the
critical section ends), and one that arrives while the trainer waits at target batch size zero. Either way the trainer has
given memory away, so from the reply on it keeps to the announced batch size, the next adjust is a request like any other
(not taken for one during the recovery of a killed batch, which is answered on the spot), and kInferExit lets the batch
grow back (pytorch/torch_col/csrc/control_stub.cc:423-593, pytorch/torch_col/colocate_ctrl.py:325-358)."""
import multiprocessing as mp
import os
import time
import uuid

import pytest

from sirius_b200.torch_col._C import CtrlEvent

BS, GLOBAL_BS, DS = 8, 32, 64


def _until(cond, what, limit_s=20.0):
    t0 = time.time()
    while not cond():
        if time.time() - t0 > limit_s:
            raise TimeoutError(what)
        time.sleep(0.001)


class _Memory:
    """Stands in for a step object: the batch size its activation set is sized for."""

    def __init__(self):
        self.held = 0

    def synchronize(self):
        pass

    def shrink_activations(self, b):
        self.held = min(self.held, b)
        return 1

    def release_activations(self):
        self.held = 0
        return 1


def _trainer(scenario, comm_name, dist_name, q):
    os.environ.update({
        "COLTRAIN_MODE": "colocate-l1", "COLTRAIN_HOOK_MODE": "xsched-sync2", "COLTRAIN_USE_XSCHED": "1",
        "COLTRAIN_HAS_INFER_SERVER": "1", "SIRIUS_B200_COMM_NAME": comm_name, "SIRIUS_B200_DIST_NAME": dist_name})
    import threading

    import torch
    from sirius_b200 import torch_col as tc
    torch.set_num_threads(1)
    srv = tc.DebugServer(1, comm_name)
    tc.setup_colocate_training(0, 1, False, False)
    model = torch.nn.Sequential(torch.nn.Flatten(), torch.nn.Linear(3 * 4 * 4, 10))
    opt = torch.optim.SGD(model.parameters(), 0.05)
    crit = torch.nn.CrossEntropyLoss()
    ctrl = tc.create_colocate_ctrl(tc.get_colocate_train_mode(), tc.get_colocate_ctrl_hook_mode(), 1, BS, stub_poll_ms=2)
    mem = _Memory()
    tc.set_train_step(mem)
    ds, mgr = tc.init_dynamic_batch(DS, tc.DatasetType.VISION, tc.VisionDatasetConfig((3, 4, 4), 10), BS,
                                    global_batch_size=GLOBAL_BS, enable_grad_accumulate=True, checkpoint_micro_batch=True)
    tc.init_train_info(BS, BS, "resnet152")
    tc.util.initialize_sgd_optimizer(model, opt)
    acc = tc.GradAccumulator(model)
    stub = ctrl._stub
    begin, end = stub.StepsNoInteruptBegin, stub.StepsNoInteruptEnd
    plan = {"at": 2 if scenario == "micro" else 4, "n": 0, "cid": None}
    sizes, log = [], []
    replied = lambda cid: any(m.id == cid for _, m in srv.events(CtrlEvent.kColocateAdjustL1Done))

    def begin_with_adjust():
        begin()
        plan["n"] += 1
        if scenario in ("micro", "last") and plan["n"] == plan["at"]:
            plan["cid"] = srv.colocate_l1([4])

    def end_after_command():
        end()
        if scenario != "zero" and plan["n"] == plan["at"]:         # the command is in before the trainer looks
            _until(lambda: stub.cmd == CtrlEvent.kColocateAdjustL1, "the control thread never took the adjust in")

    stub.StepsNoInteruptBegin, stub.StepsNoInteruptEnd = begin_with_adjust, end_after_command

    def iter_train_fn(batch):
        mem.held = max(mem.held, len(batch))
        sizes.append(len(batch))
        script(len(sizes))
        ctrl.check_kill("fwd")
        loss = mgr.scale_loss(batch, crit(model(batch["images"]), batch["labels"]))
        loss.backward()
        ctrl.check_kill("bwd")
        mgr.optimizer_step(batch, opt, grad_accumulator=acc)
        return loss.item()

    phase = {"k": 0}

    def script(n):
        """What the server does next, called inside a micro-batch."""
        if scenario == "zero":
            if n == 2:                                             # kill: nothing may stay
                plan["cid"] = srv.colocate_l1([0])
                _until(lambda: stub.cmd == CtrlEvent.kColocateAdjustL1, "first adjust not taken in")
                threading.Thread(target=server_while_waiting, daemon=True).start()
            return
        if plan["cid"] is None or plan["n"] < plan["at"]:
            return
        phase["k"] += 1
        if phase["k"] == 2:                                        # a later request that needs more
            plan["cid2"] = srv.colocate_l1([2])
            _until(lambda: stub.cmd == CtrlEvent.kColocateAdjustL1 or replied(plan["cid2"]), "second adjust not taken in")
            log.append("asked" if stub.cmd == CtrlEvent.kColocateAdjustL1 else "answered at once")
        elif phase["k"] == 4:
            srv.infer_exit([BS])
            _until(lambda: srv.comm.get_field(0, 5) == BS, "kInferExit was ignored", 5.0)

    def server_while_waiting():
        _until(lambda: replied(plan["cid"]), "first adjust not answered")
        time.sleep(0.05)                                           # the trainer waits at batch size zero
        cid = srv.colocate_l1([0])
        _until(lambda: replied(cid), "second adjust not answered")
        srv.infer_exit([BS])
        for _ in range(2000):
            if srv.comm.get_field(0, 5) == BS:
                return
            time.sleep(0.001)
        log.append("kInferExit was ignored")
        os._exit(3)                                                # the trainer would wait for good

    trainer = tc.Trainer(model, iter_train_fn)
    ctrl.train_start()
    for e in range(2):
        trainer.train_one_epoch(e)
    ctrl.train_end()
    dones = [m.id for _, m in srv.events(CtrlEvent.kColocateAdjustL1Done)]
    q.put((sizes, log, dones, plan.get("cid"), plan.get("cid2"), len(ctrl.adjust_log)))
    tc.cleanup_colocate_training(False)
    srv.close()


@pytest.mark.timeout(120)
@pytest.mark.parametrize("scenario", ["micro", "last", "zero"])
def test_adjust_that_no_killed_batch_answers(scenario):
    tag = f"{os.getpid()}_{uuid.uuid4().hex[:6]}"
    ctx = mp.get_context("spawn")
    q = ctx.Queue()
    p = ctx.Process(target=_trainer, args=(scenario, f"srt_aob_comm_{tag}", f"srt_aob_dist_{tag}", q))
    p.start()
    try:
        p.join(90)
        assert p.exitcode == 0
        sizes, log, dones, cid, cid2, adjusts = q.get(timeout=10)
    finally:
        if p.is_alive():
            p.terminate()
    assert cid in dones
    if scenario == "zero":
        assert adjusts == 2 and not log and sizes[2] == BS         # back at the full batch after kInferExit
        return
    k = 2 if scenario == "micro" else 4                            # micro-batches before the reply
    assert sizes[:k] == [BS] * k
    assert max(sizes[k:k + 2]) <= 4, sizes                         # the memory above four samples belongs to inference
    assert log == ["asked"] and cid2 in dones and adjusts == 2     # the second request is served, by a smaller set
    assert max(sizes[k + 2:k + 4]) <= 2, sizes
    assert BS in sizes[k + 4:]                                     # and given back after kInferExit
