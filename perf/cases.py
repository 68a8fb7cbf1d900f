"""The work that is timed when a change to this framework is judged by its speed.

Every case is one pass through the handles a user's program holds: the training steps of the four model families
(`ResNetStep`, `SwinStep`, `Gpt2Step`, `Qwen2Step`: forward, backward, optimizer, loss) and the forward passes of the
inference worker that runs beside them (`ResNetStep.forward_infer`, `DistilBertInfer`). Weights are random draws of
the usual initialisation and inputs are N(0,1) images or uniform token ids, as in the benchmark.
"""
import math

import numpy as np
import torch

from sirius_b200 import _lib
from sirius_b200.bert_infer import DISTILBERT_BASE, DistilBertInfer
from sirius_b200.gpt2_step import Gpt2Step
from sirius_b200.qwen2_step import QWEN2_05B, Qwen2Step
from sirius_b200.step import RESNET_LAYERS, ResNetStep
from sirius_b200.swin_step import SWIN_B, SwinStep

# Every training case is the work of one rank of a data-parallel job: srt_ddp_create() switches the CTA-pair
# filter-gradient kernel off for such a process, and so does this file, for all cases alike.
_lib.lib().srt_conv_wgrad_pairs(0)

WARM_UP_LR = 1e-6   # an early step of a warm-up: repeated passes on the same batch stay near the weights that were drawn
GPT2_SMALL = dict(n_layer=12, n_head=12, d_model=768, vocab=50257, ctx=1024)


def listed():
    return [
        # the request of the inference worker: one sentence, answered while training runs; launches and latency count
        {"name": "distilbert_b1_s128", "kind": "bert", "batch": 1, "seq": 128},
        # a few queued requests of a ragged length answered together
        {"name": "distilbert_b6_s328", "kind": "bert", "batch": 6, "seq": 328},
        # the other request of the inference worker: one image, from host memory to host memory
        {"name": "resnet152_infer_b1", "kind": "resnet_infer", "arch": "resnet152", "batch": 1, "dtype": "bf16"},
        # evaluation of a ragged last batch in the exact fp32 mode
        {"name": "resnet50_infer_f32_b5", "kind": "resnet_infer", "arch": "resnet50", "batch": 5, "dtype": "f32"},
        # the headline training step
        {"name": "resnet152_train_b64", "kind": "resnet_train", "arch": "resnet152", "batch": 64, "max_batch": 64},
        # a micro-batch of the executor built for 32 after the inference side has taken part of its memory
        {"name": "resnet50_train_b19_of_32", "kind": "resnet_train", "arch": "resnet50", "batch": 19, "max_batch": 32},
        # the image transformer at its per-GPU batch, and at the odd micro-batch of a shrunk job
        {"name": "swin_b_train_b32", "kind": "swin", "batch": 32},
        {"name": "swin_b_train_b7", "kind": "swin", "batch": 7},
        # decoder training at the benchmark's batch, and a few short sequences whose length is no multiple of a tile
        {"name": "gpt2_train_8x1024", "kind": "gpt2", "batch": 8, "seq": 1024},
        {"name": "gpt2_train_3x328", "kind": "gpt2", "batch": 3, "seq": 328},
        # grouped-query decoder: the largest step (vocabulary of 151 936), and one short sequence
        {"name": "qwen2_train_4x2048", "kind": "qwen2", "batch": 4, "seq": 2048},
        {"name": "qwen2_train_1x640", "kind": "qwen2", "batch": 1, "seq": 640},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bert", "bert", "resnet_infer", "resnet_train", "swin", "gpt2", "gpt2", "qwen2"])
    if kind == "bert":
        return {"kind": kind, "batch": _log_int(rng, 1, 16), "seq": 8 * _log_int(rng, 2, 64)}
    if kind == "resnet_infer":
        dtype = rng.choice(["bf16", "bf16", "f32"])
        return {"kind": kind, "arch": rng.choice(sorted(RESNET_LAYERS)), "batch": _log_int(rng, 1, 8 if dtype == "f32" else 32),
                "dtype": dtype}
    if kind == "resnet_train":
        batch = _log_int(rng, 2, 64)
        return {"kind": kind, "arch": rng.choice(sorted(RESNET_LAYERS)), "batch": batch, "max_batch": min(64, batch + rng.choice([0, 0, 5, 16]))}
    if kind == "swin":
        return {"kind": kind, "batch": _log_int(rng, 1, 32)}
    if kind == "gpt2":
        return {"kind": kind, "batch": _log_int(rng, 1, 8), "seq": 8 * _log_int(rng, 8, 128)}
    return {"kind": kind, "batch": _log_int(rng, 1, 4), "seq": 128 * _log_int(rng, 1, 16)}


def _weights(params, gen, std=None, residual_gain=1.0):
    """Initial values by name: norm scales 1, biases and running means 0, running variances 1, matrices and filters
    N(0, std); std None is Kaiming's fan-out rule. residual_gain: scale of the norm that ends a residual branch."""
    sd = {}
    for name, info in params.items():
        shape = tuple(info.shape if hasattr(info, "shape") else info[1])
        if len(shape) > 1:
            s = std if std is not None else math.sqrt(2.0 / (shape[0] * math.prod(shape[2:])))
            t = torch.empty(shape, device="cuda").normal_(0.0, s, generator=gen)
        elif name.endswith("running_mean") or name.endswith("bias"):
            t = torch.zeros(shape, device="cuda")
        else:
            t = torch.full(shape, residual_gain if name.endswith("bn3.weight") else 1.0, device="cuda")
        sd[name] = t
    return sd


class _Gradient:
    """The flat gradient buffer of a step, for torch.as_tensor; the tensor keeps the step alive through it."""

    def __init__(self, step):
        ptr, n = step.grad_buffer()
        self.step = step
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f4", "data": (ptr, False), "version": 2}


def _host(t):
    """Data as a loader hands it over: host memory, pinned."""
    return t.cpu().pin_memory()


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, batch = case["kind"], case["batch"]
    state = {"kind": kind, "batch": batch}
    if kind == "bert":
        step = DistilBertInfer(**DISTILBERT_BASE, max_batch=batch, seq=case["seq"])
        step.load_state_dict(_weights(step.params, gen, std=0.02))
    elif kind in ("resnet_infer", "resnet_train"):
        train = kind == "resnet_train"
        # lr 0: the first step of a linear warm-up. Repeated passes see the weights that were drawn: one weight that
        # rounds to another bf16 value is enough to give this network, at its initialisation, another gradient.
        step = ResNetStep(arch=case["arch"], max_batch=case.get("max_batch", batch), dtype=case.get("dtype", "bf16"), lr=0.0)
        step.load_state_dict(_weights(step.params, gen, residual_gain=1.0 if train else 0.25))
    elif kind == "swin":
        step = SwinStep(**SWIN_B, max_batch=batch, lr=WARM_UP_LR)
        step.load_state_dict(_weights(step.params, gen, std=0.02))
    elif kind == "gpt2":
        step = Gpt2Step(**GPT2_SMALL, max_batch=batch, seq=case["seq"], lr=WARM_UP_LR)
        step.load_state_dict(_weights(step.params, gen, std=0.02))
    else:
        step = Qwen2Step(**QWEN2_05B, max_batch=batch, seq=case["seq"], lr=WARM_UP_LR)
        step.load_state_dict(_weights(step.params, gen, std=0.02))
    if kind in ("bert", "gpt2", "qwen2"):
        ids = torch.randint(0, step.vocab, (batch, case["seq"]), device="cuda", generator=gen, dtype=torch.int32)
        state["ids"] = ids.cpu().numpy()
    else:
        images = torch.empty((batch, 3, 224, 224), device="cuda").normal_(generator=gen)
        labels = torch.randint(0, 1000, (batch,), device="cuda", generator=gen, dtype=torch.int64)
        # the ResNet trainer reads batches that a loader has put on the GPU; the others take host batches
        on_gpu = kind == "resnet_train"
        state["images"], state["labels"] = (images, labels) if on_gpu else (_host(images), _host(labels))
    if kind not in ("bert", "resnet_infer"):
        state["grad"] = torch.as_tensor(_Gradient(step), device="cuda")
    torch.cuda.synchronize()
    state["step"] = step
    return state


def run(state):
    kind, step, batch = state["kind"], state["step"], state["batch"]
    if kind == "bert":
        step.upload_tokens(state["ids"])
        step.forward()
        return step.output()
    if kind == "resnet_infer":
        step.upload_batch(state["images"], state["labels"])
        step.forward_infer(batch)
        return step.logits(batch)
    if kind == "resnet_train":
        step.set_batch_device(state["images"].data_ptr(), state["labels"].data_ptr(), batch)
        step.forward_backward(batch)
        step.optimizer_step()
        return {"loss": step.loss(), "grad": state["grad"]}
    if kind == "swin":
        return {"loss": step.train_step(state["images"], state["labels"]), "grad": state["grad"]}
    return {"loss": step.train_step(state["ids"]), "grad": state["grad"]}


def _resnet_macs(arch):
    """(multiply-adds of one image, parameters)"""
    macs, params, hw, cin = 112 * 112 * 64 * 147, 64 * 147 + 128, 56, 64
    for stage, (blocks, width) in enumerate(zip(RESNET_LAYERS[arch], (64, 128, 256, 512))):
        for b in range(blocks):
            stride = 2 if b == 0 and stage > 0 else 1
            out = hw // stride
            weights = cin * width, 9 * width * width, 4 * width * width
            macs += hw * hw * weights[0] + out * out * (weights[1] + weights[2])
            params += sum(weights) + 2 * (width + width + 4 * width)
            if b == 0:
                macs += out * out * cin * 4 * width
                params += cin * 4 * width + 8 * width
            cin, hw = 4 * width, out
    return macs + cin * 1000, params + cin * 1000 + 1000


def _swin_macs():
    tokens, macs, params, c = 56 * 56, 56 * 56 * 48 * 128, 48 * 128, 128
    for stage, depth in enumerate(SWIN_B["depths"]):
        macs += depth * tokens * (12 * c * c + 2 * 49 * c)
        params += depth * (12 * c * c + 13 * c + 169 * SWIN_B["heads"][stage])
        if stage < 3:
            tokens //= 4
            macs += tokens * 8 * c * c
            params += 8 * c * c + 8 * c
            c *= 2
    return macs + c * 1000, params + c * 1000


def _lm(case):
    """(multiply-adds, parameters) of one forward pass; attention counts the causal half."""
    b, s = case["batch"], case["seq"]
    if case["kind"] == "gpt2":
        c, layers, vocab = GPT2_SMALL["d_model"], GPT2_SMALL["n_layer"], GPT2_SMALL["vocab"]
        lin, att, tables = 12 * c * c, c, (vocab + GPT2_SMALL["ctx"]) * c
    else:
        c, layers, vocab = QWEN2_05B["hidden"], QWEN2_05B["n_layer"], QWEN2_05B["vocab"]
        lin, att, tables = c * (2 * c + 2 * 128) + 3 * c * QWEN2_05B["intermediate"], c, vocab * c
    return b * s * (layers * (lin + att * s) + vocab * c), layers * lin + tables


def work(case):
    """Bytes: what is read and written once whatever the implementation (inputs, results, weights; a training step also
    writes its gradient and updates fp32 weights and optimizer state). Operations: the model's multiply-adds, three
    times the forward pass for a training step."""
    kind, b = case["kind"], case["batch"]
    if kind == "bert":
        c, f, layers, s = DISTILBERT_BASE["dim"], DISTILBERT_BASE["hidden_dim"], DISTILBERT_BASE["n_layer"], case["seq"]
        lin = 4 * c * c + 2 * c * f
        return {"bytes": 2 * layers * lin + b * s * (4 + 2 * c + 4 * c), "flops": 2 * b * s * layers * (lin + 2 * s * c)}
    if kind == "resnet_infer":
        macs, params = _resnet_macs(case["arch"])
        return {"bytes": params * (4 if case["dtype"] == "f32" else 2) + b * 3 * 224 * 224 * 4 + b * 4000, "flops": 2 * b * macs}
    if kind == "resnet_train":
        macs, params = _resnet_macs(case["arch"])
        return {"bytes": 20 * params + b * 3 * 224 * 224 * 4, "flops": 6 * b * macs}   # SGD: P and M read, P, M and G written
    if kind == "swin":
        macs, params = _swin_macs()
        return {"bytes": 28 * params + b * 3 * 224 * 224 * 4, "flops": 6 * b * macs}   # AdamW: two moments
    macs, params = _lm(case)
    return {"bytes": 28 * params + 4 * b * case["seq"], "flops": 6 * macs}


def tolerance(case):
    """Measured: gradients of GPT-2 small against PyTorch in fp32 and under bf16 autocast differ by 1.1e-2 to 1.4e-2
    (2-norm) and by up to 1.9 times the root mean square in single entries (norm and bias gradients, sums over all
    tokens), as the two PyTorch runs do from each other. fp32 inference differs by the order of fp32 sums."""
    if case.get("dtype") == "f32":
        return {"rel": 2e-5}
    return {"rel": 0.02} if case["kind"] in ("bert", "resnet_infer") else {"rel": 0.03, "max": 0.99}
