"""What this framework is measured on: training steps and inference passes of its own networks on one GPU.

A training pass is what a training program does per iteration: queue one pinned host batch (`StepEngine.feed`), run the
step (`StepEngine.step`: input kernel, forward, loss, backward, optimizer) and go on with the updated weights on the
current stream. An inference pass is one `StepEngine.eval_batch` of a host batch, as the validation loop calls it.
Networks, input shapes and batch sizes are those of the training tools (`rembrandt_b200/cli`) and of `bench.py`.
"""
from __future__ import annotations

import math

import torch

from rembrandt_b200.api import build_replica

# model: (channels, height = width, categories, largest training batch drawn, largest inference batch drawn,
#         multiply-adds per image forward, those of the first layer (it needs no data gradient), parameters)
MODELS = {
    "lenet": (1, 28, 10, 512, 1024, 2_293_000, 288_000, 431_080),
    "cifar": (3, 32, 10, 512, 1024, 10_732_160, 2_457_600, 85_098),
    "resnet20_cifar": (3, 32, 10, 512, 1024, 40_813_184, 442_368, 274_042),
    "go_policy_resnet": (32, 19, 361, 512, 512, 546_039_936, 13_307_904, 1_518_209),
    "nin": (3, 224, 1000, 128, 256, 1_100_188_800, 101_616_768, 7_595_176),
    "alexnet": (3, 227, 1000, 256, 256, 1_135_256_096, 105_415_200, 62_378_344),
    "resnet18": (3, 256, 1000, 64, 128, 1_814_073_344, 118_013_952, 11_699_112),
    "vgg_a_avgpool": (3, 256, 1000, 64, 64, 9_777_434_624, 113_246_208, 9_733_480),
}


def listed():
    return [
        # one digit through the smallest network: nothing but launches and latency
        {"name": "lenet_infer_1", "model": "lenet", "mode": "infer", "batch": 1},
        # the MNIST tool at its default batch: a step of very small kernels
        {"name": "lenet_train_64", "model": "lenet", "mode": "train", "batch": 64},
        # the CIFAR-10 tool's two networks at its default batch
        {"name": "cifar_train_128", "model": "cifar", "mode": "train", "batch": 128},
        {"name": "resnet20_cifar_train_128", "model": "resnet20_cifar", "mode": "train", "batch": 128},
        # the Go tool's residual network at its default batch (19 x 19 boards, 128 channels)
        {"name": "go_resnet_train_256", "model": "go_policy_resnet", "mode": "train", "batch": 256},
        # ImageNet-shaped training at the batch sizes the benchmark and the tools use
        {"name": "nin_train_64", "model": "nin", "mode": "train", "batch": 64},
        {"name": "alexnet_train_128", "model": "alexnet", "mode": "train", "batch": 128},
        {"name": "resnet18_train_32", "model": "resnet18", "mode": "train", "batch": 32},
        # a ragged batch: the last one of an epoch, no multiple of any tile
        {"name": "nin_train_37", "model": "nin", "mode": "train", "batch": 37},
        # validation passes: a whole validation batch of a plain and of a batch-normalised network
        {"name": "nin_infer_100", "model": "nin", "mode": "infer", "batch": 100},
        {"name": "resnet18_infer_50", "model": "resnet18", "mode": "infer", "batch": 50},
        # the largest: a VGG-A trunk on 256 x 256 images
        {"name": "vgg_a_avgpool_train_64", "model": "vgg_a_avgpool", "mode": "train", "batch": 64},
    ]


def draw(rng):
    """A training step or (one time in three) an inference pass of one of the networks, at any batch size up to the
    largest that is used in earnest; statistics over fewer than 8 images are not trained on."""
    model = rng.choice(sorted(MODELS))
    mode = "infer" if rng.random() < 1 / 3 else "train"
    most = MODELS[model][4 if mode == "infer" else 3]
    least = 1 if mode == "infer" else 8
    batch = int(round(math.exp(rng.uniform(math.log(least), math.log(most)))))
    return {"model": model, "mode": mode, "batch": batch}


def _images(gen, n, c, hw, planes):
    if planes:                           # bit planes of a board: stones are sparse, bytes are 0 or 255
        return (torch.rand((n, c, hw, hw), generator=gen, device="cuda") < 0.25).to(torch.uint8) * 255
    # photograph-like: a smooth field per channel with some grain on top
    low = torch.rand((n, c, 8, 8), generator=gen, device="cuda") * 255
    x = torch.nn.functional.interpolate(low, size=(hw, hw), mode="bilinear", align_corners=False)
    x = x + torch.randn((n, c, hw, hw), generator=gen, device="cuda") * 16
    return x.clamp_(0, 255).to(torch.uint8)


def prepare(case, seed):
    c, hw, classes = MODELS[case["model"]][:3]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = case["batch"]
    batches = []
    for _ in range(2):                   # a loader's pinned slots, used in turn
        images = _images(gen, n, c, hw, case["model"].startswith("go_"))
        labels = torch.randint(0, classes, (n,), generator=gen, device="cuda", dtype=torch.int32)
        batches.append((images.cpu().pin_memory(), labels.cpu().pin_memory()))
    engine = build_replica(case["model"], n, device="cuda", seed=(seed * 2 + 1, 0xC0FFEE))
    torch.cuda.synchronize()
    return {"case": case, "engine": engine, "batches": batches, "at": 0}


def run(state):
    engine, net = state["engine"], state["engine"].net
    images, labels = state["batches"][state["at"] % 2]
    state["at"] += 1
    loss_op = net.loss_op
    if state["case"]["mode"] == "infer":
        loss, _ = engine.eval_batch(images, labels)
        logits = loss_op.flat if loss_op.spatial else net.hidden_ops[-1].out
        return {"loss": loss, "logits": logits}
    stream = torch.cuda.current_stream()
    engine.compute_stream.wait_stream(stream)
    engine.feed(images, labels)
    engine.step()
    stream.wait_stream(engine.compute_stream)     # the program goes on with the new weights on its own stream
    return net.params                             # weights, biases, normalisation parameters and running statistics


def work(case):
    c, hw = MODELS[case["model"]][:2]
    macs, first, params = MODELS[case["model"]][5:]
    n = case["batch"]
    pixels = n * c * hw * hw
    if case["mode"] == "infer":
        # 16-bit weights
        return {"bytes": pixels + 2 * params, "flops": 2.0 * macs * n}
    # forward, data gradient (not for the first layer), weight gradient; 32-bit weights and momentum in and out
    return {"bytes": pixels + 16 * params, "flops": 2.0 * (3 * macs - first) * n}


# What a training step leaves open, measured on the updated parameters after one and two steps at 8 images: (relative
# error, largest error over the root mean square). Seen when the same step runs with its sums in other orders (other
# tile and reduction plans, one block per output) or with the convolutions on CUDA cores; the gradients are bf16 sums
# behind ReLUs, whose signs flip where a value rounds the other way, and deep normalised networks amplify that. It
# falls with the root of the batch. For the CIFAR network: one part in a hundred of an update, what bf16 gradients give.
STEP_NOISE = {
    "lenet": (2.2e-4, 7e-3),
    "cifar": (2.5e-6, 1e-3),
    "resnet20_cifar": (9.7e-4, 2e-2),
    "go_policy_resnet": (1.8e-3, 2.4e-2),
    "nin": (1.4e-6, 1.5e-3),
    "alexnet": (3.7e-5, 1e-2),
    "resnet18": (1.4e-3, 9e-2),
    "vgg_a_avgpool": (1.7e-4, 1.4e-2),
}
# the same for the bf16 logits of an inference pass, any batch size
LOGIT_NOISE = {"go_policy_resnet": 7.2e-3, "alexnet": 4.3e-3}


def tolerance(case):
    """Four times what was seen."""
    if case["mode"] == "infer":
        return {"rel": 4 * LOGIT_NOISE.get(case["model"], 3e-3), "max": 0.1}
    rel, largest = STEP_NOISE[case["model"]]
    scale = 4 * math.sqrt(8 / case["batch"])
    return {"rel": rel * scale, "max": largest * scale}
