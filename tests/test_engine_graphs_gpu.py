"""Steps and inference passes replayed from graphs against the same engine without graphs: alternating staging slots, an
inference pass between feeding a batch and stepping on it, host batches of other label types, what the loss operator reads
changing between two inference passes."""
import pytest
import torch

from rembrandt_b200.api import build_replica
from rembrandt_b200.ops import native_ops as K
from rembrandt_b200.optim.sgd import Momentum, SgdOptConfig, StepSizeSchedule

pytestmark = pytest.mark.gpu


def _batches(n, batch, seed=3):
    g = torch.Generator().manual_seed(seed)
    return [(torch.randint(0, 256, (batch, 1, 28, 28), dtype=torch.uint8, generator=g).pin_memory(),
             torch.randint(0, 10, (batch,), dtype=torch.int32, generator=g).pin_memory()) for _ in range(n)]


def _pair(batch):
    return [build_replica("lenet", batch, use_graph=ug, seed=(5, 7)) for ug in (True, False)]


def test_steps_and_inference_passes_agree_with_eager():
    batch = 17
    seen = []
    for eng in _pair(batch):
        out = []
        for i, (x, y) in enumerate(_batches(9, batch)):
            eng.feed(x, y)
            if i % 3 == 1:                        # the staged batch must survive a validation pass
                vx, vy = _batches(1, batch, seed=50 + i)[0]
                out.append(eng.eval_batch(vx, vy.long() if i == 4 else vy))
            s = eng.step()
            if s is not None:
                out.append(s)
        out.append(eng.flush())
        eng.synchronize()
        seen.append((out, eng.net.params.clone()))
    (a, pa), (b, pb) = seen
    assert len(a) == len(b) == 12
    for (la, ca), (lb, cb) in zip(a, b):
        # the same kernels on the same data; sums of several CTAs may be added in another order
        assert abs(la - lb) < 1e-3 * max(1.0, abs(lb)) and abs(ca - cb) <= 1
    assert float((pa - pb).norm() / pb.norm()) < 1e-4


def test_an_inference_graph_follows_what_the_loss_reads():
    batch = 8
    graphed, eager = _pair(batch)
    # labels among the categories that the mask leaves: the loss is finite, and another mask gives another loss
    (x, y), (x2, y2) = [(x, (y // 2 * 2 + 1).pin_memory()) for x, y in _batches(2, batch)]
    masks = [None, torch.ones(batch, 10, dtype=torch.uint8), None]
    masks[1][:, ::2] = 0
    on_device = (x2.cuda(), y2.cuda())
    torch.cuda.synchronize()
    seen = {}
    for mask in masks:
        for eng in (graphed, eager):
            eng.net.loss_op.load_mask(mask)
        for data in ((x, y), (x2, y2), (x, y), on_device, (x2.clone(), y2.clone())):
            a, b = graphed.eval_batch(*data), eager.eval_batch(*data)
            assert abs(a[0] - b[0]) < 1e-3 * b[0] and a[1] == b[1]
            seen.setdefault(mask is None, []).append(a[0])
    # fewer categories to share the probability: every batch's loss is lower under the mask
    assert all(m < 0.99 * u for m, u in zip(seen[False], seen[True]))
    assert len(graphed._eval_graphs) == 2


@pytest.mark.parametrize("accum", [1, 3])
def test_a_changing_learning_rate_needs_no_further_capture(accum):
    """The rate changes before most iterations: the same parameters and statistics as without graphs, from at most one graph
    per staging slot and form of the step. With the sums of the convolutions and affine layers in one order: with several parts, added
    as they arrive, one value of this run lies so close to a rounding edge that any two runs of it, both without graphs too, part by
    2e-3 of the loss and 0.14 of an update in one case of six (24 runs of each kind)."""
    # small enough that training does not amplify rounding: at ten times these rates its loss grows, and differences with it
    batch, rates = 8, [2e-3, 2e-3, 1e-3, 4e-3, 4e-3, 5e-4, 0.0, 6e-3]
    seen = []
    with K.gemm_options(deterministic=1):
        for ug in (True, False):
            opt = SgdOptConfig(minibatch_size=batch * accum, step_size=StepSizeSchedule.constant(rates[0]),
                               momentum=Momentum.UPDATE_NESTEROV, mu=0.9, l2_reg_coef=1e-3, display_iters=0)
            eng = build_replica("lenet", batch, use_graph=ug, seed=(5, 7), opt=opt)
            assert eng.accum == accum
            stats, params, captured = [], [], 0
            for i, (x, y) in enumerate(_batches(len(rates) * accum, batch)):
                if i % accum == 0:
                    eng.set_lr(rates[i // accum])
                eng.feed(x, y)
                s = eng.step()
                stats += [s] if s is not None else []
                captured = max(captured, len(eng._graphs))
                if (i + 1) % accum == 0:
                    eng.synchronize()
                    params.append(eng.net.params.clone())
            stats.append(eng.flush())
            eng.synchronize()
            assert captured <= (2 if accum == 1 else 4) and (captured > 0) == ug
            seen.append((stats, params))
    (a, pa), (b, pb) = seen
    assert len(a) == len(b) == len(rates) * accum
    for (la, ca), (lb, cb) in zip(a, b):
        # fp32 sums over 8 images in another order: 4e-7 seen
        assert abs(la - lb) < 1e-5 * max(1.0, abs(lb)) and abs(ca - cb) <= 1
    for i in range(1, len(rates)):
        # Bias sums in another order leave 1e-8 of an update (seen). An update with the rate before it is off by
        # (1 + mu) * (difference of the rates) * |g|, against an update of at most (1 + mu) * rate * |g| + mu^2 * |v| with
        # |v| <= sum of mu^k * rate * |g|: a tenth and more wherever these rates change.
        assert float((pa[i] - pb[i]).norm()) < 1e-4 * float((pb[i] - pb[i - 1]).norm()), i
