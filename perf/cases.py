"""The work a user of this framework has it do, as cases that can be timed and compared.

Every case drives `StageRuntime` and the weight-stashing optimizers the way a training script does: minibatches come
from a loader of pinned host tensors, `run()` is one training step (`run_forward`, `zero_grad`, `load_old_params`,
`run_backward`, `load_new_params`, `step`), one double-buffered macrobatch of two microbatches (the GPT decoder), one
forward-only validation minibatch, or one 1F1B run of a few minibatches over a pipeline whose stages share the GPU.

Networks and their settings are the repository's own benchmark configurations:

  vgg16     224 x 224 images, 1000 classes, SGD momentum 0.9 weight decay 5e-4, dropout 0.5
  resnet50  224 x 224 images, 1000 classes, BatchNorm in training mode, SGD momentum 0.9 weight decay 1e-4
  gnmt      8 + 8 LSTM layers, hidden 1024, vocabulary 32320, dropout 0.2, label smoothing 0.1, Adam
  gpt       24 layers, hidden 1024, 16 heads, vocabulary 50257, dropout 0.1, Adam, two weight versions

The learning rates are those a warm-up starts from.  (At full rate the first steps of a freshly initialised network
amplify a last-bit difference into another trajectory, and two runs of one program could not be compared.)
"""
import math

import torch

from pipedream_b200 import adam, communication, gnmt_blocks, layers, runtime, schedule, sgd, stages

_POOL = 2                # minibatches a state's loader cycles over
_GPT_SEQ = 512           # rows of the decoder's position table: the longest sequence it takes
_LR = {"vgg16": 1e-5, "resnet50": 1e-5, "gnmt": 1e-6, "gpt": 1e-6}


def listed():
    return [
        # The headline configuration: the per-replica batch of the hybrid VGG-16 partitioning, 16-bit.
        {"name": "vgg16_train_64", "net": "vgg16", "mode": "train", "dtype": "bf16", "batch": 64},
        # A training script run without its 16-bit option: fp32 throughout, the batch of the two-rank CPU configuration.
        {"name": "vgg16_train_8_fp32", "net": "vgg16", "mode": "train", "dtype": "fp32", "batch": 8},
        # Validation between epochs: forward only, a batch of 100.
        {"name": "vgg16_eval_100", "net": "vgg16", "mode": "eval", "dtype": "bf16", "batch": 100},
        # ResNet-50 training at the benchmark's batch.
        {"name": "resnet50_train_64", "net": "resnet50", "mode": "train", "dtype": "bf16", "batch": 64},
        # The last, incomplete minibatch of an fp32 epoch.
        {"name": "resnet50_train_7_fp32", "net": "resnet50", "mode": "train", "dtype": "fp32", "batch": 7},
        # The smallest call there is: one image through the network, where launches and host work are everything.
        {"name": "resnet50_eval_1", "net": "resnet50", "mode": "eval", "dtype": "bf16", "batch": 1},
        # 1F1B with weight stashing: a straight pipeline of four stages (4, 3, 2 and 1 weight versions) in one process.
        {"name": "resnet50_pipeline_32", "net": "resnet50", "mode": "pipeline", "dtype": "bf16", "batch": 32, "stages": 4,
         "minibatches": 8},
        # Translation at the benchmark's batch and sentence lengths.
        {"name": "gnmt_train_128", "net": "gnmt", "mode": "train", "dtype": "bf16", "batch": 128, "shortest": 20,
         "longest": 50},
        # A ragged bucket of short sentences.
        {"name": "gnmt_train_21", "net": "gnmt", "mode": "train", "dtype": "bf16", "batch": 21, "shortest": 3,
         "longest": 27},
        # Validation loss of the translation model.
        {"name": "gnmt_eval_64", "net": "gnmt", "mode": "eval", "dtype": "bf16", "batch": 64, "shortest": 20,
         "longest": 50},
        # The 2BW decoder: microbatches of eight full sequences, one optimizer step for two of them.
        {"name": "gpt_train_8x512", "net": "gpt", "mode": "train", "dtype": "bf16", "batch": 8, "tokens": 512},
        # Short sequences of a length that is no multiple of a tile, as when fine-tuning on documents.
        {"name": "gpt_train_2x200", "net": "gpt", "mode": "train", "dtype": "bf16", "batch": 2, "tokens": 200},
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, spread evenly over its logarithm."""
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    net = rng.choice(["vgg16", "resnet50", "gnmt", "gpt"])
    mode = rng.choice(["train", "train", "eval"] + (["pipeline"] if net in ("vgg16", "resnet50") else []))
    # fp32 is what the image drivers run by default; the sequence models are trained in 16 bits
    dtype = "fp32" if net in ("vgg16", "resnet50") and mode != "pipeline" and rng.random() < 0.3 else "bf16"
    case = {"net": net, "mode": mode, "dtype": dtype}
    if net == "gpt":
        case["batch"] = _spread(rng, 1, 8)
        case["tokens"] = _spread(rng, 40, _GPT_SEQ)
    elif net == "gnmt":
        case["batch"] = _spread(rng, 4, 128)
        case["longest"] = rng.randint(12, 50)
        case["shortest"] = rng.randint(3, case["longest"] // 2)
    else:
        largest = {"train": 64, "eval": 128, "pipeline": 32}[mode] if dtype == "bf16" else 8
        case["batch"] = _spread(rng, 4 if net == "resnet50" and mode != "eval" else 1, largest)
        if mode == "pipeline":
            case["stages"] = 2 if net == "vgg16" else rng.randint(2, 8)
            case["minibatches"] = rng.randint(case["stages"], 8)
    return case


# ------------------------------------------------------------------------------------------------- state
class _Cycle:
    """An endless loader over a few minibatches."""

    def __init__(self, items):
        self.items = items

    def __iter__(self):
        while True:
            yield from self.items


def _sentences(case, seed):
    """Minibatches in the translation loader's format, sorted by source length.  As in a shuffled epoch the longest
    sentence, and with it every tensor's shape, changes from one minibatch to the next."""
    batch, items = case["batch"], []
    g = torch.Generator().manual_seed(1000 * seed + 1)
    zipf = torch.arange(1, 31997, dtype=torch.float32).pow(-1.1)
    for k in range(4):
        sides = []
        for longest in (case["longest"] - k, case["longest"] - 2 * k % 3):
            lengths = torch.randint(case["shortest"], longest + 1, (batch,), generator=g)
            lengths[int(torch.randint(0, batch, (1,), generator=g))] = longest
            ids = torch.multinomial(zipf, longest * batch, replacement=True, generator=g).view(longest, batch) + 4
            ids[0] = stages.SyntheticTranslation.BOS
            ids[lengths - 1, torch.arange(batch)] = stages.SyntheticTranslation.EOS
            ids[torch.arange(longest).unsqueeze(1) >= lengths] = stages.SyntheticTranslation.PAD
            sides.append((ids, lengths))
        order = torch.argsort(sides[0][1], descending=True, stable=True)
        items.append(tuple((ids[:, order].pin_memory(), lengths[order].tolist()) for ids, lengths in sides))
    return items


def _loader(case, seed):
    net, batch = case["net"], case["batch"]
    if net == "gnmt":
        items = _sentences(case, seed)
    elif net == "gpt":
        items = [(x.pin_memory(), y.pin_memory()) for x, y in stages.SyntheticTokens(
            batch, _POOL, seq_len=case["tokens"], seed=1000 * seed + 1)]
    else:
        g = torch.Generator(device="cuda").manual_seed(1000 * seed + 1)
        items = []
        for _ in range(_POOL):
            x = torch.randn(batch, 3, 224, 224, device="cuda", generator=g)
            y = torch.randint(0, 1000, (batch,), device="cuda", generator=g)
            items.append((x.cpu().pin_memory(), y.cpu().pin_memory()))
    return _Cycle(items)


def _package(case):
    net, n = case["net"], case.get("stages", 1)
    if net == "vgg16":
        return stages.vgg16("gpus=8" if n == 2 else "gpus=1"), torch.nn.CrossEntropyLoss()
    if net == "resnet50":
        return stages.resnet50(n), torch.nn.CrossEntropyLoss()
    if net == "gpt":
        return stages.gpt2(1, seq_len=_GPT_SEQ), torch.nn.CrossEntropyLoss()
    return stages.gnmt_large(), gnmt_blocks.LabelSmoothing(0, 0.1)


def _shapes(case, pkg):
    """Boundary tensors of the stages and their types, as a driver script's dry run finds them."""
    batch, real = case["batch"], torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
    if case["mode"] != "pipeline":
        return {}, {}
    if case["net"] == "vgg16":
        shapes = {"input0": (batch, 3, 224, 224), "target": (batch,), "out0": (batch, 512, 28, 28), "out1": (batch, 1000)}
    else:
        shapes = pkg.boundary_shapes(batch)
    return shapes, {k: torch.int64 if k in ("input0", "target") else real for k in shapes}


def _worker(case, seed, rank=None):
    """The runtime of one stage (rank None: of the whole network) and its optimizer."""
    net, bf16 = case["net"], case["dtype"] == "bf16"
    torch.manual_seed(seed)
    with torch.device("cuda"):
        pkg, criterion = _package(case)
        model = pkg.model(criterion)
    for stage, _, _ in model:
        for m in stage.modules():
            if isinstance(m, stages.Bottleneck):      # residual branches that start small, as is usual
                torch.nn.init.constant_(m.bn3.weight, 0.1)
    shapes, dtypes = _shapes(case, pkg)
    conf = {"module_to_stage_map": None, "stage_to_rank_map": None, "stage_to_depth_map": None}
    if rank is not None:
        conf.update({k: pkg.conf[k] for k in ("module_to_stage_map", "stage_to_rank_map")})
    inputs = {"input0": 0, "input1": 0, "input2": 0} if net == "gnmt" else {"input": 0}
    targets = {"target", "target_length"} if net == "gnmt" else {"target"}
    r = runtime.StageRuntime(
        model=model, distributed_backend=None if rank is None else communication.LOCAL, fp16=bf16, loss_scale=1,
        training_tensor_shapes=dict(shapes), eval_tensor_shapes=dict(shapes), training_tensor_dtypes=dtypes,
        inputs_module_destinations=inputs, target_tensor_names=targets, configuration_maps=conf, master_addr=None,
        rank=rank, local_rank=0, num_ranks_in_server=1, verbose_freq=0,
        model_type=runtime.TRANSLATION if net == "gnmt" else runtime.IMAGE_CLASSIFICATION)
    # dropout masks that depend on the seed alone, not on how many modules the process has built before
    k = 0
    for m in r.modules():
        for sub in m.modules():
            if isinstance(sub, layers.NativeDropout):
                k += 1
                sub.seed = 104729 * seed + 1000 * (rank or 0) + k
    if case["mode"] == "eval":
        return r, None
    args = (r.modules(), r.master_parameters, r.model_parameters, 1)
    if net == "gnmt":
        opt = adam.AdamWithWeightStashing(*args, num_versions=1, lr=_LR["gnmt"], weight_decay=1e-4)
    elif net == "gpt":
        opt = adam.AdamWithWeightStashing(*args, num_versions=2, lr=_LR["gpt"], weight_decay=0.01, macrobatch=True)
    else:
        opt = sgd.SGDWithWeightStashing(*args, num_versions=r.num_warmup_minibatches + 1, momentum=0.9,
                                        lr=_LR[net], weight_decay=5e-4 if net == "vgg16" else 1e-4)
    return r, opt


def prepare(case, seed):
    if case["mode"] == "pipeline":
        workers = [_worker(case, seed, rank) for rank in range(case["stages"])]
        workers[0][0].set_loader(_loader(case, seed))
        return {"case": case, "workers": workers, "pipeline": schedule.LocalPipeline(workers)}
    r, opt = _worker(case, seed)
    if case["mode"] == "eval":
        r.eval(1 << 30)
    else:
        r.train(1 << 30)
    r.set_loader(_loader(case, seed))
    return {"case": case, "workers": [(r, opt)]}


# --------------------------------------------------------------------------------------------------- run
def _groups(opt, flat, count):
    """A flat buffer over all parameters of a stage, cut between parameters into at most `count` consecutive pieces.
    (Gradients of different layers have different scales; a piece is compared on its own scale.)"""
    params = opt.master_parameters
    base = params[0].storage_offset()
    firsts = [i * len(params) // count for i in range(count)] if len(params) > count else range(len(params))
    edges = [params[i].storage_offset() - base for i in firsts] + [flat.numel()]
    return [flat[lo:hi] for lo, hi in zip(edges, edges[1:])]


def _updated(case, workers):
    """What a training pass leaves behind: the weights (every stashed version, and the fp32 master copy of 16-bit ones),
    and the gradients and the optimizer's moments.  The last two are left out for the 16-bit image networks: which
    ReLUs pass a gradient depends on the last bit of 16-bit activations, and after a dozen layers two correct programs
    that round at different places agree in the updated weights but not in the gradients of the early layers."""
    out, count = [], 16 // len(workers)
    for r, opt in workers:
        state = {"weights": opt.arena, "master": opt.master}
        if case["net"] in ("gnmt", "gpt") or case["dtype"] == "fp32":
            state["gradients"] = _groups(opt, opt.grad_arena, count)
            state["moments"] = _groups(opt, opt.state_a, count)
            state["squares"] = opt.state_b
        out.append(state)
    return out


def run(state):
    case, workers = state["case"], state["workers"]
    if case["mode"] == "pipeline":
        losses = []
        state["pipeline"].run([case["minibatches"]] * case["stages"], on_loss=lambda k, i, r: losses.append(r.loss))
        return {"losses": losses, "output": workers[-1][0].output, "updated": _updated(case, workers)}
    r, opt = workers[0]
    if case["mode"] == "eval":
        with torch.no_grad():
            r.run_forward()
            r.run_ack()
        return {"loss": r.loss, "output": r.output}
    losses = []
    for _ in range(opt.update_interval):
        r.run_forward()
        losses.append(r.loss)
        schedule.backward_step(r, opt)
    out = {"losses": losses, "updated": _updated(case, workers)}
    if case["net"] in ("vgg16", "resnet50"):
        out["output"] = r.output          # what the image drivers compute their accuracy from
    return out


# -------------------------------------------------------------------------------------------------- work
def _gnmt_flops(batch, length):
    """Forward flops of `batch` pairs of `length` tokens a side (2 per multiply-add)."""
    H, V, tokens = 1024, 32320, batch * length
    narrow, wide = 2 * 4 * H * (H + H), 2 * 4 * H * (2 * H + H)
    encoder = 2 * narrow + wide + 6 * narrow
    decoder = narrow + 7 * wide + 2 * H * V
    attention = 2 * 2 * H * H + length * 4 * H
    return tokens * (encoder + decoder + attention)


def work(case):
    net, batch = case["net"], case["batch"]
    size = 2 if case["dtype"] == "bf16" else 4
    if net == "vgg16":
        params, units, fwd, bwd = 138357544, batch, 30.94e9, 61.71e9
        inputs, kept, outputs = 3 * 224 * 224 * 4, 13.56e6, 1000     # kept: convolution outputs the backward pass reads
    elif net == "resnet50":
        params, units, fwd, bwd = 25557032, batch, 8.18e9, 16.12e9
        inputs, kept, outputs = 3 * 224 * 224 * 4, 11.11e6, 1000
    elif net == "gnmt":
        mean = (case["shortest"] + case["longest"]) / 2
        params, units = 193.0e6, batch
        fwd = _gnmt_flops(1, mean)
        bwd, inputs, kept, outputs = 2 * fwd, 4 * 8 * mean, mean * 1024 * 17 * 5, mean * 32320
    else:
        T, H = case["tokens"], 1024
        params, units = 405.9e6, batch * (2 if case["mode"] == "train" else 1)
        fwd = 2 * (params - (50304 + _GPT_SEQ) * H) * T + 24 * 2.0 * T * T * H
        bwd, inputs, kept, outputs = 2 * fwd, 2 * 8 * T, 24 * T * H * 12, T * 50304.0
    units *= case.get("minibatches", 1)
    if case["mode"] == "eval":
        return {"bytes": params * size + units * (inputs + outputs * size), "flops": units * fwd}
    # an optimizer step reads and writes the fp32 weights and moments, writes the gradients and, for 16-bit stages,
    # a 16-bit copy of the weights
    moments = 8 if net in ("vgg16", "resnet50") else 16
    per_param = size + 4 + 8 + moments + (2 if size == 2 else 0)
    return {"bytes": params * per_param * case.get("minibatches", 1) + units * (inputs + 2 * kept * size),
            "flops": units * (fwd + bwd)}


def tolerance(case):
    if case["dtype"] == "fp32" and case["mode"] == "eval":
        return {"rel": 1e-4}
    # 16 bits: moving every rounding by half a unit moves the logits of the image networks by 8e-3 and the gradients of
    # the sequence models by 7e-3 to 2e-2.  fp32 gradients of the image networks: a ReLU whose input is within rounding
    # of zero passes the whole gradient or none of it, so a relative change d of the activations moves the early
    # layers' gradients by about sqrt(d): 7e-3 for 1e-7.
    return {"rel": 2e-2} if case["mode"] == "eval" else {"rel": 2e-2, "max": 0.99}
