"""Recorded passes (pipedream_b200/stage_graphs.py) against the same passes run launch by launch: the recordings replay
the same kernels on the same values, so with deterministic weight gradients losses and weights are equal bit for bit -
dropout positions, BatchNorm statistics and the weight versions in flight included."""
import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("deterministic_weight_gradients")]

from pipedream_b200 import communication, layers, schedule, stage_graphs, stages      # noqa: E402
import pipeline_util as pu                                                             # noqa: E402


def _seed_dropout(workers):
    k = 0
    for r, _ in workers:
        for m in r.modules():
            for sub in m.modules():
                if isinstance(sub, layers.NativeDropout):
                    k += 1
                    sub.seed = 1000 + k


def _pipeline(kind):
    """A GPT pipeline with dropout (2BW: two slots, gradients accumulated over two microbatches), or three ResNet-50
    stages (BatchNorm; three weight versions on stage 0, so its passes read the shadow slot)."""
    schedule.reset_local()
    if kind == "gpt":
        cfg = dict(layers=2, hidden=128, heads=2, seq_len=128, vocab=250, dropout=0.1)
        pkg, n, dtype, kw = stages.gpt2(2, **cfg), 2, torch.bfloat16, dict(optimizer="adam", macrobatch=True, lr=1e-3)
        batch, data = 2, lambda steps: stages.SyntheticTokens(2, steps, cfg["seq_len"], cfg["vocab"])
    else:
        pkg, n, dtype, kw = stages.resnet50(3), 3, torch.bfloat16, dict(lr=1e-3)
        batch, data = 2, lambda steps: stages.SyntheticImages(2, steps)
    conf = dict(pkg.conf, stage_to_depth_map=None)
    shapes = {k: tuple(v) for k, v in pkg.boundary_shapes(batch).items()}
    dtypes = {k: torch.int64 if k in ("input0", "target") else dtype for k in shapes}
    workers = [pu.make_worker(pkg, conf, rank, batch, True, communication.LOCAL, shapes=(shapes, dtypes), dropout=True,
                              **kw) for rank in range(n)]
    _seed_dropout(workers)
    return schedule.LocalPipeline(workers), data


@pytest.mark.parametrize("kind", ["gpt", "resnet50"])
def test_recorded_passes_equal_launched_passes(kind, monkeypatch):
    got = {}
    for on in (True, False):
        monkeypatch.setattr(stage_graphs, "_ENABLED", on)
        pipe, data = _pipeline(kind)
        steps, losses, outputs = 24, [], []
        pipe.workers[0][0].set_loader(data(steps))
        for w in pipe.workers[1:]:
            w[0].set_loader(None)

        def on_loss(k, i, r):
            losses.append(r.loss)                    # kept unread: a later replay must not touch it
            outputs.append(r.output)
        pipe.run([steps] * len(pipe.workers), on_loss=on_loss)
        assert [r._graphs.usable for r, _ in pipe.workers] == [on] * len(pipe.workers)
        if on:
            assert all(r._graphs.count > 0 for r, _ in pipe.workers)
            assert not any(p.failed or not p.backwards for r, _ in pipe.workers
                           for have in r._graphs.passes.values() for p in have)
        state = [b.clone() for r, o in pipe.workers for b in (o.arena, o.master, o.state_a)]
        state += [b for r, _ in pipe.workers for m in r.modules() for b in m.buffers()]
        got[on] = (torch.stack(losses), torch.stack(outputs[-4:]), state)
    assert torch.equal(got[True][0], got[False][0])
    assert torch.equal(got[True][1], got[False][1])
    assert all(torch.equal(a, b) for a, b in zip(got[True][2], got[False][2]))


def test_every_batch_shape_has_its_own_recording(monkeypatch):
    """Evaluation over batches of two sizes: each is recorded once it has come three times in a row, answered by its own
    recording from then on, and the output of one pass is still there after the next."""
    torch.manual_seed(0)
    pkg = stages.resnet50(1)
    r, _ = pu.make_worker(pkg, None, None, 1, True, None, shapes=({}, {}))
    sizes = [3, 1, 3, 1, 3, 3, 3, 1, 1, 1, 3, 1, 3]
    batches = [next(iter(stages.SyntheticImages(b, 1, seed=7 + b))) for b in sizes]
    r.eval(len(batches))
    r.set_loader(batches)
    outs = []
    with torch.no_grad():
        for _ in batches:
            r.run_forward()
            outs.append(r.output)
            r.run_ack()
            assert r._graphs.count == (len(outs) > 6) + (len(outs) > 9)
    for b, out in zip(sizes, outs):
        assert torch.equal(out, outs[sizes.index(b)])
