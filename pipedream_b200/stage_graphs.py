"""CUDA graphs of a stage's forward and backward passes.

A stage launches between one hundred (VGG-16) and two thousand (the GPT decoder, per optimizer step) kernels per
minibatch from Python, most of them 2 to 30 us long, and the host needs 15 to 25 us for each (autograd node, output
allocation, launch).  ResNet-50 spent 14 ms per minibatch of 64 and 4.4 ms per single image on work the GPU finishes in
11.1 and 1.0 ms.  Shapes repeat from one minibatch to the next, so the launches are recorded once and replayed.

What a `Pass` holds is one minibatch in flight: static input buffers, the recorded forward pass with the autograd graph
and activations it left behind, and the backward passes recorded on them.  1F1B keeps several minibatches of a stage in
flight; each has a Pass of its own.  A Pass is chosen by everything a recording has baked in: shapes and strides of the
inputs, grad mode, the modules' settings, and where the weights lie.

Weights.  A recording reads the weights at fixed addresses.  With one or two weight versions a Pass is recorded per ring
slot and reads the slot in place.  With more, the number of (slot, minibatch in flight) pairs grows with the square of
the pipeline depth, so every pass first copies the slot it is meant to use into one shadow slot (a few microseconds for
the part of a network a deep pipeline's stage holds) and all recordings read that.

Python state that changes per pass (dropout stream positions, BatchNorm's batch counters, call counters, the attention
mask) is advanced as observed while recording.  Dropout kernels take their position from device memory when recorded; the
recording itself moves it on.

What is recorded and what is not: only stages all of whose leaves are this package's modules, without hooks, not
replicated (the gradient averager listens to each gradient as it is produced) and not recomputing; anything else, and
the first minibatches of every shape, run launch by launch on the same stream the recordings are made on.
"""
import contextlib
import os
import threading
import warnings

import torch
import torch.nn as nn

from . import _lib
from . import functional as pf
from . import layers

_ENABLED = os.environ.get("PD_STAGE_GRAPHS", "1") != "0"
_LOCK = threading.RLock()              # recordings are made one at a time
_STREAMS = threading.local()

MAX_PASSES = 16                        # recordings kept per stage
MAX_BACKWARDS = 4                      # recorded backward passes per Pass (accumulate or not, which slot)
_PLAIN = (nn.Identity, nn.Flatten)    # stateless torch leaves that launch plain work or none


def _stream(device):
    """The stream recordings (and the passes around them) run on: one per device and host thread."""
    table = _STREAMS.__dict__.setdefault("table", {})
    st = table.get(device.index)
    if st is None:
        st = table[device.index] = torch.cuda.Stream(device=device)
    return st


def _static_like(t):
    """A zero-filled buffer of t's shape and strides (a padded view keeps its zero border)."""
    span = 1 + sum((n - 1) * s for n, s in zip(t.shape, t.stride())) if t.numel() else 0
    pad = pf.padded_of(t) if t.is_cuda and t.dim() == 4 and not t.is_contiguous() else None
    if pad is not None:
        buf = torch.zeros(pad.shape, dtype=t.dtype, device=t.device)
        return pf.nchw_view(buf, *t.shape)
    return torch.zeros(max(span, 1), dtype=t.dtype, device=t.device).as_strided(t.shape, t.stride())


class _Backward:
    """One recorded backward pass of a Pass."""
    __slots__ = ("graph", "leaf_grads", "foreign", "written", "counts")


class Pass:
    __slots__ = ("key", "busy", "graph", "static", "data", "out", "loss", "output", "workspaces", "dropout_steps",
                 "steps_dev", "batches", "calls", "masks", "counts", "backwards", "grad_in", "failed", "last_used", "roots")

    def __init__(self, key):
        self.key, self.busy, self.failed, self.last_used = key, False, False, 0
        self.workspaces, self.backwards, self.grad_in = {}, {}, {}


class StageGraphs:
    def __init__(self, rt):
        self.device = rt.device
        self.passes = {}               # key -> [Pass]
        self.count = 0                 # recordings held
        self.seen = {}                 # key -> passes run launch by launch so far
        self.minibatches = 0
        self.last_inputs, self.steady = None, 0      # shapes of the minibatch before; minibatches that had the same in a row
        self.activation_bytes = 0
        self.shadow = None
        self.usable = _ENABLED and rt.device.type == "cuda" and rt.num_ranks_in_stage == 1
        if not self.usable:
            return
        mods = [m for top in rt.plan.modules for m in top.modules()]
        owners = {id(m.bidir) for m in mods if isinstance(m, layers.NativeEmuBidirLSTM)}     # hold parameters, never run
        mods = [m for m in mods if id(m) not in owners]
        self.params = list(rt.parameters())
        for m in mods:
            leaf = next(m.children(), None) is None
            ours = isinstance(m, layers._NATIVE_TYPES + (layers.NativeFork,) + _PLAIN)
            container = type(m).__module__.startswith("pipedream_b200.") or getattr(m, "_pd_traced", False) \
                or isinstance(m, (nn.ModuleList, nn.Sequential))
            if not (ours or (container and not leaf) or self._kept_core(m)):
                self.usable = False
                return
        self.mods = mods
        self.native = [p for p in self.params if getattr(p, "_pd_native", False)]
        self.foreign = [p for p in self.params if not getattr(p, "_pd_native", False)]
        self.dropouts = [m for m in mods if isinstance(m, layers.NativeDropout)]
        self.norms = [m for m in mods if isinstance(m, layers.NativeBatchNorm2d)]
        self.cores = [m for m in mods if isinstance(m, layers.NativeCausalAttentionCore)]
        self.attentions = [m for m in mods if isinstance(m, layers.NativeBahdanauAttention)]
        self.offsets_dev, self.offsets_host = None, None
        self.names = list(rt.plan.inputs)
        if rt.is_criterion:
            self.names += [n for n in sorted(rt.target_tensor_names) if n not in self.names]

    @staticmethod
    def _kept_core(m):
        """The plain attention core a native one keeps for the shapes its kernels do not take, and its like."""
        return type(m).__name__ == "CausalAttentionCore" and type(m).__module__.startswith("pipedream_b200.")

    # ------------------------------------------------------------------ keys
    def _settings(self):
        """Everything in the modules that a recording bakes in; None when a hook would be skipped."""
        flags = []
        for m in self.mods:
            if m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks:
                return None
            flags.append(m.training)
        return (tuple(flags), tuple([(d.p, d.seed) for d in self.dropouts]),
                tuple([(b.momentum, b.eps, b._buffers["running_mean"].data_ptr()) for b in self.norms]),
                pf._DETERMINISTIC)

    def _weights(self, rt):
        """(key part, ring optimizer whose slot has to be copied into the shadow or None)."""
        opt = rt._optimizer_ref() if rt._optimizer_ref is not None else None
        if opt is not None and opt.num_versions > 2:
            views = opt._views[opt._current_slot]
            if self.params and all(p.data_ptr() == v.data_ptr() for p, v in zip(opt.master_parameters, views)):
                return ("shadow", id(opt)), opt
        return tuple([p.data_ptr() for p in self.params]), None

    def _key(self, rt, tensors):
        if pf.timeline is not None:
            return None, None
        settings = self._settings()
        if settings is None:
            return None, None
        ins = []
        for n in self.names:
            t = tensors.get(n)
            if t is None:
                continue
            if not (torch.is_tensor(t) and t.is_cuda and t.grad_fn is None):
                return None, None
            ins.append((n, t.shape, t.stride(), t.dtype, t.requires_grad))
        weights, opt = self._weights(rt)
        return (tuple(ins), torch.is_grad_enabled(), rt.forward_only, rt.loss_scale, settings, weights), opt

    # ------------------------------------------------------------------ shadow weights
    def _shadow(self, opt):
        if self.shadow is None or self.shadow[0] is not opt.arena:
            buf = torch.zeros(opt.slot_stride, dtype=opt.dtype, device=self.device)
            views = [buf.as_strided(v.shape, v.stride(), off) for v, (off, _) in zip(opt._views[0], opt._offsets)]
            self.shadow = (opt.arena, buf, views)
        return self.shadow

    def _load_shadow(self, opt):
        self._shadow(opt)[1].copy_(opt.arena[opt._current_slot])

    @contextlib.contextmanager
    def _recording(self, p, opt, counts):
        """Around a recording: parameters on the shadow slot, workspaces of the Pass, launch accounting aside."""
        with _LOCK:
            prev_counts, _lib.COUNTERS = _lib.COUNTERS, counts
            prev_ws, pf.capture_workspaces = pf.capture_workspaces, p.workspaces
            if opt is not None:
                for q, v in zip(opt.master_parameters, self._shadow(opt)[2]):
                    q.data = v
            try:
                yield
            finally:
                if opt is not None:
                    opt._point_params(opt._current_slot)
                pf.capture_workspaces = prev_ws
                _lib.COUNTERS = prev_counts

    @staticmethod
    def _count(counts):
        if _lib.COUNTERS is not None:
            for name, n in counts.items():
                _lib.COUNTERS[name] = _lib.COUNTERS.get(name, 0) + n

    # ------------------------------------------------------------------ forward
    def forward(self, rt, tensors):
        """Runs the stage's forward pass over `tensors` (filled in place).  Returns the Pass that was replayed, or None
        when the pass ran launch by launch."""
        key, opt = self._key(rt, tensors)
        self.minibatches += 1
        self.steady = self.steady + 1 if key is not None and key[0] == self.last_inputs else 0
        self.last_inputs = key[0] if key is not None else None
        p = None
        if key is not None:
            have = self.passes.get(key)
            if have:
                p = next((q for q in have if not q.busy), None)
            fresh = p is None and self._worth_recording(rt, key)
            if fresh:
                p = self._record_forward(rt, key, opt, tensors)
            if p is not None:
                self._replay_forward(rt, p, opt, tensors, fresh)
                return p
            if len(self.seen) > 256:
                self.seen.clear()
            self.seen[key] = self.seen.get(key, 0) + 1
        new = key is not None and self.seen[key] <= 2
        before = torch.cuda.memory_allocated(self.device) if new else 0
        cur, st = torch.cuda.current_stream(self.device), _stream(self.device)
        st.wait_stream(cur)
        with torch.cuda.stream(st):
            rt._run_forward(tensors)
        cur.wait_stream(st)
        if new:
            self.activation_bytes = max(self.activation_bytes, torch.cuda.memory_allocated(self.device) - before)
        return None

    def _worth_recording(self, rt, key):
        # A recording costs about two passes run launch by launch and pays from then on, so a shape has to have come
        # back, and the pipeline to have filled and drained about once, before one is made.  Where shapes change from
        # one minibatch to the next (sentences), few come back often enough: twelve recordings of 25 to 130 ms against
        # passes of 12 ms made such a stage slower, not faster.
        if self.seen.get(key, 0) < 1 or self.minibatches <= min(8, 2 * rt.num_stages) or self.steady < 2:
            return False
        # A recording of the 24-layer decoder (1100 launches a pass, two weight slots, two backward passes each) takes 35 to
        # 170 ms, four to ten times what a minibatch gains from it: only a run that has settled makes one.
        if len(self.params) > 200 and self.steady < 64:
            return False
        if self.count >= MAX_PASSES:
            idle = [q for have in self.passes.values() for q in have if not q.busy]
            oldest = min(idle, key=lambda q: q.last_used, default=None)
            if oldest is None or self.minibatches - oldest.last_used < 8 * MAX_PASSES:
                return False
            self._drop(oldest)
        free = torch.cuda.mem_get_info(self.device)[0] + torch.cuda.memory_reserved(self.device) \
            - torch.cuda.memory_allocated(self.device)
        return free > 3 * self.activation_bytes + (2 << 30)

    def _drop(self, p):
        have = self.passes.get(p.key, [])
        if p in have:
            have.remove(p)
            self.count -= 1
            if not have:
                del self.passes[p.key]

    def _record_forward(self, rt, key, opt, tensors):
        p = Pass(key)
        p.static, p.data = {}, {}
        for n in self.names:
            t = tensors.get(n)
            if t is None:
                continue
            s = _static_like(t)
            p.data[n] = s                               # an alias with a version counter of its own
            s = s.data
            if t.requires_grad:
                s.requires_grad_()
            p.static[n] = s
        starts = [d.offset for d in self.dropouts]
        calls = [c.native_calls for c in self.cores]
        batches = [int(b.num_batches_tracked) for b in self.norms]
        if self.dropouts and self.offsets_dev is None:
            self.offsets_dev = torch.zeros(len(self.dropouts), dtype=torch.int64, device=self.device)
        p.steps_dev = torch.zeros_like(self.offsets_dev) if self.dropouts else None
        p.counts = {}
        cur, st = torch.cuda.current_stream(self.device), _stream(self.device)
        kept = (rt.__dict__.get("loss"), rt.__dict__.get("_output"))
        out = dict(p.static)
        for k, d in enumerate(self.dropouts):
            d._pd_recorded = (self.offsets_dev, k, d.offset)
        st.wait_stream(cur)
        try:
            with self._recording(p, opt, p.counts), torch.cuda.stream(st):
                p.graph = torch.cuda.CUDAGraph()
                p.graph.capture_begin(capture_error_mode="thread_local")
                try:
                    rt._run_forward(out)
                    if self.dropouts:
                        self.offsets_dev.add_(p.steps_dev)
                finally:
                    p.graph.capture_end()
        except Exception as e:
            self.usable = False                         # something in this stage cannot be recorded
            warnings.warn("forward pass not recorded, the stage runs launch by launch: %s" % e)
            for d, off in zip(self.dropouts, starts):
                d.offset = off
            for b, n in zip(self.norms, batches):
                b.num_batches_tracked.fill_(n)
            for c, n in zip(self.cores, calls):
                c.native_calls = n
            rt.loss, rt._output = kept
            return None
        finally:
            for d in self.dropouts:
                d._pd_recorded = None
        p.out = {n: v for n, v in out.items() if n not in p.static}
        p.loss, p.output = rt.loss, rt._output
        p.roots = [n for n in rt.plan.outputs if torch.is_tensor(out.get(n)) and out[n].requires_grad]
        p.dropout_steps = [d.offset - s for d, s in zip(self.dropouts, starts)]
        if self.dropouts:
            p.steps_dev.copy_(torch.tensor(p.dropout_steps, dtype=torch.int64))
            for d, off in zip(self.dropouts, starts):
                d.offset = off                          # the replay that follows moves it on
        p.batches = [b.num_batches_tracked for b, n in zip(self.norms, batches) if int(b.num_batches_tracked) != n]
        for b, n in zip(self.norms, batches):
            b.num_batches_tracked.fill_(n)
        p.masks = [(a.mask, a._ctx_len) for a in self.attentions]
        p.calls = [c.native_calls - n for c, n in zip(self.cores, calls)]
        for c, n in zip(self.cores, calls):
            c.native_calls = n
        self.passes.setdefault(key, []).append(p)
        self.count += 1
        return p

    def _replay_forward(self, rt, p, opt, tensors, fresh):
        p.last_used = self.minibatches
        for n, s in p.data.items():
            pf.copy_into(s, tensors[n])
        if opt is not None:
            self._load_shadow(opt)
        if self.dropouts:
            now = [d.offset for d in self.dropouts]
            if now != self.offsets_host:
                self.offsets_dev.copy_(torch.tensor(now, dtype=torch.int64))
        p.graph.replay()
        if self.dropouts:
            for d, step in zip(self.dropouts, p.dropout_steps):
                d.offset += step
            self.offsets_host = [d.offset for d in self.dropouts]
        if p.batches:
            torch._foreach_add_(p.batches, 1)
        for c, n in zip(self.cores, p.calls):
            c.native_calls += n
        for a, (mask, lengths) in zip(self.attentions, p.masks):
            a.mask, a._ctx_len = mask, lengths
        self._count(p.counts)
        # what leaves the pass must survive its next replay: the loss is copied here, the output when it is asked for
        # (StageRuntime.output), boundary tensors when they are sent
        for n, v in p.out.items():
            tensors[n] = v
        rt._output, rt._output_is_static = p.output, True
        if torch.is_tensor(p.loss):
            rt.loss = p.loss.detach().clone()
            name = rt.plan.last_outputs[0]
            if p.out.get(name) is p.loss:
                tensors[name] = rt.loss
            elif name in p.out:
                tensors[name] = p.out[name].detach().clone()
        else:
            rt.loss = p.loss
        p.busy = torch.is_grad_enabled() and not rt.forward_only

    # ------------------------------------------------------------------ backward
    @contextlib.contextmanager
    def around_backward(self):
        """For a backward pass that runs launch by launch: its nodes run on the stream their forward pass ran on."""
        cur, st = torch.cuda.current_stream(self.device), _stream(self.device)
        st.wait_stream(cur)
        yield
        cur.wait_stream(st)

    def backward(self, rt, p):
        """The backward pass of a replayed forward pass; fills rt.gradients for the stage's inputs."""
        grads = {}
        for n in p.roots:
            g = rt.gradients.get(n)
            if g is not None:
                s = p.grad_in.get(n)
                padded = not g.is_contiguous() and pf.padded_of(g) is not None
                if s is None or s.shape != g.shape or s.dtype != g.dtype or padded != (not s.is_contiguous()):
                    s = p.grad_in[n] = _static_like(g) if padded else torch.empty(g.shape, dtype=g.dtype, device=self.device)
                    p.backwards.clear()
                pf.copy_into(s, g)
                grads[n] = s
        weights, opt = self._weights(rt)
        if opt is not None:
            self._load_shadow(opt)
        b = None
        if not p.failed and pf.timeline is None and all(hasattr(q, "_pd_grad") for q in self.native):
            key = (weights, tuple([(q._pd_acc, q._pd_grad.data_ptr()) for q in self.native]), tuple(grads),
                   tuple([q.grad.data_ptr() if q.grad is not None else 0 for q in self.foreign]),
                   rt.loss_scale, pf._DETERMINISTIC)
            b = p.backwards.get(key)
            if b is None and len(p.backwards) < MAX_BACKWARDS:
                b = self._record_backward(rt, p, opt, grads)
                if b is not None:
                    p.backwards[key] = b
        if b is None:
            leaf = self._backward_by_launch(rt, p, grads)
        else:
            b.graph.replay()
            for q, g in b.foreign:
                q.grad = g
            for q in b.written:
                q._pd_acc = True
            self._count(b.counts)
            leaf = b.leaf_grads
        for n in rt._bwd_send:
            g = leaf.get(n)
            rt.gradients[n] = pf.copy_of(g) if g is not None else torch.zeros_like(p.static[n])
        p.busy = False

    def _roots(self, rt, p, grads):
        roots, root_grads = [], []
        for n in p.roots:
            t = p.out[n]
            if n == "loss" and rt.loss_scale != 1:
                t = t * rt.loss_scale
            roots.append(t)
            root_grads.append(grads.get(n))
        return tuple(roots), tuple(root_grads)

    def _take_leaf_grads(self, p):
        leaf = {}
        for n, s in p.static.items():
            if s.requires_grad:
                leaf[n] = s.grad
                s.grad = None
        return leaf

    def _record_backward(self, rt, p, opt, grads):
        b = _Backward()
        b.counts = {}
        before = [q._pd_acc for q in self.native]
        held = [q.grad for q in self.foreign]
        cur, st = torch.cuda.current_stream(self.device), _stream(self.device)
        st.wait_stream(cur)
        try:
            with self._recording(p, opt, b.counts), torch.cuda.stream(st):
                b.graph = torch.cuda.CUDAGraph()
                b.graph.capture_begin(pool=p.graph.pool(), capture_error_mode="thread_local")
                try:
                    roots, root_grads = self._roots(rt, p, grads)
                    torch.autograd.backward(roots, grad_tensors=root_grads, retain_graph=True)
                finally:
                    b.graph.capture_end()
        except Exception as e:
            p.failed = True
            warnings.warn("backward pass not recorded, it runs launch by launch: %s" % e)
            for q, acc in zip(self.native, before):
                q._pd_acc = acc
            for q, g in zip(self.foreign, held):
                q.grad = g
            self._take_leaf_grads(p)
            return None
        b.leaf_grads = self._take_leaf_grads(p)
        b.foreign = [(q, q.grad) for q in self.foreign]
        b.written = [q for q, acc in zip(self.native, before) if q._pd_acc and not acc]
        return b

    def _backward_by_launch(self, rt, p, grads):
        with self.around_backward():
            roots, root_grads = self._roots(rt, p, grads)
            torch.autograd.backward(roots, grad_tensors=root_grads, retain_graph=True)
        return self._take_leaf_grads(p)

    def release(self):
        """No minibatch is in flight any more (the start of an epoch)."""
        for have in self.passes.values():
            for p in have:
                p.busy = False

