"""Forward and backward of a one-rank training step as CUDA graphs.

A step of a small model is bound by its launches: the Python, autograd and driver work of one kernel
launch is about 28 us, so the 92 launches of a two-layer d = 256 step took 2.5 ms of which the GPU worked
0.5, and the 179 of a four-layer GPT-2-XL step 5.4 ms against 4.5.  On one rank a step contains no
communication and its tensors stay where they are (parameters and gradients are views of two flat
buffers), so the launches of forward and backward are recorded once per batch shape and replayed.  The
optimizer runs outside the graph: its learning rate and bias corrections change every step.

A shape is recorded after it has been run ``EAGER_STEPS`` times.  Up to ``MAX_SHAPES`` shapes are kept, and
one gives way to another only after ``IDLE_STEPS`` steps without it: a recording costs more than an eager
step, and batches of more shapes than are kept would pay for one at every step if the least recently used
made room (ten lengths of the d = 256 model in turn took 3.4 ms a step with four kept so, 2.5 eagerly,
1.1 to 2.1 now).

Steps run eagerly, as they would without this module, whenever a replay could differ from that: hooks added
to a module, to a parameter or to all modules, modules or parameters put in place of the model's own, a
``forward``, an epsilon or an entry of the configuration changed, moved storage, saved-tensor hooks,
dispatch and function modes, autocast, anomaly detection, a capture that is already under way.  A shape is
recorded again when another GEMM or attention implementation has been selected since.
A recording that fails (no memory for the graph, a call that no recording may make) is given up, the step runs
eagerly and so do all later ones.
"""
from __future__ import annotations

import contextlib
import warnings
from collections import OrderedDict

import torch
from torch import overrides
from torch.nn.modules import module
from torch.utils._device import DeviceContext

from .. import _lib
from ..ops import attention, gemm, rope


def _modes() -> bool:
    """Whether something watches or replaces every operation or saved tensor of this thread, or every module call."""
    return bool(torch._C._len_torch_dispatch_stack()
                or torch._C._autograd._top_saved_tensors_default_hooks(True) is not None
                or module._has_any_global_hook()
                # a default device is a function mode too, and changes nothing here
                or any(not isinstance(m, DeviceContext) for m in overrides._get_current_function_mode_stack()))


def _address(t):
    return None if t is None else t.data_ptr()


class _Recorded:
    __slots__ = ("graph", "ids", "loss", "key", "keep", "launches", "used")


class StepGraphs:
    EAGER_STEPS = 2
    MAX_SHAPES = 16    # all of one memory pool: they share their activations' memory
    IDLE_STEPS = 1024
    # A graph's activations live in a pool of their own beside the allocator's, which gives none of its cached
    # blocks back during a recording: recorded only where they are small against the memory that nobody has taken.
    MAX_BYTES = 8 << 30
    MAX_FREE_FRACTION = 0.125

    def __init__(self, model, flat, cfg):
        self.model, self.flat, self.cfg = model, flat, cfg
        # the model as the engine has built it; the objects are kept, so that no other one can have their identity
        self._modules = list(model.modules())
        self._params = list(model.parameters())
        self._hook_dicts = [d for m in self._modules for d in (m._forward_hooks, m._forward_pre_hooks, m._backward_hooks,
                                                               m._backward_pre_hooks)]
        self._child_dicts = [d for m in self._modules for d in (m._modules, m._parameters) if d]
        self._attrs = [m.__dict__ for m in self._modules]
        self._with_eps = [m for m in self._modules if hasattr(m, "eps")]
        self._built = self._state()
        self._seen: dict = {}
        self._recorded: OrderedDict = OrderedDict()
        self._refused: set = set()
        self._steps = 0
        self._failed = False
        self._stream = None
        self._pool = None

    # -- when a replay is the same as running the step ---------------------------------------------
    def _state(self) -> list:
        """What the model is made of, apart from the values of its parameters."""
        return [
            [key for d in self._hook_dicts if d for key in d],
            [id(x) for d in self._child_dicts for x in d.values()],
            ["forward" in d for d in self._attrs],
            [m.eps for m in self._with_eps],
            [id(d.get("cfg")) for d in self._attrs],
            list(vars(self.model.config).values()),
            [(p.data_ptr(), _address(getattr(p, "main_grad", None)), p.requires_grad, p.grad is None,
              not p._backward_hooks, not p._post_accumulate_grad_hooks) for p in self._params],
        ]

    def _key(self):
        f = self.flat
        return (f.master.data_ptr(), f.grad_master.data_ptr(), f.master_c.data_ptr(), gemm.get_backend(),
                attention._FWD_IMPL, attention._BWD_IMPL, self.model.training, self.model.activation_checkpointing)

    def _allowed(self) -> bool:
        return (torch.is_grad_enabled() and not torch.is_anomaly_enabled() and not torch.is_autocast_enabled("cuda")
                and not torch.cuda.is_current_stream_capturing() and not _modes() and self._state() == self._built)

    def _activation_bytes(self, tokens: int) -> int:
        """What forward and backward hold at once, from the tensors that the blocks save."""
        c = self.cfg
        block = 8 * c.d_model + (c.n_heads + 2 * c.n_kv_heads) * c.head_dim + 3 * c.ffn
        saved = c.n_layers * block if not self.model.activation_checkpointing else c.n_layers * 2 * c.d_model + block
        return 2 * tokens * (saved + c.vocab_size + 6 * c.ffn)

    def _host_bound(self, tokens: int) -> bool:
        """Whether the launches (about 23 a layer and 20 beside the layers, 28 us each) are more than a tenth of the GPU's
        work (products at 1.4 PFLOP/s, 14 bytes an element for the update).  Below that a replay has nothing to save, and
        recorded GEMMs hand their tiles out in a fixed order: a 34B layer at 4096 tokens took 29.0 ms eagerly and
        29.9 replayed (a twentieth), a 13B layer at 2048 tokens 7.4 and 7.2 (a sixth)."""
        n = self.cfg.num_params()
        return 10 * 28e-6 * (23 * self.cfg.n_layers + 20) > 6 * n * tokens / 1.4e15 + 14 * n / 6e12

    # -- run ---------------------------------------------------------------------------------------
    def owns(self, loss: torch.Tensor) -> bool:
        return any(r.loss is loss for r in self._recorded.values())

    def run(self, ids: torch.Tensor):
        """Forward and backward of ``ids`` by replay; None when this step has to run eagerly."""
        if self._failed or ids.dim() != 2 or ids.dtype != torch.int64:
            return None
        shape = tuple(ids.shape)
        key = self._key()
        if (shape, key) in self._refused or not self._allowed():  # the second takes 0.5 ms for a model of 48 layers
            return None
        self._steps += 1
        rec = self._recorded.get(shape)
        if rec is not None and rec.key != key:
            del self._recorded[shape]
            self._seen[shape] = 0
            rec = None
        if rec is None:
            seen = self._seen.get(shape, 0)
            if seen < self.EAGER_STEPS:
                if len(self._seen) > 256:
                    self._seen.clear()
                self._seen[shape] = seen + 1
                return None
            full = len(self._recorded) >= self.MAX_SHAPES
            if full and self._steps - next(iter(self._recorded.values())).used < self.IDLE_STEPS:
                return None
            free, _ = torch.cuda.mem_get_info(self.flat.device)
            if (not self._host_bound(ids.numel())
                    or self._activation_bytes(ids.numel()) > min(self.MAX_BYTES, self.MAX_FREE_FRACTION * free)):
                if len(self._refused) > 256:
                    self._refused.clear()
                self._refused.add((shape, key))
                return None
            if full:
                self._recorded.popitem(last=False)
            try:
                rec = self._record(shape, key)
            except Exception as e:
                warnings.warn(f"training steps run without CUDA graphs from here on: {type(e).__name__}: {e}")
                self._failed = True
                self._recorded.clear()
                return None
            self._recorded[shape] = rec
        self._recorded.move_to_end(shape)
        rec.used = self._steps
        rec.ids.copy_(ids, non_blocking=True)
        rec.graph.replay()
        _lib.add_launches(rec.launches)
        return rec.loss

    def _record(self, shape, key) -> _Recorded:
        dev = self.flat.device
        rec = _Recorded()
        rec.key = key
        rec.ids = torch.zeros(shape, dtype=torch.int64, device=dev)
        # the cached tables that the recorded launches read: made ahead of the recording, outside the graphs' memory
        rec.keep = (rope.cached_tables(shape[1], self.cfg.head_dim, self.cfg.rope_theta, rec.ids.device)
                    if self.cfg.family == "llama" else None)
        rec.graph = torch.cuda.CUDAGraph()
        if self._stream is None:
            self._stream = torch.cuda.Stream(dev)
        if not self._recorded:  # a pool ends with its last graph
            self._pool = torch.cuda.graph_pool_handle()
        cur = torch.cuda.current_stream(dev)
        before = _lib.launch_count()
        self._stream.wait_stream(cur)
        with torch.cuda.stream(self._stream):
            # thread_local: other threads (the process group's watchdog) go on calling CUDA meanwhile
            rec.graph.capture_begin(pool=self._pool, capture_error_mode="thread_local")
            try:
                out = self.model(input_ids=rec.ids, labels=rec.ids)
                self.flat.backward(out.loss)
                rec.loss = out.loss.detach()
                del out
            except BaseException:
                self.flat.drop_gradients()
                _lib.add_launches(before - _lib.launch_count())
                with contextlib.suppress(RuntimeError):  # the first error is the one to report
                    rec.graph.capture_end()
                raise
            rec.graph.capture_end()
        cur.wait_stream(self._stream)
        rec.launches = _lib.launch_count() - before
        _lib.add_launches(-rec.launches)  # recorded, not run
        return rec
