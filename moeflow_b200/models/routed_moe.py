"""Serving-side wrapper of one routed MoE layer: static buffers + one CUDA graph.

``GraphedMoELayer`` is the call a user makes on the hot path.  It captures ``FixedEPLayer.forward`` once, and then
every call is a replay on this step's hidden states and router logits.  Nothing is allocated and nothing is read back
to the host by the layer itself.  A replay cannot be captured: a larger captured decode step takes
``FixedEPLayer.forward`` instead, and these calls raise while the current stream is capturing.

Two ways to feed it:

* ``layer(x, logits, out)``: two tensors (pinned host or device);
* ``layer.step(block, out)``: ``block = layer.new_pinned_inputs()`` is one pinned host block laid out like the
  device-side input block — hidden rows, logits, row count — which the caller fills in place (``block.x``,
  ``block.logits``, ``block.set_rows(t)``) and does not touch again before the step is done.

On the cuda backend the captured graph has no buffers of its own in the way: its first kernel reads the caller's
device tensors and its last one writes the caller's output rows (device, or pinned host memory at decode sizes), by
updating the two kernel nodes' arguments when pointers or row count change.  Other inputs (host memory, other dtypes or
strides) are copied into the static buffers ``.x`` / ``.logits`` / ``.num_valid`` first, which is also what ``load`` and
``replay`` work on.  The small copies and the gap in front of the graph were 13 us of a device-fed call.  A pinned input
block is still one copy: read by the first kernel itself over PCIe, 24 rows took 43 us, the copy engine needs 9.

All calls launch one executable graph of the layer's own.  ``.graph`` is the forward on the static buffers for a holder
that replays it, whatever was called before (it is instantiated by its first replay); ``.out`` holds the rows
of ``replay`` and of the calls without ``out`` (a call with ``out`` may leave it as it was).
"""

from __future__ import annotations

import ctypes as C
import weakref
from collections import deque

import torch
import torch.distributed as dist

from ..fixed import FixedEPLayer

_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)  # handle of a device's current stream

#: Up to this many rows of pinned output are written by the forward's last kernel itself; beyond it the copy engine moves
#: them (not measured there).  us per step on 72 bf16 experts, direct / copied, the two taken in turn call by call:
#:
#:     rows                             1      2      4      8     16     24     32     64    128
#:     queued, the same output     88/ 97 126/134 175/185 234/236 333/338 394/406 407/418 445/453 472/476
#:     queued, new outputs         88/ 95 126/135 175/185 234/245 333/342 395/401 407/418 448/453 472/477
#:     waited for, same output    102/111 134/140 182/188 236/241 342/346 402/407 421/429 457/460 496/502
#:     waited for, new outputs    106/109 137/138 186/187 239/241 346/347 405/411 424/429 457/459 491/501
MAX_HOST_ROWS = 128


class PinnedInputs:
    """One step's inputs in pinned host memory, in the layout of the layer's device input block."""

    def __init__(self, raw: torch.Tensor, x: torch.Tensor, logits: torch.Tensor, rows: torch.Tensor):
        self.raw, self.x, self.logits, self._rows = raw, x, logits, rows
        self.rows = 0

    def set_rows(self, t: int) -> None:
        self.rows = int(t)
        self._rows.fill_(int(t))


class GraphedMoELayer:
    def __init__(self, layer: FixedEPLayer, bias: torch.Tensor | None, warmup: int = 2):
        self.layer, self.bias = layer, bias
        cfg, dev = layer.cfg, layer.device
        # one block: [C, H] activations | [C, E] fp32 logits | int32 row count (16-byte aligned sections)
        itemsize = torch.empty((), dtype=layer.dtype).element_size()
        self._x_bytes = layer.C * cfg.hidden_size * itemsize
        self._lg_off = (self._x_bytes + 15) // 16 * 16
        self._lg_bytes = layer.C * cfg.n_routed_experts * 4
        self._nv_off = (self._lg_off + self._lg_bytes + 15) // 16 * 16
        self.packed_bytes = self._nv_off + 16
        self._block = torch.zeros(self.packed_bytes, dtype=torch.uint8, device=dev)
        self.x, self.logits, self.num_valid = self._views(self._block)
        self.num_valid.fill_(layer.C)
        self.graph: torch.cuda.CUDAGraph | None = None
        self._nodes: dict | None = None  # kernel nodes whose arguments follow the caller's buffers
        self._exec = None                # executable graph with those arguments; only _launch uses it
        self._bound: dict = {}           # what its first and last node point at
        # pinned outputs that replays may still be writing: the latest one (with its stream), and earlier ones with an
        # event behind their last replay
        self._host_out: tuple | None = None
        self._host_refs: deque = deque()
        self._warmup = warmup

    @property
    def kernels_per_step(self) -> int:
        ly = self.layer
        fp8 = getattr(ly, "_fp8", None)
        front = 1 if getattr(ly, "fuse_meta", False) else 3 if getattr(ly, "meta_ctas", 1) > 1 else 2  # dispatch, metadata
        if fp8 is not None and not fp8["in_meta"]:
            front += 1  # quantiser of the received rows
        if getattr(ly, "_expand", None) is not None:
            front += 1 if ly._expand_beside else 2
        if getattr(ly, "permute_rows", False) and fp8 is None:
            front += 1
        tail = 1 if getattr(ly, "fuse_return", False) or getattr(ly, "fuse_combine", False) else 2
        return front + 2 + tail

    def _views(self, block: torch.Tensor):
        cfg, C = self.layer.cfg, self.layer.C
        x = block[: self._x_bytes].view(self.layer.dtype).view(C, cfg.hidden_size)
        logits = block[self._lg_off : self._lg_off + self._lg_bytes].view(torch.float32).view(C, cfg.n_routed_experts)
        rows = block[self._nv_off : self._nv_off + 4].view(torch.int32).view(())
        return x, logits, rows

    def new_pinned_inputs(self) -> PinnedInputs:
        """A pinned host block for one step's inputs (fill ``.x[:t]``, ``.logits[:t]``, then ``set_rows(t)``)."""
        raw = torch.zeros(self.packed_bytes, dtype=torch.uint8).pin_memory()
        x, logits, rows = self._views(raw)
        return PinnedInputs(raw, x, logits, rows)

    def _forward(self) -> torch.Tensor:
        return self.layer.forward(self.x, self.logits, self.bias, self.num_valid)

    def capture(self) -> "GraphedMoELayer":
        """Warm up on a side stream, then capture one forward.  Every rank must call this together."""
        self._drop()
        side = torch.cuda.Stream(device=self.layer.device)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(self._warmup):
                self._forward()
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        if dist.is_available() and dist.is_initialized():
            dist.barrier(group=self.layer.group)
        native = self.layer.backend == "cuda"
        graph = torch.cuda.CUDAGraph(keep_graph=native)
        nodes = {} if native else None
        self.layer._node_log = nodes
        try:
            with torch.cuda.graph(graph):
                self.out = self._forward()
        finally:
            self.layer._node_log = None
        if native:
            from ..ops import _lib

            for name, (node, args) in nodes.items():
                own = [type(a).from_buffer_copy(a) for a in args]
                nodes[name] = (node, own[0], (C.c_void_p * len(own))(*(C.addressof(a) for a in own)), own)
            own_exec = C.c_void_p()
            _lib.check(_lib.lib().mf_graph_instantiate(graph.raw_cuda_graph(), _lib.stream_ptr(), C.byref(own_exec)), "graph instantiation")
            self._set_args, self._graph_launch, self._check = _lib.lib().mf_graph_set_args, _lib.lib().mf_graph_launch, _lib.check
            self._exec, self._device_index = own_exec.value, self.x.device.index
            self._drop_exec = weakref.finalize(self, _lib.lib().mf_graph_destroy, own_exec.value)
            self._drop_exec.atexit = False  # the context goes first
            self._own_out = (self.layer.out.data_ptr(), 0)
            self._bound = {"first": (self.x.data_ptr(), self.logits.data_ptr(), self.layer.C, self.num_valid.data_ptr()),
                           "last": self._own_out}  # as captured
        self.graph, self._nodes = graph, nodes
        torch.cuda.synchronize()
        return self

    def _launch(self, x: int, logits: int, rows: int, out: int | None, num_valid: int | None = None) -> None:
        """Replay on the caller's buffers (addresses; ``out`` None: all rows of the layer's own buffer; ``num_valid``: the
        device word that says how many of ``rows`` are live, None: all)."""
        first, last = (x, logits, rows, num_valid), self._own_out if out is None else (out, rows)
        if first != self._bound.get("first"):
            self._update("first", first)
        if last != self._bound.get("last"):
            self._update("last", last)
        # nothing else between here and the device: a call that is waited for pays for every line (4 us with the stream
        # object and the module lookups)
        code = self._graph_launch(self._exec, _raw_stream(self._device_index))
        if code:
            self._check(code, "graph launch")

    def _update(self, name: str, key: tuple) -> None:
        node, a, arg_list, _ = self._nodes[name]
        if name == "first":
            a.x, a.logits, a.T, a.num_valid = key
        else:
            a.out, a.rows = key
        self._bound.pop(name, None)  # unknown if the update fails
        self._check(self._set_args(self._exec, node, arg_list), "graph update")
        self._bound[name] = key

    def _readable(self, x: torch.Tensor, logits: torch.Tensor) -> bool:
        """Can the captured kernels read these tensors where they are?"""
        cfg, dev = self.layer.cfg, self.x.device
        return (x.device == dev and logits.device == dev and x.dtype == torch.bfloat16 and logits.dtype == torch.float32
                and x.dim() == 2 and x.shape[1] == cfg.hidden_size and logits.shape == (x.shape[0], cfg.n_routed_experts)
                and x.is_contiguous() and logits.is_contiguous() and x.data_ptr() % 16 == 0 and 0 < x.shape[0] <= self.layer.C)

    def _writable(self, out: torch.Tensor | None, rows: int, shape_ok) -> bool:
        return (out is not None and out.dtype == torch.bfloat16 and out.is_contiguous() and out.data_ptr() % 16 == 0
                and shape_ok and (out.device == self.x.device or (out.device.type == "cpu" and rows <= MAX_HOST_ROWS and out.is_pinned())))

    def _hold(self, out: torch.Tensor | None) -> None:
        """Keep a pinned output alive until the replays that write it are done (its allocator does not know of them)."""
        refs, last = self._host_refs, self._host_out
        now = None if out is None else torch.cuda.current_stream(self.x.device)
        if last is not None and (last[0] is not out or last[1] != now):
            done = torch.cuda.Event()
            done.record(last[1])
            refs.append((done, last[0]))
        self._host_out = None if out is None else (out, now)
        while refs and refs[0][0].query():
            refs.popleft()

    def load(self, x: torch.Tensor, logits: torch.Tensor) -> int:
        """Copy one step's inputs (``[T, H]``, ``[T, E]``; host-pinned or device) into the static buffers."""
        t = x.shape[0]
        if t > self.layer.C:
            raise ValueError(f"{t} tokens exceed capacity {self.layer.C}")
        self.x[:t].copy_(x, non_blocking=True)
        self.logits[:t].copy_(logits, non_blocking=True)
        self.num_valid.fill_(t)
        return t

    def replay(self) -> torch.Tensor:
        if self.graph is None:
            self.capture()
        if self._nodes is None or torch.cuda.is_current_stream_capturing():
            self.graph.replay()
        else:  # one executable graph for all calls: replays on several streams follow one another
            self._launch(self.x.data_ptr(), self.logits.data_ptr(), self.layer.C, None, self.num_valid.data_ptr())
        return self.out

    def _replay_static(self, t: int) -> torch.Tensor:
        """The first ``t`` rows of the static input buffers; on the calls' own executable graph, which is ready since the
        capture."""
        if self._nodes is None or t < 1 or torch.cuda.is_current_stream_capturing():
            return self.replay()[:t]
        self._launch(self.x.data_ptr(), self.logits.data_ptr(), t, None)
        return self.out[:t]

    def __call__(self, x: torch.Tensor, logits: torch.Tensor, out: torch.Tensor | None = None) -> torch.Tensor:
        """One step.  With ``out`` (e.g. a pinned host tensor ``[T, H]``) the rows are copied there."""
        if self.graph is None:
            self.capture()
        t = x.shape[0]
        if self._nodes is not None and self._readable(x, logits) and not torch.cuda.is_current_stream_capturing():
            if out is not None and out.is_cuda and self._writable(out, t, tuple(out.shape) == tuple(x.shape)):
                self._launch(x.data_ptr(), logits.data_ptr(), t, out.data_ptr())
                return out
            self._launch(x.data_ptr(), logits.data_ptr(), t, None)
            res = self.out[:t]
        else:
            t = self.load(x, logits)
            res = self._replay_static(t)
        if out is not None:
            out.copy_(res, non_blocking=True)
            return out
        return res

    def step(self, inputs: PinnedInputs, out: torch.Tensor | None = None) -> torch.Tensor:
        """One step from a pinned input block; with ``out`` (``[>= T, H]``, pinned host or device) the rows go there."""
        t = inputs.rows
        if t > self.layer.C:
            raise ValueError(f"{t} tokens exceed capacity {self.layer.C}")
        if self.graph is None:
            self.capture()
        self._block.copy_(inputs.raw, non_blocking=True)
        if (self._nodes is not None and t > 0 and not torch.cuda.is_current_stream_capturing() and
                self._writable(out, t, out is not None and out.dim() == 2 and out.shape[0] >= t and out.shape[1] == self.layer.H)):
            self._launch(self.x.data_ptr(), self.logits.data_ptr(), t, out.data_ptr())
            if not out.is_cuda:
                self._hold(out)  # behind the launch: in front of it a new output cost a waited-for step 7 to 15 us more
            return out
        res = self._replay_static(t)
        if out is not None:
            out[:t].copy_(res, non_blocking=True)
            return out
        return res

    def _drop(self) -> None:
        if self._exec is not None:
            self._drop_exec()  # one still running is freed when it is done
        self.graph = self._nodes = self._exec = None
        self._bound = {}

    def close(self) -> None:
        """Drop the graph (do this before destroying the process group)."""
        if self._host_out is not None:
            self._hold(None)
        for done, _ in self._host_refs:
            done.synchronize()
        self._host_refs.clear()
        self._drop()
