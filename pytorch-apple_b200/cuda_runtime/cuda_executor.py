"""Run a ``CUDAProgram`` on one B200.

Interface of the reference executor (cuda_runtime/cuda_executor.py:66-176):
``CUDAExecutor(program)`` does all one-time work, ``run(inputs, weights)`` takes
name -> ``CUDABuffer`` dicts (weights keyed by placeholder) and returns
``{output name: CUDABuffer}``.

What happens inside is different.  The reference walks ~1.3 k Python dispatches per
decode token (NVRTC kernels and ``cupy.matmul``).  Here

1. *bind*: every step is turned once into ``(entry point, argument tuple)`` with all
   device pointers resolved - intermediates live at fixed offsets of one arena,
   inputs and weights at the addresses of the caller's buffers;
2. *launch*: the first run issues the calls one by one through ctypes; the
   second run with the same buffer addresses captures them into a CUDA graph, and
   every later run is a single graph replay;
3. weights are prepared once per weight set (dtype narrowing, batch-norm folding
   and channels-last repacking of convolution filters) by library kernels.

Outputs are views into the arena, or - for an in-place ``index_copy`` - the caller's
own input buffer; they stay valid until the next ``run`` (the reference reuses its
pool the same way, cuda_executor.py:90-95).  Not re-entrant; one executor per GPU.
"""

from __future__ import annotations

import contextlib
import ctypes as C
import operator
from typing import Any

from cuda_compiler.cuda_codegen import EW_OPCODES
from cuda_compiler.cuda_program import AliasStep, CUDAProgram, TensorView
from cuda_runtime import native
from cuda_runtime.native import DTYPE_BYTES, DTYPE_CODES, MASK_TILE, STEM_TMA_WIDTH

try:
    import torch
except ImportError:  # pragma: no cover
    torch = None


_HANDLE = operator.attrgetter("native_handle")
_CONTIGUOUS = operator.methodcaller("is_contiguous")


def _mask_key(m: TensorView) -> tuple:
    """What a prefill mask [B, 1, T, S] is: its elements, with the sequences it has of its own (one when it is shared)."""
    B, _, T, S = m.shape
    return (m.buffer, m.offset, 1 if m.strides[0] == 0 else B, T, S, m.strides[0], m.strides[2])


def _users(steps, names) -> dict[str, list[int]]:
    """Steps whose parameters hold a view of each of the buffers ``names``, in order."""
    found = {n: [] for n in names}

    def look(i, values):
        for v in values:
            kind = type(v)
            if kind is TensorView:
                if v.buffer in found and found[v.buffer][-1:] != [i]:
                    found[v.buffer].append(i)
            elif kind is dict:
                look(i, v.values())
            elif kind is list or kind is tuple:
                look(i, v)

    for i, params in steps:
        look(i, params.values())
    return found


def _find_stems(program: CUDAProgram, lib) -> list[tuple[int, int, int]]:
    """Heads of convolution networks that run as one kernel: the repack of a planar graph input to channels-last, a convolution
    of it, and a 3x3 / 2 max-pooling of the result, with nothing else reading what lies in between (256 images of a
    ResNet: 584 us as three kernels, 172 as one).  Indices of the three steps.

    Only images whose rows TMA can copy: others the kernel copies element by element (us, three kernels against one: 8 / 128
    images 223 wide 32 against 42 / 301 against 583, 256 wide 35 against 44 / 360 against 798, 33 wide 15 against 16 / 41
    against 50; 200 wide, by TMA, 30 against 12 / 259 against 81)."""
    steps = [(i, s.params) for i, s in enumerate(program.steps) if getattr(s, "params", None)]
    convs = {p["x"].buffer: i for i, p in steps if p.get("op") == "conv2d"}
    inputs = {s.name for s in program.input_specs}
    results = {program.views[s.name].buffer for s in program.output_specs if s.name in program.views}
    params, found = dict(steps), []
    for i, copy in steps:
        if copy.get("op") != "strided_copy" or copy["in_view"].buffer not in inputs or len(copy["in_view"].shape) != 4 or copy["out_view"].buffer not in convs:
            continue
        x, mid = copy["in_view"], copy["out_view"].buffer
        at = convs[mid]
        conv = params[at]
        y = conv["y"]
        if {mid, y.buffer} & results or conv["residual"] is not None:
            continue
        users = _users(steps, (mid, y.buffer))
        if users[mid] != [i, at] or users[y.buffer][:1] != [at] or len(users[y.buffer]) != 2:
            continue
        last = users[y.buffer][1]
        pool = params[last]
        if pool.get("op") != "max_pool2d" or pool["x"].buffer != y.buffer or pool["y"].buffer == y.buffer:
            continue
        N, Cn, H, W = x.shape
        O, PH, PW = y.shape[1], (y.shape[2] - 1) // 2 + 1, (y.shape[3] - 1) // 2 + 1
        cv = [conv[k] for k in ("c_pad", "out_channels", "kernel_h", "kernel_w", "stride_h", "stride_w", "pad_h", "pad_w")]
        if (W % 8 == 0 and W <= STEM_TMA_WIDTH and x.dtype == y.dtype == pool["y"].dtype and tuple(x.strides) == (Cn * H * W, H * W, W, 1) and tuple(copy["out_view"].shape) == tuple(x.shape)
                and conv["x"].offset == copy["out_view"].offset and tuple(pool["x"].shape) == tuple(y.shape)
                and tuple(pool["x"].strides) == tuple(y.strides) and pool["x"].offset == y.offset
                and [pool[k] for k in ("kernel_h", "kernel_w", "stride_h", "stride_w", "pad_h", "pad_w")] == [3, 3, 2, 2, 1, 1]
                and tuple(pool["y"].shape) == (N, O, PH, PW) and tuple(pool["y"].strides) == (PH * PW * O, 1, PW * O, O)
                and pool["y"].offset % 8 == 0 and lib.b200_conv_stem_pool_supported(Cn, H, W, *cv, DTYPE_CODES[y.dtype])):
            found.append((i, at, last))
    return found


class _Plan:
    """Launch list bound to one set of buffer addresses."""

    def __init__(self):
        self.launches: list[tuple[Any, tuple]] = []   # (cfunc, args without the trailing stream)
        self.keepalive: list[Any] = []
        self.outputs: dict[str, Any] = {}
        self.out_buffers: dict[str, Any] | None = None
        self.graph = None
        self.runs = 0
        self.n_kernels = 0
        self.masks_seen: set[tuple] = set()   # prefill masks whose tile states this launch list has already found


class CUDAExecutor:
    def __init__(self, program: CUDAProgram, device_id: int = 0, use_cuda_graph: bool = True):
        if torch is None:
            raise RuntimeError("PyTorch is not installed; it provides device memory for the CUDA executor")
        self._lib = native.load()
        self._device = native.device_string(device_id)
        self._torch_device = torch.device(self._device)
        self._on_gpu = self._device.startswith("cuda")
        if self._on_gpu and not torch.cuda.is_available():
            raise RuntimeError("no CUDA device is available")
        self._program = program
        self._compute_dtype = program.compute_dtype
        self._use_graph = use_cuda_graph and self._on_gpu
        self._allocs = {a.name: a for a in program.buffer_allocations}
        self._input_names = [s.name for s in program.input_specs]
        self._input_set = set(self._input_names)
        # zero-filled once: padding channels rely on it, everything else is overwritten before use
        self._arena = torch.zeros(max(int(program.arena_bytes), 256), dtype=torch.uint8, device=self._device)
        ws_lin = ws_att = 0
        for step in program.steps:
            p = getattr(step, "params", None) or {}
            if p.get("op") == "linear" and p.get("workspace"):
                ws_lin = max(ws_lin, int(self._lib.b200_linear_workspace_bytes(p["M"], p["N"], p["K"])))
            if p.get("op") == "attention" and p.get("workspace"):
                ws_att = max(ws_att, int(self._lib.b200_attn_decode_workspace_bytes(p["B"], p["Hq"], p["Hkv"], p["S"], p["D"])))
        # a state per 128 x 128 tile of each mask of a prefill attention, shared by the layers that read that mask
        self._tiles: dict[tuple, Any] = {}
        for step in program.steps:
            p = getattr(step, "params", None) or {}
            if p.get("op") == "attention" and not p["decode"] and p["mask"] is not None:
                key = _mask_key(p["mask"])
                if key not in self._tiles:
                    self._tiles[key] = torch.empty(key[2] * -(-key[3] // MASK_TILE) * -(-key[4] // MASK_TILE), dtype=torch.uint8, device=self._device)
        self._stems = _find_stems(program, self._lib)
        # split-K partial sums must start at zero; the kernel restores zeros before it exits
        self._ws = {"__ws_splitk": torch.zeros(max(ws_lin, 256), dtype=torch.uint8, device=self._device),
                    "__ws_attn": torch.empty(max(ws_att, 256), dtype=torch.uint8, device=self._device)}
        self._weights_seen: list[tuple[str, Any]] | None = None   # (placeholder, device tensor) of the prepared weight set
        self._weight_tensors: dict[str, Any] = {}
        self._weight_cache: dict[tuple[str, str], Any] = {}
        self._prepared: dict[str, Any] = {}
        self._plans: dict[tuple, _Plan] = {}
        self.last_launch_count = 0

    # ------------------------------------------------------------------ public
    def _device_guard(self):
        """The library launches on the current device; make it this executor's for the call."""
        return torch.cuda.device(self._device) if self._on_gpu else contextlib.nullcontext()

    def _input_tensors(self, inputs: dict[str, Any]) -> dict[str, Any]:
        tensors = {n: inputs[n].native_handle for n in self._input_names if n in inputs}
        dev = self._torch_device
        for n, t in tensors.items():   # (device objects compare in C; a decode step passes 60 buffers per call)
            if t.device != dev and not (dev.type == "cuda" and t.device.type == "cuda" and t.device.index in (None, dev.index)):
                raise ValueError(f"input '{n}' lives on {t.device}, this executor runs on {self._device}")
        return tensors

    def run(self, inputs: dict[str, Any], weights: dict[str, Any]) -> dict[str, Any]:
        with self._device_guard():
            return self._run(inputs, weights)

    def _run(self, inputs: dict[str, Any], weights: dict[str, Any]) -> dict[str, Any]:
        from cuda_runtime.cuda_backend import CUDABuffer

        self._check_weights(weights)
        tensors = self._input_tensors(inputs)
        key = tuple((n, t.data_ptr(), t.dtype) for n, t in tensors.items())
        if not all(map(_CONTIGUOUS, tensors.values())):   # not the plan of a contiguous tensor that had this address: binding refuses it
            key += tuple(n for n, t in tensors.items() if not t.is_contiguous())
        plan = self._plans.get(key)
        if plan is None:
            if len(self._plans) >= 8:
                self._plans.pop(next(iter(self._plans)))
            plan = self._bind(tensors)
            self._plans[key] = plan
        self._launch(plan)
        self.last_launch_count = plan.n_kernels
        # the same arena views on every replay of this plan: wrapped once (and again if a caller re-pointed a wrapper)
        cached = plan.out_buffers
        if cached is None or not all(map(operator.is_, map(_HANDLE, cached.values()), plan.outputs.values())):
            cached = plan.out_buffers = {name: CUDABuffer(t, logical_shape=tuple(t.shape)) for name, t in plan.outputs.items()}
        return dict(cached)

    def profile(self, inputs: dict[str, Any], weights: dict[str, Any]) -> list[tuple[str, float]]:
        """Run once without a CUDA graph, bracketing every library call with CUDA events on
        the launching stream.  Returns ``[(entry point, milliseconds), ...]`` in issue order.
        (The reference's profiler times whole runs with a host clock, npu_runtime/profiler.py:23-49.)"""
        if not self._on_gpu:
            raise RuntimeError("profile() needs a CUDA device")
        self._check_weights(weights)
        tensors = {n: inputs[n].native_handle for n in self._input_names if n in inputs}
        plan = self._bind(tensors)
        stream = torch.cuda.current_stream()
        events = []
        for fn, args in plan.launches:
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            rc = fn(*args, stream.cuda_stream)
            b.record(stream)
            if rc != 0:
                native.check(rc, fn.__name__)
            events.append((fn.__name__, a, b))
        stream.synchronize()
        return [(name, a.elapsed_time(b)) for name, a, b in events]

    def profile_entry(self, inputs: dict[str, Any], weights: dict[str, Any], entry: str, iters: int = 10) -> tuple[int, float]:
        """Time only the calls of one entry point: they are captured, in program order, into a
        CUDA graph of their own, and replays of that graph are timed with CUDA events on the
        launching stream (no host time between the launches).  Returns ``(calls per replay,
        mean milliseconds per call)``.  The calls read whatever their input buffers hold and
        write their usual outputs, so run it after the measurement proper, not in between."""
        if not self._on_gpu:
            raise RuntimeError("profile_entry() needs a CUDA device")
        self._check_weights(weights)
        tensors = {n: inputs[n].native_handle for n in self._input_names if n in inputs}
        plan = self._bind(tensors)
        calls = [(fn, args) for fn, args in plan.launches if fn.__name__ == entry]
        if not calls:
            return 0, 0.0
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(side):
            for fn, args in calls:   # warm-up outside the capture (one-off set-up inside the library)
                native.check(fn(*args, side.cuda_stream), entry)
            side.synchronize()
            with torch.cuda.graph(graph, stream=side):
                for fn, args in calls:
                    native.check(fn(*args, torch.cuda.current_stream().cuda_stream), entry)
        torch.cuda.synchronize()
        stream = torch.cuda.current_stream()
        graph.replay()
        times = []
        for _ in range(iters):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            graph.replay()
            b.record(stream)
            stream.synchronize()
            times.append(a.elapsed_time(b))
        return len(calls), float(sum(times) / len(times) / len(calls))

    # --------------------------------------------------------------- launching
    def _stream_ptr(self) -> int:
        return torch.cuda.current_stream().cuda_stream if self._on_gpu else 0

    def _issue(self, plan: _Plan, stream: int) -> None:
        for fn, args in plan.launches:
            rc = fn(*args, stream)
            if rc != 0:
                native.check(rc, getattr(fn, "__name__", "call"))

    def _launch(self, plan: _Plan) -> None:
        plan.runs += 1
        if plan.graph is not None:
            plan.graph.replay()
            return
        if self._use_graph and plan.runs == 2:
            graph = torch.cuda.CUDAGraph()
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.graph(graph, stream=side):
                self._issue(plan, torch.cuda.current_stream().cuda_stream)
            plan.graph = graph
            graph.replay()
            return
        self._issue(plan, self._stream_ptr())

    # ----------------------------------------------------------------- weights
    def _check_weights(self, weights: dict[str, Any]) -> None:
        """Prepare the weights again when any buffer of the set was replaced.  The reference reads
        the dict on every run (cuda_executor.py:153-164); here narrowed copies, folded convolution
        filters and bound pointers hang off the tensors, so the set is compared entry by entry
        (same names, same device tensors) - swapping one buffer inside the same dict counts."""
        seen = self._weights_seen
        if seen is not None and len(seen) == len(weights):
            # names as one list comparison, tensors by identity through C-level iterators: this runs before every launch
            if list(weights) == self._weights_names and all(map(operator.is_, self._weights_handles, map(_HANDLE, weights.values()))):
                return
        self._load_weights(weights)

    def _load_weights(self, weights: dict[str, Any]) -> None:
        self._weights_seen = [(n, b.native_handle) for n, b in weights.items()]
        self._weights_names = [n for n, _ in self._weights_seen]
        self._weights_handles = [t for _, t in self._weights_seen]
        self._weight_tensors = {n: b.native_handle for n, b in weights.items()}
        self._weight_cache.clear()
        self._prepared.clear()
        self._plans.clear()
        for key, const in (self._program.constants or {}).items():
            for ph, k in self._program.weight_name_mapping.items():
                if k == key and ph not in self._weight_tensors:
                    self._weight_tensors[ph] = torch.tensor(const.get("data", []), dtype=getattr(torch, const["dtype"]),
                                                            device=self._device).reshape(const["shape"])
        stream = self._stream_ptr()
        for prep in self._program.weight_preps:
            if prep.kind == "conv_fold":
                self._prep_conv(prep, stream)
            elif prep.kind == "concat_rows":
                self._prep_concat(prep)
            elif prep.kind == "interleave_rows":
                self._prep_interleave(prep)
            elif prep.kind == "scale_cols":
                self._prep_scale_cols(prep)
            else:
                raise RuntimeError(f"unknown weight preparation {prep.kind}")

    def _raw_weight(self, name: str):
        t = self._weight_tensors.get(name)
        if t is None:
            raise RuntimeError(f"weight '{name}' was not provided to CUDAExecutor.run")
        return t

    def _weight(self, name: str, dtype: str):
        """Weight ``name`` in ``dtype``; narrowed/widened once on the device if the
        upload has another floating type."""
        t = self._raw_weight(name)
        want = getattr(torch, dtype)
        if t.dtype == want and t.is_contiguous():
            return t
        cached = self._weight_cache.get((name, dtype))
        if cached is None:
            src = t if t.is_contiguous() else t.contiguous()
            cached = torch.empty(src.shape, dtype=want, device=self._device)
            self._convert(src, cached)
            self._weight_cache[(name, dtype)] = cached
        return cached

    def _convert(self, src, dst) -> None:
        """dst = cast(src) through the library's strided copy (both contiguous)."""
        n = src.numel()
        if n == 0:
            return
        a = native.make_tensor(dst.data_ptr(), str(dst.dtype).replace("torch.", ""), (n,), (1,))
        b = native.make_tensor(src.data_ptr(), str(src.dtype).replace("torch.", ""), (n,), (1,))
        native.check(self._lib.b200_strided_copy(C.byref(a), C.byref(b), self._stream_ptr()), "weight cast")

    def _scale_cols(self, mat, rows: int, cols: int, gain_name: str) -> None:
        """mat[rows, cols] *= gain[cols] (rounded to mat's dtype), in place: an RMSNorm gain folded into the
        columns of the weights that consume the normalised activations."""
        dt = str(mat.dtype).replace("torch.", "")
        gain = self._weight(gain_name, dt)
        out = native.make_tensor(mat.data_ptr(), dt, (rows, cols), (cols, 1))
        ins = (native.Tensor * 2)(native.make_tensor(mat.data_ptr(), dt, (rows, cols), (cols, 1)),
                                  native.make_tensor(gain.data_ptr(), dt, (rows, cols), (0, 1)))
        ops = (native.EwOp * 1)(native.EwOp(EW_OPCODES["MUL"], 0, 1, DTYPE_CODES[dt], 0.0))
        native.check(self._lib.b200_ew_chain(C.byref(out), ins, 2, ops, 1, self._stream_ptr()), "gain folding")

    def _prep_scale_cols(self, prep) -> None:
        p = prep.params
        src = self._weight(prep.inputs[0], p["dtype"])
        out = src.clone()      # the unscaled weight may serve other layers (a tied embedding table)
        self._scale_cols(out, p["rows"], p["cols"], prep.inputs[1])
        self._prepared[prep.outputs[0]] = out

    def _prep_concat(self, prep) -> None:
        """Row-wise concatenation of weights (merged q/k/v projection), in the compute dtype."""
        p = prep.params
        dt = getattr(torch, p["dtype"])
        cols = p["cols"]
        out = torch.empty(sum(p["rows"]) * cols, dtype=dt, device=self._device)
        at = 0
        for name, rows in zip(prep.inputs, p["rows"]):
            src = self._raw_weight(name)
            src = src if src.is_contiguous() else src.contiguous()
            if src.numel() != rows * cols:
                raise RuntimeError(f"weight '{name}' has {src.numel()} elements, expected {rows * cols}")
            self._convert(src.reshape(-1), out[at:at + rows * cols])
            at += rows * cols
        if p.get("col_scale"):
            self._scale_cols(out, sum(p["rows"]), cols, p["col_scale"])
        self._prepared[prep.outputs[0]] = out

    def _prep_interleave(self, prep) -> None:
        """Gate and up projection rows interleaved in blocks (gated-MLP GEMM), in the compute dtype."""
        p = prep.params
        rows, cols, blk = p["rows"], p["cols"], p["block"]
        out = torch.empty(2 * rows * cols, dtype=getattr(torch, p["dtype"]), device=self._device)
        for half, name in enumerate(prep.inputs):
            src = self._raw_weight(name)
            src = src if src.is_contiguous() else src.contiguous()
            if src.numel() != rows * cols:
                raise RuntimeError(f"weight '{name}' has {src.numel()} elements, expected {rows * cols}")
            dst = native.make_tensor(out.data_ptr() + half * blk * cols * out.element_size(), p["dtype"], (rows // blk, blk, cols),
                                     (2 * blk * cols, cols, 1))
            s_t = native.make_tensor(src.data_ptr(), str(src.dtype).replace("torch.", ""), (rows // blk, blk, cols), (blk * cols, cols, 1))
            native.check(self._lib.b200_strided_copy(C.byref(dst), C.byref(s_t), self._stream_ptr()), "weight interleave")
        if p.get("col_scale"):
            self._scale_cols(out, 2 * rows, cols, p["col_scale"])
        self._prepared[prep.outputs[0]] = out

    def _prep_conv(self, prep, stream: int) -> None:
        p = prep.params
        w = self._raw_weight(prep.inputs[0])
        opt = [self._raw_weight(n) if n is not None else None for n in prep.inputs[1:]]
        params = [t for t in opt if t is not None]
        pdt = params[0].dtype if params else torch.float32
        if any(t.dtype != pdt for t in params):
            raise RuntimeError("convolution bias and batch-norm parameters must share one dtype")
        out_dt = getattr(torch, p["dtype"])
        wout = torch.empty(p["O"] * p["KH"] * p["KW"] * p["I_pad"], dtype=out_dt, device=self._device)
        bout = torch.empty(p["O"], dtype=torch.float32, device=self._device)
        name = lambda t: str(t.dtype).replace("torch.", "")
        ptr = lambda t: t.data_ptr() if t is not None else None
        wc = w if w.is_contiguous() else w.contiguous()
        native.check(self._lib.b200_conv_weight_prep(
            wc.data_ptr(), ptr(opt[0]), ptr(opt[1]), ptr(opt[2]), ptr(opt[3]), ptr(opt[4]), wout.data_ptr(), bout.data_ptr(),
            p["O"], p["I"], p["KH"], p["KW"], p["I_pad"], float(p["eps"]), DTYPE_CODES[name(wc)],
            DTYPE_CODES[name(params[0])] if params else 0, DTYPE_CODES[p["dtype"]], stream), "conv weight prep")
        self._prepared[prep.outputs[0]] = wout
        self._prepared[prep.outputs[1]] = bout

    # ----------------------------------------------------------------- binding
    def _bind(self, inputs: dict[str, Any]) -> _Plan:
        plan = _Plan()
        self._cur_inputs = inputs
        self._cur_plan = plan
        self._staged: dict[str, Any] = {}
        merged = {}   # steps that one kernel stands for: nothing to bind, except at the last of them
        for at in self._stems:
            copy, conv, pool = (self._program.steps[i].params for i in at)
            if self._ptr(copy["in_view"]) % 16 == 0:   # TMA: a slice of a larger tensor may start anywhere
                merged.update({at[0]: None, at[1]: None, at[2]: (copy, conv, pool)})
        for i, step in enumerate(self._program.steps):
            if isinstance(step, AliasStep):
                continue
            p = step.params
            if i not in merged:
                getattr(self, "_bind_" + p["op"])(plan, step, p)
            elif merged[i] is not None:
                self._bind_stem_pool(plan, *merged[i])
        # every library call is one kernel, except decode attention when its splits are merged by a
        # second kernel (the library then asks for a workspace; with in-kernel merging it asks for none)
        def _two_kernels(q) -> bool:
            if not (q and q.get("op") == "attention" and q["decode"]):
                return False
            if not hasattr(self._lib, "b200_attn_decode_workspace_bytes"):
                return True
            return int(self._lib.b200_attn_decode_workspace_bytes(q["B"], q["Hq"], q["Hkv"], q["S"], q["D"])) > 0
        plan.n_kernels = len(plan.launches) + sum(1 for s in self._program.steps if _two_kernels(getattr(s, "params", None)))
        for spec in self._program.output_specs:
            view = self._program.views.get(spec.name)
            if view is None:
                continue
            plan.outputs[spec.name] = self._as_torch(view)
        return plan

    def _base(self, view: TensorView, any_dtype: bool = False):
        """(device address of element 0 of the view's buffer, dtype actually stored there)."""
        name = view.buffer
        alloc = self._allocs.get(name)
        if alloc is not None and name not in self._ws:
            return self._arena.data_ptr() + alloc.offset, view.dtype
        if name in self._ws:
            return self._ws[name].data_ptr(), view.dtype
        if name in self._input_set:
            t = self._cur_inputs.get(name)
            if t is None:
                raise RuntimeError(f"graph input '{name}' was not provided to CUDAExecutor.run")
            have = str(t.dtype).replace("torch.", "")
            if have == "bool":
                have = "uint8"
            if not t.is_contiguous():   # views are strides of the declared shape, and a conversion takes the elements as they lie
                raise RuntimeError(f"graph input '{name}' must be contiguous")
            if have == view.dtype or any_dtype:
                return t.data_ptr(), have
            staged = self._staged.get(name)
            if staged is None:  # per-run conversion into the dtype the kernels expect
                staged = torch.empty(t.shape, dtype=getattr(torch, view.dtype), device=self._device)
                self._staged[name] = staged
                n = t.numel()
                a = native.make_tensor(staged.data_ptr(), view.dtype, (n,), (1,))
                b = native.make_tensor(t.data_ptr(), have, (n,), (1,))
                self._cur_plan.keepalive += [a, b, staged]
                self._cur_plan.launches.append((self._lib.b200_strided_copy, (C.byref(a), C.byref(b))))
            return staged.data_ptr(), view.dtype
        if name in self._prepared:
            return self._prepared[name].data_ptr(), view.dtype
        return self._weight(name, view.dtype).data_ptr(), view.dtype

    def _ptr(self, view: TensorView | None) -> int | None:
        if view is None:
            return None
        base, _ = self._base(view)
        return base + view.offset * DTYPE_BYTES[view.dtype]

    def _wptr(self, name: str | None, dtype: str | None = None) -> int | None:
        if name is None:
            return None
        view = self._program.views[name]
        return self._ptr(view if dtype is None else TensorView(view.buffer, view.offset, view.shape, view.strides, dtype))

    def _tensor(self, plan: _Plan, view: TensorView, any_dtype: bool = False):
        base, dtype = self._base(view, any_dtype)
        t = native.make_tensor(base + view.offset * DTYPE_BYTES[dtype], dtype, view.shape, view.strides)
        plan.keepalive.append(t)
        return t

    def _as_torch(self, view: TensorView):
        base, dtype = self._base(view)
        name = view.buffer
        if name in self._input_set and name not in self._staged:
            root = self._cur_inputs[name]
        elif name in self._staged:
            root = self._staged[name]
        elif name in self._allocs and name not in self._ws:
            a = self._allocs[name]
            root = self._arena[a.offset:a.offset + a.size_bytes].view(getattr(torch, dtype))
        elif name in self._prepared:
            root = self._prepared[name]
        else:
            root = self._weight(name, view.dtype)
        flat = root.reshape(-1)  # as_strided offsets are absolute in the storage
        return torch.as_strided(flat, tuple(view.shape), tuple(view.strides), flat.storage_offset() + view.offset)

    # one binder per library entry point --------------------------------------------
    def _bind_ew_chain(self, plan, step, p):
        out = self._tensor(plan, p["out_view"])
        ins = (native.Tensor * len(p["in_views"]))()
        for i, v in enumerate(p["in_views"]):
            base, dtype = self._base(v, any_dtype=True)
            ins[i] = native.make_tensor(base + v.offset * DTYPE_BYTES[dtype], dtype, v.shape, v.strides)
        ops = (native.EwOp * len(p["program"]))()
        for i, (name, a, b, rd, imm) in enumerate(p["program"]):
            ops[i] = native.EwOp(EW_OPCODES[name], a, b, DTYPE_CODES[rd], float(imm))
        plan.keepalive += [ins, ops]
        plan.launches.append((self._lib.b200_ew_chain, (C.byref(out), ins, len(p["in_views"]), ops, len(p["program"]))))

    def _bind_strided_copy(self, plan, step, p):
        dst = self._tensor(plan, p["out_view"])
        src = self._tensor(plan, p["in_view"], any_dtype=True)
        plan.launches.append((self._lib.b200_strided_copy, (C.byref(dst), C.byref(src))))

    def _bind_fill(self, plan, step, p):
        y = p["y"]
        plan.launches.append((self._lib.b200_fill, (self._ptr(y), y.numel, float(p["fill_value"]), DTYPE_CODES[y.dtype])))

    def _bind_rmsnorm(self, plan, step, p):
        x, y = p["x"], p["y"]
        plan.launches.append((self._lib.b200_rmsnorm, (self._ptr(x), self._wptr(p["w"], x.dtype), self._ptr(y), p["rows"], p["cols"],
                                                       x.strides[0] if p["rows"] > 1 else p["cols"], p["cols"], float(p["eps"]),
                                                       DTYPE_CODES[x.dtype], int(p["round_mid"]))))

    def _bind_softmax(self, plan, step, p):
        x, y, m = p["x"], p["y"], p["mask"]
        d0, d1, d2 = p["dims"]
        ms = p["mask_strides"]
        plan.launches.append((self._lib.b200_softmax, (self._ptr(x), self._ptr(m), self._ptr(y), d0, d1, d2, p["cols"], ms[0], ms[1],
                                                       ms[2], float(p["scale"]), DTYPE_CODES[x.dtype],
                                                       DTYPE_CODES[m.dtype] if m is not None else 0, DTYPE_CODES[y.dtype],
                                                       int(p["round_steps"]))))

    def _bind_mean_last_dim(self, plan, step, p):
        x, y = p["x"], p["y"]
        plan.launches.append((self._lib.b200_mean_last_dim, (self._ptr(x), self._ptr(y), p["rows"], p["cols"], DTYPE_CODES[x.dtype],
                                                             DTYPE_CODES[y.dtype])))

    def _bind_argmax(self, plan, step, p):
        x, y = p["x"], p["y"]
        plan.launches.append((self._lib.b200_argmax_rows, (self._ptr(x), self._ptr(y), p["rows"], p["cols"], p["cols"],
                                                           DTYPE_CODES[x.dtype])))

    def _bind_embedding(self, plan, step, p):
        ids, y = p["ids"], p["y"]
        base, ids_dtype = self._base(ids, any_dtype=True)
        if ids_dtype not in ("int64", "int32"):
            raise RuntimeError(f"embedding indices arrived as {ids_dtype}; upload them as int64/int32")
        row_bytes = p["embed_dim"] * DTYPE_BYTES[y.dtype]
        plan.launches.append((self._lib.b200_embedding, (self._wptr(p["table"], y.dtype), base + ids.offset * DTYPE_BYTES[ids_dtype],
                                                         self._ptr(y), p["seq_len"], p["vocab"], row_bytes, DTYPE_CODES[ids_dtype])))

    def _index_ptr(self, view: TensorView):
        base, dtype = self._base(view, any_dtype=True)
        if dtype not in ("int64", "int32"):
            raise RuntimeError(f"index tensor '{view.buffer}' arrived as {dtype}; upload it as int64/int32")
        return base + view.offset * DTYPE_BYTES[dtype], DTYPE_CODES[dtype]

    def _bind_index_copy(self, plan, step, p):
        base, dst, src = p["base"], p["dst"], p["src"]
        iptr, idt = self._index_ptr(p["index"])
        plan.launches.append((self._lib.b200_index_copy, (self._ptr(base), self._ptr(dst), self._ptr(src), iptr, p["outer_size"],
                                                          p["dim_size"], p["inner_size"], p["num_indices"], src.strides[0],
                                                          src.strides[1], DTYPE_BYTES[dst.dtype], idt)))

    def _bind_rope_table(self, plan, step, p):
        pptr, pdt = self._index_ptr(p["pos"])
        plan.launches.append((self._lib.b200_rope_table, (self._wptr(p["inv_freq"], "float32"), pptr, self._ptr(p["cos"]),
                                                          self._ptr(p["sin"]), p["seq_len"], p["head_dim"], pdt,
                                                          DTYPE_CODES[p["cos"].dtype])))

    def _bind_rope_rotate(self, plan, step, p):
        x = self._tensor(plan, p["x"])
        plan.launches.append((self._lib.b200_rope_rotate, (C.byref(x), self._ptr(p["cos"]), self._ptr(p["sin"]), self._ptr(p["y"]),
                                                           None, None, 0, 0)))

    def _bind_rope_rotate_pair(self, plan, step, p):
        q, k = self._tensor(plan, p["q"]), self._tensor(plan, p["k"])
        plan.launches.append((self._lib.b200_rope_rotate_pair, (C.byref(q), C.byref(k), self._ptr(p["cos"]), self._ptr(p["sin"]),
                                                                self._ptr(p["q_out"]), self._ptr(p["k_out"]))))

    def _bind_qkv_post(self, plan, step, p):
        q, k, v = (self._tensor(plan, p[n]) for n in ("q", "k", "v"))
        iptr, idt = self._index_ptr(p["index"])
        plan.launches.append((self._lib.b200_qkv_rope_cache, (C.byref(q), C.byref(k), C.byref(v), self._ptr(p["cos"]), self._ptr(p["sin"]),
                                                              self._ptr(p["q_out"]), self._ptr(p["k_cache"]), self._ptr(p["v_cache"]), iptr,
                                                              p["cache_len"], idt)))

    def _bind_linear_qkv_rope(self, plan, step, p):
        x, r = p["x"], p["rope"]
        dt = p["y"].dtype
        epi = native.EPI_W_STATIC if (p["w"] in self._weight_tensors or p["w"] in self._prepared) else 0
        ld = lambda v: v.strides[0] if v.shape[0] > 1 else v.shape[1]
        norm = p.get("norm")
        iptr, idt = self._index_ptr(r["index"])
        plan.launches.append((self._lib.b200_linear_qkv_rope, (
            self._ptr(x), self._wptr(p["w"], dt), self._wptr(p["bias"], dt), p["M"], p["N"], p["K"], ld(x), p["K"], DTYPE_CODES[dt], DTYPE_CODES[dt],
            epi, float(norm["eps"]) if norm else 0.0, self._ptr(norm["sumsq"]) if norm else None, int(norm["cols"]) if norm else 0,
            self._ptr(r["cos"]), self._ptr(r["sin"]), self._ptr(r["q_out"]), self._ptr(r["k_cache"]), self._ptr(r["v_cache"]), iptr,
            int(r["cache_len"]), idt, int(p["Hq"]), int(p["Hkv"]))))

    def _bind_max_pool2d(self, plan, step, p):
        x, y = self._tensor(plan, p["x"]), self._tensor(plan, p["y"])
        plan.launches.append((self._lib.b200_max_pool2d, (C.byref(x), C.byref(y), p["kernel_h"], p["kernel_w"], p["stride_h"],
                                                          p["stride_w"], p["pad_h"], p["pad_w"])))

    def _bind_adaptive_avg_pool2d(self, plan, step, p):
        x, y = self._tensor(plan, p["x"]), self._tensor(plan, p["y"])
        plan.launches.append((self._lib.b200_adaptive_avg_pool2d, (C.byref(x), C.byref(y))))

    def _bind_batch_norm(self, plan, step, p):
        x, y = self._tensor(plan, p["x"]), self._tensor(plan, p["y"])
        pd = "float32"
        g = lambda n: self._weight(n, pd).data_ptr() if n is not None else None
        plan.launches.append((self._lib.b200_batch_norm, (C.byref(x), C.byref(y), g(p["gamma"]), g(p["beta"]), g(p["mean"]), g(p["var"]),
                                                          float(p["eps"]), DTYPE_CODES[pd], int(p["relu"]))))

    def _bind_linear(self, plan, step, p):
        x, y = p["x"], p["y"]
        dt = y.dtype
        res, aux = p["residual"], p["aux"]
        epi = (native.EPI_RELU if p["relu"] else 0) | (native.EPI_SILU_MUL if aux is not None else 0) | (native.EPI_GLU if p.get("glu") else 0)
        if p["w"] in self._weight_tensors or p["w"] in self._prepared:
            epi |= native.EPI_W_STATIC   # model weight: may be prefetched ahead of the previous kernel's completion
        ws = self._ws["__ws_splitk"] if p["workspace"] else None
        ld = lambda v: (v.strides[0] if v.shape[0] > 1 else v.shape[1]) if v is not None else 0
        norm, sumsq_out = p.get("norm"), p.get("sumsq_out")
        if norm is not None or sumsq_out is not None:   # decode shapes: RMSNorm folded into its neighbours
            plan.launches.append((self._lib.b200_linear_norm, (
                self._ptr(x), self._wptr(p["w"], dt), self._wptr(p["bias"], dt), self._ptr(res), self._ptr(y), p["M"], p["N"], p["K"],
                ld(x), p["K"], ld(y), ld(res), DTYPE_CODES[dt], DTYPE_CODES[dt], epi,
                float(norm["eps"]) if norm else 0.0, self._ptr(norm["sumsq"]) if norm else None, int(norm["cols"]) if norm else 0,
                self._ptr(sumsq_out))))
            return
        tail = p.get("norm_tail")
        if tail is not None:   # the RMSNorm of the result rides on the kernel that adds up the split-K partial sums
            plan.launches.append((self._lib.b200_linear_rmsnorm, (
                self._ptr(x), self._wptr(p["w"], dt), self._wptr(p["bias"], dt), self._ptr(res), self._ptr(y), p["M"], p["N"], p["K"],
                ld(x), p["K"], ld(y), ld(res), DTYPE_CODES[dt], DTYPE_CODES[dt], epi,
                ws.data_ptr() if ws is not None else None, ws.numel() if ws is not None else 0,
                self._wptr(tail["w"], dt), self._ptr(tail["y"]), p["N"], float(tail["eps"]), int(tail["round_mid"]))))
            return
        plan.launches.append((self._lib.b200_linear, (
            self._ptr(x), self._wptr(p["w"], dt), self._wptr(p["bias"], dt), self._ptr(res), self._ptr(y), p["M"], p["N"], p["K"],
            ld(x), p["K"], ld(y), ld(res), DTYPE_CODES[dt], DTYPE_CODES[dt], epi, self._ptr(aux), ld(aux),
            ws.data_ptr() if ws is not None else None, ws.numel() if ws is not None else 0)))

    def _bind_matmul(self, plan, step, p):
        a, b, y = p["a"], p["b"], p["y"]
        arr = lambda v: (C.c_int64 * 4)(*v.strides)
        sa, sb, so = arr(a), arr(b), arr(y)
        plan.keepalive += [sa, sb, so]
        plan.launches.append((self._lib.b200_matmul_strided, (self._ptr(a), self._ptr(b), self._ptr(y), p["b1"], p["b2"], p["M"], p["N"],
                                                              p["K"], sa, sb, so, DTYPE_CODES[y.dtype])))

    def _bind_conv2d(self, plan, step, p):
        x, y, res = p["x"], p["y"], p["residual"]
        epi = native.EPI_RELU if p["relu"] else 0
        plan.launches.append((self._lib.b200_conv2d_nhwc, (
            self._ptr(x), self._prepared[p["w_prepared"]].data_ptr(), self._prepared[p["bias_prepared"]].data_ptr(), self._ptr(res),
            self._ptr(y), p["batch"], p["in_h"], p["in_w"], p["c_pad"], p["c_pad"], p["out_channels"], p["kernel_h"], p["kernel_w"],
            p["stride_h"], p["stride_w"], p["pad_h"], p["pad_w"], p["out_h"], p["out_w"], DTYPE_CODES[y.dtype], epi)))

    def _bind_stem_pool(self, plan, copy, conv, pool):
        x = copy["in_view"]
        plan.launches.append((self._lib.b200_conv_stem_pool, (
            self._ptr(x), self._prepared[conv["w_prepared"]].data_ptr(), self._prepared[conv["bias_prepared"]].data_ptr(), self._ptr(pool["y"]),
            *x.shape, conv["c_pad"], conv["out_channels"], conv["kernel_h"], conv["kernel_w"], conv["stride_h"], conv["stride_w"], conv["pad_h"],
            conv["pad_w"], DTYPE_CODES[x.dtype], native.EPI_RELU if conv["relu"] else 0)))

    def _bind_attention(self, plan, step, p):
        q, k, v, m, y = p["q"], p["k"], p["v"], p["mask"], p["y"]
        dt = DTYPE_CODES[y.dtype]
        if p["decode"]:
            ws = self._ws["__ws_attn"]
            plan.launches.append((self._lib.b200_attn_decode, (
                self._ptr(q), self._ptr(k), self._ptr(v), self._ptr(m), self._ptr(y), p["B"], p["Hq"], p["Hkv"], p["S"], p["D"],
                q.strides[0], k.strides[0], k.strides[1], m.strides[0] if m is not None else 0, float(p["scale"]), dt,
                ws.data_ptr(), ws.numel())))
            return
        arr = lambda t: (C.c_int64 * 3)(*t.strides[:3])
        qs, ks, vs = arr(q), arr(k), arr(v)
        plan.keepalive += [qs, ks, vs]
        plan.launches.append((self._lib.b200_attn_prefill_tiles, (
            self._ptr(q), self._ptr(k), self._ptr(v), self._ptr(m), self._mask_tiles(plan, m), self._ptr(y), p["B"], p["Hq"], p["Hkv"], p["T"], p["S"], p["D"],
            qs, ks, vs, m.strides[0] if m is not None else 0, m.strides[2] if m is not None else 0, float(p["scale"]), dt)))

    def _mask_tiles(self, plan, m: TensorView | None) -> int | None:
        """Address of the states of a mask's tiles.  They are found once per call for all layers that share the mask: looked
        for by every head of every layer, the mask of a 2048-token prompt is 100 MB of L2 traffic per layer."""
        if m is None:
            return None
        key = _mask_key(m)
        if not self._lib.b200_attn_prefill_reads_tiles(self._ptr(m), key[4], m.strides[0], m.strides[2], DTYPE_CODES[m.dtype]):
            return None
        tiles = self._tiles[key].data_ptr()
        if key not in plan.masks_seen:
            plan.masks_seen.add(key)
            plan.launches.append((self._lib.b200_mask_tiles, (self._ptr(m), key[2], key[3], key[4], m.strides[0], m.strides[2],
                                                              DTYPE_CODES[m.dtype], tiles)))
        return tiles
