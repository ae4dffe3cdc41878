"""Decode-step execution: one cached single-token forward plus arg-max, captured once in a CUDA graph and
replayed per generated token, so that the ~50 us of weight streaming a step needs is not buried under
host-side launch overhead."""
from __future__ import annotations

from typing import List, Optional

import torch

from . import _lib, kernels
from .models.utils import RecurrentCache
from .ops.fusedbitnet import BitLinear


class GreedyDecoder:
    """Greedy decoding for a fixed batch size with device-resident state.

    `prefill(prompt)` runs the prompt once and seeds the static cache and the first token; each `step()`
    replays the captured graph: it reads `self.ids` [B,1], advances every layer's recurrent state in place,
    writes the next token to `self.next` [B], which is the same buffer as `self.ids`.
    """

    def __init__(self, model, batch_size: int, use_graph: bool = True):
        self.model, self.B = model, batch_size
        dev = next(model.parameters()).device
        self.device = dev
        # `next` [B] and `ids` [B,1] are two views of one buffer: the arg-max of a step writes the next step's input
        self.next = torch.zeros(batch_size, dtype=torch.int64, device=dev)
        self.ids = self.next.view(batch_size, 1)
        self.cache = model.model.init_cache(batch_size)
        self.graph: Optional[torch.cuda.CUDAGraph] = None
        self._graph_logits: Optional[torch.Tensor] = None     # [B, V] buffer that a replay of self.graph writes
        self._graph_reads: list = []
        self.kernels_per_step = 0
        self.last_logits: Optional[torch.Tensor] = None
        self._use_graph = use_graph
        # prompt passes of a repeated length are replayed from a graph as well: an eager pass is about 200 launches of
        # about 2 us of host time each, and a step of few sequences needs little more on the GPU
        self._prompt_seen: dict = {}       # prompt length -> times seen
        self._prompt_graphs: dict = {}     # prompt length -> (graph, static ids and logits buffers, what it reads), at most PROMPT_GRAPHS entries
        self._host_graphs: dict = {}       # (ids_host ptr, out_host ptr) -> (graph with the two copies, its logits buffer, what it reads, the host buffers)

    def _step_eager(self) -> torch.Tensor:
        """One step; returns its logits [B, V].  Inside a captured graph they are a fixed buffer that every replay of that
        graph rewrites: a caller that samples instead of taking the arg-max reads self.last_logits after step() and
        overwrites self.next."""
        out = self.model(input_ids=self.ids, past_key_values=self.cache, use_cache=True)
        logits = out.logits[:, -1]
        kernels.argmax_rows(logits, out=self.next)
        return logits

    def _read_by_graphs(self) -> list:
        """What a captured pass reads through raw addresses and the model may drop later (weights replaced or repacked): kept with
        the graph, whose replays then still compute what was captured instead of reading freed memory."""
        model = self.model
        runner = getattr(model, "_fused_runner", None)
        if runner is not None and model.fuse:
            return [runner]
        layers = bitlinear_modules(model)
        latent = {id(m.weight) for m in layers}
        return [(m._packed, m._norm_w32, m._norm_seen) for m in layers] + [p.detach() for p in model.parameters() if id(p) not in latent]

    def _prepare_step(self) -> None:
        if hasattr(self.model, "prepare_step"):    # (a model of the caller's own need not have it)
            self.model.prepare_step(self.ids)

    def _capture(self, ids_host: Optional[torch.Tensor] = None, out_host: Optional[torch.Tensor] = None):
        """Capture one decode step; returns (graph, its logits buffer, what it reads).  With pinned host buffers the copy of the input ids
        to the device and of the new tokens back are nodes of the same graph."""
        saved = [tuple(s.clone() for s in layer) for layer in self.cache.states]
        saved_ids = self.ids.clone()
        self._prepare_step()                       # here and not in the warm-up: the copy belongs to the stream that replays the step
        side = torch.cuda.Stream(device=self.device)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(2):                     # warm-up outside capture (allocator, lazy packing)
                self._step_eager()
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        before = _lib.launch_count
        # capture on the warm-up stream: its split-K workspace already exists (and is zero), so no fill of a
        # fresh workspace is recorded into the graph
        with torch.cuda.graph(graph, stream=side):
            if ids_host is not None:
                self.ids.copy_(ids_host, non_blocking=True)
            logits = self._step_eager()
            if out_host is not None:
                out_host.copy_(self.next, non_blocking=True)
        self.kernels_per_step = _lib.launch_count - before
        for layer, keep in zip(self.cache.states, saved):   # undo the warm-up steps' effect on the state
            for dst, src in zip(layer, keep):
                dst.copy_(src)
        self.ids.copy_(saved_ids)
        return graph, logits, self._read_by_graphs()

    PROMPT_GRAPH_MAX_TOKENS = 8192   # larger prompts are bound by the GPU, and their graphs would pin gigabytes
    PROMPT_GRAPHS = 4

    def _prefill_eager(self, prompt_ids: torch.Tensor, attention_mask: Optional[torch.Tensor] = None) -> torch.Tensor:
        torch._foreach_zero_([s for layer in self.cache.states for s in layer])
        out = self.model(input_ids=prompt_ids, attention_mask=attention_mask, past_key_values=self.cache, use_cache=True,
                         last_token_only=True)
        logits = out.logits[:, -1]
        kernels.argmax_rows(logits, out=self.next)
        return logits

    def _capture_prompt(self, T: int):
        ids = torch.zeros(self.B, T, dtype=torch.int64, device=self.device)
        if T == 1:                                 # (such a prompt is a step)
            self._prepare_step()
        side = torch.cuda.Stream(device=self.device)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            self._prefill_eager(ids)               # warm-up outside capture (allocator, workspace of this stream)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            logits = self._prefill_eager(ids)
        if len(self._prompt_graphs) >= self.PROMPT_GRAPHS:
            self._prompt_graphs.pop(next(iter(self._prompt_graphs)))
        self._prompt_graphs[T] = (graph, ids, logits, self._read_by_graphs())
        return self._prompt_graphs[T]

    @torch.no_grad()
    def prefill(self, prompt_ids: torch.Tensor, attention_mask: Optional[torch.Tensor] = None) -> torch.Tensor:
        """Run the prompt [B, T]; returns the first generated token [B] (also left in self.ids / self.next) and leaves
        the last position's logits [B, V] in self.last_logits.  The pass overwrites the recurrent state (a prompt starts
        from the zero state).  From the second prompt of the same length on, the pass is replayed from a CUDA graph
        (prompts with an attention_mask always run eagerly)."""
        if prompt_ids.shape[0] != self.B:
            raise ValueError(f"decoder was built for batch {self.B}, got {prompt_ids.shape[0]}")
        T = prompt_ids.shape[1]
        if self._use_graph and attention_mask is None and self.B * T <= self.PROMPT_GRAPH_MAX_TOKENS:
            entry = self._prompt_graphs.get(T)
            seen = self._prompt_seen.get(T, 0)
            self._prompt_seen[T] = seen + 1
            if entry is None and seen >= 1:
                entry = self._capture_prompt(T)
            if entry is not None:
                graph, ids, self.last_logits, _ = entry
                ids.copy_(prompt_ids)
                graph.replay()
                return self.next
        self.last_logits = self._prefill_eager(prompt_ids, attention_mask)
        return self.next

    @torch.no_grad()
    def seed(self, past_key_values, last_logits: torch.Tensor) -> torch.Tensor:
        """Take over after a prompt pass made elsewhere (e.g. one with a padding mask): copy its recurrent states
        into the static cache and pick the first token from its last-position logits [B, V], which become
        self.last_logits."""
        torch._foreach_copy_([s for layer in self.cache.states for s in layer], [s for layer in past_key_values for s in layer])
        kernels.argmax_rows(last_logits, out=self.next)
        self.last_logits = last_logits
        return self.next

    @torch.no_grad()
    def step(self) -> torch.Tensor:
        """Consume self.ids, produce the next token in self.next (and feed it back). Returns self.next."""
        if not self._use_graph:
            before = _lib.launch_count
            self.last_logits = self._step_eager()
            self.kernels_per_step = _lib.launch_count - before
        else:
            kernels.raise_if_gave_up(self.device)
            if self.graph is None:
                self.graph, self._graph_logits, self._graph_reads = self._capture()
            self.graph.replay()
            self.last_logits = self._graph_logits
        return self.next

    @torch.no_grad()
    def step_host(self, ids_host: torch.Tensor, out_host: torch.Tensor) -> None:
        """One decode step driven from the host: the token ids [B, 1] are read from `ids_host`, the new tokens [B] are
        written to `out_host` (both int64 in pinned memory); the step's logits are left in self.last_logits.  The two
        copies and the step's kernels are one CUDA graph launch; the call returns once it is enqueued — synchronise the
        stream before reading `out_host`."""
        if not (ids_host.is_pinned() and out_host.is_pinned()):
            raise ValueError("step_host needs pinned host buffers")
        if ids_host.shape != self.ids.shape or out_host.shape != self.next.shape or ids_host.dtype != torch.int64 \
                or out_host.dtype != torch.int64:
            raise ValueError(f"step_host needs int64 buffers of shape {tuple(self.ids.shape)} and {tuple(self.next.shape)}")
        if not self._use_graph:
            self.ids.copy_(ids_host, non_blocking=True)
            self.step()
            out_host.copy_(self.next, non_blocking=True)
            return
        kernels.raise_if_gave_up(self.device)
        key = (ids_host.data_ptr(), out_host.data_ptr())
        entry = self._host_graphs.get(key)
        if entry is None:
            entry = (*self._capture(ids_host, out_host), ids_host, out_host)   # the graph keeps pointing at these buffers
            self._host_graphs = {key: entry}
        entry[0].replay()
        self.last_logits = entry[1]

    @torch.no_grad()
    def generate(self, prompt_ids: torch.Tensor, max_new_tokens: int) -> torch.Tensor:
        toks = torch.empty(self.B, max_new_tokens, dtype=torch.int64, device=self.device)
        self.prefill(prompt_ids)
        for t in range(max_new_tokens):
            toks[:, t].copy_(self.next)
            if t + 1 < max_new_tokens:
                self.step()
        return torch.cat([prompt_ids, toks], dim=1)


class FusedRunner:
    """The HGRNBit forward as a chain of fused kernels: per block four BitLinear contractions, each fed int8
    codes by one fused row-wise kernel, plus the gated recurrence scan.

    Mathematically this is HGRNBitBlock.forward / HGRNBitAttention.forward / HGRNBitMLP.forward of the module
    path with the same rounding points; the i/f/g projections, which share their input row, run as one
    grouped contraction.  The chain itself is launched by native code (csrc/binding.cpp), which holds the pointers
    gathered here.  Built lazily from a model; rebuilt when a weight is repacked."""

    def __init__(self, lm):
        # (no reference to `lm`, which holds this object: a dropped model is freed at once, not by the cycle collector)
        model = lm.model
        cfg = lm.config
        self.device = model.embeddings.weight.device
        self.h = cfg.hidden_size
        self.dtype = model.embeddings.weight.dtype
        # per-layer lower bounds of the forget gates depend on parameters only: evaluated once (in the parameter
        # dtype, with the reference's op sequence) instead of on every forward
        with torch.no_grad():
            lbs = model.layer_lower_bounds()
        self.items = []                      # the packed weights of one pass, in execution order
        layers = []
        for i, blk in enumerate(model.layers):
            at, mlp = blk.attn, blk.mlp
            if at.input_dim != self.h:
                raise NotImplementedError("fused path needs expand_ratio == 1")
            ifg = kernels.stack_packed([at.i_proj.packed(), at.f_proj.packed(), at.g_proj.packed()])
            o, gate, down = at.o_proj.packed(), mlp.gate_proj.packed(), mlp.down_proj.packed()
            self.items += [ifg, o, gate, down]
            layers.append((
                self._w32(blk.attn_norm.weight), *self._linear(ifg),
                at.i_proj.norm_weight_f32(), at.f_proj.norm_weight_f32(), at.g_proj.norm_weight_f32(),
                lbs[i].contiguous() if (lbs is not None and i > 0) else None,
                self._w32(at.g_norm.weight), float(at.g_norm.eps),
                *self._linear(o), at.o_proj.norm_weight_f32(),
                self._w32(blk.mlp_norm.weight), *self._linear(gate), mlp.gate_proj.norm_weight_f32(),
                *self._linear(down), mlp.down_proj.norm_weight_f32(), float(at.i_proj.NORM_EPS)))
        head = lm.lm_head.packed()
        self.items.append(head)
        tail = (self._w32(model.norm.weight), *self._linear(head), lm.lm_head.norm_weight_f32(), float(cfg.rms_norm_eps),
                float(lm.lm_head.NORM_EPS))
        self._native = _lib.native()
        self.resident = bool(lm.resident_step)
        self.chain = self._native.chain(model.embeddings.weight, layers, tail, self.resident)
        self.watch = self._native.watch(self._slots(lm))

    @staticmethod
    def _w32(w):
        return None if w is None else w.detach().float().contiguous()

    @staticmethod
    def _linear(pw):
        return pw.packed, pw.scale, pw.N, pw.K, pw.groups

    @staticmethod
    def _slots(lm):
        """(parameter dict, name) of every parameter.  Walking the module tree costs about 2 ms on a 24-block model, so
        the slots are listed once per model object and only looked up afterwards; a replaced parameter is still seen,
        because the slot is read anew."""
        slots = lm.__dict__.get("_fused_param_slots")
        if slots is None:
            slots = [(m._parameters, n) for m in lm.modules() for n in m._parameters]
            object.__setattr__(lm, "_fused_param_slots", slots)
        return slots

    def prepare_step(self, batch: int) -> bool:
        """Do now, on the current stream, what the first decode step of `batch` sequences would do once for all: lay the weights out for
        the resident kernel.  True if those steps take it."""
        return self._native.prepare_step(self.chain, batch)

    def current(self) -> bool:
        """False once a parameter was replaced, cast or modified in place."""
        return self._native.unchanged(self.watch)

    @torch.no_grad()
    def forward(self, input_ids, inputs_embeds, states, last_only: bool, want_logits: bool = True,
                want_hidden: bool = False, attention_mask=None):
        """states: list of fp32 [B, ..., h]-shaped tensors advanced in place.  attention_mask: optional [B, T], zero at
        (left-)padding positions — their input to the recurrence is dropped, as the reference's attention layer does
        (layers/hgrn_bit.py:119-120), for a prompt inside the scan and for a single decode token inside the step kernel.
        Returns (logits | None, hidden | None)."""
        mask = None
        if attention_mask is not None:
            mask = (attention_mask.to(self.device) != 0).to(torch.uint8).contiguous()
        try:
            out = self._native.chain_forward(self.chain, input_ids, inputs_embeds, states, mask, last_only, want_logits, want_hidden)
        except _lib.MMFreeError as e:
            kernels._after_failure(e)
            raise
        _lib.launch_count += self._native.take_launches()
        return out


def fused_runner(lm) -> FusedRunner:
    """The model's cached FusedRunner, rebuilt if any parameter (or `resident_step`) changed since it was made."""
    r = getattr(lm, "_fused_runner", None)
    if r is None or r.resident != lm.resident_step or not r.current():
        r = FusedRunner(lm)
        object.__setattr__(lm, "_fused_runner", r)
    return r


def bitlinear_modules(model) -> List[BitLinear]:
    """Every BitLinear of the model in execution order."""
    return [m for m in model.modules() if isinstance(m, BitLinear)]


class WeightStreamProbe:
    """Exactly the BitLinear contractions of one decode step (the grouped i/f/g projection, o, gate, down of
    every block, then lm_head), with pre-quantised activations and nothing else, replayed from a CUDA graph so
    that their device time can be measured with CUDA events."""

    def __init__(self, lm, M: int, out_dtype: torch.dtype, use_graph: bool = True):
        self._use_graph = use_graph
        runner = fused_runner(lm)
        dev = next(lm.parameters()).device
        g = torch.Generator(device=dev).manual_seed(0)
        self.items = []
        self.packed_bytes = 0
        for pw in runner.items:
            x = torch.randn(M, pw.K, generator=g, device=dev, dtype=torch.float32).to(out_dtype)
            q, dq, rs = kernels.act_quant(x, None, 1e-6)
            if pw.groups > 1:
                q, dq, rs = q.repeat(pw.groups, 1), dq.repeat(pw.groups), rs.repeat(pw.groups)
            out = torch.empty(M, pw.N, dtype=out_dtype, device=dev)
            self.items.append((q, dq, rs, pw, out))
            self.packed_bytes += pw.packed.numel()
        self.out_dtype = out_dtype
        self.launches = len(self.items)
        self.graph = None

    def run_eager(self):
        for q, dq, rs, pw, out in self.items:
            kernels.bitlinear(q, dq, rs, pw, self.out_dtype, out=out)

    def run(self):
        if not self._use_graph:
            return self.run_eager()
        if self.graph is None:
            side = torch.cuda.Stream(device=self.items[0][0].device)
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):          # the capture reuses this stream's (zeroed) workspace
                self.run_eager()
            torch.cuda.current_stream().wait_stream(side)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=side):
                self.run_eager()
            self.graph = graph
        self.graph.replay()
