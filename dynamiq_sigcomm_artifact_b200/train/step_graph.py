"""One optimizer step as one CUDA graph.

A training step of a small model, or of any model at a small batch, is a few hundred kernels of a few microseconds:
issued one by one from Python and autograd they take longer to launch than to run (GPT-2 tiny: 277 us of kernels in
1190 us; GPT-2 small at batch 1: 3.6 ms for 1.5 ms of kernels).  On one GPU nothing in the step depends on the host -
the bucket reducer has fixed addresses, the optimizer's step-dependent scalars live in device memory
(:class:`~..ops.layers.FusedAdamW`, ``hyper``) - so forward, loss, backward and the AdamW launches on the side stream
are captured once per input shape and replayed with one call.

With several ranks the collectives take a new epoch and step every time, so the step is not captured there; the
trainer then captures the transformer blocks only.
"""
from __future__ import annotations

import gc
from typing import Optional

import torch

from ..utils import counters


class StepGraph:
    """Captured step for one (shape, dtype, labels given or not).  ``run`` returns the loss in a buffer that the next
    ``run`` overwrites."""

    def __init__(self, trainer, ids: torch.Tensor, labels: Optional[torch.Tensor], pool):
        self.ids = torch.zeros_like(ids, device=trainer.device)
        self.labels = None if labels is None else torch.zeros_like(labels, device=trainer.device)
        self._capture(trainer, pool)

    def _capture(self, tr, pool) -> None:
        reducer, opt = tr.reducer, tr.opt
        gen = tr._gen if tr.cfg.task == "mlm" else None
        rng = None if gen is None else gen.get_state()
        consumer, reducer.on_reduced = reducer.on_reduced, None
        try:
            # library plans, workspaces and lazily built tables exist before the capture; no parameter is touched
            stream = torch.cuda.Stream(tr.device)
            stream.wait_stream(torch.cuda.current_stream(tr.device))
            with torch.cuda.stream(stream):
                tr._forward_backward(self.ids, self.labels)
            torch.cuda.current_stream(tr.device).wait_stream(stream)
        finally:
            reducer.on_reduced = consumer
            reducer.arena.zero_()
        for bi, params in enumerate(reducer.bucket_params):
            opt.prepare_subset(bi, params)
        self.graph = torch.cuda.CUDAGraph()
        if gen is not None:
            self.graph.register_generator_state(gen)
        before = counters.snapshot()
        opt.use_hyper = True
        # a garbage collection inside the capture could destroy another trainer's graphs, which CUDA does not allow then
        collecting = gc.isenabled()
        gc.collect()
        gc.disable()
        try:
            # the captured kernels keep their streams' priorities: optimizer steps on the side stream only take SMs that
            # backward leaves idle
            with torch.cuda.graph(self.graph, pool=pool, stream=torch.cuda.Stream(tr.device, priority=-1),
                                  capture_error_mode="thread_local"):
                self.loss = tr._forward_backward(self.ids, self.labels)
        except Exception:
            if gen is not None:  # the registered generator still counts for the capture: eager steps get another one
                tr._gen = torch.Generator(device=tr.device)
                tr._gen.set_state(rng)
            raise
        finally:
            opt.use_hyper = False
            if collecting:
                gc.enable()
            if gen is not None:
                gen.set_state(rng)
        self.launches = counters.total() - sum(before.values())
        counters.restore(before)  # nothing ran yet
        self.addresses = tr._graph_addresses()

    def run(self, ids: torch.Tensor, labels: Optional[torch.Tensor]) -> torch.Tensor:
        self.ids.copy_(ids, non_blocking=True)
        if self.labels is not None:
            self.labels.copy_(labels, non_blocking=True)
        self.graph.replay()
        counters.add("graphed_step", self.launches)
        return self.loss
