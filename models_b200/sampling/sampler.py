"""Picks the next token of every row of a batch of logits on the device.

Rows whose options are plain greedy take the argmax kernel; the others take the sampling kernel,
which follows integrallis/models' Sampler step by step (models-runtime/.../Sampler.java:78-151).
Each request draws from its own stream: Philox keyed by its seed, counted by its draws.
"""

from __future__ import annotations

import secrets
import struct
from typing import List, Optional, Sequence

import numpy as np
import torch

from ..kernels import ops
from .options import SamplingOptions


class RequestSampling:
    """Sampling state of one request: its options, its seed, how many draws it has made."""

    def __init__(self, options: SamplingOptions, prompt: Sequence[int]):
        self.options = options
        self.seed = options.seed if options.seed is not None else secrets.randbits(62)
        self.draws = 0
        # the reference penalises every earlier token, prompt included (GenerationLoop.java:165-169)
        self.history: Optional[List[int]] = list(prompt) if options.repetition_penalty > 1.0 else None
        # the same tokens on the device (int32, room for every token the request may still get): the
        # sampling kernel reads them there and stores each new id behind them, so a step sends no history
        self.history_device: Optional[torch.Tensor] = None
        self.history_sent = 0  # tokens of the history that the device array holds


class BatchSampler:
    def __init__(self, vocab_size: int, device):
        self.vocab = vocab_size
        self.device = torch.device(device)
        self._max_sorted = None
        self._staging = None
        self._staging_next = 0

    def check(self, options: SamplingOptions) -> None:
        """Refuses what the kernel cannot do exactly, before any step runs."""
        if options.temperature == 0.0:
            return
        if self._max_sorted is None:
            self._max_sorted = ops.sample_max_sorted()
        if min(options.top_k, self.vocab) > self._max_sorted and options.top_p < 1.0:
            raise ValueError(
                f"top_p < 1 needs the candidates sorted, which the sampling kernel does for at most "
                f"{self._max_sorted} of them: use top_k <= {self._max_sorted}, or top_p = 1 (got top_k "
                f"{options.top_k}, top_p {options.top_p})")

    def sample(self, logits: torch.Tensor, requests: Sequence[RequestSampling], greedy=None) -> torch.Tensor:
        """logits: float32 [len(requests), vocab] on the device.  Returns int32 token ids on the
        device, one per request, and advances the draw counters.  `greedy(logits)`, if given,
        supplies the argmax of every row (the decode graph computes it along with the logits)."""
        rows = len(requests)
        if logits.shape[0] < rows or logits.shape[1] != self.vocab:
            raise ValueError(f"logits {tuple(logits.shape)} do not fit {rows} requests of vocabulary {self.vocab}")
        options = [r.options for r in requests]
        if all(o.greedy for o in options):
            return greedy(logits)[:rows] if greedy is not None else ops.argmax_rows(logits[:rows])
        if logits.shape[0] > rows:
            logits = logits[:rows]
        penalised = any([r.history is not None for r in requests])
        if penalised:
            for r in requests:
                if r.history is not None:
                    self._history_on_device(r)
        parameters, most = self._parameters(requests, options)
        counts = torch.empty((rows, self.vocab), dtype=torch.int32, device=self.device) if penalised else None
        work = torch.empty((rows, self.vocab), dtype=torch.float32, device=self.device)
        out = ops.sample_rows_packed(logits, work, counts, parameters, max_candidates=most, append=penalised)
        for r in requests:
            if r.options.temperature > 0.0:
                r.draws += 1
            if r.history_device is not None:
                r.history_sent += 1  # the kernel has stored this step's id behind the others
        return out

    def _history_on_device(self, r: RequestSampling) -> None:
        """The request's earlier tokens as a device array that the kernel extends by itself.  Sent once
        (the prompt); sent again only if the host's list and the device's count ever disagree, which
        happens when ids were recorded that this sampler did not draw."""
        room = len(r.history) + max(1, int(r.options.max_tokens)) + 4  # a finished request may be sampled once more
        if r.history_device is None or r.history_sent != len(r.history) or r.history_device.numel() < len(r.history) + 1:
            host = torch.zeros((room,), dtype=torch.int32)
            host[: len(r.history)] = torch.tensor(r.history, dtype=torch.int32)
            r.history_device = host.to(self.device)
            r.history_sent = len(r.history)

    def _parameters(self, requests: Sequence[RequestSampling], options: Sequence[SamplingOptions]):
        """The per-row options on the device as `ops.sample_rows_packed` takes them, sent as one asynchronous copy from pinned memory (a copy
        from ordinary memory would wait for every step that is still queued), and the largest candidate set among the rows that cut
        anything (1 if none does): it picks the kernel.  A list per option, packed at once: a walk over the rows, numpy's conversion of
        lists and a tensor for every option took 100 us of the host's time for 64 rows, twice the kernel's."""
        rows, vocab = len(requests), self.vocab
        words = ops.sample_parameter_words(rows)
        if self._staging is None or self._staging[0][0].numel() < words:
            size = max(6 * 64, words)
            self._staging = []
            for _ in range(4):
                host = torch.empty((size,), dtype=torch.int64).pin_memory()
                self._staging.append((host, host.numpy(), torch.cuda.Event()))
        host, longs, event = self._staging[self._staging_next]
        self._staging_next = (self._staging_next + 1) % len(self._staging)
        event.synchronize()  # the copy that last read this buffer, four calls ago
        top_ks = [o.top_k for o in options]
        most = max(top_ks)
        if most >= vocab:
            most = max([min(o.top_k, vocab) for o in options if o.top_k < vocab or o.top_p < 1.0], default=1)
            top_ks = [min(k, vocab) for k in top_ks]
        histories = [r.history_device for r in requests]
        addresses = [0 if h is None else h.data_ptr() for h in histories]
        lengths = [0 if h is None else r.history_sent for h, r in zip(histories, requests)]
        whole = [r.seed for r in requests] + [r.draws for r in requests] + addresses
        floats = [o.temperature for o in options] + [o.top_p for o in options] + [o.repetition_penalty for o in options]
        try:
            struct.pack_into(f"={3 * rows}q{3 * rows}f{2 * rows}i", longs, 0, *whole, *floats, *top_ks, *lengths)
        except (struct.error, OverflowError):  # numbers beyond their type: as numpy takes or refuses them
            longs[:3 * rows] = whole
            small = longs[3 * rows:words]
            small.view(np.float32)[:3 * rows] = floats
            small.view(np.int32)[3 * rows:5 * rows] = top_ks + lengths
        device = torch.empty((words,), dtype=torch.int64, device=self.device)
        device.copy_(host[:words], non_blocking=True)
        event.record(torch.cuda.current_stream(self.device))  # (without one torch asks the driver and the environment which device it is)
        return device, most

    @staticmethod
    def record(requests: Sequence[RequestSampling], tokens: Sequence[int]) -> None:
        for r, t in zip(requests, tokens):
            if r.history is not None:
                r.history.append(int(t))
