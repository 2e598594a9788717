"""From logits to one token per request.

Greedy and plain temperature sampling run in one kernel of this package (argmax; softmax of
l / T and an inverse-CDF walk in vocabulary order with the request's own uniform number), the
top-k / top-p / min-p cuts in another that follows the reference's algorithm
(crates/sglang-srt/src/model_executor.rs:471-555): sort descending; keep k; keep an item while
the mass before it is below top_p; drop items below max_p * min_p; walk the kept items in
sorted order with target = u * kept mass.  Penalties (model_executor.rs:558-590) change the logits of tokens
seen in prompt and output first, from counts kept on the device.  None of this needs a request's
tokens on the host, so steps overlap the host whatever the sampling options.

Each request draws from its own generator, seeded by its ``seed`` (or by its id), so its
tokens do not depend on what else is in the batch.
"""
from __future__ import annotations

import random
import zlib
from typing import List, Sequence

import numpy as np
import torch

from .. import ops
from .params import SamplingParams

ONE_BELOW = 1.0 - 2.0 ** -24      # the reference clamps u to [0, 1 - 2^-24] (model_executor.rs:548-555)


class RequestRandom:
    """The request's stream of uniform numbers in [0, 1)."""

    def __init__(self, request_id, seed):
        key = seed if seed is not None else zlib.crc32(repr(request_id).encode("utf-8"))
        self._generator = random.Random(int(key))

    def next_unit(self) -> float:
        return min(max(self._generator.random(), 0.0), ONE_BELOW)


class SeenCounts:
    """How often each token occurred in the prompt and output of the requests that have penalties:
    one row of ``vocab`` counts per such request, on the device.  The prompt is counted when the
    request arrives, every sampled token by the sampler as it is chosen; the row goes back when the
    request ends."""

    def __init__(self, vocab: int, device):
        self.vocab, self.device = int(vocab), device
        self.table = None                       # int32 [capacity, vocab]
        self.rows = {}                          # request id -> row
        self.free = []

    def open(self, request_id, prompt: Sequence[int]) -> None:
        if not self.free:
            old = 0 if self.table is None else self.table.shape[0]
            grown = torch.zeros((max(4, 2 * old), self.vocab), dtype=torch.int32, device=self.device)
            if old:
                grown[:old].copy_(self.table)
            self.table = grown
            self.free = list(range(grown.shape[0] - 1, old - 1, -1))
        row = self.free.pop()
        self.rows[request_id] = row
        self.table[row].zero_()
        if len(prompt):
            tokens = torch.tensor(list(prompt), dtype=torch.int32).pin_memory().to(self.device, non_blocking=True)
            ops.count_tokens(self.table[row], tokens)

    def close(self, request_id) -> None:
        row = self.rows.pop(request_id, None)
        if row is not None:
            self.free.append(row)

    def row_of(self, request_id) -> int:
        return self.rows.get(request_id, -1)


class Sampler:
    def __init__(self, device, vocab: int = 0):
        self.device = device
        self.seen = SeenCounts(vocab, device)

    def pick_on_device(self, logits: torch.Tensor, params: Sequence[SamplingParams],
                       randoms: Sequence[RequestRandom], request_ids: Sequence = ()) -> torch.Tensor:
        """One token per row: the chosen ids stay on the device (int32 [rows]); nothing waits for the
        GPU.  ``request_ids`` name the rows' requests, for those with penalties (``logits`` is then
        changed in place, and the chosen tokens are counted as seen)."""
        rows = logits.shape[0]
        temperature, uniform = [0.0] * rows, [0.0] * rows          # of the rows sampled without cuts
        cut, cut_options = [], []                                  # rows with top-k / top-p / min-p, and what they ask for
        penalised, penalties = [], []
        plain = False
        for r in range(rows):
            p = params[r]
            if p.penalised:
                seen_row = self.seen.row_of(request_ids[r]) if r < len(request_ids) else -1
                if seen_row < 0:
                    raise RuntimeError("a request with penalties has no row of counts; SeenCounts.open was not called")
                penalised.append(r)
                penalties.append((seen_row, p.presence_penalty or 0.0, p.frequency_penalty or 0.0,
                                  p.repetition_penalty if p.repetition_penalty is not None else 1.0))
            choice = p.choice
            if choice[0] == "greedy":
                continue
            uniform[r] = randoms[r].next_unit()
            if choice[0] == "cut":
                cut.append(r)
                cut_options.append(choice)
            else:
                temperature[r] = choice[1]
                plain = True
        device = self._upload(rows, temperature, uniform, cut, cut_options, penalised, penalties) \
            if plain or cut or penalised else None
        if penalised:
            seen_row, presence, frequency, repetition = device[-4:]
            ops.apply_penalties(logits, self.seen.table, seen_row.view(torch.int32), presence, frequency, repetition)
        if cut:
            # the rows with cuts first in `index`, the others behind them: every row is written by one of the two
            cut_temperature, top_p, min_p, top_k, index = device[2:7]
            index = index.view(torch.int32)
            picked = torch.empty(rows, dtype=torch.int32, device=logits.device)
            if len(cut) < rows:
                ops.sample(logits, device[0] if plain else None, device[1] if plain else None, picked, index[len(cut):])
            ops.sample_filtered(logits, index[:len(cut)], cut_temperature, top_k.view(torch.int32), top_p, min_p, device[1], picked)
        elif plain:
            picked = ops.sample(logits, device[0], device[1])
        else:
            picked = ops.sample(logits, None, None)
        if penalised:
            ops.count_picked(self.seen.table, seen_row.view(torch.int32), picked)
        return picked

    def _upload(self, rows: int, temperature, uniform, cut, cut_options, penalised, penalties):
        """What the step's kernels need per row, in one pinned buffer and one copy: float rows on the device (rows of ints
        among them, by their bits): temperature, uniform; with cuts temperature, top_p, min_p, top_k and the rows that have
        them; with penalties the rows of counts, presence, frequency and repetition."""
        count = 2 + (5 if cut else 0) + (4 if penalised else 0)
        staging = torch.empty((count, rows), dtype=torch.float32, pin_memory=True)
        floats = staging.numpy()
        ints = floats.view(np.int32)
        floats[0], floats[1] = temperature, uniform
        if cut:
            floats[2:5] = ((1.0,), (1.0,), (0.0,))                 # of the rows without cuts, which no block takes up
            ints[5:7] = 0
            at = np.asarray(cut)
            _, heat, top_k, top_p, min_p = zip(*cut_options)
            floats[2, at], floats[3, at], floats[4, at] = heat, top_p, min_p
            ints[5, at] = np.array(top_k, np.int32)                # (refuses what 32 bits do not hold)
            ints[6, :len(cut)] = at
            others = np.ones(rows, bool)
            others[at] = False
            ints[6, len(cut):] = np.flatnonzero(others)
        if penalised:
            floats[-3:] = ((0.0,), (0.0,), (1.0,))
            ints[-4] = -1
            at = np.asarray(penalised)
            seen_row, presence, frequency, repetition = zip(*penalties)
            ints[-4, at] = seen_row
            floats[-3, at], floats[-2, at], floats[-1, at] = presence, frequency, repetition
        return staging.to(self.device, non_blocking=True).unbind(0)

    def sample(self, logits: torch.Tensor, params: Sequence[SamplingParams], randoms: Sequence[RequestRandom],
               request_ids: Sequence = ()) -> List[int]:
        """The same with the chosen token ids brought to the host."""
        return self.pick_on_device(logits, params, randoms, request_ids).cpu().tolist()
