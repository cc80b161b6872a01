"""Replay of given tokens through the engine: teacher-forced steps that return logits instead of sampling.

Every step is one batch of the engine (portions of prompts beside single tokens of other requests), scheduled into
the same blocks and state slots and run by the same prefill and decode steps as generation.
"""
from __future__ import annotations

from contextlib import nullcontext
from typing import Any, Dict, List, Sequence as Seq, Tuple

import numpy as np
import torch

from ..utils.context import reset_context
from .llm_engine import LLMEngine
from .sequence import Sequence


class TokenReplay:
    def __init__(self, llm: LLMEngine):
        self.llm = llm
        self.live: Dict[str, Sequence] = {}
        self._host = self._status = None         # pinned: the logits of a step and the device status word

    # larger reads than this go through pageable memory instead of a pinned buffer that stays
    MAX_PINNED = 64 << 20

    def _read_back(self, got: torch.Tensor) -> Tuple[torch.Tensor, int]:
        """fp32 copy of `got` on the host and the device status word, with one wait for both."""
        from .. import ops
        if self._status is None:
            self._status = torch.zeros(1, dtype=torch.int32, pin_memory=True)
        if self._host is None or self._host.numel() < got.numel():
            self._host = torch.empty(got.numel(), dtype=torch.float32, pin_memory=True)
        host = self._host[: got.numel()].view(got.shape)
        host.copy_(got.float(), non_blocking=True)
        self._status.copy_(ops.ext().status_tensor(got.device.index).view(-1)[:1], non_blocking=True)
        torch.cuda.current_stream(got.device).synchronize()
        return host.clone(), int(self._status[0]) & 0xFF

    @torch.inference_mode()
    def step(self, entries: Seq[Dict[str, Any]], end: Seq[str] = ()) -> torch.Tensor:
        """Feed the next `tokens` of every entry (`id`, `tokens`, `want`) as one batch; returns the logits at the
        wanted places in order, fp32 [wanted, vocab].  The requests named in `end` give back what they hold."""
        sch, runner = self.llm.scheduler, self.llm.model_runner
        pieces = []
        for e in entries:
            if any(not 0 <= w < len(e["tokens"]) for w in e.get("want", ())):
                raise ValueError(f"request {e['id']!r}: a wanted place is not among its {len(e['tokens'])} tokens")
            seq = self.live.get(e["id"])
            if seq is None:
                seq = self.live[e["id"]] = Sequence(e["tokens"])
            pieces.append((seq, list(e["tokens"])))
        logits = torch.empty(0, self.llm.config.hf_config.vocab_size)
        status = None                            # the device status word, where it was read with the logits
        if pieces:
            seqs = sch.schedule_pieces(pieces)
            offsets = np.concatenate([[0], np.cumsum([len(t) for _, t in pieces])])
            rows = [int(o) + int(w) for o, e in zip(offsets, entries) for w in e.get("want", ())]
            stream = torch.cuda.stream(runner.main_stream) if runner.main_stream is not None else nullcontext()
            with stream:
                if all(len(t) == 1 and s.prefill_start > 0 for s, t in pieces):
                    got = runner.run_decode(seqs)
                    if not got.is_cuda or rows != list(range(len(got))):
                        got = got[rows]
                else:
                    got = runner.run_prefill(seqs, logits_rows=rows)
                if got.is_cuda and 0 < got.numel() * 4 <= self.MAX_PINNED:
                    logits, status = self._read_back(got)
                else:
                    logits = got.float().cpu()
            if runner.main_stream is not None:
                # also when nothing was read back: the next step writes the pinned buffers that this one copies from
                runner.main_stream.synchronize()
            reset_context()
            for s in seqs:
                s.num_computed_tokens, s.prefill_end = s.prefill_end, None
        if status is None or status:
            self.llm.check_device_status()
        for rid in end:
            sch.finish(self.live.pop(rid))
        return logits
