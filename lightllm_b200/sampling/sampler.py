"""Choosing the next token of every row of logits, on the device.

The reference copies each row of logits to the host and samples there
(src/engine/engine_server.cpp:2043-2051, src/ops/sampling.cpp:22-335).  Here the rows stay on
the device: greedy rows go through the argmax kernel, the rest through the sampling kernel
(temperature, top-k, top-p, min-p and the draw); only the chosen ids come back.  The uniform
number of each draw comes from the request's own counter-based stream (Philox keyed by the
request's seed and id), so a request's output does not depend on what else is in the batch.
"""
from __future__ import annotations

from typing import Dict, Hashable, List, Sequence

import numpy as np
import torch

from ..csrc import ops
from .params import GREEDY_BELOW, SamplingParams


class RequestStream:
    """The random stream of one request: draw ``n`` gives the same number whatever happened to
    other requests.  (The numbers are drawn a few dozen at a time: the generator gives the same ones as one by one, and a
    call of it costs the host a microsecond.)"""

    AHEAD = 32

    def __init__(self, seed: int, request_id: int):
        key = (int(seed) & 0xFFFF_FFFF_FFFF_FFFF, int(request_id) & 0xFFFF_FFFF_FFFF_FFFF)
        self._gen = np.random.Generator(np.random.Philox(key=np.array(key, dtype=np.uint64)))
        self._drawn: List[float] = []          # the next ones, last first

    def uniform(self) -> float:
        if not self._drawn:
            self._drawn = self._gen.random(self.AHEAD, dtype=np.float32)[::-1].tolist()
        return self._drawn.pop()


class Sampler:
    def __init__(self, device: torch.device):
        self.device = device
        self._streams: Dict[Hashable, RequestStream] = {}

    def stream(self, request_id: int, seed: int) -> RequestStream:
        s = self._streams.get(request_id)
        if s is None:
            s = self._streams[request_id] = RequestStream(seed, request_id)
        return s

    def forget(self, request_id: int) -> None:
        self._streams.pop(request_id, None)

    def sample(self, logits: torch.Tensor, request_ids: Sequence[int], params: Sequence[SamplingParams]) -> List[int]:
        """One token id per row of ``logits`` (float32 ``[R, V]`` on the device)."""
        tokens = self.sample_device(logits, request_ids, params)
        return tokens.cpu().tolist()

    def sample_device(self, logits: torch.Tensor, request_ids: Sequence[int],
                      params: Sequence[SamplingParams]) -> torch.Tensor:
        R = logits.shape[0]
        if len(request_ids) != R or len(params) != R:
            raise ValueError(f"{R} rows of logits but {len(request_ids)} requests and {len(params)} parameter sets")
        out = torch.empty(R, dtype=torch.int32, device=logits.device)
        temperature = [p.temperature for p in params]
        if all(t < GREEDY_BELOW for t in temperature):
            ops.argmax(logits, out)
            return out
        host = np.empty((5, R), dtype=np.float32)
        host[0] = temperature
        host[1] = [p.top_p for p in params]
        host[2] = [p.min_p for p in params]
        host[3] = [0.0 if t < GREEDY_BELOW else self.stream(rid, p.seed).uniform() for rid, p, t in zip(request_ids, params, temperature)]
        host[4].view(np.int32)[:] = [p.top_k for p in params]
        # (not waited for: from memory that is not pinned the driver has taken the numbers when the call returns)
        dev = torch.from_numpy(host).to(logits.device, non_blocking=True)
        ops.sample(logits, dev[0], dev[4].view(torch.int32), dev[1], dev[2], dev[3], out)
        return out
