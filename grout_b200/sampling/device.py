"""Choosing tokens on the GPU from the step's 32-bit logits."""
from __future__ import annotations

from typing import Sequence

import numpy as np
import torch

from ..kernels import ops
from .params import SamplingParams


class DeviceSampler:
    """Rows of logits -> one token per row.  Greedy rows go through the argmax
    kernel; if any row samples, all rows go through the sampling kernel, which
    treats a temperature at the floor as greedy."""

    def __init__(self, device):
        self.device = torch.device(device)

    def kernel_modules(self):
        return ("sample",)

    def choose(self, logits: torch.Tensor, params: Sequence[SamplingParams],
               draws: Sequence[float]) -> torch.Tensor:
        n = logits.shape[0]
        if len(params) != n or len(draws) != n:
            raise ValueError("one SamplingParams and one draw per row of logits are needed")
        if all(p.greedy for p in params):
            return ops.argmax(logits)
        # what the rows ask for travels with the launch: a copy to the device would wait for
        # everything queued in front of it
        return ops.sample_host(
            logits, np.array([0.0 if p.greedy else p.temperature for p in params], dtype=np.float32),
            np.array([p.top_k for p in params], dtype=np.int32),
            np.array([p.top_p for p in params], dtype=np.float32), np.array(draws, dtype=np.float32))
