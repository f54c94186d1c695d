"""Chooses the next token of every sampled request on the device, in one
launch for the whole batch.

Greedy rows and temperature rows go through the same kernel; a step whose rows
are all greedy uses the argmax kernel.  The per-row options travel as small
tensors; nothing comes back to the host but the chosen ids.  The reference
loops over rows in Python with a device-to-host transfer per row
(python/lyapunov_engine/engine/sampling.py:30-70).
"""
from __future__ import annotations

import numpy as np
import torch

from .. import ops


class Sampler:
    def __init__(self, device, max_rows: int):
        self.device = device
        self.max_rows = max_rows
        # A ring of pinned buffers: the copy to the device runs when the device gets to it, which may be after
        # the next call has been made (the engine launches steps ahead of reading their results).
        # A call's options stand one kind behind the other, as the kernel reads them: n temperatures, n top_p, n top_k,
        # n triples (seed low word, seed high word, counter).
        self._hosts = [(torch.empty(max_rows * 6, dtype=torch.int32, pin_memory=True), torch.cuda.Event()) for _ in range(4)]
        self._host_at = 0
        self._dev = torch.empty(max_rows * 6, dtype=torch.int32, device=device)
        self._out = torch.empty(max_rows, dtype=torch.int32, device=device)
        self._scratch = None

    def sample(self, logits: torch.Tensor, params: list, token_indices: list[int]) -> torch.Tensor:
        """``logits`` [n, V] float32; ``params[i]`` the SamplingParams of row i;
        ``token_indices[i]`` the index in its sequence of the token being
        chosen (the generator's counter).  Returns int32 ids [n] on the device."""
        n = logits.shape[0]
        out = self._out[:n]
        if all(p.temperature < 1e-4 for p in params):
            need = ops.argmax_scratch_floats(self.max_rows, logits.shape[1])
            if self._scratch is None or self._scratch.numel() < need:
                self._scratch = torch.empty(need, dtype=torch.float32, device=self.device)
            ops.argmax(out, logits, self._scratch)
            return out
        pinned, event = self._hosts[self._host_at]
        self._host_at = (self._host_at + 1) % len(self._hosts)
        event.synchronize()
        # (whole columns at a time: 64 rows value by value took 160 us, and two kernels to turn them into columns)
        host = pinned.numpy()
        floats = host.view(np.float32)
        floats[:n] = [p.temperature for p in params]
        floats[n:2 * n] = [p.top_p for p in params]
        host[2 * n:3 * n] = np.array([p.top_k for p in params], dtype=np.int32)
        triples = host[3 * n:6 * n].reshape(n, 3)
        seeds = np.array([int(p.seed) & 0xFFFFFFFFFFFFFFFF for p in params], dtype=np.uint64)
        triples[:, :2] = seeds.view(np.int32).reshape(n, 2)          # (low word first)
        triples[:, 2] = np.array(token_indices[:n], dtype=np.int32)
        d = self._dev[:6 * n]
        d.copy_(pinned[:6 * n], non_blocking=True)
        event.record()
        temperature, top_p = d[:2 * n].view(torch.float32).view(2, n)
        top_k, seeds = d[2 * n:3 * n], d[3 * n:].view(n, 3)
        ops.sample(out, logits, temperature, top_p, top_k, seeds)
        return out
