"""Choosing the next token from logits, for a batch of requests at once.

Greedy at temperature 0, otherwise temperature and optional top-k with a per-request
random stream (src/flexengine/engine/sampling/sampler.py:7-22; per-request seeds
src/flexengine/engine/runtime.py:112-116).  The reference draws on the CPU with one
``torch.Generator`` per request; here the draw is a kernel keyed by (request seed, number
of the draw), which gives the same property: a request's tokens do not depend on what
else is in the batch or on how the scheduler cut the work.
"""
from __future__ import annotations

from array import array

import numpy as np
import torch


def validate_sampling(temperature: float, top_k: int) -> None:
    if temperature < 0 or top_k < 0:
        raise ValueError("temperature and top_k must be >= 0")


def _none_negative(values, n: int) -> bool:
    """Whether a list or tuple of ``n`` certainly holds nothing below zero, in one pass (a first NaN is not certain: it hides what
    follows)."""
    return type(values) in (list, tuple) and len(values) == n and (n == 0 or bool(min(values) >= 0))


def _fill(words, values, dtype) -> None:
    """``values`` into the numpy array ``words``: a list or tuple that numpy takes for numbers of the kind in one conversion;
    anything else as a tensor of ``dtype``, which takes, broadcasts and refuses what a tensor does."""
    try:
        given = np.array(values) if type(values) in (list, tuple) else None
    except (TypeError, ValueError):
        given = None
    if given is not None and given.shape == words.shape and given.dtype.kind in ("fi" if dtype is torch.float32 else "i"):
        words[:] = given
    else:
        torch.from_numpy(words)[:] = torch.tensor(list(values), dtype=dtype)


def _arrays(n, temperatures, top_ks, seeds, draws):
    """The four as arrays of the kernel's types, where they are lists or tuples of ``n`` plain numbers that fit; None otherwise."""
    for values in (top_ks, seeds, draws):
        if type(values) not in (list, tuple) or len(values) != n or set(map(type, values)) != {int}:
            return None
    if type(temperatures) not in (list, tuple) or not set(map(type, temperatures)) <= {int, float}:
        return None
    try:
        return array("f", temperatures), array("i", top_ks), array("q", seeds), array("q", draws)
    except OverflowError:
        return None


class Sampler:
    def __init__(self, ops=None):
        if ops is None:
            from .. import ops as cuda_ops
            ops = cuda_ops
        self.ops = ops
        self._zeros = {}

    def sample(self, logits: torch.Tensor, temperatures, top_ks, seeds, draws) -> list:
        """logits float32 [R, V]; the other arguments are sequences of length R.  Returns R token ids."""
        return self.sample_on_device(logits, temperatures, top_ks, seeds, draws).tolist()

    def sample_on_device(self, logits: torch.Tensor, temperatures, top_ks, seeds, draws) -> torch.Tensor:
        """As ``sample`` but the token ids stay where the logits are (int32 [R]); nothing waits for the device."""
        if logits.dim() != 2 or logits.shape[0] != len(temperatures):
            raise ValueError("Expected logits [requests, vocab]")
        n = len(temperatures)
        if not (_none_negative(temperatures, n) and _none_negative(top_ks, n)):
            for t, k in zip(temperatures, top_ks):
                validate_sampling(t, k)
        dev = logits.device
        if all(t == 0.0 for t in temperatures):
            # greedy rows need no parameters: zeros kept on the device, no copy per step
            key = (str(dev), n)
            if key not in self._zeros:
                self._zeros[key] = (torch.zeros(n, dtype=torch.float32, device=dev),
                                    torch.zeros(n, dtype=torch.int32, device=dev),
                                    torch.zeros(n, dtype=torch.int64, device=dev))
            temperature, top_k, zero64 = self._zeros[key]
            return self.ops.sample(logits, temperature, top_k, zero64, zero64)
        # Plain lists go with the launch as far as they fit into its parameters: no buffer, no copy, no views
        # (64 rows, with the kernel's own gain: a call among others 50 to 52 -> 40 us, alone 95 to 100 -> 65)
        listed = getattr(self.ops, "sample_listed", None)
        if listed is not None and 0 < n <= self.ops.SAMPLE_LISTED_ROWS and dev.type == "cuda":
            arrays = _arrays(n, temperatures, top_ks, seeds, draws)
            if arrays is not None:
                return listed(logits, *arrays)
        # One host buffer, one copy, no kernel to take it apart: [seeds | draws | temperatures | top_ks] as 8, 8, 4 and 4 bytes
        # each (four conversions and two kernels before: the host took longer than the device, 106 us for 64 rows)
        packed = torch.empty(3 * n, dtype=torch.int64, pin_memory=dev.type == "cuda")
        host = packed.numpy()
        with np.errstate(over="ignore"):                 # a temperature beyond float32 is an infinite one
            _fill(host[:n], seeds, torch.int64)
            _fill(host[n:2 * n], draws, torch.int64)
            _fill(host[2 * n:].view(np.float32)[:n], temperatures, torch.float32)
            _fill(host[2 * n:].view(np.int32)[n:], top_ks, torch.int64)
        on_dev = packed.to(dev, non_blocking=True)
        small = on_dev[2 * n:].view(torch.int32)
        return self.ops.sample(logits, small[:n].view(torch.float32), small[n:], on_dev[:n], on_dev[n:2 * n])
