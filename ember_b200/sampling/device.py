"""Device sampler: one kernel launch for all rows of a step."""
from __future__ import annotations

import functools
import struct
from operator import attrgetter
from typing import Optional, Sequence

import torch

from .. import ops, transfers
from .params import SamplingParams

_U64 = (1 << 64) - 1


@functools.lru_cache(maxsize=64)
def _rows_struct(rows: int) -> struct.Struct:
    return struct.Struct("<" + "fiffQQ" * rows)     # temperature, top_k, top_p, min_p, seed, counter: 32 bytes a row


_fields = attrgetter("temperature", "top_k", "top_p", "min_p", "seed")


def pack_params(params: Sequence[SamplingParams], counters: Sequence[int]) -> bytes:
    values = []
    for p, c in zip(params, counters):
        values += _fields(p)
        values.append(c)
    try:
        return _rows_struct(len(params)).pack(*values)
    except struct.error:                            # numbers of other types, seeds and counters outside 64 bits
        for i in range(0, len(values), 6):
            t, k, top, low, seed, c = values[i:i + 6]
            values[i:i + 6] = float(t), int(k), float(top), float(low), int(seed) & _U64, int(c) & _U64
        return _rows_struct(len(params)).pack(*values)


_scratch = {}


def _argmax_scratch(device, rows: int):
    got = _scratch.get(device)
    if got is None or got[0].numel() < rows * 32:
        n = max(rows, 64) * 32
        got = (torch.empty(n, dtype=torch.float32, device=device), torch.empty(n, dtype=torch.int32, device=device))
        _scratch[device] = got
    return got


def sample(logits: torch.Tensor, params: Sequence[SamplingParams], counters: Sequence[int],
           out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """One token id per row of ``logits`` [rows, vocab] (fp32, device); returns int32 [rows] on the device."""
    rows, vocab = logits.shape
    if len(params) != rows or len(counters) != rows:
        raise ops.KernelError(f"sample: {len(params)} parameter sets for {rows} rows")
    if out is None:
        out = torch.empty(rows, dtype=torch.int32, device=logits.device)
    if all(p.greedy for p in params):
        # argmax needs no parameters on the device and is spread over many blocks per row
        part_v, part_i = _argmax_scratch(logits.device, rows)
        ops.argmax(logits, out, rows, part_v, part_i)
        return out
    packed = pack_params(params, counters)
    ops.sample_host(logits, packed, out, rows)
    transfers.add_h2d(len(packed))
    return out
