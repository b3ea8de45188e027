"""A step's tokens cut into chunks of a fixed number of tokens, per request in order: what the scans over long portions
(the minGRU's, the matrix-state mixers') walk side by side.  Made once per step on the host and shared by the layers."""
from __future__ import annotations

import numpy as np
import torch

from .base import StepContext


def _staged(ctx: StepContext, key, *tables):
    """int32 [rows, width] tables on the device, from pinned memory and without waiting for the device (a pageable copy would stall the
    launches behind it)."""
    pinned = torch.from_numpy(np.concatenate([np.asarray(t, dtype=np.int32).reshape(-1) for t in tables])).pin_memory()
    dev = pinned.to(ctx.token_ids.device, non_blocking=True)
    ctx.derived[key + ("staged",)] = pinned
    out, at = [], 0
    for t in tables:
        out.append(dev[at:at + len(t) * len(t[0])].view(len(t), len(t[0])))
        at += len(t) * len(t[0])
    return tuple(out)


def token_chunks(ctx: StepContext, chunk: int):
    """(chunk_meta int32 [chunks, 4] = (first token, tokens, request, first chunk of its request ? 1 : 0),
    req_chunks int32 [requests, 2] = (first chunk, chunks)), both on the device."""
    key = ("token_chunks", chunk)
    if key not in ctx.derived:
        meta, per_req = [], []
        for r, (s, n) in enumerate(zip(ctx.q_start, ctx.q_len)):
            first = len(meta)
            for off in range(0, n, chunk):
                meta.append((s + off, min(chunk, n - off), r, int(off == 0)))
            per_req.append((first, len(meta) - first))
        ctx.derived[key] = _staged(ctx, key, meta, per_req)
    return ctx.derived[key]


def split_portions(ctx: StepContext, chunk: int, at_least: int):
    """The portions of at least ``at_least`` tokens (there is one) in chunks, the others for a walk over tokens: (chunk_meta, req_chunks) as
    of ``token_chunks``, where a walked request has 0 chunks, and int32 [requests, 4] = (first token, tokens, tokens held, 0), where a
    chunked request has 0 tokens, or None if none is walked."""
    key = ("split_portions", chunk, at_least)
    if key not in ctx.derived:
        meta, per_req, walk = [], [], []
        for r, (s, n, held) in enumerate(zip(ctx.q_start, ctx.q_len, ctx.kv_len)):
            first = len(meta)
            if n >= at_least:
                for off in range(0, n, chunk):
                    meta.append((s + off, min(chunk, n - off), r, int(off == 0)))
            per_req.append((first, len(meta) - first))
            walk.append((s, 0 if n >= at_least else n, held, 0))
        tables = _staged(ctx, key, meta, per_req, walk)
        ctx.derived[key] = tables if any(w[1] for w in walk) else (tables[0], tables[1], None)
    return ctx.derived[key]
