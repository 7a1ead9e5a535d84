"""Key / value caches that grow in place while generating.

A layer's cache is the tensor it returns as ``present``: ``[2, n, b, heads, hn]``.  Here that tensor is the front of a
buffer with room for more rows, so a step writes its own rows behind the ones that are there instead of copying the
whole cache (concatenating k and v and stacking them moves every cached byte twice per step).

Only the tensor that the layer returned last, unchanged in length and on the same stream, is extended in place; an older
one (a second continuation of the same prefix), another layer's or a caller's own is copied into a buffer of its own, so
no ``present`` ever sees rows that were appended to another.  So is one that was returned in inference mode once that
mode has ended: its memory may not be written any more.  Nothing is grown in place while a graph is captured, and
nothing that a captured step returned is (on the stream of the steps around it, where the stream would not tell them
apart): every replay writes that step's rows again.

A grown cache shares its front with the shorter one it came from, and its storage holds room for more rows: clone a cache
to change or to save it by itself.
"""
from __future__ import annotations

import threading
import weakref

import torch

_LOCK = threading.Lock()
#: layer -> [weak reference to the cache it returned last or None, stream]; the cache itself is held by whoever uses it
_LAST: "weakref.WeakKeyDictionary" = weakref.WeakKeyDictionary()
_MIN_ROOM = 256


def _stream(t):
    return torch._C._cuda_getCurrentRawStream(t.get_device()) if t.is_cuda else 0


def _slot(layer):
    with _LOCK:
        slot = _LAST.get(layer)
        if slot is None:
            slot = _LAST[layer] = [None, None]
        return slot


def _claim(slot, past, stream) -> bool:
    """Whether ``past`` is the cache the layer returned last; the answer is yes once per returned cache."""
    with _LOCK:
        ref, st = slot
        if ref is None or ref() is not past or st != stream:
            return False
        if past.is_inference() and not torch.is_inference_mode_enabled():
            return False                # its buffer may not be written outside inference mode
        slot[0] = None
        return True


def extend(layer, past, rows: int, like: torch.Tensor, shape=None) -> torch.Tensor:
    """The cache ``[2, n + rows, b, heads, hn]`` whose first n rows are ``past``'s (None or empty: n = 0) and whose last
    ``rows`` rows the caller fills.  ``like``: a tensor of the cache's dtype and device, [*, b, heads, hn] unless ``shape``
    gives (b, heads, hn)."""
    n = 0 if past is None else past.shape[1] if torch.is_tensor(past) else past[0].shape[0]
    shape = tuple(like.shape[1:]) if shape is None else shape
    stream, total = _stream(like), n + rows
    present, slot = None, _slot(layer)
    capturing = like.is_cuda and torch.cuda.is_current_stream_capturing()
    if torch.is_tensor(past) and past.dtype == like.dtype and past.device == like.device and not capturing \
            and past.shape[2:] == shape and _claim(slot, past, stream):
        stride = past.stride()
        if total <= stride[0] // stride[1]:
            present = past.as_strided((2, total) + shape, stride)
    if present is None:
        if n and not (past[0].shape == past[1].shape == (n,) + shape):
            # (the copies would broadcast the cache of another batch or head count)
            raise RuntimeError("kv_cache: the cache holds keys %s and values %s, this step appends rows of %s"
                               % (tuple(past[0].shape), tuple(past[1].shape), shape))
        buf = torch.empty((2, total + max(_MIN_ROOM, total // 4)) + shape, device=like.device, dtype=like.dtype)
        if n:
            buf[0, :n].copy_(past[0])
            buf[1, :n].copy_(past[1])
        present = buf[:, :total]
    if not capturing:
        with _LOCK:
            slot[0], slot[1] = weakref.ref(present), stream
    return present
