"""The launches of a layer, recorded while it runs once and handed to the library for the layers that are like it.

Within a step, layers of one shape make the same calls with the same arguments but for the addresses of their weights and
pages.  `Recording` collects a layer's calls as the words that `sb_run_calls` takes (csrc/run_calls.cu) and finds in them
the places that hold the layer's own addresses; `run` fills in another layer's and launches all of it in one call.  A
recording lives for one step: nothing is kept from one step to the next, and buffers, scratch, sizes and the stream are the
step's.

Which layers are alike is read off the layers themselves in every step (`layer_facts`): a class says with `@replayable`
what its calls depend on.
"""

from __future__ import annotations

import ctypes
import struct
from operator import attrgetter
from typing import Callable, Dict, List, Optional, Sequence, Tuple

import numpy as np
import torch

from .library import F, P, Counters, KernelError, _SIGNATURES, library, set_recorder

# the entry points that a recorded layer may consist of, by their number in run_calls.cu
ENTRIES = {"sb_add_rmsnorm": 0, "sb_gemm_tcgen05": 1, "sb_gemm_simt": 2, "sb_qk_norm_rope_kvwrite": 3, "sb_silu_mul": 4,
           "sb_attention_simt": 5, "sb_attention_prefill_tcgen05": 6, "sb_attention_prefill_mma": 7,
           "sb_attention_balanced": 8, "sb_attention_decode_mma": 9, "sb_attention_decode_stream": 10}
# host-only questions that a layer may ask while it is recorded
_QUESTIONS = ("_supports", "_splits", "_parts", "_shares", "_kernels", "_blocks_per_sm", "sb_last_error",
              "sb_set_dependent_launch")


# class -> (method, its function, an instance's constants, its tensors, those it may lack, the parts inside it)
_REPLAYABLE: Dict[type, Tuple[str, Callable, Callable, Callable, Callable, Callable]] = {}


def replayable(method: str, constants: Sequence[str] = (), tensors: Sequence[str] = (), optional: Sequence[str] = (),
               parts: Callable = lambda self: ()):
    """Class decorator: what `method` launches depends on the instance through the attributes named here (`tensors`, and
    `optional` ones that may be None) and the `parts` inside it alone.  It holds for the very class (a subclass may launch
    other things) and for the very function."""
    def getter(names):
        get = attrgetter(*names) if names else None
        return (lambda self: ()) if get is None else get if len(names) > 1 else (lambda self: (get(self),))

    def mark(cls):
        _REPLAYABLE[cls] = (method, cls.__dict__[method], getter(constants), getter(tensors), getter(optional), parts)
        return cls
    return mark


def layer_facts(part, facts: list, tensors: list) -> bool:
    """Append what the calls of `part` depend on: `tensors` whose addresses stand in them, and everything else to `facts`
    (two layers with equal facts make the same calls but for these addresses).  False: that is not known, because
    something in the layer is no replayable class or lacks a tensor, or a method was replaced or wrapped, on the class or on
    the instance."""
    known = _REPLAYABLE.get(type(part))
    if known is None:
        return False
    method, function, constants, own, optional, parts = known
    if type(part).__dict__.get(method) is not function or method in part.__dict__:
        return False
    facts.append(type(part))
    facts.append(constants(part))
    for t in own(part):
        if t is None:
            return False
        tensors.append(t)
    for t in optional(part):
        facts.append(t is None)
        if t is not None:
            tensors.append(t)
    for inner in parts(part):
        if not layer_facts(inner, facts, tensors):
            return False
    return True


class _Recorder:
    """Stands in for the library: entry points run as ever and leave their name and arguments."""

    def __init__(self, lib):
        self.lib = lib
        self.calls: List[Tuple[str, tuple]] = []
        self.complete = True            # False once something ran that cannot be repeated from words

    def __getattr__(self, name):
        real = getattr(self.lib, name)
        if name in ENTRIES:
            def entry(*args):
                self.calls.append((name, args))
                return real(*args)
            return entry
        if not name.endswith(_QUESTIONS):
            self.complete = False
        return real


def _word(kind, value, keep: list) -> int:
    if kind is F:
        return struct.unpack("<I", struct.pack("<f", value))[0]
    if kind is P:
        if value is None:
            return 0
        if not isinstance(value, int):                      # byref(c_int): a number on the host, as the call left it
            keep.append(value._obj)
            return ctypes.addressof(value._obj)
    return int(value)


class Recording:
    """`with Recording(addresses):` runs a layer; `addresses` are the layer's own device addresses, in an order that
    other layers' follow."""

    def __init__(self, addresses: Sequence[int]):
        self.addresses = list(addresses)
        self.words: Optional[np.ndarray] = None
        self._keep: list = []

    def __enter__(self) -> "Recording":
        self._recorder = _Recorder(library())
        self._launches = Counters.launches
        set_recorder(self._recorder)
        return self

    def __exit__(self, kind, value, trace):
        set_recorder(None)
        self.launches = Counters.launches - self._launches
        if kind is not None or not self._recorder.complete or len(set(self.addresses)) != len(self.addresses):
            return False
        index: Dict[int, int] = {a: i for i, a in enumerate(self.addresses)}
        words, places, which = [], [], []
        for name, args in self._recorder.calls:
            words.append(ENTRIES[name])
            for t, v in zip(_SIGNATURES[name], args):
                if t is P and isinstance(v, int) and v in index:
                    places.append(len(words))
                    which.append(index[v])
                words.append(_word(t, v, self._keep))
        self.words = np.array([w - (1 << 64) if w >= 1 << 63 else w for w in words], dtype=np.int64)
        self._places, self._which = np.array(places, dtype=np.intp), np.array(which, dtype=np.intp)
        self._done = ctypes.c_int(0)
        return False

    @property
    def usable(self) -> bool:
        return self.words is not None

    def run(self, addresses: Sequence[int]) -> None:
        """The recorded calls with another layer's addresses."""
        words = self.words
        words[self._places] = np.array(addresses, dtype=np.int64)[self._which]
        lib = library()
        rc = lib.sb_run_calls(words.ctypes.data, len(words), ctypes.byref(self._done))
        if rc != 0:
            raise KernelError(f"call {self._done.value} of a recorded layer: "
                              f"{lib.sb_last_error().decode(errors='replace')} (code {rc})")
        Counters.launches += self.launches
