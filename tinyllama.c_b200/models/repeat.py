"""The calls of one layer made again for the layers that are like it.

CodeClaper/tinyllama.c walks a static list of nodes for every step (graph.c:1278-1302).  Here a layer's forward() is
Python that checks its operands and makes a dozen calls of the kernel library, and for prompts of up to a few hundred
tokens that is slower than the kernels: 24 layers of the 1.5B sizes took the host 4 ms, 13 us a call, where the GPU
needs 1 to 2.5.  Where all layers of the run order are alike (the same parts of the same sizes and constants, tensors of the same
types, shapes and strides), the first one runs as ever and its calls are noted; the others' are the same calls with their
own weights and their own part of the cache in place of the first one's, and are made by the library in one go.

Nothing is kept from one step for the next but the description of the layers, which is made anew when a part of theirs, a list
of parts or numbers, or the list of the layers itself has been edited; the tensors' addresses, types, shapes and strides are
read in every step.  A pointer that is neither one of the first layer's tensors nor something that all layers share (the
stream of rows, the step's tables and temporaries) ends the attempt, and so does a caller's stream that is one of the first
layer's own: the layers then run one by one, as they do under capture, on other devices and with parts that do not say that
they can be repeated.
"""
from __future__ import annotations

from operator import attrgetter, getitem, itemgetter
from types import FunctionType
from typing import List, Optional, Tuple

import numpy as np
import torch

from .. import ops
from ..parts.base import Editable, LayerCache, StepInfo, current_stream, used_on


_PLAIN = (type(None), bool, int, float, str, torch.dtype, torch.device)
_LOW = np.uint64(15)
_edits = attrgetter("edits")
_ptr, _size, _stride, _dtype = torch.Tensor.data_ptr, torch.Tensor.size, torch.Tensor.stride, attrgetter("dtype")
_dense = torch.Tensor.is_contiguous


# The wrappers of the kernel library as they are defined: the functions that name one of its calls, and those that they go through.
_OPS = {k: f for k, f in vars(ops).items() if isinstance(f, FunctionType) and
        (k in ("_call", "record_event", "wait_event") or any(isinstance(c, str) and c in ops.REPEATABLE for c in f.__code__.co_consts))}
# methods that a step has no use for
_NOT_IN_A_STEP = {"__init__", "bind", "weight_specs", "cache_requests", "step_requests", "shapes_from", "parts", "repeats", "add", "fuse_bound",
                  "fuse_bound_inputs", "out_features", "__setattr__", "__delattr__", "__init_subclass__"}


class _Description:
    """What a layer is made of: a form that is equal for two layers whose calls differ in their tensors' addresses alone, where
    its tensors are (a part's attributes and the name, in the order in which they come up: none is held here), and what an
    edit goes through: the parts (their attributes) and the lists."""

    def __init__(self, layer, parts: List[Editable], lists: list, classes: set):
        self.tensors: List[Tuple[dict, str]] = []
        self.parts, self.lists, self.classes = parts, lists, classes
        self.known, self.inside = True, set()            # known: whether every part says that it can be repeated
        self.form = self._of(layer)

    def _of(self, obj):
        if isinstance(obj, _PLAIN):
            return type(obj), obj
        if isinstance(obj, torch.Tensor):
            return "tensor", obj.dtype, tuple(obj.shape), obj.stride(), obj.device
        if id(obj) in self.inside or not isinstance(obj, (list, tuple, dict, Editable)):
            self.known = False
            return type(obj), id(obj)
        self.inside.add(id(obj))
        try:
            if not isinstance(obj, Editable):
                items = list(obj.values() if isinstance(obj, dict) else obj)
                if any(isinstance(v, torch.Tensor) for v in items):
                    self.known = False                    # (compared with a list of old, a tensor compares its values)
                elif not isinstance(obj, tuple):
                    self.lists.append(obj)
                return type(obj), tuple(obj) if isinstance(obj, dict) else None, tuple(map(self._of, items))
            self.parts.append(obj)
            self.classes.update(c for c in type(obj).__mro__ if issubclass(c, Editable))
            aside = obj.repeats()
            if aside is None or "repeats" not in type(obj).__dict__:      # (a class derived from such a part speaks for itself)
                self.known, aside = False, ()
            names = [k for k in sorted(vars(obj)) if k not in aside and k != "edits"]
            self.tensors += [(vars(obj), k) for k in names if isinstance(vars(obj)[k], torch.Tensor)]
            return type(obj), tuple((k, self._of(vars(obj)[k])) for k in names)
        finally:
            self.inside.remove(id(obj))


def _items(places: List[int]):
    """What takes the values at these places out of a list."""
    if len(places) > 1:
        return itemgetter(*places)
    return (lambda values: (values[places[0]],)) if places else (lambda values: ())


def _of_cache(view: LayerCache) -> Tuple[tuple, List[torch.Tensor]]:
    """(what must be equal, tensors) of a layer's part of the cache."""
    tensors = []
    for kv in view.kv.values():
        tensors += [kv.k_pages, kv.block_table] if kv.v_pages is None else [kv.k_pages, kv.block_table, kv.v_pages]
    tensors += view.state.values()
    return (view.writes, view.kv_writes, [(k, kv.window, kv.v_pages is None) for k, kv in view.kv.items()], list(view.state)), tensors


class RepeatedLayers:
    """The layers of a run order that are alike."""

    # Where a layer keeps the GPU longer than Python takes for one (0.22 ms), the layers run one by one: while the first one's calls
    # are looked through the GPU waits for 0.3 ms, which pays where the GPU would wait for every layer.  That is so up to the
    # rows that make a layer's products take LONG_LAYER at the rates below (the norms, the scan and attention come on top) and up
    # to LONG_STEP rows at most.  Milliseconds a prompt, repeated and one by one: 1.5B sizes, 600 / 700 / 1,000 / 2,048 rows 5.13 / 5.28 /
    # 5.55 / 8.2 and 5.35 / 5.30 / 5.27 / 8.0; 3B, 250 / 270 / 700 6.54 / 7.54 / 8.7 and 6.75 / 7.14 / 8.4; 7B, 125 / 140 / 333 7.7 /
    # 9.60 / 11.3 and 9.1 / 9.52 / 11.0; 1.5B in 32 bits, 5 / 10 / 20 4.25 / 6.27 / 5.71 and 4.78 / 6.02 / 5.44.
    LONG_STEP, LONG_LAYER = 1024, 87e-6
    READ_RATE, RATE_16, RATE_32 = 6.5e12, 1e15, 1.4e13        # bytes, operations of 16-bit and of few-row 32-bit products a second

    @staticmethod
    def of(layers, schedule) -> Optional["RepeatedLayers"]:
        """None where the run order is more than one pass of like layers, each with a cache of its own."""
        found = RepeatedLayers(layers, schedule)
        return found if found.alike else None

    def __init__(self, layers, schedule):
        self.order = layers, schedule
        self.all_edits = Editable.all_edits[0]            # (ahead of the look)
        self.parts, self.lists = [], [layers, schedule]
        self.layers = [layers[r.layer] for r in schedule]
        classes = set()
        found = [_Description(layer, self.parts, self.lists, classes) for layer in self.layers]
        self.written = [(vars(ops), list(_OPS), list(_OPS.values()))]
        for c in classes:
            methods = {k: f for k, f in c.as_written.items() if k not in _NOT_IN_A_STEP}
            if methods:
                self.written.append((vars(c), list(methods), list(methods.values())))
        self.tensors = [d.tensors for d in found]
        self.holders = [[attributes for attributes, _ in t] for t in self.tensors]
        self.read_s = self.row_s = 0.0                     # a layer's matrices read once, and what every row adds, in seconds
        spans, end = [], 0
        for t in (attributes[name] for attributes, name in self.tensors[0]) if self.tensors else ():
            if t.dim() == 2 and t.numel():
                n = 1 + sum((size - 1) * stride for size, stride in zip(t.shape, t.stride()))
                spans.append((t.data_ptr(), t.data_ptr() + n * t.element_size(), t.dtype))
        for lo, hi, dtype in sorted(spans, key=lambda s: s[:2]):
            n, end = max(0, hi - max(lo, end)), max(hi, end)      # (a product's parts keep ranges of its matrix)
            self.read_s += n / self.READ_RATE
            self.row_s += 2 * n / 4 / self.RATE_32 if dtype == torch.float32 else 2 * n / 2 / self.RATE_16
        self.alike = len(found) >= 3 and all(d.known and d.form == found[0].form for d in found) \
            and not any(r.cache is not None or r.kv_cache is not None or r.add is not None or r.add_embedding for r in schedule)
        self.edits, self.copies = list(map(_edits, self.parts)), [l if isinstance(l, tuple) else l.copy() for l in self.lists]

    def run(self, x: torch.Tensor, step: StepInfo, cache) -> Tuple[int, bool]:
        """Runs the first layer, and the others if they can be repeated; (how many entries of the run order have run,
        whether the last of them has left the next one's input)."""
        views = [cache.layer_view(r, True, None) for r in range(len(self.layers))]
        with ops.noting() as notes:
            left = self.layers[0].forward(x, step, views[0], False, self.layers[1].entry)
        if left or not notes.complete:
            return 1, left
        done, n = 1, len(self.layers)
        form, mine = _of_cache(views[0])
        n_own = len(self.tensors[0])
        firsts = [attributes[name] for attributes, name in self.tensors[0]] + mine
        at, also = {}, {}                                  # address -> which of the first layer's tensors; which others start there
        addresses = list(map(_ptr, firsts))
        for i, p in enumerate(addresses):
            if p and at.setdefault(p, i) != i:
                also.setdefault(p, []).append(i)
        handles = [layer.handles(x.device) if notes.forks else () for layer in self.layers]
        if notes.forks and ops.stream_handle() in handles[0]:
            return done, left       # the caller's stream (one of the few that torch hands out) is the first layer's own: a word cannot say which is meant
        for i, p in enumerate(handles[0]):
            at[p] = len(firsts) + i
        common = self._shared(x, step, notes)
        shared = notes.handles.difference(handles[0]).union((0,), map(_ptr, common))
        ranges = None
        places, which = [], []                             # words to replace, and by which tensor's address
        for w in notes.pointers:
            word = notes.words[w]
            if word in shared:
                continue
            i = at.get(word)
            if i is not None:
                places.append(w)
                which.append(i)
                continue
            if ranges is None:
                ranges = [(_ptr(t), _ptr(t) + t.untyped_storage().nbytes() - t.storage_offset() * t.element_size()) for t in common]
            if not any(lo <= word < hi for lo, hi in ranges):
                return done, left
        # a word says which address is meant, not which of the tensors that start there: they have to in every layer
        used = sorted(set(which))
        rank = {i: n for n, i in enumerate(used)}
        ties = [(rank[i], j) for i in used if i < len(firsts) for j in also.get(addresses[i], ())]
        tensors = [i for i in used if i < len(firsts)]      # (the layers' own streams and events come behind them)
        like = self._meta([firsts[i] for i in tensors])
        place = self.tensors[0]
        own, own_names = _items([i for i in tensors if i < n_own]), [place[i][1] for i in tensors if i < n_own]
        cached = _items([i - n_own for i in tensors if i >= n_own])
        tied, tied_names = _items([j for _, j in ties if j < n_own]), [place[j][1] for _, j in ties if j < n_own]
        tied_cached = _items([j - n_own for _, j in ties if j >= n_own])
        tied_to = _items([n for n, j in ties if j < n_own] + [n for n, j in ties if j >= n_own])
        own_handles = _items([i - len(firsts) for i in used[len(tensors):]])
        base = np.array([addresses[i] for i in tensors], dtype=np.uint64)
        first, functions = np.array(notes.words, dtype=np.uint64), np.array(notes.functions, dtype=np.int32)
        # The calls' own scratch came from the stream that the first layer made them on; the others use it on theirs.
        if notes.owned:
            used_on(current_stream(x.device), notes.owned)
        columns, places = np.array([rank[i] for i in which], dtype=np.intp), np.array(places, dtype=np.intp)
        # the next layer at once, so that the GPU has work while the others' addresses are gathered, then a few, then the rest
        while done < n:
            end = min(n, done + (1 if done < 3 else 4 if done < 6 else n))
            table = np.empty((end - done, len(used)), dtype=np.uint64)
            for r in range(done, end):
                other, theirs = _of_cache(views[r])
                holders = self.holders[r]
                row = list(map(getitem, own(holders), own_names))
                row += cached(theirs)
                if other != form or self._meta(row) != like:
                    return done, left
                row = list(map(_ptr, row))
                if ties and tuple(map(_ptr, (*map(getitem, tied(holders), tied_names), *tied_cached(theirs)))) != tied_to(row):
                    return done, left
                row += own_handles(handles[r])
                table[r - done] = row
            if np.count_nonzero((table[:, :len(tensors)] ^ base) & _LOW) or np.count_nonzero(table) != table.size:
                return done, left                          # (the calls may choose by how their operands are aligned)
            words = np.empty((end - done, first.size), dtype=np.uint64)
            words[:] = first
            words[:, places] = table[:, columns]
            ops.replay(functions, words, end - done)
            done = end
        return n, False

    def is_long(self, rows: int) -> bool:
        """Whether a step of that many rows waits for the GPU and not for the host (its layers run one by one, and nothing is
        looked at)."""
        return rows >= self.LONG_STEP or self.read_s + rows * self.row_s >= self.LONG_LAYER

    def stands(self, layers=None, schedule=None) -> bool:
        """Whether nothing has been edited since the layers were looked at: no attribute of a part, no list or what is in it, and
        these (where given) are the lists that were looked at."""
        if (layers is not None and layers is not self.order[0]) or (schedule is not None and schedule is not self.order[1]) or self.lists != self.copies:
            return False
        now = Editable.all_edits[0]
        if now != self.all_edits:                          # a part of some model
            if list(map(_edits, self.parts)) != self.edits:
                return False
            self.all_edits = now
        return True

    def untouched(self) -> bool:
        """Whether the layers' methods and the wrappers of the kernel library are those that the source has.  A function that a
        program puts around one of them (to trace, to time, to gather statistics) is called for every layer."""
        return all(list(map(holder.get, names)) == functions for holder, names, functions in self.written)

    @staticmethod
    def _meta(tensors):
        """Sizes, types and strides (of dense tensors the sizes say them)."""
        dense = list(map(_dense, tensors))
        return list(map(_size, tensors)), list(map(_dtype, tensors)), dense, None if all(dense) else list(map(_stride, tensors))

    @staticmethod
    def _shared(x: torch.Tensor, step: StepInfo, notes) -> List[torch.Tensor]:
        """What all layers of the step read or write alike."""
        out = [x, step.tokens, step.positions, step.row_seq, step.cu_seqlens, step.slots, step.start_pos]
        for table in step.chunks.values():
            out += table or ()
        return out + [t for t in list(step.scratch.values()) + notes.owned if isinstance(t, torch.Tensor)]
