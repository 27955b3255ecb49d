"""Layers whose calls are made again from the first one's (models/repeat.py)."""
import ctypes
import random
import weakref
from types import SimpleNamespace

import pytest
import torch

import tinyllama_c_b200 as tlc
from tinyllama_c_b200 import ops
from tinyllama_c_b200.models import repeat
from tinyllama_c_b200.config import config_from_dict
from tinyllama_c_b200.engine import StepEntry
from tinyllama_c_b200.models.repeat import RepeatedLayers
from tinyllama_c_b200.parts.base import Editable, LayerCache, LayerRun, StepInfo, step_scratch
from tinyllama_c_b200.weights import build_model

import configs

# the kernels of long prompts, of short ones and the general ones; more than two layers
SIZES = {"tensor cores": dict(configs.TINY_D, num_hidden_layers=4, mamba_d_head=64, mamba_d_ssm=128, mamba_d_state=128),
         "odd": dict(configs.TINY_C, num_hidden_layers=3), "small": dict(configs.TINY_A, num_hidden_layers=8)}


def _model(name, dtype, device):
    model = build_model(config_from_dict(dict(SIZES[name])))
    g = torch.Generator().manual_seed(3)
    tensors = {}
    for s in model.weight_specs():
        t = torch.randn(s.shape, generator=g) * 0.2
        tensors[s.name] = 1.0 + t if s.init == "ones" else t.abs() if s.init == "a_log" else t
        if s.init == "normal":
            tensors[s.name] = tensors[s.name].bfloat16()
    model.bind({k: v.to(device) for k, v in tensors.items()}, dtype, torch.device(device))
    return model


@pytest.mark.parametrize("name", list(SIZES))
def test_like_layers_are_found_and_an_edit_is_noticed(name):
    model = _model(name, torch.bfloat16, "cpu")
    found = RepeatedLayers.of(model.layers, model.schedule)
    assert found is not None and found.stands() and len(found.layers) == SIZES[name]["num_hidden_layers"]
    assert len({len(t) for t in found.tensors}) == 1
    # one layer's constant, one layer's weight type, one layer's shape: each makes the layers unlike
    last = model.layers[-1]
    for part, attribute, value in ((last.mixers[1], "eps", 0.5), (last.ffn.down, "weight", last.ffn.down.weight.float()),
                                   (last.mixer_norm, "weight", last.mixer_norm.weight[:-4]), (last.mixers[0], "window", 7)):
        before = getattr(part, attribute)
        setattr(part, attribute, value)
        assert not found.stands() and RepeatedLayers.of(model.layers, model.schedule) is None, attribute
        setattr(part, attribute, before)
        found = RepeatedLayers.of(model.layers, model.schedule)
        assert found is not None and found.stands()


def test_edits_in_lists_are_noticed_and_one_that_is_undone_stands_again():
    model, other = _model("small", torch.bfloat16, "cpu"), _model("small", torch.bfloat16, "cpu")
    layers, block = model.layers, model.layers[2]
    look = lambda: RepeatedLayers(model.layers, model.schedule)  # noqa: E731
    stands = lambda found: found.stands(model.layers, model.schedule)  # noqa: E731
    # a list (or the model's attribute), what is put in its place, and whether the layers are alike then
    for where, at, new, alike in ((layers, 2, other.layers[2], True), (block.mixers, 0, other.layers[2].mixers[0], True),
                                  (block.out_scales, 1, 0.5, False), (block.out_offsets, 0, (8, 64), False),
                                  (model.schedule, 1, LayerRun(1, cache=0), False)):
        found, before = look(), where[at]
        assert found.alike and stands(found)
        where[at] = new
        assert not stands(found) and look().alike == alike
        edited = look()
        where[at] = before
        assert not stands(edited) and look().alike
    found = look()
    model.layers = list(layers)
    assert not stands(found) and look().alike
    found = look()
    model.layers.append(model.layers.pop())
    assert stands(found)                                  # (the same again)
    model.layers.append(other.layers[0])
    assert not stands(found) and look().alike
    found = look()
    del block.ffn.limit
    assert not stands(found) and not look().alike


@pytest.mark.gpu
def test_a_step_runs_the_layers_and_mixers_that_are_there_now():
    """A layer and a mixer put in another's place count from the next prompt on, and so does taking them back."""
    model = _model("tensor cores", torch.bfloat16, "cuda:0")
    other = _model("tensor cores", torch.bfloat16, "cuda:0")
    for layer in other.layers:
        layer.ffn.down.weight = layer.ffn.down.weight * 0.5
        layer.mixers[1].D = layer.mixers[1].D + 1.0
    llm = tlc.LLM(model, dtype="bfloat16", max_tokens=64 * 8, max_seqs=2)

    def logits():
        slot = llm.cache.acquire()
        out = llm.step([StepEntry(slot, list(range(1, 60)), (58,))]).clone()
        llm.cache.release(slot)
        return out

    first = logits()
    for where, at, new in ((model.layers, 2, other.layers[2]), (model.layers[1].mixers, 1, other.layers[1].mixers[1])):
        before, where[at] = where[at], new
        changed = logits()
        repeated, model.repeated = model.repeated, None
        one_by_one = logits()
        model.repeated = repeated
        assert torch.equal(changed, one_by_one) and not torch.equal(changed, first)
        where[at] = before
        assert torch.equal(logits(), first) and model.repeated.alike


def test_a_copy_that_torch_makes_ends_the_attempt(monkeypatch):
    """A weight that is multiplied by as a dense copy: the copy's address stands for nothing in the other layers."""
    monkeypatch.setattr(ops, "linear", lambda *args: None)
    down = _model("small", torch.bfloat16, "cpu").layers[0].ffn.down
    for weight, complete in ((down.weight, True), (down.weight.t().contiguous().t(), False)):
        down.weight = weight
        with ops.noting() as notes:
            down.forward(None, None)
        assert notes.complete == complete


def test_a_mixers_own_projection_lives_as_long_as_the_step(monkeypatch):
    """A mixer that is the only one of its layer projects for itself; its calls are made again for the other layers."""
    mixer = next(m for m in _model("small", torch.float32, "cpu").layers[0].mixers if type(m).__name__ == "Mamba2Mixer")
    i32, seen = torch.zeros(4, dtype=torch.int32), []
    step = StepInfo(3, 1, i32, i32, i32, i32, i32, i32)
    monkeypatch.setattr(ops, "linear", lambda x, w, out, *args: seen.append(out))
    monkeypatch.setattr(type(mixer), "forward_projected", lambda self, proj, *args: seen.append(proj))
    with step_scratch(step):
        mixer.forward(torch.zeros(3, mixer.in_proj.in_features), step, None, None)
    assert len(seen) == 2 and all(any(t is held for held in step.scratch.values()) for t in seen)


def test_numbers_are_noted_as_the_library_gets_them():
    """A number beyond the 32-bit range is infinite for the call (a clamp that is meant to be none), and so it is when noted."""
    with ops.noting() as notes:
        for v in (0.5, -0.0, 3, 1e39, -1e39, float("inf"), 1e-46):
            notes.add("tlc_glu", (16, 0, 8, 1, 0, 32, 0, 4, 1, v, 1.0, 0))
    got = [notes.words[12 * i + 9] for i in range(7)]
    assert got == [0x3F000000, 0x80000000, 0x40400000, 0x7F800000, 0xFF800000, 0x7F800000, 0]


@pytest.mark.gpu
def test_layers_whose_weights_are_all_laid_out_otherwise_run_one_by_one():
    model, got = _model("tensor cores", torch.bfloat16, "cuda:0"), []
    repeated = model.repeated
    for turned in (False, True):
        for layer in model.layers if turned else ():
            layer.ffn.down.weight = layer.ffn.down.weight.t().contiguous().t()
        for model.repeated in (model.repeated, None):
            llm = tlc.LLM(model, dtype="bfloat16", max_tokens=64 * 8, max_seqs=2)
            got.append(llm.step([StepEntry(llm.cache.acquire(), list(range(1, 60)), (58,))]).clone())
        model.repeated = repeated
    assert all(torch.equal(got[0], other) for other in got[1:])


def test_no_weight_is_held_beside_the_layer_that_has_it():
    """A model that is bound again, or whose weights a program sets to something else, has room for one set of weights."""
    model = _model("small", torch.bfloat16, "cpu")
    found = RepeatedLayers.of(model.layers, model.schedule)
    part = model.layers[1].ffn.down
    old = weakref.ref(part.weight)
    part.weight = part.weight.clone()
    assert old() is None and not found.stands()
    old = [weakref.ref(l.ffn.down.weight) for l in model.layers]
    alive = []

    class Tensors(dict):
        def __getitem__(self, name):
            alive.append(sum(w() is not None for w in old))
            return super().__getitem__(name)

    specs = model.weight_specs()
    model.repeated = found
    model.bind(Tensors({s.name: torch.ones(s.shape) for s in specs}), torch.bfloat16, torch.device("cpu"))
    assert alive[0] == len(old) and alive[-1] == 0


def test_functions_put_around_a_layers_methods_or_the_kernels_wrappers_are_noticed(monkeypatch):
    model = _model("small", torch.bfloat16, "cpu")
    found = RepeatedLayers.of(model.layers, model.schedule)
    layer = model.layers[0]
    assert found.untouched()
    assert {n for n in ops._SIGNATURES if ops.library().tlc_replay_index(n.encode()) >= 0} == ops.REPEATABLE
    for owner, name in ((type(layer), "forward"), (type(layer.ffn), "forward"), (type(layer.mixers[0]), "mix"),
                        (type(layer), "entry"), (ops, "linear"), (ops, "attention"), (ops, "_call")):
        with monkeypatch.context() as m:
            old = getattr(owner, name)
            m.setattr(owner, name, lambda *args: old(*args))
            assert not found.untouched(), name
        assert found.untouched() and found.stands()


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["a layer", "a kernel"])
def test_a_function_put_around_the_layers_is_called_for_every_one(monkeypatch, where):
    model = _model("small", torch.bfloat16, "cuda:0")
    llm = tlc.LLM(model, dtype="bfloat16", max_tokens=64 * 8, max_seqs=2)
    calls, got = [], []
    owner, name, times = (type(model.layers[0]), "forward", 1) if where == "a layer" else (ops, "linear_swiglu", 1)
    old = getattr(owner, name)
    for traced in (False, True, False):
        with monkeypatch.context() as m:
            if traced:
                m.setattr(owner, name, lambda *args, **more: (calls.append(1), old(*args, **more))[1])
            slot = llm.cache.acquire()
            got.append(llm.step([StepEntry(slot, list(range(1, 60)), (58,))]).clone())
            llm.cache.release(slot)
    assert len(calls) == times * len(model.layers) and torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])


def test_steps_that_wait_for_the_gpu_are_told_by_rows_and_weights():
    """From a number of rows on that falls with the size of a layer's matrices, and with their type's rate."""
    layers = [_Forks(i) for i in range(4)]
    look = lambda: RepeatedLayers.of(layers, [LayerRun(i) for i in range(len(layers))])  # noqa: E731
    assert not look().is_long(1023) and look().is_long(1024)
    first = {}
    for dtype in (torch.float32, torch.bfloat16):
        for n in (2048, 4096):
            for layer in layers:
                layer.weight = torch.empty(n, n, dtype=dtype)
                layer.gain = layer.weight[:n // 2]              # (rows of the same matrix: counted once)
            first[dtype, n] = next(rows for rows in range(1, 1025) if look().is_long(rows))
    assert first[torch.float32, 4096] < first[torch.float32, 2048] < first[torch.bfloat16, 4096] <= first[torch.bfloat16, 2048] == 1024


@pytest.mark.gpu
def test_long_steps_run_layer_by_layer(monkeypatch):
    model, got, times = _model("tensor cores", torch.bfloat16, "cuda:0"), [], []
    table = ops.replay
    monkeypatch.setattr(ops, "replay", lambda functions, words, n: (times.append(n), table(functions, words, n)))
    for limit, repeated in ((1024, 3), (60, 3), (59, 0)):
        model.repeated.LONG_STEP = limit
        llm = tlc.LLM(model, dtype="bfloat16", max_tokens=64 * 8, max_seqs=2)
        got.append(llm.step([StepEntry(llm.cache.acquire(), list(range(1, 60)), (58,))]).clone())
        assert sum(times) == repeated
        times.clear()
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])


def test_parts_that_say_nothing_are_not_repeated():
    model = _model("small", torch.float32, "cpu")

    class Own(type(model.layers[1].ffn)):
        pass

    model.layers[1].ffn.__class__ = Own
    assert RepeatedLayers.of(model.layers, model.schedule) is None


def test_the_table_of_calls_is_checked_before_the_first_call():
    lib = ops.library()
    assert lib.tlc_replay_index(b"tlc_linear") >= 0 and lib.tlc_replay_index(b"tlc_argmax") == -1
    words = (ctypes.c_ulonglong * 4)()
    for functions, n_words in (([lib.tlc_replay_index(b"tlc_event_record")], 4), ([99], 4), ([-1], 0)):
        fns = (ctypes.c_int * len(functions))(*functions)
        assert lib.tlc_replay(fns, words, n_words, len(functions), 1) < 0 and b"replay" in lib.tlc_last_error()
    assert lib.tlc_replay(None, None, 0, 0, 3) == 0


class _Forks(Editable):
    """A layer of four calls on the host: one on the caller's stream, one on a stream of its own between two events."""
    entry = None

    def __init__(self, number):
        self.weight, self.gain = torch.ones(8), torch.ones(8)
        self.side, self.fork, self.done = [0x1000 * (number + 1) + 0x100 * i for i in range(3)]

    def repeats(self):
        return frozenset(("side", "fork", "done"))

    def handles(self, device):
        return [self.side, self.fork, self.done]

    def forward(self, x, step, cache, ready, wanted, scratch=()):
        stream = lambda h: SimpleNamespace(cuda_stream=h)  # noqa: E731
        event = lambda h: SimpleNamespace(cuda_event=h, record=lambda s: None)  # noqa: E731
        waiting = lambda h: SimpleNamespace(cuda_stream=h, wait_event=lambda e: None)  # noqa: E731
        norm = lambda w, h: ops._notes.calls.add("tlc_rmsnorm", (x.data_ptr(), 8, None, w.data_ptr(), 1e-5, 1, 8, x.data_ptr(), 0, h))  # noqa: E731
        norm(self.weight, ops.stream_handle())
        ops.record_event(event(self.fork), stream(ops.stream_handle()))
        ops.wait_event(waiting(self.side), event(self.fork))
        ops._note_owned(*scratch)
        norm(self.gain, self.side)
        ops.record_event(event(self.done), stream(self.side))
        ops.wait_event(waiting(ops.stream_handle()), event(self.done))
        return False


def _run_on_the_host(monkeypatch, layers, stream):
    """(entries that ran, [stream of every norm call made again]) of a step on a stream of that handle, and the words."""
    got = []
    monkeypatch.setattr(ops, "stream_handle", lambda: stream)
    monkeypatch.setattr(ops, "replay", lambda functions, words, times: got.append((functions.copy(), words.copy())))
    found = RepeatedLayers.of(layers, [LayerRun(i) for i in range(len(layers))])
    i32 = torch.zeros(4, dtype=torch.int32)
    step = StepInfo(1, 1, i32, i32, i32, i32, i32, i32)
    done, left = found.run(torch.zeros(1, 8), step, SimpleNamespace(layer_view=lambda r, writes, kv: LayerCache()))
    rows = [row for _, words in got for row in words.tolist()]
    return done, rows


def test_the_callers_stream_is_never_taken_for_a_layers_own(monkeypatch):
    """torch hands out 32 streams in turn, and the layers have some of them: a step may run on a layer's own stream."""
    layers = [_Forks(i) for i in range(4)]
    norm_words, event_words = 10, 2
    first, second = norm_words - 1, 2 * norm_words + 2 * event_words - 1     # where the streams of the two norm calls stand
    for stream in (0, 0x77, layers[2].side):
        done, rows = _run_on_the_host(monkeypatch, layers, stream)
        assert done == 4 and [row[first] for row in rows] == [stream] * 3
        assert [row[second] for row in rows] == [layer.side for layer in layers[1:]]
    # the first layer's own: the words do not say which of the two is meant, so the layers run one by one
    done, rows = _run_on_the_host(monkeypatch, layers, layers[0].side)
    assert (done, rows) == (1, [])


def test_scratch_of_repeated_calls_is_kept_until_the_callers_stream_is_through(monkeypatch):
    """It was allocated on the first layer's own stream, where others may be handed it, and every layer's stream uses it."""
    seen = []

    class OnGpu(torch.Tensor):
        is_cuda = True

        def record_stream(self, stream):
            seen.append((self.data_ptr(), stream))

    scratch = torch.zeros(8).as_subclass(OnGpu)

    class Layer(_Forks):
        def repeats(self):
            return super().repeats()

        def forward(self, *args):
            return super().forward(*args, scratch=(scratch,))

    monkeypatch.setattr(repeat, "current_stream", lambda device: "the caller's")
    done, rows = _run_on_the_host(monkeypatch, [Layer(i) for i in range(3)], 0x77)
    assert done == 3 and len(rows) == 2 and seen == [(scratch.data_ptr(), "the caller's")]


def test_tensors_that_share_an_address_in_one_layer_only(monkeypatch):
    """Two weights of the first layer that are one tensor: its calls do not say which is meant."""
    tied = [_Forks(i) for i in range(4)]
    for layer in tied:
        layer.gain = layer.weight
    done, rows = _run_on_the_host(monkeypatch, tied, 0x77)
    assert done == 4 and [(row[3], row[17]) for row in rows] == [(l.weight.data_ptr(),) * 2 for l in tied[1:]]
    others = [_Forks(i) for i in range(4)]
    others[2].gain = others[2].weight                    # (its own words say so)
    done, rows = _run_on_the_host(monkeypatch, others, 0x77)
    assert done == 4 and [(row[3], row[17]) for row in rows] == [(l.weight.data_ptr(), l.gain.data_ptr()) for l in others[1:]]
    first = [_Forks(i) for i in range(4)]
    first[0].gain = first[0].weight
    assert _run_on_the_host(monkeypatch, first, 0x77) == (1, [])
    tied[3].gain = torch.ones(8)                         # the last one's are two: the layers before it are repeated
    done, rows = _run_on_the_host(monkeypatch, tied, 0x77)
    assert done == 1 + len(rows) <= 3


@pytest.mark.gpu
def test_a_step_on_a_layers_own_stream_gives_the_same_bits():
    model = _model("tensor cores", torch.bfloat16, "cuda:0")
    r = random.Random(6)
    tokens = [[r.randrange(SIZES["tensor cores"]["vocab_size"]) for _ in range(n)] for n in (40, 150, 20)]
    got = []
    for stream in (lambda: torch.cuda.current_stream(), lambda: model.layers[0]._side[0], lambda: model.layers[2]._side[0]):
        llm = tlc.LLM(model, dtype="bfloat16", max_tokens=64 * 16, max_seqs=3)
        slots = [llm.cache.acquire() for _ in tokens]
        torch.cuda.synchronize()
        with torch.cuda.stream(stream()):
            out = [llm.step([StepEntry(s, t, (len(t) - 1,)) for s, t in zip(slots, tokens)]) for _ in range(2)]
        torch.cuda.synchronize()
        got.append([t.clone() for t in out] + [g.data.clone() for g in llm.cache.state_groups])
    for other in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0], other))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("name", list(SIZES))
def test_repeated_layers_give_the_same_bits_as_layers_one_by_one(name, dtype):
    """Prompts in batches (row by row, in chunks, longer than a chunk), a further turn, single tokens without a captured
    step: logits and the whole cache, on the default stream and on another."""
    model = _model(name, getattr(torch, dtype), "cuda:0")
    assert model.repeated is not None
    V, r = SIZES[name]["vocab_size"], random.Random(5)
    ids = lambda n: [r.randrange(V) for _ in range(n)]  # noqa: E731
    steps = [[ids(n) for n in lens] for lens in ((5, 1, 3), (40, 150, 20), (1, 1, 1), (33, 1, 260), (500, 30, 600))]
    got, calls = [], []
    for repeated in (model.repeated, None):
        for stream in (torch.cuda.current_stream(), torch.cuda.Stream()):
            model.repeated = repeated
            llm = tlc.LLM(model, dtype=dtype, max_tokens=64 * 64, max_seqs=3)
            slots = [llm.cache.acquire() for _ in range(3)]
            before = ops.launch_count()
            torch.cuda.synchronize()
            with torch.cuda.stream(stream):
                out = [llm.step([StepEntry(s, t, (len(t) - 1,)) for s, t in zip(slots, step)]) for step in steps]
            torch.cuda.synchronize()
            calls.append(ops.launch_count() - before)
            got.append([t.clone() for t in out] + [g.k.clone() for g in llm.cache.kv_groups] + [g.v.clone() for g in llm.cache.kv_groups]
                       + [g.data.clone() for g in llm.cache.state_groups])
    assert len(set(calls)) == 1
    for other in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0], other))


@pytest.mark.gpu
def test_every_layer_of_a_repeated_step_goes_through_the_library_once():
    """The first layer's calls through Python, the others' from the table; tensors that change their place between steps are
    found again."""
    model = _model("tensor cores", torch.bfloat16, "cuda:0")
    llm = tlc.LLM(model, dtype="bfloat16", max_tokens=64 * 8, max_seqs=2)
    table, times = ops.replay, []
    ops.replay = lambda functions, words, n: (times.append(n), table(functions, words, n))
    try:
        tokens = list(range(1, 60))

        def logits():
            slot = llm.cache.acquire()
            out = llm.step([StepEntry(slot, tokens, (58,))]).clone()
            llm.cache.release(slot)
            return out

        first = logits()
        assert times == [1, 1, 1]
        w = model.layers[2].ffn.down
        w.weight = w.weight.clone()                     # an edit: found alike again, at the new place
        assert torch.equal(first, logits()) and times == [1, 1, 1] * 2
        w.weight = w.weight.t().contiguous().t()        # other strides in one layer: one by one
        assert torch.equal(first, logits()) and times == [1, 1, 1] * 2
    finally:
        ops.replay = table
