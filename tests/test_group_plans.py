"""The native plans of the optimizer's shape groups: what is kept, and when the engine's own entry points are bypassed."""
import contextlib
import copy
import functools
import pickle
import threading
import types

import pytest
import torch

from i8muon_b200 import CutlassNSInt8, Muon, engine as engine_module, optimizer, recommend_coefficients
from i8muon_b200.engine import coefficient_array

C5 = recommend_coefficients(5)


@pytest.fixture
def host_only(monkeypatch):
    """``muon_step`` on CPU tensors with the library's calls recorded instead of made: the host's decisions alone."""
    calls = []
    word = torch.zeros(1, dtype=torch.int32)

    def call(name, *args):
        calls.append((name, args))
    monkeypatch.setattr(optimizer.native, "call", call)
    monkeypatch.setattr(optimizer.native, "group_bytes", lambda plan: calls.append(("group_bytes", ())) or 256)
    monkeypatch.setattr(optimizer, "validate_ns_device", lambda *a: None)
    monkeypatch.setattr(optimizer, "matrix_spec", lambda *a: None)
    monkeypatch.setattr(optimizer, "on_device", lambda index: contextlib.nullcontext())
    monkeypatch.setattr(optimizer, "raw_stream", lambda index: 0)
    monkeypatch.setattr(optimizer, "status_word", lambda device: word)
    monkeypatch.setattr(optimizer, "status_host", lambda index: word)
    monkeypatch.setattr(optimizer, "post_status", lambda device: None)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    return calls


def step(engine, shapes=((64, 96),) * 2, **settings):
    tensors = [[torch.ones(s) for s in shapes] for _ in range(3)]
    optimizer.muon_step(*tensors, **{**dict(lr=0.02, weight_decay=0.01, momentum=(0.95, 0.95), ns_coefficients=C5, eps=1e-7,
                                            adjust_lr_fn="none", precision="float16", ns_engine=engine), **settings})


# where a caller can put code of their own between the optimizer and the library
@pytest.mark.parametrize("where,name,precision", [
    ("class", "_regular_prec", "float16"), ("class", "_regular_bq", "fp8"), ("class", "_run", "float16"),
    ("class", "_call", "int8"), ("class", "_regular_i8", "int8_bq"), ("instance", "_regular_i8", "int8"),
    ("instance", "_regular_i8", "int8_bq"), ("instance", "_run", "float16"),
    ("instance", "_call", "float16"), ("router", "_regular_prec", "float16")])
def test_code_put_in_place_of_the_engines_own_is_called(monkeypatch, host_only, where, name, precision):
    engine, seen = CutlassNSInt8(), []
    if where == "router":                     # routes to the entry point of another engine
        other = CutlassNSInt8(fp16_first=False)
        monkeypatch.setattr(other, "_run", lambda route, x, *args: seen.append(x.shape) or x.clone())
        engine.router = other.router
    else:
        own = getattr(CutlassNSInt8, name)

        @functools.wraps(own)                 # keeps the name
        def wrapper(*args, **kwargs):
            x = next(a for a in args if isinstance(a, torch.Tensor))
            seen.append(x.shape)
            return x.clone()
        monkeypatch.setattr(CutlassNSInt8 if where == "class" else engine, name, wrapper)
    step(engine, precision=precision)
    assert [tuple(s)[-2:] for s in seen] == [(64, 96)]
    assert "i8m_group_step" not in [c[0] for c in host_only]


def test_an_engine_as_it_comes_takes_one_native_call_per_group(host_only):
    step(CutlassNSInt8(), ((64, 96), (64, 96), (32, 32)))
    assert [c[0] for c in host_only if c[0] != "group_bytes"] == ["i8m_group_step"] * 2


@pytest.mark.parametrize("shapes,posts", [(((64, 96), (32, 32)), 1), (((32, 32), (64, 96)), 0), (((64, 96), (64, 96)), 0),
                                          (((32, 32), (32, 32)), 1)])
def test_the_last_kernels_of_a_step_are_followed_by_a_copy_of_the_status_word(monkeypatch, host_only, shapes, posts):
    """A native group posts the word with its own last kernel; what runs after it on the device needs another copy."""
    posted = []
    monkeypatch.setattr(optimizer, "post_status", posted.append)
    engine = CutlassNSInt8()

    def router(rows, cols, precision, use_gram, threshold):
        if rows == 32:
            return (lambda x, **kwargs: x.clone()), "float16"
        return engine._regular_prec, "float16"
    engine.router = router
    step(engine, shapes)
    assert len(posted) == posts


def test_a_momentum_schedule_keeps_one_plan(host_only):
    engine = CutlassNSInt8()
    for mu, mu2 in ((0.85, 0.9), (0.9, 0.95), (0.95, 0.95)):
        step(engine, momentum=(mu, mu2))
        name, args = host_only[-1]
        assert name == "i8m_group_step" and args[-5:-3] == (1.0 - mu2, mu)
    assert len(engine._group_plans) == 1 and [c[0] for c in host_only].count("group_bytes") == 1
    step(engine, momentum=(0.9,))             # without Nesterov: another kernel argument of the plan
    assert len(engine._group_plans) == 2


def test_plans_survive_more_schedules_than_their_table_holds(host_only):
    engine = CutlassNSInt8()
    for i in range(300):
        coefficient_array([(2.0 + i, -1.5, 0.5)])
    late = [(9.0, -1.5, 0.5)]
    for _ in range(3):
        step(engine, ns_coefficients=late)
    assert len(engine._group_plans) == 1 and [c[0] for c in host_only].count("group_bytes") == 1
    for i in range(optimizer.MAX_GROUP_PLANS + 5):
        step(engine, ns_coefficients=[(2.0 + i, -1.5, 0.25)])
    assert len(engine._group_plans) == optimizer.MAX_GROUP_PLANS


def test_an_epsilon_held_in_a_tensor_is_read_at_every_step(host_only):
    engine, eps = CutlassNSInt8(), torch.tensor(1e-7)
    step(engine, eps=eps)
    eps.fill_(1e-3)
    step(engine, eps=eps)
    assert sorted(plan[2].eps for plan in engine._group_plans.values()) == pytest.approx([1e-7, 1e-3])


@pytest.mark.parametrize("duplicate", [copy.copy, copy.deepcopy, lambda engine: pickle.loads(pickle.dumps(engine))])
def test_a_used_engine_can_be_copied_and_pickled_without_its_native_state(host_only, duplicate):
    """Plans and kept call geometries hold addresses of this process and of this engine's tables."""
    engine = CutlassNSInt8(fp16_first=False)
    step(engine)
    engine._specs[("some call",)] = (1, 64, 96, 0, 256, 0x7f0000000000)
    twin = duplicate(engine)
    assert twin.fp16_first is False and twin.tiles == engine.tiles
    assert not twin._specs and not twin._group_plans and len(engine._specs) == len(engine._group_plans) == 1
    step(twin)
    assert [c[0] for c in host_only].count("i8m_group_step") == 2 and len(engine._group_plans) == 1


@pytest.mark.parametrize("which", ["status_word", "status_host"])
def test_threads_that_come_first_together_share_one_status_word(monkeypatch, which):
    """Plans keep the words' addresses, so a word that one thread was given may not be replaced by another thread's."""
    meet, real = threading.Barrier(2), torch.zeros

    def zeros(*args, **kwargs):
        meet.wait(10)                        # both threads have found no word
        return real(*args, **{**kwargs, "device": "cpu"})
    for table in ("_STATUS_WORDS", "_STATUS_HOST", "_STATUS_VIEWS"):
        monkeypatch.setattr(engine_module, table, {})
    monkeypatch.setattr(engine_module.torch, "zeros", zeros)
    monkeypatch.setattr(torch.Tensor, "pin_memory", lambda self: self)
    make, got = getattr(engine_module, which), []
    argument = torch.device("cuda", 0) if which == "status_word" else 0
    threads = [threading.Thread(target=lambda: got.append(make(argument))) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(got) == 2 and got[0] is got[1] is make(argument)
    if which == "status_host":
        got[0].fill_(7)
        assert engine_module._STATUS_VIEWS[0].value == 7


@pytest.mark.parametrize("known", [False, True])
def test_a_plan_made_under_a_capture_allocates_no_pinned_memory(monkeypatch, known):
    word = torch.zeros(1, dtype=torch.int32)
    pinned = []

    def status_host(index):
        pinned.append(index)
        return word
    monkeypatch.setattr(optimizer, "_STATUS_HOST", {0: word} if known else {})
    monkeypatch.setattr(optimizer, "status_host", status_host)
    monkeypatch.setattr(optimizer, "status_word", lambda device: word)
    monkeypatch.setattr(optimizer, "matrix_spec", lambda *a: None)
    monkeypatch.setattr(optimizer.native, "group_bytes", lambda plan: 256)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    array, steps = coefficient_array(C5)
    settings = (tuple(C5), 1e-7, True, True, 1, True, 0)
    engine = CutlassNSInt8()
    plan, size = optimizer._group_plan(engine, "_regular_prec", "float16", settings, (array, steps), torch.device("cuda", 0),
                                       torch.float32, torch.float32, torch.Size((64, 64)), 2, 1, True)
    assert size == 256
    assert bool(plan._obj.status_host) == known and pinned == ([0] if known else [])
    assert len(engine._group_plans) == int(known)


@pytest.mark.gpu
def test_an_entry_point_replaced_on_the_engine_is_called(cuda_device):
    gen = torch.Generator().manual_seed(3)
    grads = [torch.randn(64, 96, generator=gen).to(cuda_device) for _ in range(2)]
    calls, results = [], []

    def entry(self, x, *args, **kwargs):
        calls.append(tuple(x.shape))
        return CutlassNSInt8._regular_prec(self, x, *args, **kwargs)
    entry.__name__ = "_regular_prec"
    for replaced in (False, True):
        params = [torch.nn.Parameter(torch.ones(64, 96, device=cuda_device)) for _ in grads]
        for p, g in zip(params, grads):
            p.grad = g.clone()
        muon = Muon(params, lr=0.02, weight_decay=0.01, precision="float16")
        if replaced:
            muon._ns._regular_prec = types.MethodType(entry, muon._ns)
            muon._ns._routes.clear()          # routes looked up before the replacement keep what they found
        muon.step()
        results.append([p.detach() for p in params])
    assert len(calls) == 1 and calls[0][-2:] == (64, 96)
    assert all(torch.equal(a, b) for a, b in zip(*results))
