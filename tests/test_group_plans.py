"""The native plans of the optimizer's shape groups: what is kept, and when the engine's own entry points are bypassed."""
import types

import pytest
import torch

from i8muon_b200 import CutlassNSInt8, Muon, optimizer, recommend_coefficients
from i8muon_b200.engine import coefficient_array

C5 = recommend_coefficients(5)


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
    settings = (0, steps, 1e-7, True, 0.95, 0.95, True, 1, True, 0)
    engine = CutlassNSInt8()
    plan, size = optimizer._group_plan(engine, "_regular_prec", "float16", settings, array, torch.device("cuda", 0),
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
