"""A runner that captures its step again replays the new graph: the handle of the first, which is freed with it, is not used."""
import contextlib
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from llamatov_b200 import _lib, dev_residency as dr, synth


class Graph:
    handles = 0

    def __init__(self):
        Graph.handles += 1
        self.handle = Graph.handles

    def raw_cuda_graph_exec(self):
        return self.handle


def test_replays_take_the_handle_of_the_last_capture(monkeypatch):
    launched = []
    real_zeros = torch.zeros
    monkeypatch.setattr(torch.cuda, "CUDAGraph", Graph)
    monkeypatch.setattr(torch.cuda, "graph", lambda g, stream=None: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "synchronize", lambda: None)
    monkeypatch.setattr(torch, "zeros", lambda *a, device=None, **k: real_zeros(*a, **k))
    monkeypatch.setattr(dr, "_FUSED_STEP", False)
    monkeypatch.setattr(dr, "_ensure_argmax_buf", lambda: 0)
    monkeypatch.setattr(dr, "_LOGITS_BUF", SimpleNamespace(n=4, ptr=0))
    monkeypatch.setattr(_lib, "call", lambda name, handle, *a: launched.append((name, handle.value)))
    r = object.__new__(dr.GraphRunner)
    r.kv, r.E, r.captured, r.graph, r.stream = [], 8, False, None, SimpleNamespace(cuda_stream=0)
    r.arch = SimpleNamespace(fused_step=False, device_token=True)
    r._forward_on_device_token = lambda *a: None
    r._ensure_pinned = lambda: None
    r._pin_tok_np = r._pin_idx_np = np.zeros(1, np.int32)
    for _ in range(2):
        r.capture(torch.tensor([1]), torch.tensor([0]))
        launched.clear()
        r.replay_token(1)
        r.replay_logits(1)
        assert launched == [("lt_graph_replay_token", r.graph.handle), ("lt_graph_replay_logits", r.graph.handle)]


@pytest.mark.gpu
@pytest.mark.parametrize("again", [False, True])
def test_second_capture_equals_a_fresh_runner(again):
    def start():
        kv = [None] * cfg["n_layers"]
        g = dr.GraphRunner(w, cfg, kv)
        g.seed(torch.tensor([3, 5]), torch.arange(2))
        g.capture(torch.tensor([7]), torch.tensor([2]))
        return g
    dr.reset_engine_state()
    dr.apply_production_profile()
    w, cfg = synth.reference_weights(synth.make_model("tiny-llama", seed=3))
    r = start()
    got = [r.replay_logits(7), r.replay_token(9)]
    if again:
        r.capture(torch.tensor([11]), torch.tensor([4]))
    got += [r.replay_logits(11), r.replay_token(13), r.kv[0].length]
    fresh = start()
    want = [fresh.replay_logits(7), fresh.replay_token(9), fresh.replay_logits(11), fresh.replay_token(13), fresh.kv[0].length]
    for a, b in zip(got, want):
        assert torch.equal(a, b) if isinstance(a, torch.Tensor) else a == b
    assert _lib.device_status() == set()
