"""The row offsets of products grouped by head are kept between steps; a recorded decode step holds their addresses."""
import gc

import pytest
import torch


def test_offsets_a_recording_asked_for_are_not_given_up(monkeypatch):
    from dlm_b200.ops.native import NativeOps
    ops, recording = NativeOps.__new__(NativeOps), [False]
    monkeypatch.setattr(NativeOps, "_capturing", staticmethod(lambda device: recording[0]), raising=False)
    monkeypatch.setattr(NativeOps, "most_head_offsets", 8, raising=False)
    first = ops.head_offsets(4, 2, "cpu")
    assert first.tolist() == [0, 2, 4, 6, 8] and ops.head_offsets(4, 2, "cpu") is first
    recording[0] = True
    assert ops.head_offsets(4, 2, "cpu") is first
    made = ops.head_offsets(3, 5, "cpu")          # first asked for by a recording: nothing has filled it yet
    recording[0] = False
    assert ops.head_offsets(3, 5, "cpu") is not made
    for t in range(1, 5000):
        ops.head_offsets(6, t, "cpu")
    assert ops.head_offsets(4, 2, "cpu") is first
    assert len(ops._head_offsets) <= 8


@pytest.mark.gpu
def test_a_replayed_step_after_its_offsets_were_given_up(tmp_path):
    """A decode step is recorded, the kept offsets are pushed out, and what they held is written over: replays give the
    tokens of an engine that records nothing."""
    from dlm_b200.engine import Engine
    from zesapel_models import CONFIGS, tokens, write_model
    folder = str(tmp_path / "Y")
    write_model(CONFIGS["Y"], folder, seed=5)
    prompts = [tokens(60, 70, CONFIGS["Y"]["vocab"]), tokens(61, 30, CONFIGS["Y"]["vocab"])]

    def run(graphs):
        eng = Engine.from_pretrained(folder, dtype="bfloat16", device="cuda:0", page_size=16, num_pages=64, max_requests=2,
                                     max_context=256)
        eng.use_graphs = graphs
        ids = [eng.submit(p, max_new_tokens=24) for p in prompts]
        junk, logits = [], []
        while eng.scheduler.has_work():
            eng.run_step()
            logits.append(eng.last_logits.clone())
            if eng.graphs_recorded and not junk:
                ops = eng.rt.ops
                assert ops._graph_head_offsets
                ops.most_head_offsets = 1
                for t in (1001, 1002, 1003):
                    ops.head_offsets(2, t, torch.device("cuda:0"))
                gc.collect()
                junk = [torch.full((n,), 7, dtype=torch.int32, device="cuda:0") for n in (2, 4, 8, 16, 32) for _ in range(64)]
        assert not graphs or eng.graphs_recorded > 0
        return [eng.result(i) for i in ids], logits

    eager, replayed = run(False), run(True)
    assert eager[0] == replayed[0]
    for a, b in zip(eager[1], replayed[1]):
        assert torch.allclose(a, b, atol=2e-2, rtol=2e-2)
