"""Sequences taken on one stream and stepped on another, what an engine leaves behind it when it goes, and steps that do not wait."""
import gc

import pytest
import torch

from helpers import model_folder, prompts_for

pytestmark = pytest.mark.gpu
LATE = 500_000_000          # cycles of a stream that is busy with something else: a quarter of a second, so that a slow host is still in time


def engine(dtype):
    from x0ne_engine_b200 import Engine
    return Engine.from_folder(model_folder("B", dtype), dtype=dtype, max_tokens=2048)


@pytest.mark.parametrize("taken_on", ["a stream", "the default stream"])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_a_sequence_taken_behind_other_work_of_another_stream(dtype, taken_on):
    eng = engine(dtype)
    ids, more = prompts_for(eng.vocab_size, [150, 3], seed=2)
    first = eng.new_sequence(160)
    want = [eng.step([first], [ids]).clone(), eng.step([first], [more]).clone()]
    torch.cuda.synchronize()
    one = torch.cuda.Stream() if taken_on == "a stream" else torch.cuda.default_stream()
    other = torch.cuda.Stream()
    with torch.cuda.stream(one):
        torch.cuda._sleep(LATE)
        slot = eng.new_sequence(160)
    with torch.cuda.stream(other):
        got = [eng.step([slot], [ids]), eng.step([slot], [more])]
    torch.cuda.synchronize()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    eng.cache.settle()
    assert len(eng.cache._pushed) <= 1          # streams that are through are forgotten


def test_an_engine_that_goes_waits_for_the_copies_out_of_its_pinned_tables():
    eng = engine("float32")
    slot = eng.new_sequence(64)
    eng.step([slot], [[1, 2, 3]])           # (what is loaded and allocated once is there)
    torch.cuda.synchronize()
    torch.cuda._sleep(LATE)
    eng.step([slot], [[1, 2, 3]])
    events = eng._stage_events
    assert any(e is not None and not e.query() for e in events)
    del eng
    gc.collect()
    assert all(e is None or e.query() for e in events)


def test_a_32_bit_step_returns_with_its_work_queued_and_the_next_one_reports():
    from x0ne_engine_b200 import Engine, Qwen3Config
    from x0ne_engine_b200.csrc import ops
    cfg = Qwen3Config(hidden_size=512, intermediate_size=576, num_hidden_layers=1, num_attention_heads=4, num_key_value_heads=2, head_dim=64, vocab_size=128,
                      max_position_embeddings=256, rms_norm_eps=1e-6, rope_theta=10000.0, tie_word_embeddings=False, dtype="float32")
    eng = Engine.random(cfg, seed=3, dtype="float32", max_tokens=256)
    slot = eng.new_sequence(64)
    want = eng.step([slot], [[1, 2, 3]]).clone()
    eng.free_sequence(slot)
    slot = eng.new_sequence(64)
    torch.cuda.synchronize()
    torch.cuda._sleep(LATE)
    got, queued = eng.step([slot], [[1, 2, 3]]), torch.cuda.Event()
    queued.record()
    assert not queued.query()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    ops.gemm_tc_status(eng.device).fill_(1 << 20)           # as a wait that ran out leaves it
    eng.step([slot], [[4]])
    torch.cuda.synchronize()
    with pytest.raises(ops.KernelError, match="an earlier step"):
        eng.step([slot], [[5]])
    eng.step([slot], [[5]])
    torch.cuda.synchronize()
    eng.step([slot], [[6]])


def test_the_word_for_waits_is_there_before_a_capture():
    from x0ne_engine_b200.csrc import ops
    from x0ne_engine_b200.engine.workspace import Workspace
    kept, ops._tc_status = ops._tc_status, {}
    try:
        ws = Workspace(8, torch.device("cuda:0"))
        x, w, y = ws.buffer("x", (8, 512), torch.float32).normal_(), torch.randn(96, 512, device="cuda:0"), ws.buffer("y", (8, 96), torch.float32)
        word = ops._tc_status[0]
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            ops.gemm_f32_nt(x, w, y, 8)
        assert ops._tc_status[0] is word
        word.fill_(1 << 20)
        graph.replay()
        assert int(word) == 1 << 20 and torch.allclose(y, x @ w.T, rtol=1e-4, atol=1e-3)          # (a replay leaves a report as it is)
    finally:
        ops._tc_status = kept


def test_a_sequence_is_not_taken_inside_a_capture():
    """A captured copy of the page table's row would be made from whatever the row holds when the graph is replayed."""
    from x0ne_engine_b200.csrc import ops
    eng = engine("bfloat16")
    ids = prompts_for(eng.vocab_size, [20], seed=4)[0]
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        graph = torch.cuda.CUDAGraph()
        graph.capture_begin()
        with pytest.raises(ops.KernelError, match="captured"):
            eng.new_sequence(64)
        graph.capture_end()
    torch.cuda.synchronize()
    slot = eng.new_sequence(64)
    assert bool(torch.isfinite(eng.step([slot], [ids])).all())
