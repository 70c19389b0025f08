"""The single upload of a ragged forward (engine/runner.py `forward_rows`): every field where it belongs, whatever the slot lists are."""
import pytest
import torch

from hibana_b200.engine.context import VERIFY
from hibana_b200.engine.executor import Executor
from hibana_b200.models.dense import DenseModel
from hibana_b200.target import dense_tiny


@pytest.fixture
def runner():
    t = dense_tiny()
    return Executor(DenseModel(t, "cpu", seed=0), max_batch=8, max_ctx=128, kv_slots=512, radix_cache=False).runner


def _fields(runner, *args, **kw):
    seen = {}

    def forward(ids, ctx):
        seen.update(ids=ids, ctx=ctx)
        return torch.zeros(1, runner.model.target.hidden, dtype=torch.bfloat16)

    runner._forward = forward
    runner.forward_rows(*args, want="none", **kw)
    return seen["ids"], seen["ctx"]


def test_fields_of_run_fragmented_and_empty_lists(runner):
    rows = [runner.alloc_row() for _ in range(4)]
    run, taken = runner.kv.alloc(5), runner.kv.alloc(40)
    assert run.run_start == run[0]
    fragments = [taken[9], taken[2], taken[30]]
    tokens = [[11, 12, 13, 14, 15], [], [21, 22, 23], [31]]
    starts, slots = [7, 3, 0, 64], [run, [], fragments, [taken[20]]]
    ids, ctx = _fields(runner, rows, tokens, starts, slots, mode=VERIFY, state_slots=[4, 5, 6, 7], has_initial_state=[1, 0, 0, 1])
    assert ids.dtype == torch.int64 and ids.tolist() == sum(tokens, [])
    want = {"positions": [7, 8, 9, 10, 11, 0, 1, 2, 64], "slots": list(run) + fragments + [taken[20]], "q_indptr": [0, 5, 5, 8, 9],
            "ctx_len": [12, 3, 3, 65], "seq_rows": rows, "state_slots": [4, 5, 6, 7], "has_initial_state": [1, 0, 0, 1]}
    for name, values in want.items():
        got = getattr(ctx, name)
        assert got.dtype == torch.int32 and got.tolist() == values, name
    assert ctx.max_rows == 5 and ctx.max_ctx_host == 65 and ctx.seq_starts_host == [5, 0, 3, 1]
    assert ctx.state_slots_host == [4, 5, 6, 7] and ctx.batch == 4
    assert runner.block_table[rows[0], 7:12].tolist() == list(run) and runner.block_table[rows[2], :3].tolist() == fragments
    assert int(runner.block_table[rows[3], 64]) == taken[20]
    # a run changed in place goes up as it is now
    run[1], run[3] = run[3], run[1]
    _, ctx = _fields(runner, rows[:1], tokens[:1], [7], [run])
    assert ctx.slots.tolist() == list(run)


def test_last_rows(runner):
    rows = [runner.alloc_row() for _ in range(2)]
    seen = []
    runner._forward = lambda ids, ctx: seen.append(ctx.sample_rows) or torch.zeros(2, runner.model.target.hidden, dtype=torch.bfloat16)
    runner.forward_rows(rows, [[1, 2, 3], [4]], [0, 0], [runner.kv.alloc(3), runner.kv.alloc(1)])
    assert seen[0].dtype == torch.int64 and seen[0].tolist() == [2, 3]


@pytest.mark.parametrize("broken", ["one slot for many tokens", "a run that is too short", "a run that is too long", "a start too few",
                                    "a row too many", "one state slot for two"])
def test_lists_that_do_not_fit_are_refused(runner, broken):
    rows = [runner.alloc_row() for _ in range(2)]
    tokens, starts, states = [[1, 2, 3], [4]], [0, 0], None
    slots = [runner.kv.alloc(3), runner.kv.alloc(1)]
    if broken == "one slot for many tokens":
        slots[0] = [9]
    elif broken == "a run that is too short":
        slots[0] = runner.kv.alloc(2)
    elif broken == "a run that is too long":
        slots[0] = runner.kv.alloc(4)
    elif broken == "a start too few":
        starts = [0]
    elif broken == "a row too many":
        rows.append(runner.alloc_row())
    else:
        states = [5]
    table = runner.block_table.clone()
    with pytest.raises(ValueError, match="forward_rows"):
        _fields(runner, rows, tokens, starts, slots, state_slots=states)
    assert torch.equal(table, runner.block_table)
