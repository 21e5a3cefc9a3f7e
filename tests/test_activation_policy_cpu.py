"""How many layers keep their activations: the loss chunk at its size, the allocator's own memory, and one answer for the ranks
that recompute together."""
import os
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from causal_trainer_dev_b200.models.config import preset
from causal_trainer_dev_b200.training import engine as E
from causal_trainer_dev_b200.training.memory_plan import (Lattice, backward_working_set_bytes, head_logit_bytes,
                                                          layer_activation_bytes, plan)

ROOT = Path(__file__).resolve().parents[1]
TOKENS = 16384


def _engine(cls=E.LayerwiseEngine, local=True, **options):
    engine = cls.__new__(cls)
    engine.cfg, engine.options = preset("llama3-8b"), E.EngineOptions(**options)
    engine.provider = E.LocalProvider.__new__(E.LocalProvider) if local else object()
    engine._decided = {}
    return engine


def _memory(monkeypatch, free, pool=(0, 0)):
    """The driver's free bytes (None: it must not be asked) and what the allocator has reserved and allocated."""
    def driver():
        if free is None:
            raise AssertionError("the driver was asked")
        return free, 0

    monkeypatch.setattr(torch.cuda, "mem_get_info", driver)
    monkeypatch.setattr(torch.cuda, "memory_reserved", lambda: pool[0])
    monkeypatch.setattr(torch.cuda, "memory_allocated", lambda: pool[1])
    monkeypatch.setattr(E, "_pool_bytes", lambda: pool)


def test_kept_logits_take_four_bytes():
    cfg = preset("llama3-8b")
    assert head_logit_bytes(cfg, TOKENS, 4096) == 4 and head_logit_bytes(preset("tiny"), 512, 4096) == 2
    assert head_logit_bytes(cfg, TOKENS, 100) == 2 and head_logit_bytes(cfg, 100, 4096) == 4       # chunks of whole blocks
    two, four = (backward_working_set_bytes(cfg, TOKENS, 4096, n) for n in (2, 4))
    assert four - two == 4096 * 128256 * 2
    alone = plan(cfg, seq_len=4096, micro_rows=4)
    assert alone["backward_working_set"] == four
    assert plan(cfg, seq_len=4096, micro_rows=4, lattice=Lattice(2))["backward_working_set"] == two    # a gathered head


def test_policy_counts_the_slab_that_the_loss_allocates(monkeypatch):
    cfg = preset("llama3-8b")
    per_layer = layer_activation_bytes(cfg, TOKENS)
    for engine, logit in ((_engine(), 4), (_engine(local=False), 2), (_engine(loss_backend="logits"), 2)):
        working = backward_working_set_bytes(cfg, TOKENS, 4096, logit)
        for spare in (0, per_layer - 1):
            _memory(monkeypatch, working + engine.options.memory_reserve_bytes + 5 * per_layer + spare)
            assert engine._layers_to_keep(TOKENS) == 5 and engine._room_for_logits
        _memory(monkeypatch, working + engine.options.memory_reserve_bytes - 1)
        assert engine._layers_to_keep(TOKENS) == 0 and not engine._room_for_logits


def _free_for(layers, pool=(0, 0)):
    cfg = preset("llama3-8b")
    return (backward_working_set_bytes(cfg, TOKENS, 4096, 4) + E.EngineOptions().memory_reserve_bytes
            + layers * layer_activation_bytes(cfg, TOKENS) - (pool[0] - pool[1]))


def test_a_pass_that_has_fitted_is_not_asked_for_again(monkeypatch):
    gb, engine = 1 << 30, _engine()
    for layers, used, room in ((5, 20 * gb, True), (0, 21 * gb, False)):
        pool = (30 * gb, used)
        _memory(monkeypatch, _free_for(layers, pool) - (not room), pool)
        assert engine._layers_to_keep(TOKENS) == layers and engine._room_for_logits == room
        engine._room_for_logits = not room
        for later in (pool, (30 * gb, used - gb), (30 * gb, used + E.POOL_DRIFT_BYTES)):
            _memory(monkeypatch, None, later)
            assert engine._layers_to_keep(TOKENS) == layers and engine._room_for_logits == room
        engine._decided.clear()


def test_another_state_of_the_allocator_or_another_size_asks(monkeypatch):
    gb, engine = 1 << 30, _engine()
    pool = (30 * gb, 20 * gb)
    _memory(monkeypatch, _free_for(5, pool), pool)
    assert engine._layers_to_keep(TOKENS) == 5
    for later in ((30 * gb + 1, 20 * gb), (30 * gb - 1, 20 * gb)):
        _memory(monkeypatch, _free_for(3, later), later)
        assert engine._layers_to_keep(TOKENS) == 3
        _memory(monkeypatch, _free_for(5, pool), pool)
        assert engine._layers_to_keep(TOKENS) == 5
    later = (30 * gb, 20 * gb + E.POOL_DRIFT_BYTES + 1)
    _memory(monkeypatch, _free_for(3, later), later)
    assert engine._layers_to_keep(TOKENS) == 3
    pool = later
    _memory(monkeypatch, None, pool)
    for change in (lambda e: e._layers_to_keep(TOKENS - 128), lambda e: (setattr(e.options, "memory_reserve_bytes", gb), e._layers_to_keep(TOKENS))):
        with pytest.raises(AssertionError, match="driver was asked"):
            change(engine)
    for tokens in range(128, 128 * 200, 128):                    # the memory of decisions is bounded
        _memory(monkeypatch, _free_for(5, pool), pool)
        engine._layers_to_keep(tokens)
    assert len(engine._decided) <= 64


@pytest.mark.parametrize("which", ["provider", "subclass", "empty"])
def test_only_one_replica_remembers(monkeypatch, which):
    class Other(E.LayerwiseEngine):
        pass

    pool = (0, 0) if which == "empty" else (30 << 30, 20 << 30)
    engine = _engine(Other) if which == "subclass" else _engine(local=which != "provider")
    _memory(monkeypatch, _free_for(5, pool), pool)
    engine._layers_to_keep(TOKENS)
    _memory(monkeypatch, None, pool)
    with pytest.raises(AssertionError, match="driver was asked"):
        engine._layers_to_keep(TOKENS)


def test_what_the_allocator_says(monkeypatch):
    current = lambda n: {"all": {"current": n}}  # noqa: E731
    stats = dict(reserved_bytes=current(1000), allocated_bytes=current(300))
    monkeypatch.setattr(torch.cuda, "memory_stats_as_nested_dict", lambda: stats)
    assert E._pool_bytes() == (1000, 300)
    monkeypatch.setattr(torch.cuda, "memory_stats_as_nested_dict", dict)
    assert E._pool_bytes() == (0, 0)


WORKER = r'''
import sys
import torch
import torch.distributed as dist
sys.path.insert(0, sys.argv[1])
from causal_trainer_dev_b200.models.config import preset
from causal_trainer_dev_b200.training import engine as E
from causal_trainer_dev_b200.training.memory_plan import backward_working_set_bytes, layer_activation_bytes
from causal_trainer_dev_b200.training.sp_engine import SpLayerwiseEngine
from causal_trainer_dev_b200.training.tp_engine import TpLayerwiseEngine

dist.init_process_group("gloo")
rank, group = dist.get_rank(), dist.group.WORLD
cfg = preset("llama3-8b")


class Sharded:
    fused, group = False, group


for cls, options in ((TpLayerwiseEngine, {}), (SpLayerwiseEngine, {}), (E.LayerwiseEngine, dict(remat_group_size=2))):
    engine = cls.__new__(cls)
    engine.cfg, engine.options, engine.provider = cfg, E.EngineOptions(**options), Sharded()
    engine.tp_group = engine.sp_group = group
    engine.tp_world = 1
    tokens = 16384
    per_layer = layer_activation_bytes(cfg, tokens)
    base = backward_working_set_bytes(cfg, tokens, 4096) + engine.options.memory_reserve_bytes + per_layer // 2
    torch.cuda.mem_get_info = lambda: (base + (7 + 3 * rank) * per_layer, 0)      # this rank alone: 7 or 10 layers
    torch.cuda.memory_reserved = torch.cuda.memory_allocated = lambda: 0
    assert engine._layers_to_keep(tokens) == 7, (cls, rank)
    engine.options.remat = "none"
    assert engine._layers_to_keep(tokens) == cfg.num_hidden_layers
engine.options.remat, engine.options.remat_group_size = "auto", 1
assert engine._layers_to_keep(tokens) == 7 + 3 * rank                             # nothing is recomputed together
print("DONE", rank)
dist.destroy_process_group()
'''


def test_ranks_that_recompute_together_keep_the_same_layers(tmp_path):
    script = tmp_path / "worker.py"
    script.write_text(WORKER)
    env = {**os.environ, "OMP_NUM_THREADS": "1", "CUDA_VISIBLE_DEVICES": ""}
    out = subprocess.run([sys.executable, "-m", "torch.distributed.run", "--standalone", "--local-addr", "127.0.0.1",
                          "--nproc-per-node", "2", str(script), str(ROOT)], capture_output=True, text=True, env=env, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.count("DONE") == 2
