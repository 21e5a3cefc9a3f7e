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
    return engine


def _memory(monkeypatch, free, unused=0):
    def driver():
        if free is None:
            raise AssertionError("the driver was asked")
        return free, 0

    monkeypatch.setattr(torch.cuda, "mem_get_info", driver)
    monkeypatch.setattr(torch.cuda, "memory_reserved", lambda: unused)
    monkeypatch.setattr(torch.cuda, "memory_allocated", lambda: 0)
    monkeypatch.setattr(E, "_unused_pool_bytes", lambda: unused)


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


def test_a_whole_pass_in_the_allocator_needs_no_question(monkeypatch):
    cfg = preset("llama3-8b")
    need = cfg.num_hidden_layers * layer_activation_bytes(cfg, TOKENS) + backward_working_set_bytes(cfg, TOKENS, 4096, 4)
    _memory(monkeypatch, None, need)
    engine = _engine()
    engine._room_for_logits = False
    assert engine._layers_to_keep(TOKENS) == cfg.num_hidden_layers and engine._room_for_logits
    _memory(monkeypatch, 0, need - 1)                       # less: the reserve counts
    assert 0 < engine._layers_to_keep(TOKENS) < cfg.num_hidden_layers


@pytest.mark.parametrize("which", ["provider", "subclass"])
def test_only_one_replica_answers_from_the_allocator_alone(monkeypatch, which):
    class Other(E.LayerwiseEngine):
        pass

    cfg = preset("llama3-8b")
    need = cfg.num_hidden_layers * layer_activation_bytes(cfg, TOKENS) + backward_working_set_bytes(cfg, TOKENS, 4096, 4)
    _memory(monkeypatch, 0, need)
    engine = _engine(local=False) if which == "provider" else _engine(Other)
    assert engine._layers_to_keep(TOKENS) < cfg.num_hidden_layers


def test_pieces_of_segments_in_use_do_not_count(monkeypatch):
    current = lambda n: {"all": {"current": n}}  # noqa: E731
    stats = dict(reserved_bytes=current(1000), allocated_bytes=current(300), inactive_split_bytes=current(450))
    monkeypatch.setattr(torch.cuda, "memory_stats_as_nested_dict", lambda: stats)
    assert E._unused_pool_bytes() == 250
    monkeypatch.setattr(torch.cuda, "memory_stats_as_nested_dict", dict)
    assert E._unused_pool_bytes() == 0


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
