"""Latent attention's long steps of requests that begin are replayed; a replay with another cut of the rows is the same step."""
import pytest
import torch

import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arch", ["dimuvik", "zoporax"])
def test_replayed_long_steps_equal_launched_ones(arch):
    from cajeta_llm_b200 import bench_design as B
    from cajeta_llm_b200.config import parse_config_dict
    from cajeta_llm_b200.engine.model import random_model
    from cajeta_llm_b200.engine.step import ModelRunner, StepEntry
    from cajeta_llm_b200.parts.base import Runtime
    config = getattr(B, f"{arch}_config")(dict(width=256, layers=2, heads=2, rank=128, experts=4, top=2, eff=128, ff=256, state=64))
    config["vocab"] = 500
    model = random_model(parse_config_dict(config), Runtime("bfloat16"), 5)
    cuts = [(300, 20), (20, 300), (160, 160), (300, 20), (320,), (1, 319)]       # 320 rows each, shared out differently
    outs = {}
    for graphs in (True, False):
        r = ModelRunner(model, max_seqs=2, max_tokens_per_seq=700, cuda_graphs=graphs)
        assert r.capture_max_rows < 320
        outs[graphs] = []
        for i, lengths in enumerate(cuts):
            slots = [r.admit() for _ in lengths]
            toks = [helpers.random_tokens(500, n, seed=10 * i + j) for j, n in enumerate(lengths)]
            outs[graphs].append(r.step([StepEntry(s, t, list(range(len(t)))) for s, t in zip(slots, toks)]))
            # a second long portion, now with cached tokens before it: launched kernel by kernel, not replayed
            before = r.graph_replays
            outs[graphs].append(r.step([StepEntry(s, t, [len(t) - 1]) for s, t in zip(slots, toks)]))
            assert r.graph_replays == before
            for s in slots:
                r.release(s)
        assert (r.graph_replays > 0) == graphs
    for a, b in zip(outs[True], outs[False]):
        assert torch.equal(a, b)
