"""Portions long enough for the kernels of long portions, through whole models: the recurrences in chunks and the latent attention
on tcgen05, alone in a step, beside single tokens, in recorded and in eager steps."""
import numpy as np
import pytest
import torch

import helpers
import test_fanidra_gpu as fanidra
import test_norelix_gpu as norelix
import test_pikadra_gpu as pikadra

pytestmark = pytest.mark.gpu

HGRN2 = dict(architecture="Fanidra", vocab=200, width=64, norm={"eps": 1e-5},
             layers=[fanidra.with_mlp(fanidra.layer_hgrn2(heads=1, dim=128, vdim=36), 96),
                     fanidra.with_mlp(fanidra.layer_hgrn2(heads=3, dim=64, vdim=64), None)])
DELTA = dict(architecture="Norelix", vocab=200, width=64, norm={"eps": 1e-5}, layers=[
    norelix.gated(2, 1, 16, 24, 0.25, None, norelix.dense(48, 2.5)),
    norelix.pair(norelix.left(2, 2, 32, 16, 0.18, 40, 9, 16, 1e4), norelix.right(2, 1, 64, 36, 4), 1.1, 0.9, None)])
LATENT = dict(architecture="Pikadra", vocab=200, width=64, norm={"eps": 1e-5},
              layers=[pikadra.layer(pikadra.mixer(16, 16, 64, 16, 320, 24, 0.15), {"kind": "dense", "ff": 96})])


def folder(root, config, cfg, seed, std):
    """A model folder with random weights; decays slow enough that a lost state shows."""
    from swifttransformer_b200.config import save_config
    from swifttransformer_b200.models import build_model_def
    from swifttransformer_b200.weights.random_init import random_tensors
    from swifttransformer_b200.weights.safetensors_io import write_safetensors
    cfg = config.from_dict(cfg)
    save_config(cfg, str(root))
    write_safetensors(str(root / "model.safetensors"),
                      [(s.name, (t.float() - 4.0).to(torch.bfloat16) if s.name.endswith(".A_log") else t)
                       for s, t in random_tensors(build_model_def(cfg).param_specs(), seed, std, "cpu")])
    return str(root)


def beside(reqs, cuts):
    """Steps that bring the next portion of every request at once (cuts: per request)."""
    steps, at = [], {r: 0 for r in reqs}
    for k in range(max(map(len, cuts.values()))):
        entries = [dict(id=r, tokens=reqs[r][at[r]:at[r] + c[k]], want=list(range(c[k]))) for r, c in cuts.items() if k < len(c)]
        for e in entries:
            at[e["id"]] += len(e["tokens"])
        steps.append(dict(entries=entries, end=[e["id"] for e in entries if at[e["id"]] == len(reqs[e["id"]])]))
    assert all(at[r] == len(reqs[r]) for r in reqs)
    return steps


def compare(mod, path, reqs, got, dtype, what):
    """As the design's own tests in float32.  In bfloat16 a model of recurrences alone is further off at single positions, with the
    walk as with the chunks (0.076 and 0.071 of the largest logit at worst, 5 of 691 positions above 0.05, median 0.0037)."""
    if dtype == "float32":
        return mod.compare(path, reqs, got, dtype, what)
    for rid, toks in reqs.items():
        ref = mod.plain_logits(path, toks)
        err = np.abs(got[rid] - ref).max(axis=1) / np.abs(ref).max()
        assert np.median(err) < 0.01 and (err > 0.05).mean() <= 0.03 and err.max() < 0.2, (what, rid, np.median(err), err.max())


def run(path, steps, dtype, graphs=True, page_size=16):
    from swifttransformer_b200.engine.replay import TraceSession
    s = TraceSession(path, dtype, helpers.live_token_need(steps), page_size=page_size, max_requests=8)
    s.runner.use_cuda_graphs = s.runner.use_cuda_graphs and graphs
    return helpers.replay(s, steps)


# per request: its portions in steps that all share; long ones beside single tokens and short ones, twice with a state before them
CUTS = dict(a=[130, 400, 97, 64], b=[1, 1, 1, 300], c=[95, 96, 1], d=[288, 1, 256, 1])


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("design", ["hgrn2", "delta"])
def test_recurrences(design, dtype, tmp_path, monkeypatch):
    from swifttransformer_b200 import ops
    from swifttransformer_b200.config import FanidraConfig, NorelixConfig
    mod, config, cfg = {"hgrn2": (fanidra, FanidraConfig, HGRN2), "delta": (norelix, NorelixConfig, DELTA)}[design]
    path = folder(tmp_path, config, cfg, 5, 0.08)
    reqs = {r: helpers.random_tokens(200, sum(c), seed=i) for i, (r, c) in enumerate(CUTS.items())}
    chunked = []
    for name in ("st_hgrn2_chunks", "st_delta_rule"):
        call = getattr(ops.lib(), name)
        monkeypatch.setattr(ops.lib(), name, lambda *a, call=call: (chunked.append(a), call(*a))[1])
    compare(mod, path, reqs, run(path, beside(reqs, CUTS), dtype), dtype, f"{design} beside one another")
    assert chunked
    compare(mod, path, reqs, run(path, helpers.trace_whole(reqs), dtype), dtype, f"{design} whole")


def test_recorded_and_eager_steps_take_the_same_form(tmp_path):
    """128 tokens of one request and four of 100: scratch and padding do not change the numbers of a float32 recurrence."""
    from swifttransformer_b200.config import FanidraConfig
    path = folder(tmp_path, FanidraConfig, HGRN2, 6, 0.12)
    for lens in ((128,), (100,) * 4, (300, 1, 1, 1)):
        reqs = {f"r{i}": helpers.random_tokens(200, n, seed=i) for i, n in enumerate(lens)}
        steps = beside(reqs, {r: [len(t)] for r, t in reqs.items()})
        outs = [run(path, steps, "float32", graphs) for graphs in (True, False)]
        for r in reqs:
            assert np.array_equal(outs[0][r], outs[1][r])


def test_latent_prompts(tmp_path, monkeypatch):
    from swifttransformer_b200 import ops
    from swifttransformer_b200.config import PikadraConfig
    path = folder(tmp_path, PikadraConfig, LATENT, 7, 0.12)
    taken = []
    call = ops.lib().st_latent_attention_tc
    monkeypatch.setattr(ops.lib(), "st_latent_attention_tc", lambda *a: (taken.append(1), call(*a))[1])
    cuts = dict(a=[400, 350], b=[1, 1], c=[37, 90])
    reqs = {r: helpers.random_tokens(200, sum(c), seed=i) for i, (r, c) in enumerate(cuts.items())}
    pikadra.compare(path, reqs, run(path, beside(reqs, cuts), "bfloat16"), "bfloat16", "latent beside one another")
    assert taken
    pikadra.compare(path, reqs, run(path, helpers.trace_whole(reqs), "bfloat16"), "bfloat16", "latent whole")
