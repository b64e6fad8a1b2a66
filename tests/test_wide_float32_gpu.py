"""Float32 models of every design at widths where their products run on the tensor cores and leave parts (inner sizes of 1,024 and
more; the designs' own test models are narrower), against the plain restatements: prompts together, portions, single tokens."""
import importlib

import pytest
import torch

import dryft_challenge_htn_2026_b200 as dk
import plain_qwen3
from dryft_challenge_htn_2026_b200.csrc import api
from dryft_challenge_htn_2026_b200.engine import Runner, load_model
from helpers import random_tokens
from test_fukatar_gpu import att as fukatar_att
from test_fukatar_gpu import lat, tol
from test_fukatar_gpu import par as fukatar_par
from test_mozutar_gpu import mem
from test_mozutar_gpu import par as mozutar_par
from test_nevotar_gpu import att as nevotar_att
from test_nevotar_gpu import hg
from test_nevotar_gpu import moe as nevotar_moe
from test_nevotar_gpu import par as nevotar_par
from test_nilivik_gpu import layer_cfg
from test_pibulix_gpu import attn as pibulix_attn
from test_pibulix_gpu import gla
from test_pibulix_gpu import moe as pibulix_moe
from test_venidra_gpu import attn as venidra_attn
from test_venidra_gpu import latent

pytestmark = pytest.mark.gpu
DENSE = {"kind": "dense", "ff": 1088}
BASE = dict(vocab=200, width=1024, norm={"eps": 1e-5})
MODELS = {
    "qwen3": dict(architectures=["Qwen3ForCausalLM"], vocab_size=200, hidden_size=1024, intermediate_size=1088, num_hidden_layers=2,
                  num_attention_heads=16, num_key_value_heads=4, head_dim=64, rms_norm_eps=1e-6, rope_theta=10000.0,
                  tie_word_embeddings=False, max_position_embeddings=1024),
    "nilivik": dict(BASE, architecture="Nilivik", embedding={"scale": 5.0}, logit_softcap=8.0,
                    layers=[layer_cfg(16, 4, 64, 64, 48, 16, 32, 64, 0.95, 1088), layer_cfg(20, 4, 32, 56, 24, 18, 16, 60, 0.9, None)]),
    "pibulix": dict(BASE, architecture="Pibulix", postln_alpha=2.0, decay_rank=[None, 16],
                    layers=[pibulix_attn(16, 4, 64, 64, 3, 0.2, 30.0, (32, 10000.0), (24, 3), DENSE),
                            gla(16, 32, 64, 4.0, pibulix_moe(6, 40, 2, 1, 1, 1.0, 1088))]),
    "venidra": dict(BASE, architecture="Venidra", embedding={"scale": 2.0}, logit_scale=0.5, logit_softcap=20.0,
                    layers=[latent(16, 32, 16, 64, 288, 96, 0.2, 10000.0, 40, DENSE),
                            venidra_attn(16, 4, 64, 64, 0.2, (32, 10000.0), 24, True, DENSE),
                            venidra_attn(18, 6, 32, 64, 0.2, (16, 500.0), 64, False, None)]),
    "nevotar": dict(BASE, architecture="Nevotar", norm={"eps": 1e-5, "groups": 4},
                    layers=[nevotar_att(16, 4, 16, 64, 0.25, 0.7, (0.3, 5), nevotar_moe(6, 40, 2.0, 2, (1088, 1.5))), hg(16, 32, 64, None),
                            nevotar_par((16, 4, 32, 64, 0.18, (16, 10000.0), 24), (16, 64, 16, 2, 3, 4), 0.5, 1.25, None)]),
    "fukatar": dict(BASE, architecture="Fukatar", logit_softcap=12.0,
                    embedding={"scale": 3.0, "bigram": {"buckets": 97, "mul_prev": 13, "mul_cur": 5}},
                    layers=[lat(16, 32, 64, 96, 0.3, DENSE), fukatar_att(16, 4, 32, 64, 0.5, (16, 500.0), 9.0, DENSE),
                            fukatar_par((16, 4, 32, 64, 0.3, (8, 50.0), None), (16, 4, 32, 64, 3), None)]),
    "mozutar": dict(BASE, architecture="Mozutar", embedding={"scale": 3.0}, loop={"start": 0, "stop": 1, "times": 2}, decay_rank=[None, 8],
                    layers=[mem(16, 32, 64, 8.0, DENSE), mozutar_par((16, 4, 64, 0.3, (32, 500.0), 9.0), (16, 32, 64, 4.0), DENSE)]),
}


def plain_logits(design, folder, tokens):
    if design != "qwen3":
        return importlib.import_module(f"test_{design}_gpu").plain_logits(folder, tokens)
    cfg, t = plain_qwen3.read_model(folder, torch.float64)
    return plain_qwen3.forward(cfg, t, tokens)


@pytest.mark.parametrize("design", list(MODELS))
def test_wide_models_in_float32(tmp_path, monkeypatch, design):
    made, real = [], api.gemm_f32_tc

    def noted(*a, **kw):
        out = real(*a, **kw)
        made.append(isinstance(out, api.Partial))
        return out

    monkeypatch.setattr(api, "gemm_f32_tc", noted)
    folder = str(tmp_path / design)
    dk.write_random_model(dk.config_from_dict(MODELS[design]), folder, seed=3, dtype=torch.float32, matrix_std=0.03)
    runner = Runner(load_model(folder, torch.float32), 64 * 12, 3)
    seqs = [random_tokens(200, n, 30 + n) for n in (90, 9, 130)]
    ref = [plain_logits(design, folder, s).double() for s in seqs]

    def check(out, places):
        for row, (i, p) in zip(out.double().cpu(), places, strict=True):
            err = float((row - ref[i][p].cpu()).abs().max())
            assert err <= tol("float32", ref[i]), (design, i, p, err)

    slots, cut = [runner.begin() for _ in seqs], [60, 5, 100]
    check(runner.step([(s, t[:c], [0, c - 1]) for s, t, c in zip(slots, seqs, cut)]), [(i, p) for i, c in enumerate(cut) for p in (0, c - 1)])
    check(runner.step([(slots[0], seqs[0][60:80], [3, 19]), (slots[2], seqs[2][100:120], [0])]), [(0, 63), (0, 79), (2, 100)])
    for k in range(4):
        check(runner.step([(s, [t[a + k]], [0]) for s, t, a in zip(slots, seqs, (80, 5, 120))]), [(i, a + k) for i, a in enumerate((80, 5, 120))])
    assert set(made) == {True, False}          # products in parts and whole ones
