"""The designs' 32-bit prompts with every product of more than 16 rows in three bfloat16 parts, whatever its weights' size (``Linear`` leaves the small ones,
which these models have, to the multiply-adds): the bounds of the designs' own tests hold."""
from __future__ import annotations

import importlib

import pytest

from conftest import token_ids

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("design,name", [("famalorn", "p"), ("famalorn", "t"), ("neruzen", "a"), ("neruzen", "d"), ("kerepel", "a"), ("kerepel", "b"), ("kerepel", "c"),
                                         ("sogidra", "a"), ("sogidra", "b"), ("zuvepel", "a"), ("zezilix", "a")])
def test_prompts_with_every_product_in_parts(tmp_path, monkeypatch, design, name):
    from thintensor_b200.engine.engine import Entry
    from thintensor_b200.kernels import api

    module = importlib.import_module(f"test_{design}_gpu")
    calls = []
    product = api.gemm_split
    monkeypatch.setattr(api, "gemm_split_pays", lambda tokens, features, k: tokens > 16)
    monkeypatch.setattr(api, "gemm_split", lambda *operands: (calls.append(operands[0].shape), product(*operands)))
    folder = module.write_model(tmp_path / design, name, "float32")
    judge = module.Judge("float32", folder)
    engine = module.load(folder, "float32").new_engine(max_tokens=512, max_sequences=2)
    for seed, length in enumerate([17, 65, 150, 230]):
        tokens = token_ids(module.CONFIGS[name]["vocab"], length, 100 + seed)
        slot = engine.open()
        logits = engine.step([Entry(slot, tokens, list(range(length)))])
        engine.close(slot)
        engine.check_status()
        judge.add(logits, tokens, range(length), f"{design} {name}, {length} tokens")
    judge.done()
    assert len(calls) >= 4 * len(module.CONFIGS[name]["layers"])
