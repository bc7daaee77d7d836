"""A replayed decode step chooses its chunks of keys from its shape alone: the same bits whatever lengths its graph was captured with, and the
chunk of the longest sequence, while a step that runs once takes the lengths that are there."""
import pytest
import torch

from helpers import random_ids
from tiny import make_model_dir

pytestmark = pytest.mark.gpu
CFG = {
    "architectures": ["LlamaForCausalLM"], "hidden_size": 256, "num_hidden_layers": 2, "num_attention_heads": 8, "num_key_value_heads": 8, "head_dim": 64,
    "intermediate_size": 256, "vocab_size": 128, "rope_theta": 10000.0, "rope_scaling": None, "rms_norm_eps": 1e-5, "max_position_embeddings": 4096,
    "tie_word_embeddings": True, "torch_dtype": "bfloat16", "eos_token_id": 7}
EQUAL, UNEQUAL = [1900] * 10, [1900] + [100] * 9            # one block-table width


def test_the_lengths_of_the_capture_leave_no_trace(tmp_path, monkeypatch):
    from ithaca_b200 import Engine
    from ithaca_b200.csrc import attention_bf16, ops
    d = make_model_dir(tmp_path, CFG, seed=2)
    chunks, run = [], attention_bf16.decode
    monkeypatch.setattr(attention_bf16, "decode", lambda *a, **k: (chunks.append(k["chunk_pages"]), run(*a, **k))[1])
    results = []
    for order in ((EQUAL, UNEQUAL), (UNEQUAL, EQUAL)):
        eng, rows = Engine(d, dtype="bfloat16", max_tokens=32768), {}
        for lens in order:
            slots = [eng.alloc_slot() for _ in lens]
            for i, (s, n) in enumerate(zip(slots, lens)):
                eng.step([s], [random_ids(n, CFG["vocab_size"], i)], None)
            logits, _ = eng._decoder.step(slots, [[5]] * len(lens))
            rows[len(set(lens))] = logits.clone()
            eng.stepper.check_status()
            for s in slots:
                eng.free_slot(s)
        assert len(eng._decoder.graphs) == 1
        results.append(rows)
    for kind in (1, 2):
        assert torch.equal(results[0][kind], results[1][kind])
    bound = attention_bf16.decode_chunk_pages(10, 8, 8, 32 * 64)
    pages = [-(-(n + 1) // 64) for n in UNEQUAL]
    assert set(chunks) == {bound} and attention_bf16.decode_chunk_pages_uneven(pages, 8, 8, attention_bf16.decode_chunk_pages(10, 8, 8, 30 * 64), ops.sm_count()) != bound
