"""Which portions of a step take the latent prompt form, with how much memory, and what the engine leaves for it."""
import random
from types import SimpleNamespace

import pytest
import torch

from mstar_b200 import ops
from mstar_b200.config import layout as L

HEADS, DIM, RANK = 16, 128, 512


def plan(q_lens, kv_lens, window=0, first=0):
    room = ops.latent_prompt_room(q_lens, HEADS, RANK)
    return ops.latent_prompt_groups(q_lens, kv_lens, window, HEADS * DIM, first, HEADS, room), room


def test_made_keys_and_values_take_no_more_than_the_folded_form_or_the_floor():
    rng = random.Random(1)
    for _ in range(300):
        q_lens = [rng.choice([1, 7, 31, 32, 300, 2048, 8000]) for _ in range(rng.randint(1, 6))]
        kv_lens = [q + rng.choice([0, 5, 1000, 30000, 120000]) for q in q_lens]
        window = rng.choice([0, 0, 1024])
        groups, room = plan(q_lens, kv_lens, window)
        folded = 10 * HEADS * RANK * sum(q for q in q_lens if q >= 32)
        assert room == max(256 << 20, folded)
        seen = []
        for first, count, keys in groups:
            assert all(q >= 32 or n <= 2048 or window for q, n in zip(q_lens[first:first + count], kv_lens[first:]))
            at_once = max(1, min(HEADS, room // (16 * DIM * keys)))
            assert 16 * DIM * keys * at_once <= room and (count == 1 or at_once == HEADS)
            seen += range(first, first + count)
        assert seen == sorted(set(seen))
        # what is left over is short (beside many keys or other short ones), or too long for the room with one head
        for i in set(range(len(q_lens))) - set(seen):
            short = q_lens[i] < 32 and (kv_lens[i] > 2048 or max(q_lens) < 32)
            assert short or 16 * DIM * kv_lens[i] > room


def test_each_portion_decides_for_itself():
    assert plan([2, 2048, 20, 40], [16002, 2048, 20, 40])[0] == [(1, 3, 2108)]
    assert plan([40, 20, 40], [40, 2049, 40])[0] == [(0, 1, 40), (2, 1, 40)]
    assert plan([1, 1, 64, 64], [900, 900, 64, 96], first=2)[0] == [(2, 2, 160)]
    assert plan([31, 5], [31, 5])[0] == []
    assert plan([64], [200], window=70)[0] == [(0, 1, 200 - 64)]      # past 136: keys from 67 on, a whole tile back


@pytest.mark.parametrize("dtype,v_dim,need", [(torch.bfloat16, 128, 256 << 20), (torch.float32, 128, 0),
                                              (torch.bfloat16, 64, 0)])
def test_the_cache_leaves_room_for_prompts(dtype, v_dim, need, monkeypatch):
    from mstar_b200.engine.llm import LLM
    from mstar_b200.engine.model import Model
    from mstar_b200.parts.base import CacheNeed, KVNeed
    from mstar_b200.parts.registry import mixer_workspace_bytes

    latent = L.LatentAttentionSpec(hidden_size=64, num_heads=2, qk_dim=128, rot_dim=64, v_dim=v_dim, kv_rank=64)
    assert mixer_workspace_bytes(latent, dtype) == need
    assert mixer_workspace_bytes(L.ParallelMixerSpec(hidden_size=64, branches=(latent, L.SelectiveScanSpec())), dtype) == need
    model = SimpleNamespace(layout=SimpleNamespace(blocks=[SimpleNamespace(mixer=L.SelectiveScanSpec()),
                                                           SimpleNamespace(mixer=latent)]),
                            runtime=SimpleNamespace(dtype=dtype),
                            cache_needs=[CacheNeed(kv=KVNeed(num_kv_heads=1, head_dim=128, planes=1))])
    model.workspace_bytes = lambda: Model.workspace_bytes(model)
    llm = LLM.__new__(LLM)
    llm.model, llm.device = model, torch.device("cpu")
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: (1 << 30, 1 << 31))
    page = 16 * 128 * dtype.itemsize
    assert llm._pages_from_memory(16, 0.9) == [int(((1 << 30) - need) * 0.9) // page]


def test_splits_of_a_token_s_keys():
    """A tile of 32 keys a split, or two where the CUDA-core kernels' blocks of heads fill the SMs by themselves."""
    plan = ops.latent_attention_plan
    assert plan(7, 16, 512, 70, sms=148)[1] == 3 and plan(64, 16, 512, 70, sms=148)[1] == 3
    assert plan(7, 16, 512, 70, sms=148, tensor=False)[1] == 3
    assert plan(64, 16, 512, 70, sms=148, tensor=False)[1] == 1 and plan(64, 16, 512, 200, sms=148, tensor=False)[1] == 3
    assert plan(1, 16, 512, 5, sms=148)[1] == plan(64, 16, 512, 20, sms=148, tensor=False)[1] == 1
