"""The form of decode attention is chosen by one rule: a step run kernel by kernel (as a captured graph does) and the same
step run a layer at a time take the same kernel with the same splits, also in large batches under a large context limit."""
import types

import pytest
import torch

from flexengine_b200 import ops

# clusters resident at once by cluster size, as a B200 answers for the decode kernel at head size 128
HELD = {2: 296, 3: 187, 4: 142, 5: 112, 6: 93, 7: 78, 8: 71, 9: 60, 10: 56, 11: 45, 12: 42, 13: 38, 14: 35, 15: 31, 16: 31}


@pytest.mark.parametrize("requests,nq,nkv", [(16, 40, 8), (32, 28, 4), (64, 28, 4), (64, 40, 8), (15, 40, 8), (64, 12, 2), (9, 12, 2)])
@pytest.mark.parametrize("limit", [512, 3072, 4096, 8192, 32768])
def test_eager_and_captured_steps_take_the_same_form(requests, nq, nkv, limit, monkeypatch):
    d, ps, taken = 8, 16, []
    for name, value in (("_need_cuda", lambda *t: None), ("sm_count", lambda *a: 148), ("_ptr", lambda t: None),
                        ("clusters_resident", lambda r, q, k, size, splits: HELD[splits]),
                        ("_bf16", lambda: types.SimpleNamespace(fe_paged_decode_scratch_bytes=lambda *a: 16, fe_layer_workspace_bytes=lambda *a: 16)),
                        ("scratch", lambda device, n: torch.empty(n, dtype=torch.uint8)), ("status_word", lambda device: None),
                        ("paged_decode_cluster", lambda *a, **k: taken.append((0, a[14]))),
                        ("paged_decode_mma", lambda *a, **k: taken.append((1, a[14])))):
        monkeypatch.setattr(ops, name, value)
    ctx = types.SimpleNamespace(max_q_len=1, max_ctx_len=limit, cu_q=torch.arange(requests + 1, dtype=torch.int32),
                                q_start=None, positions=None, token_request=None, host_lengths=None, host_starts=None)
    qkv, cache = torch.empty(requests, nq * d, dtype=torch.bfloat16), torch.empty(4, nkv, ps, d, dtype=torch.bfloat16)
    table = torch.zeros(requests, 4, dtype=torch.int32)
    ops.paged_attention(qkv, cache, cache, table, ctx, nq, nkv, d, ps, 1.0, 0)
    group = types.SimpleNamespace(slot_mapping=None, block_table=table, page_size=ps, storage=torch.empty(1, 2, 4))
    layer = types.SimpleNamespace(nq=nq, nkv=nkv, d=d, hidden=64, intermediate=64, window=0)
    step = ops.native_step(ctx, group, layer, torch.empty(requests, 64), write_cache=False)
    assert taken == [(step.attention, step.splits)]
