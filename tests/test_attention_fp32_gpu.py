"""The two kernels of 32-bit attention give a row the same bits.  Values that start on no 16-byte boundary are taken by the one
that reads them one by one, so that shifting the cache's values by one element runs a call through the other kernel."""
import types

import pytest
import torch

import kernel_refs
from test_kernels_gpu import DEV, bar, gen, ops, rand      # noqa: F401  (gen is a fixture)

pytestmark = pytest.mark.gpu

PORTIONS = {"prompts": [(0, 33), (0, 200), (0, 1), (0, 64), (0, 65)], "decoded": [(s, 1) for s in (0, 15, 16, 31, 32, 63, 64, 127, 300)],
            "later portions": [(300, 40), (63, 2), (64, 129), (17, 15)]}
SCORES = {"softmax": {}, "sink": {"sink": True}, "window": {"window": 70}, "narrow window": {"window": 5}, "window of a tile": {"window": 64},
          "chunk": {"window": -50}, "kept": {"window": 40, "keep": 7}, "kept tile": {"window": 100, "keep": 65}, "sigmoid": {"sigmoid": True, "bias": True},
          "squashed": {"softcap": 5.0, "scales": True}, "scaled": {"scales": True, "window": 33, "keep": 3}}


def _case(nq, nkv, d, portions, gen, ps=16):
    lengths = [s + n for s, n in portions]
    pages = [-(-n // ps) for n in lengths]
    kc, vc = (rand((sum(pages), nkv, ps, d), torch.float32, gen) for _ in range(2))
    table = torch.full((len(portions), max(pages)), -1, dtype=torch.int32)
    order, at = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(7)).to(torch.int32), 0
    for r, n in enumerate(pages):
        table[r, :n] = order[at:at + n]
        at += n
    cu = [0]
    for _, n in portions:
        cu.append(cu[-1] + n)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)      # noqa: E731
    ctx = types.SimpleNamespace(cu_q=i32(cu), q_start=i32([s for s, _ in portions]), max_ctx_len=max(lengths),
                                token_request=i32([r for r, (_, n) in enumerate(portions) for _ in range(n)]))
    return rand((cu[-1], nq * d), torch.float32, gen), kc, vc, table.to(DEV), ctx


def _run(q, kc, vc, table, ctx, nq, nkv, d, kind, gen_state):
    g = torch.Generator(DEV).manual_seed(gen_state)
    per_head = torch.rand(nq, generator=g, device=DEV) + 0.5
    return ops().paged_attention_simt(q, q.stride(0), kc, vc, table, ctx.cu_q, ctx.q_start, ctx.token_request, q.shape[0], nq, nkv, d, 16,
                                      d ** -0.5, kind.get("window", 0), sink=kind.get("sink", False), sigmoid=kind.get("sigmoid", False),
                                      head_bias=per_head if kind.get("bias") else None, softcap=kind.get("softcap", 0.0),
                                      head_scales=per_head if kind.get("scales") else None, keep=kind.get("keep", 0), max_ctx_len=ctx.max_ctx_len)


def _shifted(values):
    other = torch.empty(values.numel() + 1, device=DEV)[1:].view(values.shape)
    other.copy_(values)
    assert other.data_ptr() % 16 == 4
    return other


@pytest.mark.parametrize("nq,nkv,d", [(4, 4, 128), (12, 2, 128), (6, 1, 48), (7, 1, 80), (4, 2, 16), (2, 1, 96)])
@pytest.mark.parametrize("portions", PORTIONS)
@pytest.mark.parametrize("score", SCORES)
def test_both_kernels_give_a_row_the_same_bits(nq, nkv, d, portions, score, gen):
    q, kc, vc, table, ctx = _case(nq, nkv, d, PORTIONS[portions], gen)
    got = _run(q, kc, vc, table, ctx, nq, nkv, d, SCORES[score], 3)
    assert torch.equal(_run(q, kc, _shifted(vc), table, ctx, nq, nkv, d, SCORES[score], 3), got)
    ops().check_status(DEV)


@pytest.mark.parametrize("requests,keys", [(48, 64), (128, 17), (128, 130), (3, 16)])
def test_many_short_requests(requests, keys, gen):
    """Batches that the kernel of one warp a row takes, against the plain reference and a request by itself (which shares its keys'
    tiles where it sees more than a few)."""
    nq = nkv = 16
    q, kc, vc, table, ctx = _case(nq, nkv, 128, [(keys - 1, 1)] * requests, gen)
    got = _run(q, kc, vc, table, ctx, nq, nkv, 128, {}, 3)
    want = kernel_refs.paged_attention(q, kc, vc, table, ctx, nq, nkv, 128, 16, 128 ** -0.5, 0)
    torch.testing.assert_close(got, want, **bar(torch.float32))
    for r in (0, requests - 1):
        one = types.SimpleNamespace(cu_q=torch.tensor([0, 1], dtype=torch.int32, device=DEV), q_start=ctx.q_start[r:r + 1].contiguous(),
                                    token_request=torch.zeros(1, dtype=torch.int32, device=DEV), max_ctx_len=2000)
        alone = _run(q[r:r + 1].contiguous(), kc, vc, table[r:r + 1].contiguous(), one, nq, nkv, 128, {}, 3)
        assert torch.equal(alone[0], got[r]), r


def test_values_of_larger_heads_need_no_boundary_either(gen):
    for dtype in (torch.float32, torch.bfloat16):
        q, kc, vc, table, ctx = _case(2, 1, 320, [(0, 9), (40, 1)], gen)
        q, kc, vc = q.to(dtype), kc.to(dtype), vc.to(dtype)
        other = torch.empty(vc.numel() + 1, dtype=dtype, device=DEV)[1:].view(vc.shape)
        other.copy_(vc)
        assert torch.equal(_run(q, kc, other, table, ctx, 2, 1, 320, {}, 3), _run(q, kc, vc, table, ctx, 2, 1, 320, {}, 3))
