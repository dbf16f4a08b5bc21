"""Kernels at the sizes where their tiles, rings and lists begin and end, against the plain references."""
import math

import pytest
import torch

import kernel_refs
from test_kernels_gpu import DEV, _attention_case, bar, gen, ops, rand      # noqa: F401  (gen is a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [63, 64, 132, 515])
@pytest.mark.parametrize("N", [129, 2049, 4800, 40000])
def test_gemm_fp32_tiles(N, K, gen):
    """Rows around every tile's edge: one chain of multiply-adds an output whichever kernel ran, so that a row is the same
    bit for bit in every batch, and within float32 of the 64-bit product (K terms of unit variance, as in the test of the
    product itself)."""
    x, w, b = rand((300, K), torch.float32, gen), rand((N, K), torch.float32, gen), rand((N,), torch.float32, gen)
    want = x.double() @ w.double().T + b.double()
    full = ops().linear(x, w, b)
    torch.testing.assert_close(full.double(), want, atol=2e-6 * math.sqrt(K) * 4, rtol=1e-5)
    for M in (1, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 128, 129, 256):
        assert torch.equal(ops().linear(x[:M].contiguous(), w, b), full[:M]), M
    # rows that start on no 16-byte boundary
    shifted = torch.empty(40 * K + 1, device=DEV)[1:].view(40, K)
    shifted.copy_(x[:40])
    assert torch.equal(ops().linear(shifted, w, b), full[:40])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nq,nkv,d", [(4, 2, 64), (12, 2, 128), (7, 1, 128)])
@pytest.mark.parametrize("window", [0, 70])
def test_attention_of_many_requests(dtype, nq, nkv, d, window, gen):
    """More requests than a warp has lanes, portions and decoded tokens around the tiles' edges (rows of 32 and of 256, keys of
    64): every row finds its request and its keys."""
    chunks = [(s, n) for s in (0, 1, 63, 64, 127, 300) for n in (1, 2, 5, 37, 64, 65)] + [(0, 171), (200, 86), (0, 1), (511, 1)]
    got, want, _ = _attention_case(dtype, nq, nkv, d, 16, chunks, window, gen, tcgen05=dtype == torch.bfloat16)
    torch.testing.assert_close(got.float(), want.float(), **bar(dtype))
    ops().check_status(DEV)


def test_attention_fp32_does_not_depend_on_the_portions(gen):
    """The same 200 tokens in one portion and as the last of portions cut anywhere: a row is the same bit for bit.  Values of keys
    that a row does not see may be anything."""
    import types
    nq, nkv, d, ps, n = 6, 2, 48, 16, 200
    pages = -(-n // ps)
    kc, vc = rand((pages, nkv, ps, d), torch.float32, gen), rand((pages, nkv, ps, d), torch.float32, gen)
    qkv = rand((n, (nq + 2 * nkv) * d), torch.float32, gen)
    bt = torch.arange(pages, dtype=torch.int32, device=DEV)[None]

    def run(first, last, values):
        ctx = types.SimpleNamespace(cu_q=torch.tensor([0, last - first], dtype=torch.int32, device=DEV),
                                    q_start=torch.tensor([first], dtype=torch.int32, device=DEV),
                                    token_request=torch.zeros(last - first, dtype=torch.int32, device=DEV))
        part = qkv[first:last].contiguous()
        return ops().paged_attention_simt(part, part.stride(0), kc, values, bt, ctx.cu_q, ctx.q_start, ctx.token_request,
                                          last - first, nq, nkv, d, ps, d ** -0.5, 0)
    whole = run(0, n, vc)
    for first, last in ((0, 1), (0, 33), (63, 65), (64, 129), (130, 200), (199, 200)):
        later = vc.clone()
        later.view(-1)[:] = vc.view(-1)
        for t in range(last, n):
            later[t // ps, :, t % ps] = float("inf")
        assert torch.equal(run(first, last, later), whole[first:last]), (first, last)


@pytest.mark.parametrize("V", [1000, 152064, 152063])
def test_sample_short_list_and_its_limits(V):
    """Top-k rows whose list of candidates fits, just fits or does not fit (all logits equal, the largest ones in one thread's share,
    k beyond the list's): the token is the reference's, and the same with every number of blocks."""
    torch.manual_seed(3)
    rows = [torch.randn(V) for _ in range(8)]
    rows[1][:] = 1.0                                            # every logit ties at the threshold
    rows[2][: min(V, 3000)] = 5.0                               # more ties than the list holds
    rows[3][::4096] += 50.0                                     # large ones in one thread's share
    rows[4][:] = torch.linspace(0, 3, V)
    rows[5][:] = float("-inf")
    rows[5][V // 2: V // 2 + 40] = torch.randn(40)              # fewer finite logits than k
    logits = torch.stack(rows).to(DEV)
    for k in (1, 2, 50, 511, 512, 513, 1025):
        if k >= V:
            continue
        n = len(rows)
        temperature = torch.full((n,), 0.8, device=DEV)
        top_k = torch.full((n,), k, dtype=torch.int32, device=DEV)
        seed = torch.arange(n, dtype=torch.int64, device=DEV) + k
        draw = torch.full((n,), 5, dtype=torch.int64, device=DEV)
        got = ops().sample(logits, temperature, top_k, seed, draw)
        for blocks in (1, 2, 4, 8):
            assert torch.equal(ops().sample(logits, temperature, top_k, seed, draw, blocks=blocks), got), (k, blocks)
        for r in range(n):
            x = rows[r].double() / float(temperature[r])
            order = torch.sort(rows[r], descending=True, stable=True).indices[:k]
            keep = torch.zeros(V, dtype=torch.bool)
            keep[order] = True
            token = int(got[r])
            assert keep[token], (k, r)
            mass = torch.where(keep, torch.exp(x - x.max()), torch.zeros_like(x))
            cum = torch.cumsum(mass, 0)
            target = kernel_refs.uniform_from(int(seed[r]), 5) * float(cum[-1])
            slack = 1e-5 * float(cum[-1])          # float32 sums of up to 1,025 masses: well below 1,025 * 2^-24
            assert (float(cum[token - 1]) if token else 0.0) - slack <= target <= float(cum[token]) + slack, (k, r)


@pytest.mark.parametrize("K", [64, 68, 67, 259])
def test_gemm_fp32_at_the_lines_of_its_rules(K, gen):
    """Widths on both sides of every line of the choice between the kernels for up to 16 rows: a row is the same bit for bit in every
    batch, rows that start on no 16-byte boundary included."""
    sms = ops().sm_count()
    for line in (8, 16, 32, 44, 64, 128, 256):
        w = rand((line * sms + 1, K), torch.float32, gen)
        x = rand((17, K), torch.float32, gen)
        for N in (line * sms, line * sms + 1):
            full = ops().linear(x, w[:N])
            torch.testing.assert_close(full.double(), x.double() @ w[:N].double().T, atol=2e-6 * math.sqrt(K) * 4, rtol=1e-5)
            for M in (1, 3, 5, 9, 16):
                assert torch.equal(ops().linear(x[:M].contiguous(), w[:N]), full[:M]), (N, M)


@pytest.mark.parametrize("V", [2047, 2048, 2049, 32000])
@pytest.mark.parametrize("k", [216, 217, 400, 401, 512, 513])
def test_sample_on_both_sides_of_the_lists_rule(V, k):
    """A top-k of which the list is tried with as many blocks a row and not with more: the tokens are the same with every number of blocks,
    and one of the k largest."""
    gen = torch.Generator(DEV).manual_seed(k)
    logits = torch.randn((3, V), generator=gen, device=DEV)
    temperature, top_k = torch.full((3,), 0.9, device=DEV), torch.full((3,), k, dtype=torch.int32, device=DEV)
    seed, draw = torch.arange(3, dtype=torch.int64, device=DEV), torch.full((3,), 7, dtype=torch.int64, device=DEV)
    got = ops().sample(logits, temperature, top_k, seed, draw, blocks=1)
    for blocks in (2, 4, 8):
        assert torch.equal(ops().sample(logits, temperature, top_k, seed, draw, blocks=blocks), got), blocks
    kth = logits.topk(k).values[:, -1]
    assert bool((logits.gather(1, got[:, None].long())[:, 0] >= kth).all())


@pytest.mark.parametrize("nq,nkv,d", [(12, 2, 128), (16, 16, 64), (5, 1, 128)])
@pytest.mark.parametrize("start,n", [(0, 1), (0, 255), (0, 256), (0, 700), (900, 64), (63, 257)])
def test_prefill_attention_of_one_request(nq, nkv, d, start, n, gen):
    """A step's only request finds its row tiles without a search: against the plain reference, with split keys and without, and bit for
    bit what it is beside a request that has no tokens in the step."""
    import types
    ps = 16
    pages = -(-(start + n) // ps)
    kc, vc = (rand((pages, nkv, ps, d), torch.bfloat16, gen) for _ in range(2))
    qkv = rand((n, nq * d), torch.bfloat16, gen)
    table = torch.arange(pages, dtype=torch.int32, device=DEV)[None].repeat(2, 1).contiguous()
    cu, starts = torch.tensor([0, n, n], dtype=torch.int32, device=DEV), torch.tensor([start, 0], dtype=torch.int32, device=DEV)
    ctx = types.SimpleNamespace(cu_q=cu[:2].contiguous(), q_start=starts[:1].contiguous(), token_request=torch.zeros(n, dtype=torch.int32, device=DEV))
    want = kernel_refs.paged_attention(qkv, kc, vc, table[:1], ctx, nq, nkv, d, ps, d ** -0.5, 0)
    for splits in (1, 3):
        def run(requests):
            return ops().paged_prefill_tcgen05(qkv, qkv.stride(0), kc, vc, table[:requests].contiguous(), cu[:requests + 1].contiguous(),
                                               starts[:requests].contiguous(), n, requests, n, nq, nkv, d, ps, d ** -0.5, 0, splits=splits)
        got = run(1)
        torch.testing.assert_close(got.float(), want.float(), **bar(torch.bfloat16))
        assert torch.equal(run(2), got)
    ops().check_status(DEV)
