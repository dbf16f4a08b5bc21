"""The 32-bit product in three bfloat16 parts: as close to 64 bits as the chain of multiply-adds, the same row in every batch."""
import pytest
import torch

from flexengine_b200.bench.shapes import SHAPES
from test_kernels_gpu import DEV, gen, ops, rand      # noqa: F401  (gen is a fixture)

pytestmark = pytest.mark.gpu


def chain(x, w):
    """The chain of multiply-adds of csrc/gemm_fp32.cu."""
    o = ops()
    out = torch.empty((x.shape[0], w.shape[0]), dtype=torch.float32, device=DEV)
    o._run(o._core(), "fe_gemm_fp32", o._ptr(x), o._ptr(w), None, o._ptr(out), o._c_int(x.shape[0]), o._c_int(w.shape[0]), o._c_int(x.shape[1]), o._stream())
    return out


@pytest.mark.parametrize("N,K", [(8192, 1024), (8199, 1028), (20000, 1091), (32768, 1024), (2017, 4160), (1024, 8192), (129, 65537)])
@pytest.mark.parametrize("sign", ["both", "positive"])
def test_split_product(N, K, sign, gen):
    """Rows around every tile's edge, K around a chunk's (64) and a segment's, rows on no 16-byte boundary; values of one sign, whose
    sums are longest and whose roundings towards zero would add up."""
    assert ops().split_ok(N, K) and not ops().split_ok(N, 1023) and not ops().split_ok(32769, K)
    x, w, b = rand((200, K), torch.float32, gen), rand((N, K), torch.float32, gen), rand((N,), torch.float32, gen)
    if sign == "positive":
        x, w = x.abs(), w.abs()
    want = x.double() @ w.double().T
    full = ops().linear(x, w)
    assert float((full.double() - want).norm()) <= float((chain(x, w).double() - want).norm())
    torch.testing.assert_close(ops().linear(x, w, b), full + b, atol=0, rtol=0)
    for M in (1, 16, 17, 64, 65, 128, 129):
        assert torch.equal(ops().linear(x[:M].contiguous(), w), full[:M]), M
    shifted = torch.empty(40 * K + 1, device=DEV)[1:].view(40, K)
    shifted.copy_(x[:40])
    assert torch.equal(ops().linear(shifted, w), full[:40])
    ops().check_status(DEV)


def test_what_is_no_finite_number_comes_out_as_from_the_chain(gen):
    x, w = rand((20, 1024), torch.float32, gen), rand((8200, 1024), torch.float32, gen)
    x[3, 5], x[4, 6], w[7, 9] = float("inf"), float("nan"), float("-inf")
    w[11, 0], x[6, 0] = 1e-30, 1e-30              # lost beside ordinary numbers (whole rows of small ones have tests of their own)
    got, want = ops().linear(x, w), chain(x, w)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isposinf(got), torch.isposinf(want))
    assert torch.equal(torch.isneginf(got), torch.isneginf(want))
    finite = torch.isfinite(want)
    torch.testing.assert_close(got[finite], want[finite], atol=1e-3, rtol=1e-5)
    x[5], w[9] = 3e38, 2.0                        # a sum beyond the largest number
    assert float(ops().linear(x, w)[5, 9]) == float("inf")


FEW = [(8200, 1024), (1536, 8960), (129, 65537)]              # one segment, several, rows on no 16-byte boundary


def both(x, w):
    """The product's result and the chain's, with what 64 bits give."""
    return ops().linear(x, w), chain(x, w), x.double() @ w.double().T


@pytest.mark.parametrize("N,K", FEW)
@pytest.mark.parametrize("nonzeros", [1, 2, 8, 16])
def test_rows_of_few_numbers_are_as_close_as_by_multiply_adds(N, K, nonzeros, gen):
    """What a product leaves out, a sum of few products shows.  One product: the four sums of a chunk (the larger by 2^7 each) are exact
    but for their last places, so that a result is rounded once to float32, after a sum rounded 2^-7 below it: (1 + 2^-4) 2^-24."""
    x = torch.zeros(80, K, device=DEV)
    for r in range(80):
        x[r, torch.randperm(K, device=DEV, generator=gen)[:nonzeros]] = rand((nonzeros,), torch.float32, gen)
    x[0, x[0] != 0] = 1 + 2 ** -7 - 2 ** -23                  # all places below the first eight at their largest
    w = rand((N, K), torch.float32, gen)
    w[:64] = 1 + 2 ** -7 - 2 ** -23
    got, by_chain, want = both(x, w)
    if nonzeros == 1:
        assert bool(((got.double() - want).abs() <= (1 + 2 ** -4) * 2 ** -24 * want.abs()).all())
    # 1 %: the second rounding, and how far norms of this many errors are from their mean
    assert float((got.double() - want).norm()) <= 1.01 * float((by_chain.double() - want).norm())


@pytest.mark.parametrize("N,K", FEW)
@pytest.mark.parametrize("scales", [(-30, 0), (-34, 0), (-36, 0), (-38, 0), (-41, 0), (0, -36), (-37, 37), (37, -37), (-18, -18), (-20, -20)])
def test_small_numbers_keep_their_places(N, K, scales, gen):
    """Rows or matrices whose third parts, or second ones, are below what bfloat16 holds (1e-40), alone or met by large numbers."""
    def scaled(shape, e):
        v = rand(shape, torch.float32, gen)
        return v * 10.0 ** (e / 2) * 10.0 ** (e / 2)
    x, w = scaled((20, K), scales[0]), scaled((N, K), scales[1])
    x[3] = 0
    w[5] = 0
    got, by_chain, want = both(x, w)
    assert float((got.double() - want).norm()) <= 1.01 * float((by_chain.double() - want).norm())
    assert not bool(got[3].any()) and not bool(got[:, 5].any())
    assert torch.equal(ops().linear(x[:9].contiguous(), w), got[:9])


def test_a_small_number_beside_ordinary_ones_counts_where_the_others_meet_zeros(gen):
    """Also where what meets it is a large number, so that the result is an ordinary one."""
    x, w = rand((20, 8960), torch.float32, gen), rand((1536, 8960), torch.float32, gen)
    x[4, 7], w[9], w[9, 7] = 1.2345678e-36, 0.0, 1.0
    x[5, 8], w[10], w[10, 8] = 1.2345678e-36, 0.0, 7.6543211e36
    got, by_chain, _ = both(x, w)
    assert float(got[4, 9]) == float(by_chain[4, 9]) and float(got[5, 10]) == float(by_chain[5, 10])


def test_not_finite_over_several_segments(gen):
    x, w = rand((20, 8960), torch.float32, gen), rand((1536, 8960), torch.float32, gen)
    x[3, 5], x[4, 6], w[7, 9], w[8, 8000] = float("inf"), float("nan"), float("-inf"), float("inf")
    x[5, 100], x[5, 8900] = float("inf"), float("-inf")        # both signs, in segments of their own
    x[6, 100], x[6, 8900], w[9] = 3e38, -3e38, 2.0             # beyond the largest number on the way, not at the end
    got, want, exact = both(x, w)
    for test in (torch.isnan, torch.isposinf, torch.isneginf):
        keep = torch.ones_like(got, dtype=torch.bool)
        keep[6] = False
        assert torch.equal(test(got)[keep], test(want)[keep])
    finite = torch.isfinite(want) & torch.isfinite(got)
    assert float((got[finite].double() - exact[finite]).norm()) <= float((want[finite].double() - exact[finite]).norm())


def test_every_sm_has_work_at_few_rows():
    """The layers' matrices of the benchmark's three shapes: a step of few rows is within a quarter of its chunks dealt out evenly."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for cfg in SHAPES.values():
        h, i = cfg["hidden_size"], cfg["intermediate_size"]
        heads = cfg["num_attention_heads"] * cfg["head_dim"]
        for N, K in ((heads + 2 * cfg["num_key_value_heads"] * cfg["head_dim"], h), (h, heads), (2 * i, h), (h, i)):
            segments = int(ops()._core().fe_gemm_split_segments(N, K))
            tiles, chunks = -(-N // 128), -(-K // 64)
            if ops().split_ok(N, K):
                assert -(-tiles * segments // sms) * -(-chunks // segments) <= 1.25 * tiles * chunks / sms + 1, (N, K, segments)


@pytest.mark.parametrize("N,K,M", [(1536, 8960, 1300), (5120, 13824, 450), (129, 65537, 20000)])
def test_room_for_segments_is_bounded_whatever_the_rows(N, K, M, gen):
    """The rows go in parts that share one room of 64 MiB; each row as it is by itself."""
    x, w = rand((M, K), torch.float32, gen) if N != 129 else torch.zeros(M, K, device=DEV), rand((N, K), torch.float32, gen)
    if N == 129:
        x[::37] = rand((x[::37].shape[0], K), torch.float32, gen)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    full = ops().linear(x, w)
    torch.cuda.synchronize()
    assert torch.cuda.max_memory_allocated() - before <= 4 * M * N + (64 << 20) + (1 << 21)
    for at in (0, 5, M // 2 - 3, M - 70, M - 9):
        assert torch.equal(ops().linear(x[at:at + 67].contiguous(), w), full[at:at + 67]), at
        assert torch.equal(ops().linear(x[at:at + 9].contiguous(), w), full[at:at + 9]), at
    ops().check_status(DEV)


@pytest.mark.parametrize("N,K", [(8200, 1024), (1536, 8960)])
def test_numbers_that_lose_places_are_found_in_every_tile(N, K, gen):
    """One small number each in a few rows, far apart in rows and in K: a block's later tiles, segments and places that were used before."""
    x, w = rand((200, K), torch.float32, gen), rand((N, K), torch.float32, gen)
    rows, columns, ks = [0, 63, 64, 150, 199], [1, 127, 128, 700, N - 1], [3, 64, K // 2, K - 65, K - 1]
    for m, k in zip(rows, ks):
        x[m], x[m, k] = 0.0, 1.2345678e-37
    for n, k in zip(columns, reversed(ks)):
        w[n], w[n, k] = 0.0, 7.6543211e-39
    got, by_chain, want = both(x, w)
    for m in rows:                                # sums of one product: the same rounding, or 64 bits' own
        assert float((got[m].double() - want[m]).norm()) <= 1.01 * float((by_chain[m].double() - want[m]).norm()), m
    for n in columns:
        assert float((got[:, n].double() - want[:, n]).norm()) <= 1.01 * float((by_chain[:, n].double() - want[:, n]).norm()), n
    for M in (1, 16, 65):
        assert torch.equal(ops().linear(x[:M].contiguous(), w), got[:M])
