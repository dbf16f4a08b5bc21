"""The 32-bit product in three bfloat16 parts: as close to 64 bits as the chain of multiply-adds, the same row in every batch."""
import pytest
import torch

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
    w[11, 0], x[6, 0] = 1e-30, 1e-30              # a part below the smallest normal number
    got, want = ops().linear(x, w), chain(x, w)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isposinf(got), torch.isposinf(want))
    assert torch.equal(torch.isneginf(got), torch.isneginf(want))
    finite = torch.isfinite(want)
    torch.testing.assert_close(got[finite], want[finite], atol=1e-3, rtol=1e-5)
    x[5], w[9] = 3e38, 2.0                        # a sum beyond the largest number
    assert float(ops().linear(x, w)[5, 9]) == float("inf")
