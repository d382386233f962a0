"""The TMA-store epilogue of the bf16 GEMMs at the edges of its 32-row x 128-byte blocks, and the
plain-store path it leaves to unaligned outputs."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from hyper_parallel_b200.ops import functional as Fn
from hyper_parallel_b200.ops import native

# a bf16 result carries one rounding (2^-9 relative, each element); an fp32 one the order of at most
# K additions of exact bf16 products: K * 2^-24 relative to the sum of magnitudes, below 1e-5 in 2-norm
TOL = {torch.bfloat16: 2.0 ** -8, torch.float32: 1e-5}


@pytest.mark.parametrize("pair", ["0", "1"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (31, 40, 72), (33, 72, 64), (127, 264, 128), (129, 248, 200),
                                   (257, 520, 64), (300, 1000, 24)])
# out is a window of a larger buffer: (columns in front of it, extra columns in a row)
# ((1, 7), (6, 2): rows a multiple of 16 bytes apart whose first one is not on such a boundary)
@pytest.mark.parametrize("front,extra", [(0, 0), (8, 24), (1, 2), (8, 1), (1, 7), (6, 2)])
def test_store_window(pair, dtype, M, N, K, front, extra):
    gen = torch.Generator(device="cuda").manual_seed(M * N + K)
    a = torch.randn(M, K, device="cuda", generator=gen).to(torch.bfloat16)
    b = torch.randn(N, K, device="cuda", generator=gen).to(torch.bfloat16)
    buf = torch.full((M + 2, front + N + extra), 7.0, device="cuda", dtype=dtype)
    out = buf[1:M + 1, front:front + N]
    Fn.set_gemm_pair_mode(pair)
    try:
        Fn.gemm(a, b, out=out)
    finally:
        Fn.set_gemm_pair_mode("auto")
    native.check_status()
    ref = a.double() @ b.double().t()
    assert ((out.double() - ref).norm() / ref.norm()).item() < TOL[dtype]
    rest = buf.clone()
    rest[1:M + 1, front:front + N] = 7.0
    assert (rest == 7.0).all()                 # nothing outside the window was written


@pytest.mark.parametrize("pair", ["0", "1"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,N", [(1, 1), (33, 41), (130, 67), (257, 1003)])
@pytest.mark.parametrize("front", [0, 8])
def test_columns_that_end_inside_a_vector(pair, dtype, M, N, front):
    """TMA stores into rows of whole 16-byte vectors, clipped in the middle of one: the columns behind stay."""
    gen = torch.Generator(device="cuda").manual_seed(M + N)
    a = torch.randn(M, 72, device="cuda", generator=gen).to(torch.bfloat16)
    b = torch.randn(N, 72, device="cuda", generator=gen).to(torch.bfloat16)
    buf = torch.full((M + 2, front + (N + 7) // 8 * 8 + 8), 7.0, device="cuda", dtype=dtype)
    out = buf[1:M + 1, front:front + N]
    assert out.data_ptr() % 16 == 0 and out.stride(0) * out.element_size() % 16 == 0
    Fn.set_gemm_pair_mode(pair)
    try:
        Fn.gemm(a, b, out=out)
    finally:
        Fn.set_gemm_pair_mode("auto")
    native.check_status()
    ref = a.double() @ b.double().t()
    assert ((out.double() - ref).norm() / ref.norm()).item() < TOL[dtype]
    rest = buf.clone()
    rest[1:M + 1, front:front + N] = 7.0
    assert (rest == 7.0).all()


@pytest.mark.parametrize("pair", ["0", "1"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("front,extra", [(0, 0), (1, 7), (6, 2), (3, 0)])
def test_accumulate_window(pair, dtype, front, extra):
    M, N, K = 257, 264, 72
    gen = torch.Generator(device="cuda").manual_seed(front)
    a = torch.randn(M, K, device="cuda", generator=gen).to(torch.bfloat16)
    b = torch.randn(N, K, device="cuda", generator=gen).to(torch.bfloat16)
    buf = torch.randn(M + 2, front + N + extra, device="cuda", generator=gen).to(dtype)
    before = buf.clone()
    out = buf[1:M + 1, front:front + N]
    Fn.set_gemm_pair_mode(pair)
    try:
        Fn.gemm(a, b, out=out, accumulate=True)
    finally:
        Fn.set_gemm_pair_mode("auto")
    native.check_status()
    ref = before[1:M + 1, front:front + N].double() + a.double() @ b.double().t()
    assert ((out.double() - ref).norm() / ref.norm()).item() < TOL[dtype]
    before[1:M + 1, front:front + N] = out
    assert torch.equal(buf, before)
