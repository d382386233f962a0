"""The 128x256 fp8 GEMM against the 128x128 one (same products, same order of additions: same bits) and
the dequantised product, at remainders of its tile and with fewer, as many and more tiles than SMs."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from hyper_parallel_b200.ops import fp8, native


def _run(name, aq, sa, bq, sb):
    (M, K), N = aq.shape, bq.shape[0]
    out = torch.full((M + 2, N), 7.0, device="cuda", dtype=torch.bfloat16)
    c = out[1:M + 1]
    fn = getattr(fp8._lib(), name)
    native.check(fn(aq.data_ptr(), sa.data_ptr(), bq.data_ptr(), sb.data_ptr(), c.data_ptr(), N, M, N, K,
                    native.status_word("cuda").data_ptr(), native.sm_count("cuda"), native.stream()), name)
    native.check_status()
    assert (out[0] == 7.0).all() and (out[M + 1] == 7.0).all()
    return c


@pytest.mark.parametrize("M,N,K", [(1, 8, 128), (31, 136, 256), (128, 256, 128), (129, 264, 384), (300, 1000, 1280),
                                   (97, 40, 2048), (2048, 4096, 512), (2500, 2056, 896)])
def test_wide_tile(M, N, K):
    gen = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randn(M, K, device="cuda", generator=gen)
    x *= 4.0 ** torch.randint(-3, 4, (M, K // 128, 1), device="cuda", generator=gen).expand(M, K // 128, 128).reshape(M, K)
    w = torch.randn(N, K, device="cuda", generator=gen) * 0.05
    w *= 4.0 ** torch.randint(-3, 4, (1, K // 128, 1), device="cuda", generator=gen).expand(N, K // 128, 128).reshape(N, K)
    aq, sa = fp8.quantize_act_1x128(x.to(torch.bfloat16))
    bq, sb = fp8.quantize_weight_128x128(w.to(torch.bfloat16))
    wide, small = _run("hpb_gemm_fp8_blockscale_wide", aq, sa, bq, sb), _run("hpb_gemm_fp8_blockscale", aq, sa, bq, sb)
    assert torch.equal(wide, small) and torch.equal(fp8.gemm_fp8(aq, sa, bq, sb), small)
    want = fp8.dequantize(aq, scale_act=sa).double() @ fp8.dequantize(bq, scale_w=sb).double().t()
    # one rounding of the result to bf16 (2^-9 per element) on top of the tensor core's sums of 128
    assert ((wide.double() - want).norm() / want.norm()).item() < 2.0 ** -8
