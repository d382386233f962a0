"""The fp8 quantisers: the scales and bytes of the same steps on the CPU at row / column remainders
(8 or 32 rows x 256 columns per CTA for activations, 128 x 128 for weights), on unaligned and strided input."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from hyper_parallel_b200.ops import fp8


def _want(x, rows):
    """scale = max(amax, 1e-10) / 448 and x * (1 / scale) in fp32, rounded to e4m3: the kernels' steps."""
    M, K = x.shape
    pad = -M % rows
    xb = torch.nn.functional.pad(x.float(), (0, 0, 0, pad)).view((M + pad) // rows, rows, K // 128, 128)
    scale = xb.abs().amax(dim=(1, 3)).clamp_min(1e-10) / 448.0
    q = (xb * (1.0 / scale)[:, None, :, None]).clamp(-448.0, 448.0).view(M + pad, K)[:M].to(torch.float8_e4m3fn)
    return q, scale if rows > 1 else scale.t()


def _same(got, want):
    assert torch.equal(got[1].cpu(), want[1])
    assert torch.equal(got[0].cpu().view(torch.uint8), want[0].view(torch.uint8))


@pytest.mark.parametrize("M,K", [(1, 128), (31, 384), (32, 256), (33, 128), (129, 640), (200, 7168),
                                 (9, 256), (4099, 1408)])
@pytest.mark.parametrize("form", ["plain", "strided", "offset", "special"])
def test_quantisers(M, K, form):
    gen = torch.Generator(device="cuda").manual_seed(M + K)
    x = (torch.randn(M, K, device="cuda", generator=gen) * 3).to(torch.bfloat16)
    if form == "strided":
        x = torch.cat([x, x], dim=1)[:, K:]
    elif form == "offset":
        buf = torch.empty(M * K + 4, device="cuda", dtype=torch.bfloat16)
        buf[4:] = x.reshape(-1)
        x = buf[4:].view(M, K)                                  # contiguous, 8 bytes off
    elif form == "special":
        x[0] = 0
        x[-1, 5] = 3e38
        x[M // 2, :128] = 1e-30
    _same(fp8.quantize_act_1x128(x), _want(x.cpu(), 1))
    _same(fp8.quantize_weight_128x128(x), _want(x.cpu(), 128))


def test_more_column_blocks_than_a_grid_has_rows():
    """One row of 2^24 + 128 columns: 131073 blocks of columns (a grid's second dimension ends at 65535)."""
    K = (1 << 24) + 128
    x = torch.randn(1, K, device="cuda").to(torch.bfloat16)
    q, s = fp8.quantize_act_1x128(x)
    wq, ws = _want(x.cpu(), 1)
    _same((q, s), (wq, ws))
