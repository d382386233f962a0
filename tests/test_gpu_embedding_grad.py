"""Weight gradient of the embedding at the edges of its scan (1024 counts per block), its row groups
(1 or 2 rows), its column slices (256 vectors) and its bucket lengths."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from hyper_parallel_b200 import ops
from hyper_parallel_b200.ops import native


@pytest.mark.parametrize("V", [1, 7, 20, 1023, 1024, 1025, 5003, 16385])
@pytest.mark.parametrize("H,T", [(8, 1), (2048, 333), (2056, 2100), (4096, 17)])
def test_weight_gradient(V, H, T):
    gen = torch.Generator().manual_seed(V + H)
    tok = torch.randint(0, V, (T,), generator=gen)
    tok[: T // 3] = V - 1                                      # one long bucket (up to 700 tokens)
    tok[T // 3: T // 3 + 9] = V // 2                           # one just over the unrolled eight
    dy = torch.randn(T, H, generator=gen).to(torch.bfloat16)
    w = torch.zeros(V, H, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    ops.embedding(tok.cuda(), w).backward(dy.cuda())
    native.check_status()
    # fp32 additions in token order: up to 1024 tokens of a row the very same bits
    want = torch.zeros(V, H)
    for t in range(T):
        want[tok[t]] += dy[t].float()
    got = w.grad.cpu()
    rows = torch.bincount(tok, minlength=V) <= 1024
    assert torch.equal(got[rows], want.to(torch.bfloat16)[rows])
    # longer buckets: any order, one rounding to bf16 on top of T * 2^-24
    assert ((got.float() - want).norm() / want.norm()).item() < 2.0 ** -8


def test_more_column_slices_than_a_grid_has_rows():
    H = 8 * 256 * 65535 + 8
    w = torch.zeros(1, H, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    dy = torch.randn(1, H, device="cuda").to(torch.bfloat16)
    ops.embedding(torch.zeros(1, dtype=torch.int64, device="cuda"), w).backward(dy)
    native.check_status()
    assert torch.equal(w.grad, dy)
