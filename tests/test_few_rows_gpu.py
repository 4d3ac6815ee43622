"""Products of up to 16 rows against 64 bits: every split of features and reduction among CTAs and warps, and where the library
takes over.  Tolerance: one rounding of the result beside fp32 sums (gated: of both products before the activation)."""
import pytest
import torch
import torch.nn.functional as F

from minivllm_b200.layers import linear as L


@pytest.mark.parametrize("n,k,gated,pay", [(4096, 12288, False, True), (4096, 12352, False, False), (2048, 18944, False, True),
                                           (2048, 19008, False, False), (4736, 1024, False, True), (4744, 512, False, False),
                                           (6144, 1024, False, True), (6144, 704, False, False), (6152, 1024, False, False),
                                           (32768, 256, False, False), (12288, 512, True, True), (12304, 256, True, False),
                                           (6144, 1024, True, True), (12288, 768, True, False)])
def test_where_the_kernel_is_the_faster_one(n, k, gated, pay):
    assert L._few_rows_pay(n, k, gated) is pay


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n,k", [(16, 64), (48, 128), (1184, 576), (1200, 2048), (2368, 64), (2384, 192), (4096, 1024), (1024, 3072)])
def test_few_rows(n, k, dtype):
    g = torch.Generator(device="cuda").manual_seed(n)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    w = (rnd(n, k) * k ** -0.5).to(dtype)
    u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for rows in (1, 7, 8, 9, 16):
        x = rnd(rows, k + 8).to(dtype)[:, :k]                 # rows of a wider product
        assert L._few_rows(x, w, False) is not None
        want = x.double() @ w.double().t()
        err = (L.linear(x, w).double() - want).abs()
        assert float((err - u * want.abs()).max()) < 1e-5
        want = F.silu(want[:, :n // 2]) * want[:, n // 2:]
        got = L.swiglu_linear(x, w).double()
        assert float((got - want).norm() / want.norm()) < 2 * u
        assert float(((got - want).abs() - 4 * u * want.abs()).max()) < 2 * u


@pytest.mark.gpu
def test_what_the_library_takes():
    w = torch.randn(64, 128, device="cuda").bfloat16()
    x = torch.randn(17, 128, device="cuda").bfloat16()
    big = torch.empty(8192, 2048, device="cuda", dtype=torch.bfloat16)
    for a, b in ((x, w), (x[:4].float(), w.float()), (x[:4, :96], w[:, :96]), (x[:4], w[:60]), (x[:4], w.t().contiguous().t()),
                 (torch.empty(2, 2048, device="cuda", dtype=torch.bfloat16), big), (x[:4].clone().requires_grad_(), w)):
        assert L._few_rows(a, b, False) is None
        assert L.linear(a, b).shape == (a.shape[0], b.shape[0])
    assert L.linear(x[:0], w).shape == (0, 64)
