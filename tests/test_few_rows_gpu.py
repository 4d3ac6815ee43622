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


class _Seen(torch.utils._python_dispatch.TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.ops = getattr(self, "ops", []) + [str(func)]
        return func(*args, **(kwargs or {}))


def test_who_must_see_a_product_gets_the_library_s():
    """Modes, transforms, forward mode, tracing and subclasses; the same calls on the CPU."""
    from torch.autograd import forward_ad
    x, w = torch.randn(3, 64), torch.randn(16, 64)
    assert L._eager(x, w) and L._eager(x, torch.nn.Parameter(w))
    with _Seen() as seen:
        assert not L._eager(x, w)
        L.linear(x, w)
    assert seen.ops
    with forward_ad.dual_level():
        y = L.linear(forward_ad.make_dual(x, torch.ones_like(x)), w)
        assert not L._eager(x, w) and torch.equal(forward_ad.unpack_dual(y).tangent, F.linear(torch.ones_like(x), w))
    asked = []
    assert torch.allclose(torch.func.vmap(lambda r: (asked.append(L._eager(r, w)), L.linear(r[None], w)[0])[1])(x), F.linear(x, w), atol=1e-5)
    assert asked == [False]
    assert not L._eager(x.as_subclass(type("Sub", (torch.Tensor,), {})), w)
    torch.jit.trace(lambda a: (asked.append(L._eager(a, w)), L.linear(a, w))[1], x, check_trace=False)
    assert asked == [False, False]
    assert L._eager(x, w)


@pytest.mark.gpu
def test_autocast_and_forward_mode_on_gpu():
    from torch.autograd import forward_ad
    x, w = torch.randn(4, 128, device="cuda").bfloat16(), torch.randn(64, 128, device="cuda").bfloat16()
    assert L._few_rows(x, w, False) is not None
    with torch.autocast("cuda", torch.float16):
        assert L.linear(x, w).dtype == F.linear(x, w).dtype == torch.float16
    with forward_ad.dual_level():
        y = L.linear(forward_ad.make_dual(x, x), w)
        assert torch.equal(forward_ad.unpack_dual(y).tangent, F.linear(x, w))
    assert torch.equal(torch.func.vmap(L.linear, (0, None))(x.view(2, 2, 128), w), torch.func.vmap(F.linear, (0, None))(x.view(2, 2, 128), w))
