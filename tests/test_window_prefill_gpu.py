"""window_prefill at heads of 128 in groups (persistent CTAs) against plain attention in 64 bits: windows around the edges of
tiles, portions behind cached keys, tables longer and shorter than the window, groups of odd size, sequences that end inside
the eight rows that leave together, more and fewer sequences than are sorted."""
import pytest
import torch

from minivllm_b200.layers import window_attention as WA

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _want(q, k, v, window, scale, bias, sink):
    n, H, _ = q.shape
    m, G, _ = k.shape
    k, v = (t.double().repeat_interleave(H // G, 1).permute(1, 0, 2) for t in (k, v))
    s = q.double().permute(1, 0, 2) @ k.transpose(1, 2) * scale
    d = (torch.arange(n, device=DEV) + m - n)[:, None] - torch.arange(m, device=DEV)[None, :]
    if bias is not None:
        s += bias.double()[:, d.clamp(0, bias.shape[1] - 1)]
    s = s.masked_fill((d < 0) | (d >= window), float("-inf"))
    if sink is not None:
        s = torch.cat([s, sink.double()[:, None, None].expand(H, n, 1)], 2)
    return (s.softmax(2)[:, :, :m] @ v).permute(1, 0, 2).reshape(n, -1)


@pytest.mark.parametrize("heads,kv,spans,window,distances,sink", [
    (16, 4, [(0, 700), (0, 1), (0, 129), (0, 128)], 300, 129, True),
    (16, 4, [(500, 140), (130, 7), (0, 9), (1, 300)], 128, 129, True),        # distances cut by the window
    (6, 2, [(255, 130), (0, 250), (640, 1)], 129, 40, True),                  # a group of three heads
    (4, 2, [(0, 300), (90, 33)], 1, 129, False),                              # a row sees itself alone
    (8, 2, [(0, 900)], 1 << 30, 512, True),                                   # the longest table
    (8, 4, [(300, 500)], 513, 0, False),                                      # no bias
    (16, 4, [(0, n) for n in (15, 16, 17, 200, 0, 31, 8, 257, 1, 100, 64)], 100, 129, True),
    (32, 4, [(0, 600), (200, 520), (0, 77)], 1000, 200, True),                # more units than SMs
])
def test_window_prefill_of_grouped_heads(heads, kv, spans, window, distances, sink):
    g = torch.Generator(device=DEV).manual_seed(3)
    rnd = lambda *s, dtype=torch.bfloat16: torch.randn(*s, generator=g, device=DEV).to(dtype)
    nq, nk = sum(n for _, n in spans), sum(b + n for b, n in spans)
    q, rows = rnd(nq, heads * 128), rnd(nk, kv * 256)
    bias = rnd(heads, distances, dtype=torch.float32) if distances else None
    sk = rnd(heads) if sink else None
    cu_q, cu_k = (torch.tensor([0] + c).cumsum(0).to(torch.int32).to(DEV) for c in ([n for _, n in spans], [b + n for b, n in spans]))
    got = WA.window_prefill(q, rows, cu_q, cu_k, kv, 128, 128, window, 128 ** -0.5, bias, sk)
    torch.cuda.synchronize()
    assert int(WA._error_word(q.device).item()) == 0
    at, kt = 0, 0
    for b, n in spans:
        if n == 0:
            continue
        k, v = rows[kt:kt + b + n].split(kv * 128, 1)
        want = _want(q[at:at + n].view(n, heads, 128), k.reshape(-1, kv, 128), v.reshape(-1, kv, 128), window, 128 ** -0.5, bias, sk)
        # P in bf16 (2^-9 relative a weight, which average out) and the result's rounding
        err = (got[at:at + n].double() - want).abs()
        assert float((err - 2.0 ** -8 * want.abs()).max()) < 1e-2 and float(err.norm() / want.norm()) < 4e-3
        at, kt = at + n, kt + b + n
