"""The tensor-memory walk over chunks (csrc/chunk_walk.cuh) where sequences are cut into segments: few long sequences, ragged
ends of segments and chunks, empty sequences, states that go on, narrow last column blocks."""
import pytest
import torch

from oracle import dafotar_oracle, fozerax_oracle, subivik_oracle

pytestmark = pytest.mark.gpu
BF, F64 = torch.bfloat16, torch.float64


def _rnd(seed, *shape, scale=1.0, mean=0.0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale + mean


def _i32(x):
    return torch.tensor(x, dtype=torch.int32, device="cuda")


def _rel(got, want):
    got, want = got.double().cpu(), want.double()
    return float((got - want).norm() / want.norm())


# heads, dim, vdim, lengths of the first and the second portion of each sequence
CASES = [(1, 128, 256, [700], [513]), (2, 64, 128, [1025, 0, 300], [1, 640, 0]), (1, 96, 136, [64 * 9], [64 * 5 + 1]),
         (3, 40, 72, [899, 257], [63, 64]), (1, 128, 128, [3001], [17])]


@pytest.mark.parametrize("kind", ["gla", "time", "mlstm"])
@pytest.mark.parametrize("H,K,V,first,second", CASES, ids=str)
def test_segments(kind, H, K, V, first, second):
    """Read-outs within the rounding of bf16 results and operands, states within that of operands in two terms, as for whole
    sequences (tests of the chunked kernels)."""
    from minivllm_b200.layers import gla, mlstm, time_mix
    n, lens = len(first), [a + b for a, b in zip(first, second)]
    q, k, v = ([_rnd(10 * s + i, lens[s], H, D).to(BF) for s in range(n)] for i, D in enumerate((K, K, V)))
    S = torch.full((n, H, K, V), float("nan"), device="cuda")
    d = lambda t: t.double()
    if kind == "gla":
        z = [_rnd(10 * s + 5, lens[s], H, K, mean=3.0).to(BF) for s in range(n)]
        ref = [fozerax_oracle.gla_scan(d(a) * K ** -0.5, d(b), d(c), fozerax_oracle.channel_decay(d(x), 4.0)) for a, b, c, x in zip(q, k, v, z)]
    elif kind == "time":
        z, w0, bonus = [_rnd(10 * s + 5, lens[s], H, K, mean=-3.0) for s in range(n)], _rnd(3, H * K).to(BF), _rnd(4, H, K).to(BF)
        ref = [subivik_oracle.bonus_scan(d(a), d(b), d(c), torch.exp(-torch.exp(d(x) + d(w0).view(H, K))), d(bonus)) for a, b, c, x in zip(q, k, v, z)]
    else:
        z, zero = [_rnd(10 * s + 5, lens[s], 2 * H, mean=0.0) for s in range(n)], torch.zeros(H)
        f_b = torch.full((H,), 3.0)
        cap = lambda x: 9.0 * torch.tanh(x / 9.0)
        ref = [dafotar_oracle.mlstm_scan(d(a) * K ** -0.5, d(b), d(c), cap(d(x[:, :H])), torch.nn.functional.logsigmoid(cap(d(x[:, H:]) + 3.0)))
               for a, b, c, x in zip(q, k, v, z)]
        nv, m = torch.full((n, H, K), float("nan"), device="cuda"), torch.full((n, H), float("nan"), device="cuda")
    slots, at = _i32(list(range(n))), [0] * n
    for part in (first, second):
        cut = lambda x: torch.cat([x[s][at[s]:at[s] + part[s]].flatten(1) for s in range(n)]).cuda()
        p = torch.cat([cut(q), cut(k), cut(v)], 1)
        a, b, c = p.split([H * K, H * K, H * V], 1)
        cu, starts = _i32([0] + torch.tensor(part).cumsum(0).tolist()), _i32(at)
        if kind == "gla":
            got = gla.gla_scan(a, b, c, cut(z), 4.0, cu, slots, starts, S, H, K, V, chunked=True).view(-1, H, V)
        elif kind == "time":
            got = time_mix.time_scan(a, b, c, cut(z), w0.cuda(), bonus.cuda(), cu, slots, starts, S, H, K, V, chunked=True).view(-1, H, V)
        else:
            chain = mlstm.mlstm_gates(cut(z), zero.to(BF).cuda(), f_b.to(BF).cuda(), 9.0, cu, slots, starts, m, H)
            o, den = mlstm.mlstm_scan(a, b, c, chain, cu, slots, starts, S, nv, H, K, V, chunked=True)
            got = o.view(-1, H, V).double() / den.double()[..., None]
        want = torch.cat([ref[s][0][at[s]:at[s] + part[s]] for s in range(n)])
        assert _rel(got, want) < 6e-3, part
        at = [x + y for x, y in zip(at, part)]
    for s in range(n):
        if kind == "mlstm":
            want = ref[s][1]
            shift = torch.exp(m[s].cpu().double() - want[2])
            assert _rel(S[s].cpu().double() * shift[:, None, None], want[0]) < 1e-4 and _rel(nv[s].cpu().double() * shift[:, None], want[1]) < 1e-4
        else:
            assert _rel(S[s], ref[s][1]) < 2e-4, s


# Both sides of the lines between whole sequences and segments, and between the walk and the register form: one and two chunks of
# narrow heads, heads that are not made of slabs, few and many sequences.
@pytest.mark.parametrize("kind", ["gla", "time", "mlstm"])
@pytest.mark.parametrize("H,K,V,first,second", [(1, 64, 128, [64 * 12], [64 * 12 + 1]), (1, 128, 128, [64 * 8], [64 * 8 + 1]),
                                                (2, 64, 128, [2100, 1, 700], [900, 0, 40]), (4, 64, 72, [64] * 3, [65] * 3),
                                                (33, 64, 128, [17] * 16, [96] * 16), (5, 128, 256, [33] * 16, [32] * 16),
                                                (8, 48, 96, [500] * 7, [100] * 7)], ids=str)
def test_forms_and_lengths(kind, H, K, V, first, second):
    test_segments(kind, H, K, V, first, second)


def test_decays_are_no_further_off_than_32_bits_need():
    """The logarithms of 63 decays, summed, from a state that decays from one token on: their mean error over heads and channels, to a
    sum of about 40.  A logarithm's relative error is 4e-8 rms with a mean of 3e-9, the factor log2(e) of all has -1.4e-8, 5e-7
    here; an exponential from ex2.approx and a division in the logarithm had -5.8e-8, 2.3e-6 here."""
    from minivllm_b200.layers import gla
    H, K, V, n, tau = 16, 128, 128, 8, 0.125          # exact, as is its reciprocal
    T = 64 * n
    g = torch.Generator().manual_seed(2)
    z = (torch.randn(T, H * K, generator=g) + 3).to(BF)
    q, k, v = torch.zeros(T, H * K, dtype=BF), torch.zeros(T, H * K, dtype=BF), torch.zeros(T, H * V, dtype=BF)
    k[::64], v[::64] = 1.0, 1.0
    a, b, c = torch.cat([q, k, v], 1).cuda().split([H * K, H * K, H * V], 1)
    S = torch.zeros(n, H, K, V, device="cuda")
    gla.gla_scan(a, b, c, z.cuda(), tau, _i32([64 * i for i in range(n + 1)]), _i32(list(range(n))), _i32([0] * n), S, H, K, V, chunked=True)
    want = torch.nn.functional.logsigmoid(z.double()).view(n, 64, H, K)[:, 1:].sum(1) / tau
    assert -60 < float(want.mean()) < -30
    err = torch.log(S[..., 0].double().cpu()) - want
    assert abs(float(err.mean())) < 1e-6 and float(err.square().mean().sqrt()) < 1e-5


@pytest.mark.parametrize("kind", ["gla", "mlstm"])
@pytest.mark.parametrize("lens", [[300, 200], [1024]], ids=["whole", "segments"])
def test_a_wait_that_runs_out_ends_the_walk(kind, lens):
    """One arrival is withheld for one call: the wait for it ends after 200 ms, the error word says so, the recurrence it befell
    keeps the state it had (in segments, where every state depends on the first pass, all of them do), and the next call is
    clean."""
    import ctypes
    from minivllm_b200 import _cabi
    from minivllm_b200.layers import attention, gla, mlstm
    H, K, V, n, T = 2, 128, 128, len(lens), sum(lens)
    word = attention._error_word(torch.device("cuda", torch.cuda.current_device()))
    q, k, v = (_rnd(i, T, H * D).to(BF).cuda() for i, D in enumerate((K, K, V)))
    p = torch.cat([q, k, v], 1)
    q, k, v = p.split([H * K, H * K, H * V], 1)
    cu, slots, starts = _i32([0] + torch.tensor(lens).cumsum(0).tolist()), _i32(list(range(n))), _i32([0] * n)
    gates = _rnd(9, T, 2 * H).cuda() if kind == "mlstm" else _rnd(9, T, H * K, mean=3.0).to(BF).cuda()

    def run():
        S, nv, m = (torch.full((n, H) + x, 7.0, device="cuda") for x in ((K, V), (K,), ()))
        if kind == "gla":
            return S, nv, gla.gla_scan(q, k, v, gates, 4.0, cu, slots, starts, S, H, K, V, chunked=True)
        zero = torch.zeros(H, dtype=BF, device="cuda")
        chain = mlstm.mlstm_gates(gates, zero, zero + 3, 9.0, cu, slots, starts, m, H)
        return S, nv, *mlstm.mlstm_scan(q, k, v, chain, cu, slots, starts, S, nv, H, K, V, chunked=True)

    want = run()
    assert int(word.item()) == 0
    assert _cabi.lib().mv_debug_walk_inject(ctypes.c_int(1)) == 0
    S, nv, *_ = run()
    code = int(word.item())
    word.zero_()
    assert code >> 8 == 1, f"error word {code:#x}"
    hit = torch.zeros(n, H, dtype=torch.bool)
    hit[0, 0] = True
    if len(lens) == 1:
        hit[:] = True
    for s in range(n):
        for h in range(H):
            for got, ref in ((S, want[0]), (nv, want[1])):
                assert torch.equal(got[s, h], torch.full_like(got[s, h], 7.0) if hit[s, h] else ref[s, h]), (s, h)
    for got, ref in zip(run(), want):
        assert torch.equal(got, ref)
    assert int(word.item()) == 0
