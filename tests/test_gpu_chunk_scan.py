"""Long runs of a retention, state space or gated delta layer in chunks of 64 tokens on tcgen05 against the recurrence in 64 bits over the same prepared rows: runs at
the edges of a chunk and of the rule that takes them (32 tokens), a batch below the rule, short runs in the same batch, continued runs, sequences with states of their own in a
shuffled order, states of fewer than 128 rows, decays of exactly zero, and 32-bit storage, which keeps the token-by-token scan."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _tables(lens, pos0, dev):
    i = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    start = [sum(lens[:e]) for e in range(len(lens))]
    slots = list(range(len(lens)))[::-1]
    return (i([e for e, n in enumerate(lens) for _ in range(n)]), i([p + k for n, p in zip(lens, pos0) for k in range(n)]), i(start), i(lens), i(slots), i(pos0)), start, slots


def _check(o, state, q, g, v, b, a, skip, S0, lens, pos0, start, slots):
    """q, g [T][H][D], v [T][H][Dv], b, a [T][H] as prepared; o [T][H][Dv], state and S0 [slots][H][D][Dv]."""
    for e, n in enumerate(lens):
        S = S0[slots[e]].double() if pos0[e] else torch.zeros_like(S0[0], dtype=torch.float64)
        M = S.abs()  # the same recurrence over absolute values: what the roundings of the sums are relative to
        O, OM = [], []
        for t in range(start[e], start[e] + n):
            qt, gt, vt, at = q[t].double(), g[t].double(), v[t].double(), a[t].double()[:, None, None]
            u = b[t].double()[:, None] * vt
            S = at * S + gt[..., None] * u[:, None]
            M = at * M + gt.abs()[..., None] * u.abs()[:, None]
            O.append(torch.einsum("hdv,hd->hv", S, qt) + skip[:, None] * vt)
            OM.append(torch.einsum("hdv,hd->hv", M, qt.abs()) + (skip[:, None] * vt).abs())
        O, OM, got = torch.stack(O), torch.stack(OM), o[start[e]:start[e] + n].double()
        # a product over K numbers adds its six parts in K / 16 steps, each of which drops less than 2^-23 of the running sum: 48 steps for the state's 128
        # rows, 24 for a chunk's 64 tokens and as many for its addition to the state, which itself is rounded once a chunk; parts left out weigh 2^-24
        eps = 2.0 ** -23 * (48 + 24 + 24 + 2 * (n // 64 + 1) + 8)
        assert ((got - O).abs() <= eps * OM + 1e-30).all(), (lens, e, ((got - O).abs() / OM).max().item())
        assert ((state[slots[e]].double() - S).abs() <= eps * M + 1e-30).all(), (lens, e)
        # and as independent errors: 16 units of fp32 (a lost middle part would be 2^-17)
        for x, ref in ((got, O), (state[slots[e]].double(), S)):
            assert (x - ref).norm() <= 2.0 ** -20 * ref.norm(), (lens, e, ((x - ref).norm() / ref.norm()).item())


RUNS = [([31, 32, 33, 800], [0, 0, 9, 0]), ([63, 449], [0, 7]), ([64, 65, 640], [7, 0, 0]), ([128, 1, 129, 766], [0, 12, 3, 0]), ([300], [0]), ([255], [5]), ([128], [3])]


@pytest.mark.parametrize("lens,pos0", RUNS)
@pytest.mark.parametrize("H,G,N,P,dtype", [(4, 2, 128, 64, BF), (6, 1, 104, 64, BF), (2, 2, 72, 128, BF), (3, 1, 128, 64, BF), (4, 2, 100, 64, BF), (4, 2, 128, 64, torch.float32)])
def test_state_space(lens, pos0, H, G, N, P, dtype):
    from qserve_b200._lib import check, lib

    dev, taps = "cuda", 4
    gen = torch.Generator(device=dev).manual_seed(sum(lens) + N)
    r = lambda *s: torch.randn(*s, device=dev, generator=gen)
    T, E, inner = sum(lens), len(lens), H * P
    C = inner + 2 * G * N
    W = (inner + C + H + 7) // 8 * 8
    proj, cw, cb, cs = r(T, W).to(dtype), r(C, taps) * 0.5, r(C) * 0.1, r(E, taps - 1, C)
    a_log, dt_bias, skip, nw = r(H) * 0.5, r(H) * 0.5 - 2, 1 + 0.1 * r(H), torch.ones(inner, device=dev)
    a_log[0] = 60.0  # this head's decays are exp(-dt e^60) = 0
    if H > 1:
        a_log[1] = -30.0  # and this one's 1
    S0 = r(E, H, N, P) * 0.3
    state = S0.clone()
    tab, start, slots = _tables(lens, pos0, dev)
    R = int(lib.qs_hyb_state_space_prep_floats(H, G, N, P))
    prep, o, out = torch.full((T, R), float("nan"), device=dev), torch.full((T, inner), float("nan"), device=dev), torch.zeros(T, inner, dtype=dtype, device=dev)
    p = lambda t: t.data_ptr()
    check(lib.qs_hyb_state_space(p(out), inner, p(prep), p(o), p(proj), W, p(cw), p(cb), p(cs), p(state), p(a_log), p(dt_bias), p(skip), p(nw), G, 1.0,
                                 *map(p, tab), T, E, H, G, N, P, taps, 1e-5, 0 if dtype is BF else 1, torch.cuda.current_stream().cuda_stream))
    x, GN = prep[:, :inner].view(T, H, P), G * N
    B, Q = (prep[:, inner + k * GN:inner + (k + 1) * GN].view(T, G, N).repeat_interleave(H // G, 1) for k in (0, 1))
    at = inner + 2 * GN
    _check(o.view(T, H, P), state, Q, B, x, prep[:, at:at + H], prep[:, at + H:at + 2 * H], skip.double(), S0, lens, pos0, start, slots)
    assert torch.isfinite(out).all()


@pytest.mark.parametrize("lens,pos0", RUNS)
@pytest.mark.parametrize("H,D,Dv,dtype", [(3, 128, 128, BF), (2, 72, 128, BF), (2, 128, 64, BF), (2, 128, 128, torch.float32)])
def test_retention(lens, pos0, H, D, Dv, dtype):
    from qserve_b200._lib import check, lib

    dev = "cuda"
    gen = torch.Generator(device=dev).manual_seed(sum(lens) + D)
    r = lambda *s: torch.randn(*s, device=dev, generator=gen)
    T, E, W = sum(lens), len(lens), 2 * H * D + H * Dv
    proj, S0 = r(T, W).to(dtype), r(E, H, D, Dv) * 0.3
    decay = torch.tensor([1.0, 0.0, 0.9][:H], device=dev)
    state, (tab, start, slots) = S0.clone(), _tables(lens, pos0, dev)
    prep, o, out = torch.full((T, W), float("nan"), device=dev), torch.full((T, H * Dv), float("nan"), device=dev), torch.zeros(T, H * Dv, dtype=dtype, device=dev)
    p = lambda t: t.data_ptr()
    check(lib.qs_hyb_retention(p(out), H * Dv, p(prep), p(o), p(proj), W, p(decay), None, 0, D ** -0.5, 0, p(state), *map(p, tab[1:]), T, E, H, D, Dv, 1e-5,
                               0 if dtype is BF else 1, torch.cuda.current_stream().cuda_stream))
    q, k, v = prep[:, :H * D].view(T, H, D), prep[:, H * D:2 * H * D].view(T, H, D), prep[:, 2 * H * D:].view(T, H, Dv)
    one = torch.ones(T, H, device=dev)
    _check(o.view(T, H, Dv), state, q, k, v, one, decay * one, torch.zeros(H, dtype=torch.float64, device=dev), S0, lens, pos0, start, slots)
    assert torch.isfinite(out).all()


@pytest.mark.parametrize("lens,pos0", RUNS)
@pytest.mark.parametrize("H,G,D,Dv,dtype", [(8, 2, 128, 128, BF), (4, 4, 72, 128, BF), (12, 2, 128, 128, BF), (4, 1, 104, 128, BF), (2, 1, 128, 128, BF), (4, 2, 128, 64, BF), (4, 2, 128, 128, torch.float32)])
def test_gated_delta(lens, pos0, H, G, D, Dv, dtype):
    from qserve_b200._lib import check, lib

    dev, taps = "cuda", 4
    gen = torch.Generator(device=dev).manual_seed(sum(lens) + D + H)
    r = lambda *s: torch.randn(*s, device=dev, generator=gen)
    T, E, C = sum(lens), len(lens), 2 * G * D + H * Dv
    W = (C + H * Dv + 2 * H + 7) // 8 * 8
    proj, cw, cs = r(T, W).to(dtype), r(C, taps) * 0.5, r(E, taps - 1, C)
    a_log, dt_bias, nw = r(H) * 0.5, r(H) * 0.5, torch.ones(Dv, device=dev)
    a_log[0], a_log[1] = 60.0, -30.0  # decays of 0 and of 1
    S0 = r(E, H, D, Dv) * 0.3
    state = S0.clone()
    tab, start, slots = _tables(lens, pos0, dev)
    prep, o, out = torch.full((T, C + 2 * H), float("nan"), device=dev), torch.full((T, H * Dv), float("nan"), device=dev), torch.zeros(T, H * Dv, dtype=dtype, device=dev)
    p = lambda t: t.data_ptr()
    check(lib.qs_hyb_gated_delta(p(out), H * Dv, p(prep), p(o), p(proj), W, p(cw), p(cs), p(state), p(a_log), p(dt_bias), p(nw), *map(p, tab), T, E, H, G, D, Dv,
                                 taps, 1e-6, 1e-5, 0 if dtype is BF else 1, torch.cuda.current_stream().cuda_stream))
    q, k = (prep[:, i * G * D:(i + 1) * G * D].view(T, G, D).repeat_interleave(H // G, 1).double() for i in (0, 1))
    v, b, a = prep[:, 2 * G * D:C].view(T, H, Dv).double(), prep[:, C:C + H].double(), prep[:, C + H:C + 2 * H].double()
    for e, n in enumerate(lens):
        S = S0[slots[e]].double() if pos0[e] else torch.zeros_like(S0[0], dtype=torch.float64)
        O = []
        for t in range(start[e], start[e] + n):
            S = a[t][:, None, None] * S
            u = b[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
            S = S + k[t][..., None] * u[:, None]
            O.append(torch.einsum("hdv,hd->hv", S, q[t]))
        # keys are unit vectors and write strengths below one, so a step does not enlarge an error: what a chunk's sums add (a few units of fp32 of the
        # state's size, as for the other recurrences) meets at most sqrt(chunks) of its kind
        eps = 2.0 ** -20 * max(1.0, (n / 64) ** 0.5)
        O, got = torch.stack(O), o.view(T, H, Dv)[start[e]:start[e] + n].double()
        scale = max(O.norm() / O.numel() ** 0.5, S.norm() / S.numel() ** 0.5)
        assert (got - O).norm() <= eps * scale * O.numel() ** 0.5, (e, ((got - O).norm() / O.norm()).item())
        assert (state[slots[e]].double() - S).norm() <= eps * S.norm(), (e, ((state[slots[e]].double() - S).norm() / S.norm()).item())
        for h in range(H):  # each head by itself: the largest error of a number against the head's own size
            assert (got[:, h] - O[:, h]).abs().max() <= 16 * eps * max(O[:, h].abs().max(), S[h].abs().max()), (e, h)
    assert torch.isfinite(out).all()
