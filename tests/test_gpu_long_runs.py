"""Recurrences over long runs (retention, state space, gated delta rule) against the same recurrence in 64 bits over the same prepared rows: unequal
runs, short runs in the same batch, continued runs, sequences with states of their own in a shuffled order, states of fewer than 128 rows, decays of
exactly zero and one, 16- and 32-bit storage.  The recurrence is fp32 arithmetic token by token whatever the storage: a result does not depend on where a
prompt was cut or on what else is in the step, and a value that is not finite reaches no token ahead of it."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF, F32 = torch.bfloat16, torch.float32
DEV = "cuda"


def _tables(lens, pos0, slots):
    i = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    start = [sum(lens[:e]) for e in range(len(lens))]
    return (i([e for e, n in enumerate(lens) for _ in range(n)]), i([p + k for n, p in zip(lens, pos0) for k in range(n)]), i(start), i(lens), i(slots),
            i(pos0)), start


class _Layer:
    """One recurrence: `proj` rows -> `step` over runs, which updates `state` (and the convolution's state) and returns (prep, o, out)."""

    def rand(self, *s):
        return torch.randn(*s, device=DEV, generator=self.gen)

    def __init__(self, seed, dtype, slots):
        self.gen, self.dtype, self.dt, self.slots = torch.Generator(device=DEV).manual_seed(seed), dtype, 0 if dtype is BF else 1, slots

    def buffers(self, T, prep_width, out_width):
        nan = float("nan")
        return (torch.full((T, prep_width), nan, device=DEV), torch.full((T, out_width), nan, device=DEV),
                torch.zeros(T, out_width, dtype=self.dtype, device=DEV))

    def stream(self):
        return torch.cuda.current_stream().cuda_stream


class StateSpace(_Layer):
    def __init__(self, seed, dtype, slots, H, G, D, Dv):
        super().__init__(seed, dtype, slots)
        self.H, self.G, self.D, self.Dv, self.taps = H, G, D, Dv, 4
        r, inner = self.rand, H * Dv
        C = self.C = inner + 2 * G * D
        self.W, self.value_at = (inner + C + H + 7) // 8 * 8, inner
        self.conv_w, self.conv_b, self.conv = r(C, 4) * 0.5, r(C) * 0.1, r(slots, 3, C)
        self.a_log, self.dt_bias, self.skip, self.norm_w = r(H) * 0.5, r(H) * 0.5 - 2, 1 + 0.1 * r(H), torch.ones(inner, device=DEV)
        self.a_log[0] = 60.0   # this head's decays are exp(-dt e^60) = 0
        if H > 1:
            self.a_log[1] = -30.0  # and this one's 1
        self.state = r(slots, H, D, Dv) * 0.3

    def step(self, proj, lens, pos0, slots):
        from qserve_b200._lib import check, lib

        tab, _ = _tables(lens, pos0, slots)
        T, inner, p = sum(lens), self.H * self.Dv, lambda t: t.data_ptr()
        prep, o, out = self.buffers(T, int(lib.qs_hyb_state_space_prep_floats(self.H, self.G, self.D, self.Dv)), inner)
        check(lib.qs_hyb_state_space(p(out), inner, p(prep), p(o), p(proj), proj.stride(0), p(self.conv_w), p(self.conv_b), p(self.conv), p(self.state), p(self.a_log),
                                     p(self.dt_bias), p(self.skip), p(self.norm_w), self.G, 1.0, *map(p, tab), T, len(lens), self.H, self.G, self.D, self.Dv,
                                     self.taps, 1e-5, self.dt, self.stream()))
        return prep, o, out

    def split(self, prep):  # q, g, v, b, a per head
        T, H, G, D, Dv = prep.shape[0], self.H, self.G, self.D, self.Dv
        inner, GD = H * Dv, G * D
        g, q = (prep[:, inner + k * GD:inner + (k + 1) * GD].view(T, G, D).repeat_interleave(H // G, 1) for k in (0, 1))
        at = inner + 2 * GD
        return q, g, prep[:, :inner].view(T, H, Dv), prep[:, at:at + H], prep[:, at + H:at + 2 * H]


class Retention(_Layer):
    def __init__(self, seed, dtype, slots, H, G, D, Dv):
        super().__init__(seed, dtype, slots)
        self.H, self.G, self.D, self.Dv = H, G, D, Dv
        self.W, self.value_at = 2 * H * D + H * Dv, 2 * H * D
        self.decay = torch.tensor([0.0, 1.0, 0.9][:H], device=DEV)
        self.skip, self.conv = torch.zeros(H, device=DEV), torch.zeros(1, device=DEV)
        self.state = self.rand(slots, H, D, Dv) * 0.3

    def step(self, proj, lens, pos0, slots):
        from qserve_b200._lib import check, lib

        tab, _ = _tables(lens, pos0, slots)
        T, p = sum(lens), lambda t: t.data_ptr()
        prep, o, out = self.buffers(T, self.W, self.H * self.Dv)
        check(lib.qs_hyb_retention(p(out), self.H * self.Dv, p(prep), p(o), p(proj), proj.stride(0), p(self.decay), None, 0, self.D ** -0.5, 0, p(self.state),
                                   *map(p, tab[1:]), T, len(lens), self.H, self.D, self.Dv, 1e-5, self.dt, self.stream()))
        return prep, o, out

    def split(self, prep):
        T, H, D = prep.shape[0], self.H, self.D
        q, g, v = prep[:, :H * D].view(T, H, D), prep[:, H * D:2 * H * D].view(T, H, D), prep[:, 2 * H * D:].view(T, H, self.Dv)
        one = torch.ones(T, H, device=DEV)
        return q, g, v, one, self.decay * one


class GatedDelta(_Layer):
    def __init__(self, seed, dtype, slots, H, G, D, Dv):
        super().__init__(seed, dtype, slots)
        self.H, self.G, self.D, self.Dv, self.taps = H, G, D, Dv, 4
        r = self.rand
        C = self.C = 2 * G * D + H * Dv
        self.W, self.value_at = (C + H * Dv + 2 * H + 7) // 8 * 8, 2 * G * D
        self.conv_w, self.conv = r(C, 4) * 0.5, r(slots, 3, C)
        self.a_log, self.dt_bias, self.norm_w = r(H) * 0.5, r(H) * 0.5, torch.ones(Dv, device=DEV)
        self.a_log[0], self.a_log[1] = 60.0, -30.0  # decays of 0 and of 1
        self.state = r(slots, H, D, Dv) * 0.3

    def step(self, proj, lens, pos0, slots):
        from qserve_b200._lib import check, lib

        tab, _ = _tables(lens, pos0, slots)
        T, p = sum(lens), lambda t: t.data_ptr()
        prep, o, out = self.buffers(T, self.C + 2 * self.H, self.H * self.Dv)
        check(lib.qs_hyb_gated_delta(p(out), self.H * self.Dv, p(prep), p(o), p(proj), proj.stride(0), p(self.conv_w), p(self.conv), p(self.state), p(self.a_log),
                                     p(self.dt_bias), p(self.norm_w), *map(p, tab), T, len(lens), self.H, self.G, self.D, self.Dv, self.taps, 1e-6, 1e-5,
                                     self.dt, self.stream()))
        return prep, o, out

    def split(self, prep):
        T, H, G, D, Dv = prep.shape[0], self.H, self.G, self.D, self.Dv
        q, g = (prep[:, i * G * D:(i + 1) * G * D].view(T, G, D).repeat_interleave(H // G, 1) for i in (0, 1))
        return q, g, prep[:, 2 * G * D:self.C].view(T, H, Dv), prep[:, self.C:self.C + H], prep[:, self.C + H:self.C + 2 * H]


def _recurrence(layer, prep, S):
    """The recurrence over one run's prepared rows in 64 bits: o [n, H, Dv] and the last state."""
    q, g, v, b, a = (x.double() for x in layer.split(prep))
    delta, O = isinstance(layer, GatedDelta), []
    skip = layer.skip.double()[:, None] if isinstance(layer, StateSpace) else 0.0
    for t in range(prep.shape[0]):
        S = a[t][:, None, None] * S
        u = v[t] - torch.einsum("hdv,hd->hv", S, g[t]) if delta else v[t]
        S = S + g[t][..., None] * (b[t][:, None] * u)[:, None]
        O.append(torch.einsum("hdv,hd->hv", S, q[t]) + skip * v[t])
    return torch.stack(O), S


RUNS = [([31, 32, 33, 800], [0, 0, 9, 0]), ([63, 449], [0, 7]), ([64, 65, 640], [7, 0, 0]), ([128, 1, 129, 766], [0, 12, 3, 0]), ([300], [0]), ([255], [5]), ([2048], [3])]
LAYERS = [(StateSpace, 4, 2, 128, 64), (StateSpace, 4, 1, 104, 64), (StateSpace, 4, 2, 72, 128), (StateSpace, 3, 1, 128, 64), (StateSpace, 4, 2, 100, 64),
          (Retention, 3, 3, 128, 128), (Retention, 2, 2, 72, 128), (Retention, 2, 2, 128, 64),
          (GatedDelta, 8, 2, 128, 128), (GatedDelta, 4, 4, 72, 128), (GatedDelta, 4, 1, 104, 128), (GatedDelta, 4, 2, 128, 64)]


@pytest.mark.parametrize("lens,pos0", RUNS)
@pytest.mark.parametrize("dtype", [BF, F32])
@pytest.mark.parametrize("kind,H,G,D,Dv", LAYERS)
def test_against_64_bits(kind, H, G, D, Dv, dtype, lens, pos0):
    slots = list(range(len(lens)))[::-1]
    layer = kind(sum(lens) + D + H, dtype, len(lens), H, G, D, Dv)
    proj, S0 = layer.rand(sum(lens), layer.W).to(dtype), layer.state.clone()
    prep, o, out = layer.step(proj, lens, pos0, slots)
    assert torch.isfinite(out).all()
    start = 0
    for e, n in enumerate(lens):
        S = S0[slots[e]].double() if pos0[e] else torch.zeros_like(S0[0], dtype=torch.float64)
        rows = slice(start, start + n)
        start += n
        O, S = _recurrence(layer, prep[rows], S)
        got, state = o[rows].view(n, H, Dv).double(), layer.state[slots[e]].double()
        if n < 16:  # a read-out of few tokens may cancel: nothing to measure its error by
            continue
        for h in range(H):
            err_o, err_s = ((got[:, h] - O[:, h]).norm() / O[:, h].norm()).item(), ((state[h] - S[h]).norm() / S[h].norm()).item()
            # a step rounds the decayed state and what it adds once each: independent errors of up to half a unit of fp32 (2^-24), which add up as sqrt(2 n) / 2
            # units where nothing is forgotten (head 1).  Elsewhere a few steps count: three units for a state (measured 0.3e-7 to 1.4e-7), and two for a
            # read-out, whose 128 products are added in parts and a tree (0.5e-7 to 1.0e-7; with operands in three bfloat16 terms on the tensor cores
            # 1.5e-7 to 1.8e-7)
            kept = 8 + (2 * n) ** 0.5 / 2
            assert err_o <= 2.0 ** -24 * (kept if h == 1 else 2) and err_s <= 2.0 ** -24 * (kept if h == 1 else 3), (h, n, err_o, err_s)



LONG = [(StateSpace, 4, 2, 128, 64), (Retention, 3, 3, 128, 128), (GatedDelta, 8, 2, 128, 128)]


@pytest.mark.parametrize("dtype", [BF, F32])
@pytest.mark.parametrize("kind,H,G,D,Dv", LONG)
def test_cuts_and_neighbours(kind, H, G, D, Dv, dtype):
    """A run of 800 tokens whole, in portions, and beside a single token and a run of 500: the same bits.  (Retention and state space have scans of their own
    for steps of fewer than 32 tokens a sequence, which add in another order; the delta rule has not.)"""
    def fresh():
        return kind(5, dtype, 3, H, G, D, Dv)

    layer = fresh()
    proj = layer.rand(1301, layer.W).to(dtype)
    mine = proj[501:]
    _, o, out = layer.step(mine, [800], [0], [1])
    cut, at = fresh(), 0
    for n in (300, 63, 1, 436) if kind is GatedDelta else (300, 63, 437):
        _, o2, out2 = cut.step(mine[at:at + n], [n], [at], [1])
        assert torch.equal(o2, o[at:at + n]) and torch.equal(out2, out[at:at + n])
        at += n
    beside = fresh()
    _, o2, out2 = beside.step(proj, [1, 500, 800], [4, 7, 0], [2, 0, 1])
    assert torch.equal(o2[501:], o) and torch.equal(out2[501:], out)
    for other in (cut, beside):
        assert torch.equal(other.state[1], layer.state[1])


@pytest.mark.parametrize("kind,H,G,D,Dv", LONG)
def test_a_value_that_is_not_finite(kind, H, G, D, Dv):
    """Infinity in one value of one token: nothing ahead of it changes, nor any other column of the state."""
    clean, hit, n, t, h, c = kind(6, BF, 1, H, G, D, Dv), kind(6, BF, 1, H, G, D, Dv), 400, 200, 2, 5
    proj = clean.rand(n, clean.W).to(BF)
    bad = proj.clone()
    bad[t, clean.value_at + h * Dv + c] = float("inf")
    o, o_bad = (layer.step(x, [n], [0], [0])[1].view(n, H, Dv) for layer, x in ((clean, proj), (hit, bad)))
    assert torch.isfinite(o).all() and not torch.isfinite(o_bad[t, h, c])
    assert torch.equal(o_bad[:t], o[:t])
    keep = torch.ones(H, Dv, dtype=torch.bool, device=DEV)
    keep[h, c] = False
    assert torch.equal(o_bad[:, keep], o[:, keep])
    assert torch.equal(hit.state[0].movedim(1, 2)[keep], clean.state[0].movedim(1, 2)[keep])
