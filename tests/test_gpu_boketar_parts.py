"""Each mechanism of the Boketar parts alone against its plain function (GPU): the kernels are
called as the parts call them, on inputs made so that a fault shows."""
import math

import pytest
import torch

from plain import boketar_plain as P

from poor_mans_mamba_b200.kernels import ops as K

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DTYPES = [torch.float32, torch.bfloat16]


def rnd(*shape, seed=0, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).to(torch.bfloat16).float()


def close(got, want, dtype, what, f32=2e-5, bf16=2e-2):
    got, want = got.double().cpu(), want.double()
    tol = (f32 if dtype == torch.float32 else bf16) * max(1.0, float(want.abs().max()))
    err = float((got - want).abs().max())
    assert err <= tol, f"{what}: {err:.3e} > {tol:.3e}"


def batch_index(lens, slots):
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    seq_of = torch.cat([torch.full((n,), i, dtype=torch.int32) for i, n in enumerate(lens)]).to(DEV)
    return cu, seq_of, torch.tensor(slots, dtype=torch.int32, device=DEV)


# ----------------------------------------------------------------------------- residual lanes
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n,D", [(1, 48), (2, 256), (3, 100), (8, 64), (2, 77), (5, 50)])
def test_lanes_mix_and_norm(dtype, n, D):
    T = 7
    x = rnd(n, T, D, seed=1)
    y = rnd(T, D, seed=2)
    mix, ow, iw, nw = rnd(n, n, seed=3), rnd(n, seed=4), rnd(n, seed=5), rnd(D, seed=6) + 1.0
    new = torch.einsum("st,sij->tij", mix.double(), x.double()) + ow.double().view(n, 1, 1) * y.double()
    want = P.norm_plain(torch.einsum("s,sij->ij", iw.double(), new), nw.double(), 1e-5)
    lanes = x.to(DEV).clone()
    out = torch.empty(T, D, dtype=dtype, device=DEV)
    K.hc_mix_norm(lanes, lanes, y.to(DEV, dtype), mix.reshape(-1).to(DEV), ow.to(DEV), iw.to(DEV), nw.to(DEV), 1e-5, out)
    close(lanes, new, torch.float32, "lanes")
    close(out, want, dtype, "normed")
    # all lanes start from one stream; listed rows only, lanes untouched
    h = rnd(T, D, seed=7).to(DEV)
    rows = torch.tensor([5, 0, 5], dtype=torch.int32, device=DEV)
    out2 = torch.empty(3, D, dtype=dtype, device=DEV)
    K.hc_mix_norm(h.unsqueeze(0).expand(n, T, D), None, y.to(DEV, dtype), mix.reshape(-1).to(DEV), ow.to(DEV),
                  torch.ones(n, device=DEV), nw.to(DEV), 1e-5, out2, rows)
    new2 = mix.double().sum(0).view(n, 1, 1) * h.cpu().double() + ow.double().view(n, 1, 1) * y.double()
    close(out2, P.norm_plain(new2.sum(0), nw.double(), 1e-5)[[5, 0, 5]], dtype, "rows")


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("D", [4, 1020, 1024, 2052])
def test_lanes_rows_on_and_off_their_boundaries(dtype, D):
    """Four values at a time where a row of the sublayer's result starts on a 16-byte boundary, one where it does not."""
    n, T = 2, 9
    x, y = rnd(n, T, D, seed=1), rnd(T, D, seed=2).to(dtype)
    mix, ow, iw, nw = rnd(n, n, seed=3), rnd(n, seed=4), rnd(n, seed=5), rnd(D, seed=6) + 1.0
    new = torch.einsum("st,sij->tij", mix.double(), x.double()) + ow.double().view(n, 1, 1) * y.double()
    want = P.norm_plain(torch.einsum("s,sij->ij", iw.double(), new), nw.double(), 1e-5)
    for shift in (0, 1):
        flat = torch.zeros(T * D + 1, dtype=dtype, device=DEV)
        flat[shift:shift + T * D] = y.reshape(-1).to(DEV)
        lanes, out = x.to(DEV).clone(), torch.empty(T, D, dtype=dtype, device=DEV)
        K.hc_mix_norm(lanes, lanes, flat[shift:shift + T * D].view(T, D), mix.reshape(-1).to(DEV), ow.to(DEV), iw.to(DEV), nw.to(DEV), 1e-5, out)
        close(lanes, new, torch.float32, "lanes")
        close(out, want, dtype, "normed")


@pytest.mark.parametrize("dtype", DTYPES)
def test_normed_sum_of_branches(dtype):
    T, D = 5, 72
    a, b, wa, wb = rnd(T, D, seed=1, scale=3.0), rnd(T, D, seed=2, scale=0.1), rnd(D, seed=3), rnd(D, seed=4)
    wide = torch.zeros(T, 2 * D + 8, dtype=dtype, device=DEV)  # branches as column slices
    wide[:, :D], wide[:, D + 8:] = a.to(DEV, dtype), b.to(DEV, dtype)
    out = torch.empty(T, D, dtype=dtype, device=DEV)
    K.normed_sum([(wide[:, :D], wa.to(DEV)), (wide[:, D + 8:], wb.to(DEV))], 1e-6, 0.5, out)
    want = 0.5 * (P.norm_plain(a.double(), wa.double(), 1e-6) + P.norm_plain(b.double(), wb.double(), 1e-6))
    close(out, want, dtype, "normed sum")
    bias = rnd(D, seed=5)  # a branch's bias joins it before its norm
    K.normed_sum([(wide[:, :D], wa.to(DEV)), (wide[:, D + 8:], wb.to(DEV))], 1e-6, 0.5, out, biases=[None, bias.to(DEV)])
    want = 0.5 * (P.norm_plain(a.double(), wa.double(), 1e-6) + P.norm_plain(b.double() + bias.double(), wb.double(), 1e-6))
    close(out, want, dtype, "normed sum with a bias")


# ----------------------------------------------------------------------------- matrix-state recurrences
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("H,G,d,dv", [(4, 2, 24, 16), (2, 2, 64, 40), (3, 1, 128, 96), (1, 1, 8, 8), (2, 1, 200, 33)])
def test_gated_delta_rule_in_portions(dtype, H, G, d, dv):
    """Three sequences of unequal length, in two steps that cut them at odd places, in slots that
    are not in order; the state of a slot that is used again starts from zero."""
    lens = [37, 1, 22]
    T = sum(lens)
    q, k, v = rnd(T, G * d, seed=1), rnd(T, G * d, seed=2), rnd(T, H * dv, seed=3)
    beta, a = rnd(T, H, seed=4), rnd(T, H * d, seed=5)
    dt_bias, a_log = rnd(H * d, seed=6) - 1.0, rnd(H, seed=7) * 0.5
    g = torch.exp(-torch.exp(a_log.double())[None, :, None] * P.softplus(a.double() + dt_bias.double()).view(T, H, d))
    qd, kd = q.double().view(T, G, d), k.double().view(T, G, d)
    qn = (qd / torch.sqrt((qd * qd).sum(-1, keepdim=True) + 1e-6) * d ** -0.5).repeat_interleave(H // G, dim=1)
    kn = (kd / torch.sqrt((kd * kd).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, dim=1)
    want, t0 = [], 0
    for n in lens:
        s = slice(t0, t0 + n)
        want.append(P.gated_delta_rule(qn[s], kn[s], v.double().view(T, H, dv)[s], torch.sigmoid(beta.double())[s], g[s]))
        t0 += n
    want = torch.cat(want).reshape(T, H * dv)
    state = torch.full((5, H, d, dv), 7.0, device=DEV)  # stale values of earlier owners
    slots = [3, 0, 4]
    for s in slots:
        state[s].zero_()
    out = torch.empty(T, H * dv, device=DEV)
    dev = lambda t: t.to(DEV, dtype)
    first = [20, 1, 2]  # tokens of each sequence in the first step (the second sequence ends there)
    starts = [0, 37, 38]
    for part in (0, 1):
        rows, ls, sl = [], [], []
        for i, n in enumerate(lens):
            lo, hi = (0, first[i]) if part == 0 else (first[i], n)
            if hi > lo:
                rows += list(range(starts[i] + lo, starts[i] + hi))
                ls.append(hi - lo)
                sl.append(slots[i])
        idx = torch.tensor(rows)
        cu, _, sl_t = batch_index(ls, sl)
        o = torch.empty(len(rows), H * dv, device=DEV)
        K.delta_scan(dev(q[idx]), dev(k[idx]), dev(v[idx]), dev(beta[idx]), dev(a[idx]), dt_bias.to(DEV), a_log.to(DEV),
                     state, cu, sl_t, len(ls), o, H, G, d, dv, 1e-6, d ** -0.5)
        out[idx.to(DEV)] = o
    close(out, want, torch.float32, "delta rule", f32=1e-4)  # inputs are exact in both types; the state is float
    assert float(state[1].min()) == 7.0 and float(state[2].max()) == 7.0  # other slots untouched


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("H,d,dv", [(2, 16, 24), (4, 32, 32), (1, 100, 7), (3, 4, 130)])
def test_decayed_linear_attention_far_back(dtype, H, d, dv):
    """600 tokens in portions of changing size with a decay of one on the first head: the first
    token weighs as much as the last."""
    T = 600
    q, k, v = rnd(T, H * d, seed=1), rnd(T, H * d, seed=2), rnd(T, H * dv, seed=3)
    decay = [1.0] + [0.97] * (H - 1)
    want = P.decayed_linear_attention(P.silu(q.double()).view(T, H, d), P.silu(k.double()).view(T, H, d),
                                      P.silu(v.double()).view(T, H, dv), decay).reshape(T, H * dv)
    state = torch.zeros(2, H, d, dv, device=DEV)
    out = torch.empty(T, H * dv, device=DEV)
    t0 = 0
    for n in [1, 2, 16, 17, 64, 100, 1, 1, 398]:
        cu, _, sl = batch_index([n], [1])
        K.decay_scan(q[t0:t0 + n].to(DEV, dtype), k[t0:t0 + n].to(DEV, dtype), v[t0:t0 + n].to(DEV, dtype),
                     torch.tensor(decay, device=DEV), state, cu, sl, 1, out[t0:t0 + n], H, d, dv)
        t0 += n
    close(out, want, torch.float32, "decayed linear attention", f32=1e-4)
    assert float(state[0].abs().max()) == 0.0


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("H,G,d,dv", [(4, 2, 24, 16), (2, 2, 64, 40), (3, 1, 128, 96), (1, 1, 8, 8), (2, 1, 192, 33)])
def test_gated_delta_rule_in_chunks(dtype, H, G, d, dv):
    """Sequences of 1, 63, 64, 65 and 200 tokens (chunk edges), the longest cut into two steps at an odd
    place, strong and weak decays side by side: the chunked kernels against the plain recurrence and
    against the token-serial kernel, state included."""
    lens = [200, 1, 63, 64, 65]
    T = sum(lens)
    q, k, v = rnd(T, G * d, seed=1), rnd(T, G * d, seed=2), rnd(T, H * dv, seed=3)
    beta, a = rnd(T, H, seed=4), rnd(T, H * d, seed=5, scale=3.0)
    dt_bias, a_log = rnd(H * d, seed=6) - 1.0, rnd(H, seed=7) * 0.5 + 1.0   # decays from 1 down to e^-12 a token
    g = torch.exp(-torch.exp(a_log.double())[None, :, None] * P.softplus(a.double() + dt_bias.double()).view(T, H, d))
    assert float(g.min()) < 1e-3 and float(g.max()) > 0.99
    qd, kd = q.double().view(T, G, d), k.double().view(T, G, d)
    qn = (qd / torch.sqrt((qd * qd).sum(-1, keepdim=True) + 1e-6) * d ** -0.5).repeat_interleave(H // G, dim=1)
    kn = (kd / torch.sqrt((kd * kd).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, dim=1)
    want, t0 = [], 0
    for n in lens:
        sl = slice(t0, t0 + n)
        want.append(P.gated_delta_rule(qn[sl], kn[sl], v.double().view(T, H, dv)[sl], torch.sigmoid(beta.double())[sl], g[sl]))
        t0 += n
    want = torch.cat(want).reshape(T, H * dv)
    dev = lambda t: t.to(DEV, dtype)
    slots = [4, 0, 2, 1, 3]
    results = {}
    for kind in ("chunked", "serial"):
        state = torch.zeros(6, H, d, dv, device=DEV)
        out = torch.empty(T, H * dv, device=DEV)
        first = [77, 1, 63, 64, 65]
        starts = [0, 200, 201, 264, 328]
        for part in (0, 1):
            rows, ls, sl = [], [], []
            for i, n in enumerate(lens):
                lo, hi = (0, first[i]) if part == 0 else (first[i], n)
                if hi > lo:
                    rows += list(range(starts[i] + lo, starts[i] + hi))
                    ls.append(hi - lo)
                    sl.append(slots[i])
            idx = torch.tensor(rows)
            cu, _, sl_t = batch_index(ls, sl)
            o = torch.empty(len(rows), H * dv, device=DEV)
            if kind == "chunked":
                scratch = torch.empty(K.recurrent_chunked_scratch_floats(ls, H, d, dv, True), device=DEV)
                K.recurrent_chunked(dev(q[idx]), dev(k[idx]), dev(v[idx]), state, cu, sl_t, ls, o, scratch, H, G, d, dv,
                                    beta=dev(beta[idx]), a=dev(a[idx]), dt_bias=dt_bias.to(DEV), a_log=a_log.to(DEV),
                                    unit_eps=1e-6, q_scale=d ** -0.5)
            else:
                K.delta_scan(dev(q[idx]), dev(k[idx]), dev(v[idx]), dev(beta[idx]), dev(a[idx]), dt_bias.to(DEV),
                             a_log.to(DEV), state, cu, sl_t, len(ls), o, H, G, d, dv, 1e-6, d ** -0.5)
            out[idx.to(DEV)] = o
        close(out, want, torch.float32, f"delta rule, {kind}", f32=1e-4)
        results[kind] = state
    close(results["chunked"], results["serial"].cpu(), torch.float32, "states", f32=1e-4)
    assert float(results["chunked"][5].abs().max()) == 0.0


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("d,dv,shift", [(64, 64, 0), (64, 61, 1), (128, 8, 0), (128, 130, 3), (244, 17, 2), (4, 4, 0)])
def test_gated_delta_rule_in_chunks_of_views(dtype, d, dv, shift):
    """Every form of the chunked delta rule (key sizes known when compiling and others, one and two buffers in the chain,
    rows on and off boundaries of four elements, value columns that are no whole tile, more values than keys) on both sides
    of a chunk's edge against the token-serial kernel.  Tolerance: float sums of up to 130 tokens and 244 channels in another
    order, relative to the largest entry."""
    H, G = 2, 1
    for n in (1, 2, 7, 8, 9, 64, 129):
        width = 2 * G * d + H * dv + H * d + H
        rows = (rnd(n, width + 8, seed=n) * torch.linspace(0.5, 2.0, n)[:, None]).to(DEV, dtype)[:, shift:shift + width]
        q, k, v, a, beta = rows.split([G * d, G * d, H * dv, H * d, H], dim=1)
        dt_bias, a_log = (rnd(H * d, seed=6) * 4.0 - 1.0).to(DEV), (rnd(H, seed=7) + 1.0).to(DEV)
        got = {}
        for kind in ("chunked", "serial"):
            state = (rnd(2, H, d, dv, seed=8) * 0.1).to(DEV)
            out = torch.empty(n, H * dv, device=DEV)
            cu, _, sl = batch_index([n], [1])
            if kind == "chunked":
                scratch = torch.full((K.recurrent_chunked_scratch_floats([n], H, d, dv, True),), float("nan"), device=DEV)
                K.recurrent_chunked(q, k, v, state, cu, sl, [n], out, scratch, H, G, d, dv, beta=beta, a=a, dt_bias=dt_bias,
                                    a_log=a_log, unit_eps=1e-6, q_scale=d ** -0.5)
            else:
                K.delta_scan(q, k, v, beta, a, dt_bias, a_log, state, cu, sl, 1, out, H, G, d, dv, 1e-6, d ** -0.5)
            got[kind] = (out, state)
        for x, y in zip(got["chunked"], got["serial"]):
            assert float((x - y).abs().max()) <= 2e-5 * max(1.0, float(y.abs().max())), (n, float((x - y).abs().max()))


@pytest.mark.parametrize("d", [64, 128, 244])
def test_gated_delta_rule_solve_rounds_a_row_once(d):
    """Nearly orthogonal keys without decay, a chunk of 64 tokens: the rows solved before take almost nothing off a row, so what
    is left of the error is how often the solve rounds a whole row.  Once (the sum of the small terms is taken off at the end),
    with the roundings of key, product and state beside it, is below 2.2 half units in the last place (1.3e-7); a subtraction a
    term measured 1.7e-7."""
    H, n, dv = 2, 64, 64
    k = torch.eye(n, d).repeat(1, H) + 0.001 * rnd(n, H * d, seed=d)
    v = rnd(n, H * dv, seed=d + 1)
    state, out = torch.zeros(2, H, d, dv, device=DEV), torch.empty(n, H * dv, device=DEV)
    cu, _, sl = batch_index([n], [1])
    scratch = torch.empty(K.recurrent_chunked_scratch_floats([n], H, d, dv, True), device=DEV)
    K.recurrent_chunked(k.to(DEV), k.to(DEV), v.to(DEV), state, cu, sl, [n], out, scratch, H, H, d, dv,
                        beta=torch.full((n, H), 30.0, device=DEV), a=torch.zeros(n, H * d, device=DEV),
                        dt_bias=torch.full((H * d,), -30.0, device=DEV), a_log=torch.zeros(H, device=DEV))
    kk = k.double().view(n, H, d)
    kk = kk / kk.norm(dim=-1, keepdim=True)
    vv = v.double().view(n, H, dv)
    s64 = torch.zeros(H, d, dv, dtype=torch.float64)
    for t in range(n):
        u = vv[t] - (s64 * kk[t].unsqueeze(-1)).sum(1)
        s64 = s64 + kk[t].unsqueeze(-1) * u.unsqueeze(1)
    assert float((state[1].cpu().double() - s64).norm() / s64.norm()) < 2.2 * 2.0 ** -24


@pytest.mark.parametrize("d", [224, 244])
def test_gated_delta_rule_read_out_of_long_keys(d):
    """A given state read out by keys of 224 entries and more, no decay, no writes (beta zero, values zero): a sum of d random
    terms.  One after the other they measured 2.8e-7, in fours 1.7e-7; the bound lies between, at 3.7 half units in the last place."""
    H, n, dv = 4, 64, 64
    q, s0 = rnd(n, H * d, seed=d), torch.randn(2, H, d, dv, generator=torch.Generator().manual_seed(d + 1))
    state, out = s0.to(DEV), torch.empty(n, H * dv, device=DEV)
    cu, _, sl = batch_index([n], [1])
    scratch = torch.empty(K.recurrent_chunked_scratch_floats([n], H, d, dv, True), device=DEV)
    K.recurrent_chunked(q.to(DEV), q.to(DEV), torch.zeros(n, H * dv, device=DEV), state, cu, sl, [n], out, scratch, H, H, d, dv,
                        beta=torch.full((n, H), -200.0, device=DEV), a=torch.zeros(n, H * d, device=DEV),
                        dt_bias=torch.full((H * d,), -30.0, device=DEV), a_log=torch.zeros(H, device=DEV))
    qq = q.double().view(n, H, d)
    want = torch.einsum("nhd,hdv->nhv", qq / qq.norm(dim=-1, keepdim=True), s0[1].double()).reshape(n, H * dv)
    assert float((out.cpu().double() - want).norm() / want.norm()) < 3.7 * 2.0 ** -24


def _delta_operands(lens, H, d, dv, dtype=torch.float32):
    T = sum(lens)
    q, k, v, a, beta = (rnd(T, n, seed=i).to(DEV, dtype) for i, n in enumerate((H * d, H * d, H * dv, H * d, H)))
    state = (rnd(len(lens) + 1, H, d, dv, seed=8) * 0.1).to(DEV)
    cu, _, sl = batch_index(lens, list(range(1, len(lens) + 1)))
    return q, k, v, a, beta, (rnd(H * d, seed=6) - 1.0).to(DEV), rnd(H, seed=7).to(DEV), state, cu, sl


@pytest.mark.parametrize("d,dv", [(64, 64), (128, 40), (244, 8)])
def test_gated_delta_rule_chunks_that_are_not_full(d, dv):
    """Portions on both sides of every sixteen rows, alone and behind a full chunk, in one batch: the rows behind a portion's last
    sixteen are neither made nor read (the scratch is not a number).  Tolerance: float sums of up to 80 tokens and 244 channels
    in another order, relative to the largest entry."""
    H, lens = 2, [1, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65, 80]
    q, k, v, a, beta, dt_bias, a_log, state, cu, sl = _delta_operands(lens, H, d, dv)
    serial, out, want = state.clone(), torch.empty(sum(lens), H * dv, device=DEV), torch.empty(sum(lens), H * dv, device=DEV)
    scratch = torch.full((K.recurrent_chunked_scratch_floats(lens, H, d, dv, True),), float("nan"), device=DEV)
    K.recurrent_chunked(q, k, v, state, cu, sl, lens, out, scratch, H, H, d, dv, beta=beta, a=a, dt_bias=dt_bias, a_log=a_log,
                        unit_eps=1e-6, q_scale=d ** -0.5)
    K.delta_scan(q, k, v, beta, a, dt_bias, a_log, serial, cu, sl, len(lens), want, H, H, d, dv, 1e-6, d ** -0.5)
    for x, y in ((out, want), (state, serial)):
        assert float((x - y).abs().max()) <= 2e-5 * max(1.0, float(y.abs().max()))


def test_gated_delta_rule_of_lone_tokens_is_not_a_whole_chunk_each():
    """Requests with one token beside a prompt portion go through the chunked form with it: what they cost is their rows', not 64
    rows' (the ratio of a step of lone tokens to one of whole chunks, medians on the device: 0.82 where every chunk's 64 rows are
    made, 0.51 where 16 are)."""
    H, d, dv = 4, 244, 64
    took = {}
    for n in (1, 64):
        lens = [n] * 128
        q, k, v, a, beta, dt_bias, a_log, state, cu, sl = _delta_operands(lens, H, d, dv)
        out = torch.empty(sum(lens), H * dv, device=DEV)
        scratch = torch.empty(K.recurrent_chunked_scratch_floats(lens, H, d, dv, True), device=DEV)
        times = []
        for _ in range(9):
            t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            t0.record()
            K.recurrent_chunked(q, k, v, state, cu, sl, lens, out, scratch, H, H, d, dv, beta=beta, a=a, dt_bias=dt_bias,
                                a_log=a_log, unit_eps=1e-6, q_scale=d ** -0.5)
            t1.record()
            torch.cuda.synchronize()
            times.append(t0.elapsed_time(t1))
        took[n] = sorted(times)[4]
    assert took[1] < 0.65 * took[64], took


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("H,d,dv", [(2, 16, 24), (4, 32, 32), (1, 100, 7), (3, 4, 130)])
def test_decayed_linear_attention_in_chunks(dtype, H, d, dv):
    T = 600
    q, k, v = rnd(T, H * d, seed=1), rnd(T, H * d, seed=2), rnd(T, H * dv, seed=3)
    decay = [1.0] + [0.97, 0.5, 0.0][:H - 1]
    want = P.decayed_linear_attention(P.silu(q.double()).view(T, H, d), P.silu(k.double()).view(T, H, d),
                                      P.silu(v.double()).view(T, H, dv), decay).reshape(T, H * dv)
    state = torch.zeros(2, H, d, dv, device=DEV)
    out = torch.empty(T, H * dv, device=DEV)
    t0 = 0
    for n in [1, 65, 64, 270, 200]:
        cu, _, sl = batch_index([n], [1])
        scratch = torch.empty(K.recurrent_chunked_scratch_floats([n], H, d, dv, False), device=DEV)
        K.recurrent_chunked(q[t0:t0 + n].to(DEV, dtype), k[t0:t0 + n].to(DEV, dtype), v[t0:t0 + n].to(DEV, dtype), state,
                            cu, sl, [n], out[t0:t0 + n], scratch, H, H, d, dv, decay=torch.tensor(decay, device=DEV))
        t0 += n
    close(out, want, torch.float32, "decayed linear attention in chunks", f32=1e-4)
    assert float(state[0].abs().max()) == 0.0


@pytest.mark.parametrize("d,dv", [(8, 8), (64, 72), (64, 76), (72, 64), (128, 128), (136, 128), (128, 200)])
def test_chunk_states_in_the_prepare_launch_and_beside_it(d, dv):
    """The state's part made by the prepare kernel (sizes in whole eights whose operands leave room for two blocks an SM) and by
    its own launch, column tiles of 64 and what is left of them, inner slices of 32 and what is left, portions that end anywhere
    in a chunk; values that are infinite after a portion's last token of the chunk reach nothing."""
    H, T = 2, 230
    q, k, v = rnd(T, H * d, seed=1), rnd(T, H * d, seed=2), rnd(T, H * dv, seed=3)
    decay = [0.97, 0.5]
    want = P.decayed_linear_attention(P.silu(q.double()).view(T, H, d), P.silu(k.double()).view(T, H, d),
                                      P.silu(v.double()).view(T, H, dv), decay).reshape(T, H * dv)
    state = torch.zeros(2, H, d, dv, device=DEV)
    out = torch.full((T, H * dv), float("nan"), device=DEV)
    t0 = 0
    for n in [1, 64, 129, 36]:
        cu, _, sl = batch_index([n], [1])
        scratch = torch.full((K.recurrent_chunked_scratch_floats([n], H, d, dv, False),), float("inf"), device=DEV)
        K.recurrent_chunked(q[t0:t0 + n].to(DEV), k[t0:t0 + n].to(DEV), v[t0:t0 + n].to(DEV), state, cu, sl, [n],
                            out[t0:t0 + n], scratch, H, H, d, dv, decay=torch.tensor(decay, device=DEV))
        t0 += n
    close(out, want, torch.float32, "rows", f32=1e-4)
    s64 = torch.zeros(H, d, dv, dtype=torch.float64)
    for t in range(T):
        kk, vv = P.silu(k[t].double()).view(H, d), P.silu(v[t].double()).view(H, dv)
        s64 = torch.tensor(decay, dtype=torch.float64).view(H, 1, 1) * s64 + kk.unsqueeze(2) * vv.unsqueeze(1)
    close(state[1], s64, torch.float32, "state", f32=1e-4)


def test_decayed_sum_of_more_column_tiles_than_a_grid_is_deep():
    """65,536 tiles of 64 value columns and one column more: three tokens against the formula, rows and state."""
    H, n, d, dv = 1, 3, 4, 65536 * 64 + 1
    q, k = rnd(n, d, seed=1), rnd(n, d, seed=2)
    v = torch.randn(n, dv, generator=torch.Generator(device=DEV).manual_seed(3), device=DEV)
    state, out = torch.zeros(1, H, d, dv, device=DEV), torch.full((n, dv), float("nan"), device=DEV)
    cu, _, sl = batch_index([n], [0])
    scratch = torch.empty(K.recurrent_chunked_scratch_floats([n], H, d, dv, False), device=DEV)
    K.recurrent_chunked(q.to(DEV), k.to(DEV), v, state, cu, sl, [n], out, scratch, H, H, d, dv, decay=torch.tensor([0.5], device=DEV))
    s64 = torch.zeros(d, dv, dtype=torch.float64, device=DEV)
    for t in range(n):
        s64 = 0.5 * s64 + P.silu(k[t].double()).to(DEV).unsqueeze(1) * P.silu(v[t].double()).unsqueeze(0)
        want = (P.silu(q[t].double()).to(DEV).unsqueeze(1) * s64).sum(0)
        assert float((out[t].double() - want).abs().max()) <= 1e-5 * float(want.abs().max())
    assert float((state[0, 0].double() - s64).abs().max()) <= 1e-5 * float(s64.abs().max())


@pytest.mark.parametrize("H,lens,d,dv", [(2, [1], 64, 128), (8, [640], 64, 64), (8, [576], 64, 136), (8, [640], 64, 136), (74, [130, 64, 63, 1], 32, 64),
                                         (75, [130, 64, 63, 1], 32, 64), (16, [1793], 32, 40), (2, [64 * 112], 40, 128)])
def test_chunk_read_out_and_state_on_both_sides_of_their_grids(H, lens, d, dv):
    """The read-out with four and eight rows a thread (up to 444 blocks and beyond) and the state's part in the prepare launch (from 80
    chunks, or small states) and in its own, beside the token-serial kernel.  Tolerance: float sums of up to 7,168 decayed tokens in
    another order, relative to the largest entry."""
    T = sum(lens)
    q, k, v = (rnd(T, H * w, seed=i).to(DEV) for i, w in enumerate((d, d, dv)))
    decay = torch.linspace(0.6, 0.99, H).to(DEV)
    cu, _, sl = batch_index(lens, list(range(len(lens))))
    got = {}
    for kind in ("chunked", "serial"):
        state, out = torch.zeros(len(lens), H, d, dv, device=DEV), torch.full((T, H * dv), float("nan"), device=DEV)
        if kind == "chunked":
            scratch = torch.full((K.recurrent_chunked_scratch_floats(lens, H, d, dv, False),), float("nan"), device=DEV)
            K.recurrent_chunked(q, k, v, state, cu, sl, lens, out, scratch, H, H, d, dv, decay=decay)
        else:
            K.decay_scan(q, k, v, decay, state, cu, sl, len(lens), out, H, d, dv)
        got[kind] = (out, state)
    for x, y in zip(got["chunked"], got["serial"]):
        assert float((x - y).abs().max()) <= 2e-5 * max(1.0, float(y.abs().max()))


def test_chunked_sums_of_two_threads_with_different_values(monkeypatch):
    """Two host threads launch the decayed sum with 64 and 128 value columns, whose prepare blocks differ in shared memory, as fast as
    they can: neither may lower what the other's launch was allowed between that thread's asking and its launch."""
    import threading
    H, n, d = 2, 3, 64
    calls, kept = {}, []
    for dv in (64, 128):
        q, k, v = (rnd(n, H * w, seed=w).to(DEV) for w in (d, d, dv))
        state, out = torch.zeros(1, H, d, dv, device=DEV), torch.empty(n, H * dv, device=DEV)
        cu, _, sl = batch_index([n], [0])
        scratch = torch.empty(K.recurrent_chunked_scratch_floats([n], H, d, dv, False), device=DEV)
        decay = torch.tensor([0.9, 0.5], device=DEV)
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream), monkeypatch.context() as m:
            m.setattr(K, "_call", lambda name, *args: calls.__setitem__(dv, args))
            K.recurrent_chunked(q, k, v, state, cu, sl, [n], out, scratch, H, H, d, dv, decay=decay)
        kept.append((q, k, v, state, out, cu, sl, scratch, decay, stream))
    launch = K._fn("pmm_recurrent_chunked")
    torch.cuda.synchronize()
    codes, ready = {}, threading.Barrier(2)

    def serve(dv):
        ready.wait(30)
        codes[dv] = {launch(*calls[dv]) for _ in range(10000)}

    threads = [threading.Thread(target=serve, args=(dv,)) for dv in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert codes == {64: {0}, 128: {0}}, codes


# ----------------------------------------------------------------------------- window attention pieces
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("H,G,d,dv,rot", [(4, 2, 16, 32, 8), (2, 2, 48, 48, 48), (3, 1, 64, 16, 0), (8, 4, 64, 48, 64)])
def test_pair_rotation_and_padded_pages(dtype, H, G, d, dv, rot):
    T, page = 9, 4
    Dp = (max(d, dv) + 15) // 16 * 16
    q, k, v = rnd(T, H * d, seed=1), rnd(T, G * d, seed=2), rnd(T, G * dv, seed=3)
    positions = torch.tensor([0, 1, 2, 3, 4, 5, 1000, 1001, 70000], dtype=torch.int32)
    pool = torch.full((8, 2, page, G * Dp), 9.0, dtype=dtype, device=DEV)
    table = torch.zeros(1, 20000, dtype=torch.int32, device=DEV)
    table[0, :2] = torch.tensor([5, 2]); table[0, 250] = 7; table[0, 17500] = 1
    inv = None
    if rot:
        inv = torch.pow(torch.tensor(777.0, dtype=torch.float64), -2.0 * torch.arange(rot // 2, dtype=torch.float64) / rot)
        inv = inv.float().to(DEV)
    q_out = torch.empty(T, H * Dp, dtype=dtype, device=DEV)
    K.rope_pairs_store(q.to(DEV, dtype), k.to(DEV, dtype), v.to(DEV, dtype), inv, rot, positions.to(DEV),
                       torch.zeros(T, dtype=torch.int32, device=DEV), table, pool, q_out, H, G, d, dv, Dp)
    qr = P.rotate_pairs(q.double().view(T, H, d), positions, rot, 777.0) if rot else q.double().view(T, H, d)
    kr = P.rotate_pairs(k.double().view(T, G, d), positions, rot, 777.0) if rot else k.double().view(T, G, d)
    # angles are float: at position 70,000 the angle's rounding alone is 4e-3 radians
    tol = dict(f32=2e-5, bf16=1e-2)
    close(q_out.view(T, H, Dp)[:6, :, :d], qr[:6], dtype, "q", **tol)
    close(q_out.view(T, H, Dp)[6:8, :, :d], qr[6:8], dtype, "q at 1000", f32=2e-4)
    close(q_out.view(T, H, Dp)[8:, :, :d], qr[8:], dtype, "q at 70000", f32=2e-2, bf16=3e-2)
    assert float(q_out.view(T, H, Dp)[:, :, d:].abs().max() if Dp > d else 0.0) == 0.0
    where = {0: (5, 0), 3: (5, 3), 4: (2, 0), 6: (7, 0), 7: (7, 1), 8: (1, 0)}
    for t, (pg, r) in where.items():
        krow, vrow = pool[pg, 0, r].view(G, Dp), pool[pg, 1, r].view(G, Dp)
        close(krow[:, :d], kr[t], dtype, f"key {t}", f32=2e-2 if t == 8 else 2e-4, bf16=3e-2)
        close(vrow[:, :dv], v.double().view(T, G, dv)[t], dtype, f"value {t}", f32=0.0, bf16=1e-2)
        assert float(vrow[:, dv:].abs().max() if Dp > dv else 0.0) == 0.0


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("window", [1, 5, 16, 17, 40, 0])
def test_window_edge_and_sink_stand_out(dtype, window):
    """One key just inside the window and one just outside it carry scores far above the rest, and the
    sink is large: a window that is one token off, or a sink left out, changes the result by order one.
    Prompt rows and rows decoded one by one, across page borders, with key ranges."""
    H, G, Dh, page, T = 4, 2, 32, 16, 150
    q, k, v = rnd(T, H * Dh, seed=1, scale=0.3), rnd(T, G * Dh, seed=2, scale=0.3), rnd(T, G * Dh, seed=3)
    qh, kh = q.view(T, H, Dh), k.view(T, G, Dh)
    w = window if window > 0 else T
    for i in range(T):  # the keys at distance w - 1 (seen) and w (not seen) match the query's direction
        for j in (i - w + 1, i - w):
            if j >= 0 and j != i:
                kh[j] += 0.05 * qh[i, ::2] / (qh[i, ::2].norm(dim=-1, keepdim=True) ** 2) * 40.0
    k = kh.reshape(T, G * Dh).to(torch.bfloat16).float()
    sink = torch.tensor([3.0, -2.0, 0.5, 6.0])
    scale = 0.7
    want = P.windowed_sink_attention(q.double().view(T, H, Dh), k.double().view(T, G, Dh), v.double().view(T, G, Dh),
                                     scale, w, sink.double()).reshape(T, H * Dh)
    other = P.windowed_sink_attention(q.double().view(T, H, Dh), k.double().view(T, G, Dh), v.double().view(T, G, Dh),
                                      scale, w + 1, sink.double()).reshape(T, H * Dh)
    if window > 0:
        assert float((want - other).abs().max()) > 0.3  # the test can tell the two apart
    n_pages = (T + page - 1) // page
    pool = torch.zeros(n_pages + 2, 2, page, G * Dh, dtype=dtype, device=DEV)
    table = torch.tensor([list(range(n_pages, 0, -1))], dtype=torch.int32, device=DEV)  # pages out of order
    qd = torch.empty(T, H * Dh, dtype=dtype, device=DEV)
    pos = torch.arange(T, dtype=torch.int32, device=DEV)
    seq0 = torch.zeros(T, dtype=torch.int32, device=DEV)
    K.rope_pairs_store(q.to(DEV, dtype), k.to(DEV, dtype), v.to(DEV, dtype), None, 0, pos, seq0, table, pool, qd,
                       H, G, Dh, Dh, Dh)
    for n_splits, split_len in ((1, 0), (3, 64)):
        out = torch.empty(T, H * Dh, dtype=dtype, device=DEV)
        scratch = torch.empty(K.attention_scratch_floats(T, H, Dh, n_splits), device=DEV) if n_splits > 1 else None
        K.paged_attention(qd, pool, table, pos, seq0, out, H, G, Dh, scale, window=window, n_splits=n_splits,
                          split_len=split_len, scratch=scratch, sink=sink.to(DEV))
        close(out, want, dtype, f"prompt rows, {n_splits} key ranges", f32=2e-5, bf16=3e-2)
        one = torch.empty(1, H * Dh, dtype=dtype, device=DEV)
        for t in (0, 1, w - 1, w, w + 1, 15, 16, 17, T - 1):
            if 0 <= t < T:
                K.paged_attention(qd[t:t + 1], pool, table, pos[t:t + 1], seq0[:1], one, H, G, Dh, scale, window=window,
                                  n_splits=n_splits, split_len=split_len, scratch=scratch, sink=sink.to(DEV))
                close(one, want[t:t + 1], dtype, f"row {t} alone", f32=2e-5, bf16=3e-2)


@pytest.mark.parametrize("window", [40, 64, 65, 200, 0])
@pytest.mark.parametrize("H,G,Dh", [(4, 2, 64), (8, 1, 64), (2, 2, 128)])
def test_tensor_core_attention_with_sink_and_window(window, H, G, Dh, monkeypatch):
    """The same standing-out keys and sinks through every bfloat16 attention kernel: tcgen05 and
    mma.sync prompt tiles, decode tiles with TMA and with cp.async gathers, one and several key ranges."""
    dtype, page, T = torch.bfloat16, 64, 330
    q, k, v = rnd(T, H * Dh, seed=1, scale=0.3), rnd(T, G * Dh, seed=2, scale=0.3), rnd(T, G * Dh, seed=3)
    qh, kh = q.view(T, H, Dh), k.view(T, G, Dh)
    w = window if window > 0 else T
    rep = H // G
    for i in range(T):
        for j in (i - w + 1, i - w):
            if j >= 0 and j != i:
                kh[j] += qh[i, ::rep] / (qh[i, ::rep].norm(dim=-1, keepdim=True) ** 2) * 2.0
    k = kh.reshape(T, G * Dh).to(torch.bfloat16).float()
    sink = torch.linspace(-2.0, 5.0, H)
    scale = 0.9
    args = (q.double().view(T, H, Dh), k.double().view(T, G, Dh), v.double().view(T, G, Dh), scale)
    want = P.windowed_sink_attention(*args, w, sink.double()).reshape(T, H * Dh)
    if window > 0:
        assert float((want - P.windowed_sink_attention(*args, w + 1, sink.double()).reshape(T, H * Dh)).abs().max()) > 0.15
    assert float((want - P.windowed_sink_attention(*args, w, sink.double() - 50.0).reshape(T, H * Dh)).abs().max()) > 0.3
    n_pages = (T + page - 1) // page
    pool = torch.zeros(n_pages + 2, 2, page, G * Dh, dtype=dtype, device=DEV)
    table = torch.tensor([list(range(n_pages, 0, -1))], dtype=torch.int32, device=DEV)
    qd = torch.empty(T, H * Dh, dtype=dtype, device=DEV)
    pos = torch.arange(T, dtype=torch.int32, device=DEV)
    seq0 = torch.zeros(T, dtype=torch.int32, device=DEV)
    cu = torch.tensor([0, T], dtype=torch.int32, device=DEV)
    K.rope_pairs_store(q.to(DEV, dtype), k.to(DEV, dtype), v.to(DEV, dtype), None, 0, pos, seq0, table, pool, qd,
                       H, G, Dh, Dh, Dh)
    counter = torch.zeros(4096, dtype=torch.int32, device=DEV)
    sk = sink.to(DEV)
    for n_splits, split_len in ((1, 0), (3, 128)):
        scratch = torch.empty(K.attention_scratch_floats(T, H, Dh, n_splits), device=DEV) if n_splits > 1 else None
        out = torch.zeros(T, H * Dh, dtype=dtype, device=DEV)
        K.attention_tc(qd, pool, table, pos, cu, [T], out, H, G, Dh, scale, window=window, n_splits=n_splits,
                       split_len=split_len, scratch=scratch, split_counter=counter, sink=sk)
        close(out, want, dtype, f"tcgen05 prompt rows, {n_splits} key ranges", bf16=3e-2)
        out.zero_()
        K.paged_attention(qd, pool, table, pos, seq0, out, H, G, Dh, scale, window=window, n_splits=n_splits,
                          split_len=split_len, scratch=scratch, cu_seqlens=cu, new_lens=[T], split_counter=counter, sink=sk)
        close(out, want, dtype, f"mma.sync prompt rows, {n_splits} key ranges", bf16=3e-2)
        for tma in (True, False):
            monkeypatch.setattr(K, "_TMA_DECODE", tma)
            for t in (0, 1, w - 1, w, w + 1, 63, 64, 65, 127, 128, T - 1):
                if 0 <= t < T:
                    one = torch.zeros(1, H * Dh, dtype=dtype, device=DEV)
                    K.flash_decode_attention(qd[t:t + 1], None, None, 1.0, 1.0, 1.0, None, pool, table, pos[t:t + 1], one,
                                             H, G, Dh, scale, window=window, n_splits=n_splits, split_len=split_len,
                                             scratch=scratch, split_counter=counter, sink=sk)
                    close(one, want[t:t + 1], dtype, f"decode row {t}, tma {tma}, {n_splits} key ranges", bf16=3e-2)
    assert int(counter.abs().sum()) == 0
    K.check_status(DEV, wait=True)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("taps", [1, 2, 3, 5])
def test_convolution_without_activation_carries_its_window(dtype, taps):
    C, lens = 24, [11, 1, 6]
    T = sum(lens)
    x, w, b = rnd(T, C, seed=1), rnd(C, taps, seed=2), rnd(C, seed=3)
    want, t0 = [], 0
    for n in lens:
        want.append(P.causal_conv(x[t0:t0 + n].double() + b.double(), w.double()))
        t0 += n
    want = torch.cat(want)
    window = torch.full((4, taps - 1, C), 5.0, device=DEV)
    slots = [2, 0, 3]
    for s in slots:
        window[s].zero_()
    ones = torch.ones(C, device=DEV)
    out = torch.empty(T, C, dtype=dtype, device=DEV)
    xd = x.to(DEV, dtype)
    # first step: 4, 1 and 2 tokens; then the rest of the first and third one token at a time
    first = [4, 1, 2]
    starts = [0, 11, 12]
    rows = [r for i in range(3) for r in range(starts[i], starts[i] + first[i])]
    cu, seq_of, sl = batch_index(first, slots)
    o = torch.empty(len(rows), C, dtype=dtype, device=DEV)
    xin = xd[torch.tensor(rows, device=DEV)].contiguous()
    K.conv1d_fwd(xin, ones, b.to(DEV), w.to(DEV), None, window, seq_of, cu, sl, o, weight_t=w.t().contiguous().to(DEV),
                 activation=False)
    K.conv1d_window_update(xin, ones, b.to(DEV), window, cu, sl, 3, taps)
    out[torch.tensor(rows, device=DEV)] = o
    for step in range(7):
        rows = [starts[0] + 4 + step] + ([starts[2] + 2 + step] if step < 4 else [])
        sl = torch.tensor([2, 3][:len(rows)], dtype=torch.int32, device=DEV)
        o = torch.empty(len(rows), C, dtype=dtype, device=DEV)
        K.conv1d_decode(xd[torch.tensor(rows, device=DEV)].contiguous(), ones, b.to(DEV), w.to(DEV), None, window, sl, o,
                        activation=False)
        out[torch.tensor(rows, device=DEV)] = o
    close(out, want, dtype, "convolution", f32=1e-5, bf16=2e-2)
    if taps > 1:
        assert float(window[1].min()) == 5.0


@pytest.mark.parametrize("dtype", DTYPES)
def test_gated_norm_with_sigmoid_gate_on_float_rows(dtype):
    T, H, dv = 6, 3, 40
    o, z, w = rnd(T, H * dv, seed=1, scale=5.0), rnd(T, H * dv, seed=2), rnd(dv, seed=3) + 1.0
    want = (P.rms_unit(o.double().view(T, H, dv), 1e-5) * w.double() * torch.sigmoid(z.double()).view(T, H, dv))
    out = torch.empty(T, H * dv, dtype=dtype, device=DEV)
    K.gated_norm(o.to(DEV), z.to(DEV, dtype), 1.0, None, w.repeat(H).to(DEV), 1e-5, H, True, out, gate="sigmoid")
    close(out, want.reshape(T, H * dv), dtype, "per-head norm with sigmoid gate")
    want1 = P.norm_plain(o.double(), w.repeat(H).double(), 1e-5) * torch.sigmoid(z.double())
    K.gated_norm(o.to(DEV), z.to(DEV, dtype), 1.0, None, w.repeat(H).to(DEV), 1e-5, 1, True, out, gate="sigmoid")
    close(out, want1, dtype, "norm over all heads with sigmoid gate")
