"""The token-by-token scans over long portions (a warp's columns) beside the ones for a few tokens: the same bits however a
prompt is cut between them, and both against the recurrence in 64 bits.

Bounds: states and sums are 32-bit sums of at most 256 products and as many tokens; inputs of size 1.  A rounding is 2^-24
of a partial sum; over a few hundred of them the error grows as their root: 1e-5 of an output's own size, 1e-4 with margin
for the activations' 2^-21 in float32."""

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops():
    from turingserve_b200 import kernels
    return kernels.ops()


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def steps(lens, cuts):
    """[(rows, step)] of requests of ``lens`` tokens in portions: ``cuts`` are places (of every request) a step ends at."""
    starts = [sum(lens[:i]) for i in range(len(lens))]
    out, at = [], 0
    for end in list(cuts) + [max(lens)]:
        part = [(min(n, at), min(n, end)) for n in lens]
        here = [i for i, (a, e) in enumerate(part) if e > a]
        if here:
            n = [part[i][1] - part[i][0] for i in here]
            rows = torch.cat([torch.arange(starts[i] + part[i][0], starts[i] + part[i][1], device=DEV) for i in here])
            step = SimpleNamespace(q_start=i32([sum(n[:k]) for k in range(len(n) + 1)]), state_slots=i32([2 * i + 1 for i in here]),
                                   num_requests=len(here), max_q_len=max(n),
                                   token_request=i32([k for k, m in enumerate(n) for _ in range(m)]))
            out.append((rows, step))
        at = end
    return out


CUTS = [(), (63,), (64, 65), (1, 17, 90), (16, 32, 160)]


def close(got, want):
    return torch.allclose(got.double(), want, rtol=1e-4, atol=1e-4 * float(want.abs().max()))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,D,V", [(2, 128, 128), (3, 64, 40), (1, 8, 8), (2, 40, 24), (1, 256, 16), (2, 136, 8)])
def test_linear_attention_long_portions(ops, monkeypatch, dtype, H, D, V):
    lens, width = [150, 64, 7, 200], H * (2 * D + V)
    g = torch.Generator(device=DEV).manual_seed(D + V)
    proj = torch.randn(sum(lens), width + 16, generator=g, device=DEV).to(dtype)
    decay = 1 - torch.rand(H, generator=g, device=DEV) * 0.2
    first = torch.randn(9, H, D, V, generator=g, device=DEV)
    monkeypatch.setattr(ops, "lightning_long_tokens", 128)
    assert ops.lib.ts_lightning_long_supported(D, V, width + 16, 128, int(dtype == torch.bfloat16))
    results = []
    for cuts in CUTS:
        state, out = first.clone(), torch.full((sum(lens), H * V), float("nan"), device=DEV)
        for rows, step in steps(lens, cuts):
            p = proj[rows].contiguous()
            o = torch.empty(len(rows), H * V, device=DEV)
            ops.lightning(o, p[:, :width], state, decay, step, H, D, V)
            out[rows] = o
        results.append((out, state))
    act = torch.nn.functional.silu(proj.double()).to(dtype).double()
    q, k, v = (act[:, a:b].view(-1, H, (b - a) // H) for a, b in ((0, H * D), (H * D, 2 * H * D), (2 * H * D, width)))
    at = 0
    for i, n in enumerate(lens):
        S, o = first[2 * i + 1].double(), []
        for t in range(at, at + n):
            S = decay.double()[:, None, None] * S + k[t][:, :, None] * v[t][:, None, :]
            o.append(torch.einsum("hdv,hd->hv", S, q[t]).reshape(-1))
        tol = 1.0 if dtype == torch.float32 else 30.0     # (a bfloat16 activation may round the other way: 2^-9 of a term)
        for got, want in ((results[0][0][at:at + n], torch.stack(o)), (results[0][1][2 * i + 1], S)):
            assert torch.allclose(got.double(), want, rtol=1e-4 * tol, atol=1e-4 * tol * float(want.abs().max()))
        assert torch.equal(results[0][1][2 * i], first[2 * i])
        at += n
    for out, state in results[1:]:
        assert torch.equal(out, results[0][0]) and torch.equal(state, results[0][1])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,P,N,G,taps,skipped", [(4, 64, 128, 2, 4, True), (2, 40, 64, 1, 1, False), (2, 4, 12, 2, 3, True),
                                                 (2, 20, 256, 1, 4, True), (2, 8, 132, 2, 8, False)])
def test_state_space_long_portions(ops, dtype, H, P, N, G, taps, skipped):
    lens, inner = [150, 64, 7, 200], H * P
    channels = inner + 2 * G * N
    g = torch.Generator(device=DEV).manual_seed(P + N)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    proj = rnd(sum(lens), 2 * inner + 2 * G * N + H).to(dtype)
    conv_w, conv_b, a_log, dt_bias = rnd(channels, taps) * 0.5, rnd(channels) * 0.2, rnd(H) * 0.3, rnd(H) - 2.0
    skip = rnd(H) if skipped else None
    assert (channels + 2 * H) % 4 == 0 and N % 4 == 0 and P % 4 == 0
    first = rnd(9, H * N * P + (taps - 1) * channels)
    results = []
    for cuts in CUTS:
        state, out = first.clone(), torch.full((sum(lens), inner), float("nan"), device=DEV)
        rows_of = []
        for rows, step in steps(lens, cuts):
            p = proj[rows].contiguous()
            ready = torch.empty(len(rows), channels + 2 * H, device=DEV)
            ops.ssm_prepare(ready, p, inner, inner + channels, conv_w, conv_b, a_log, dt_bias, state, H * N * P, step, H, channels, taps)
            o = torch.empty(len(rows), inner, device=DEV)
            ops.ssm_scan(o, ready, p, inner, state, skip, step, H, G, N, P, taps)
            out[rows] = o
            rows_of.append((rows, ready))
        results.append((out, state, torch.cat([r for r, _ in rows_of]), torch.cat([x for _, x in rows_of])))
    ready = torch.empty_like(results[0][3])
    ready[results[0][2]] = results[0][3]
    ready = ready.double()
    x, dt, a = ready[:, :inner].view(-1, H, P), ready[:, channels:channels + H], ready[:, channels + H:]
    B, C = (ready[:, inner + i * G * N:inner + (i + 1) * G * N].view(-1, G, N).repeat_interleave(H // G, 1) for i in (0, 1))
    at = 0
    for i, n in enumerate(lens):
        S, o = first[2 * i + 1, :H * N * P].view(H, N, P).double(), []
        for t in range(at, at + n):
            S = a[t][:, None, None] * S + (dt[t][:, None] * B[t])[:, :, None] * x[t][:, None, :]
            o.append((torch.einsum("hnp,hn->hp", S, C[t]) + (0 if skip is None else skip.double()[:, None] * x[t])).reshape(-1))
        assert close(results[0][0][at:at + n], torch.stack(o)) and close(results[0][1][2 * i + 1, :H * N * P], S.reshape(-1))
        assert torch.equal(results[0][1][2 * i], first[2 * i])
        at += n
    for r in results[1:]:
        assert torch.equal(r[0], results[0][0]) and torch.equal(r[1], results[0][1])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,D,V,taps,pad", [(4, 2, 128, 128, 4, 2), (2, 1, 64, 40, 3, 3), (3, 3, 8, 4, 1, 3), (2, 1, 100, 20, 2, 3),
                                             (2, 1, 128, 24, 8, 3), (2, 1, 64, 40, 3, 0)])
def test_delta_rule_portions(ops, dtype, H, G, D, V, taps, pad):
    """Rows on 16-byte boundaries (``pad``) go to the kernel of eight lanes a column, others do not; portions of any lengths
    from two tokens give the same bits."""
    lens, C = [150, 64, 9, 200], 2 * G * D + H * V
    width = C + 2 * H + G
    assert pad == 0 or (width + pad) % 4 == 0
    g = torch.Generator(device=DEV).manual_seed(D + V)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    proj = rnd(sum(lens), C + H * V + 2 * H).to(dtype)
    conv_w, a_log, dt = rnd(C, taps) * 0.5, rnd(H) * 0.3, rnd(H) - 2.0
    first = rnd(9, H * D * V + (taps - 1) * C)
    results = []
    for cuts in ((), (63,), (2, 66), (64, 70, 90), (16, 32, 148)):
        state, out, kept = first.clone(), torch.full((sum(lens), H * V), float("nan"), device=DEV), torch.empty(sum(lens), width, device=DEV)
        for rows, step in steps(lens, cuts):
            p = proj[rows].contiguous()
            ready = torch.full((len(rows), width + pad), float("nan"), device=DEV)[:, :width]
            ops.delta_prepare(ready, p, conv_w, a_log, dt, state, step, H, G, D, V, taps, 1e-6)
            o = torch.empty(len(rows), H * V, device=DEV)
            ops.delta_scan(o, ready, p, state, step, H, G, D, V, taps)
            out[rows], kept[rows] = o, ready
        results.append((out, state, kept))
    r = results[0][2].double()
    q, k = (r[:, i * G * D:(i + 1) * G * D].view(-1, G, D).repeat_interleave(H // G, 1) for i in (0, 1))
    v, fade, w = r[:, 2 * G * D:C].view(-1, H, V), r[:, C:C + H], r[:, C + H:C + 2 * H]
    at = 0
    for i, n in enumerate(lens):
        S, o = first[2 * i + 1, :H * D * V].view(H, D, V).double(), []
        for t in range(at, at + n):
            S = fade[t][:, None, None] * S
            u = w[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
            S = S + k[t][:, :, None] * u[:, None, :]
            o.append(torch.einsum("hdv,hd->hv", S, q[t]).reshape(-1))
        assert close(results[0][0][at:at + n], torch.stack(o)) and close(results[0][1][2 * i + 1, :H * D * V], S.reshape(-1))
        assert torch.equal(results[0][1][2 * i], first[2 * i])
        at += n
    for r in results[1:]:
        assert torch.equal(r[0], results[0][0]) and torch.equal(r[1], results[0][1])


@pytest.mark.parametrize("D", [8, 64, 104, 136])
@pytest.mark.parametrize("kind", ["linear", "state_space", "delta"])
def test_infinite_values_in_narrow_states(ops, monkeypatch, kind, D):
    """An infinite value in one column, keys and queries positive: that column's output is infinite from there on (in the delta
    rule at that token), not NaN, although a state of fewer rows than the lanes hold leaves some of them without any."""
    monkeypatch.setattr(ops, "lightning_long_tokens", 128)
    T, V, at, col = 150, 16, 70, 5
    g = torch.Generator(device=DEV).manual_seed(D)
    some = lambda *s: torch.rand(*s, generator=g, device=DEV) * 0.2 + 0.1
    step = SimpleNamespace(q_start=i32([0, T]), state_slots=i32([0]), num_requests=1, max_q_len=T, token_request=i32([0] * T))
    out, inf = torch.empty(T, V, device=DEV), float("inf")
    if kind == "linear":
        proj, state = some(T, 2 * D + V), torch.zeros(1, 1, D, V, device=DEV)
        proj[at, 2 * D + col] = inf
        ops.lightning(out, proj, state, some(1), step, 1, D, V)
    elif kind == "state_space":
        H, P = 2, V // 2                                   # (rows of 16 + 2 D + 4: on their boundaries)
        ready, proj, state = some(T, V + 2 * D + 2 * H), some(T, 2 * V + 2 * D + H), torch.zeros(1, H * D * P + 3 * (V + 2 * D), device=DEV)
        ready[at, col] = inf
        ops.ssm_scan(out, ready, proj, V, state, some(H), step, H, 1, D, P, 4)
    else:
        width = 2 * D + V + 3
        if D > 128:
            pytest.skip("wider keys go to another kernel")
        ready, proj = some(T, width + (-width) % 4)[:, :width], some(T, 2 * D + 2 * V + 2)
        state = torch.zeros(1, D * V + 3 * (2 * D + V), device=DEV)
        ready[at, 2 * D + col] = inf
        ops.delta_scan(out, ready, proj, state, step, 1, 1, D, V, 4)
    others = [c for c in range(V) if c != col]
    assert bool(out[:, others].isfinite().all()) and bool(out[:at, col].isfinite().all())
    assert bool((out[at:at + 1 if kind == "delta" else T, col] == inf).all())


def test_delta_rule_single_tokens_beside_portions(ops):
    """Steps in which every request brings one token sum a row in another order than portions do (four lanes of 32 rows, not
    eight of 16): an uncut run and one with such steps agree to 32-bit roundings, outputs and states."""
    H, G, D, V, taps, lens = 4, 2, 128, 64, 4, [150, 67]
    C = 2 * G * D + H * V
    width = C + 2 * H + G
    g = torch.Generator(device=DEV).manual_seed(5)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    proj, conv_w, a_log, dt = rnd(sum(lens), C + H * V + 2 * H), rnd(C, taps) * 0.5, rnd(H) * 0.3, rnd(H) - 2.0
    first = rnd(9, H * D * V + (taps - 1) * C)
    results = []
    for cuts in ((), (1, 2, 66), (64, 65, 100, 101)):
        state, out = first.clone(), torch.full((sum(lens), H * V), float("nan"), device=DEV)
        for rows, step in steps(lens, cuts):
            p = proj[rows].contiguous()
            ready = torch.empty_strided((len(rows), width), (width + -width % 4, 1), dtype=torch.float32, device=DEV)
            ops.delta_prepare(ready, p, conv_w, a_log, dt, state, step, H, G, D, V, taps, 1e-6)
            o = torch.empty(len(rows), H * V, device=DEV)
            ops.delta_scan(o, ready, p, state, step, H, G, D, V, taps)
            out[rows] = o
        results.append((out, state))
    for out, state in results[1:]:
        assert close(out, results[0][0].double()) and close(state, results[0][1].double())
