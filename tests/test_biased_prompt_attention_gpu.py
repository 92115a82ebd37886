"""The tcgen05 kernel for prompt portions of the attention with caps, biases, windows, sinks and latent rows: against each
request alone in 64 bits, at the edges of its tiles (128 query rows, 64 or 128 keys, boxes of 16 to 64 keys) and with each option.

Bounds: operands and results are bfloat16 (the result's rounding: 2^-9 relative); the weights enter the product as two
bfloat16 terms (2^-17), their sums are 32-bit.  So an element is off by at most 2^-8 of itself plus 2^-15 of the largest
value of its head times a few sums: rtol 2^-8, atol 2e-3 for values of size 1."""

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


def exact(q, k, v, first, scale, cap, slopes, window, block_of, keep, sinks, freq, gate):
    """q [n, H, Dk] at positions first.., k [m, KVH, Dk], v [m, KVH, Dv] -> [n, H, Dv] in 64 bits."""
    n, H, _ = q.shape
    per = H // k.shape[1]
    i, j = torch.arange(n, device=DEV)[:, None] + first, torch.arange(k.shape[0], device=DEV)[None, :]
    seen = j <= i
    if window:
        seen = seen & ((j > i - window) | (j < keep))
    if block_of:
        seen = seen & (j >= i // block_of * block_of)
    out = []
    for h in range(H):
        s = (q[:, h].double() @ k[:, h // per].double().T) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        if slopes is not None:
            s = s - slopes[h].double() * (i - j)
        s = s.masked_fill(~seen, float("-inf"))
        m = s.max(-1, keepdim=True).values
        if sinks is not None:
            m = torch.maximum(m, sinks[h].double())
        e = torch.exp(s - m)
        total = e.sum(-1, keepdim=True) + (torch.exp(sinks[h].double() - m) if sinks is not None else 0)
        out.append((e / total) @ v[:, h // per].double().masked_fill(~seen.any(0)[:, None], 0.0))
    o = torch.stack(out, 1)
    if freq is not None:
        a = i[:, :, None] * freq.double()
        u, w = o.chunk(2, -1)
        o = torch.cat([u * torch.cos(a) + w * torch.sin(a), w * torch.cos(a) - u * torch.sin(a)], -1)
    return o if gate is None else o * torch.sigmoid(gate.double())[..., None]


CASES = [
    # H, KVH, Dk, Dv, page, (tokens, context) per request, options
    (6, 2, 128, 128, 64, [(300, 0), (129, 70), (22, 1)], {}),
    (6, 2, 128, 128, 16, [(43, 0), (85, 411)], dict(cap=20.0, slopes=True, window=100)),
    (12, 2, 128, 128, 48, [(64, 64), (2, 500), (65, 5)], dict(sinks=True, gate=True)),
    (4, 1, 128, 128, 32, [(257, 130)], dict(window=64, keep=70, sinks=True, freq=True)),
    (4, 1, 128, 128, 16, [(150, 333)], dict(window=33, keep=5, freq=True, gate=True)),
    (6, 2, 128, 128, 64, [(200, 100), (64, 1)], dict(block_of=96, sinks=True)),
    (2, 2, 128, 128, 16, [(129, 0)], dict(big=True)),
    (8, 2, 64, 64, 16, [(130, 0), (33, 95)], dict(window=50, keep=3, freq=True)),
    (8, 2, 64, 64, 128, [(64, 200)], dict(cap=5.0)),
    (12, 1, 576, 512, 64, [(128, 0), (11, 300), (64, 64)], {}),
    (5, 1, 576, 512, 16, [(77, 0), (26, 131)], dict(window=70, sinks=True, gate=True)),
    (3, 1, 576, 512, 32, [(43, 21)], dict(big=True)),
    (28, 1, 576, 512, 16, [(40, 129)], dict(window=1024, sinks=True, gate=True)),
    (4, 2, 320, 256, 16, [(65, 0), (33, 66)], dict(window=40, keep=20, freq=True)),
]


@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("H,KVH,Dk,Dv,page,reqs,opt", CASES)
def test_prompt_portions_by_tcgen05(ops, H, KVH, Dk, Dv, page, reqs, opt, shuffled):
    """Behind every request's last key its page holds NaN, and so does the null page (entries past the table): none of it
    may reach a result.  ``big``: scores in the tens of thousands."""
    g = torch.Generator(device=DEV).manual_seed(H * Dk + page)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    assert ops.lib.ts_attention_biased_tc_supported(H, KVH, Dk, Dv, int(Dv != Dk), page, 1)
    n_pages = [-(-(n + c) // page) for n, c in reqs]
    ids = torch.randperm(sum(n_pages), generator=g, device=DEV).tolist() if shuffled else list(range(sum(n_pages)))
    width = max(n_pages) + 1
    pool_k = torch.full((sum(n_pages) + 1, KVH, page, Dk), float("nan"), device=DEV).bfloat16()
    pool_v = None if Dv != Dk else torch.full((sum(n_pages) + 1, KVH, page, Dv), float("nan"), device=DEV).bfloat16()
    tables, ks, vs = [], [], []
    for (n, c), m in zip(reqs, n_pages):
        table = [ids.pop(0) + 1 for _ in range(m)]
        k = (rnd(n + c, KVH, Dk) * (30.0 if opt.get("big") else 1.0)).bfloat16()
        v = k[:, :, :Dv] if pool_v is None else rnd(n + c, KVH, Dv).bfloat16()
        at = torch.arange(n + c, device=DEV)
        pages = torch.tensor(table, device=DEV)[at // page]
        pool_k[pages, :, at % page] = k
        if pool_v is not None:
            pool_v[pages, :, at % page] = v
        tables.append(table + [0] * (width - m)), ks.append(k), vs.append(v)
    lens = [n for n, _ in reqs]
    starts = [sum(lens[:i]) for i in range(len(lens) + 1)]
    step = SimpleNamespace(q_start=i32(starts), seq_lens=i32([n + c for n, c in reqs]), num_requests=len(reqs), num_decode=0,
                           max_q_len=max(lens), max_seq_len=max(n + c for n, c in reqs))
    T = sum(lens)
    q = rnd(T, H, Dk + 8).mul(30.0 if opt.get("big") else 1.0).bfloat16()[:, :, 8:]
    out = torch.full((T, H, Dv + 8), -7.0, device=DEV).bfloat16()
    slopes = torch.tensor([2.0 ** (-8.0 * (h + 1) / H) for h in range(H)], device=DEV) if opt.get("slopes") else None
    sinks = rnd(H) if opt.get("sinks") else None
    freq = 0.3 * torch.rand(Dv // 2, generator=g, device=DEV) if opt.get("freq") else None
    gate = rnd(T, H).bfloat16() if opt.get("gate") else None
    scale = Dk ** -0.5
    window, block_of, keep = opt.get("window"), opt.get("block_of"), opt.get("keep", 0)
    keys, ops.biased_tc_keys = ops.biased_tc_keys, 1
    try:
        ops.attention_biased(out[:, :, :Dv], q, pool_k, pool_v, i32(tables), step, KVH, page, scale, opt.get("cap", 0.0), slopes,
                             window, chunk=block_of, sinks=sinks, keep=keep, out_freq=freq, gate=gate)
    finally:
        ops.biased_tc_keys = keys
    assert ops.tc_status() == 0
    assert float((out[:, :, Dv:].float() + 7.0).abs().max()) == 0.0
    for (n, c), at, k, v in zip(reqs, starts, ks, vs):
        want = exact(q[at:at + n], k, v, c, scale, opt.get("cap"), slopes, window, block_of, keep, sinks, freq,
                     None if gate is None else gate[at:at + n])
        size = 30.0 if opt.get("big") and pool_v is None else 1.0
        got = out[at:at + n, :, :Dv].double()
        # (scores in the tens of thousands: a 32-bit sum of them is off by up to 1e-2, and so is a weight)
        assert torch.allclose(got, want, rtol=2 ** -8, atol=2e-3 * size * (20 if opt.get("big") else 1)), (n, c, float((got - want).abs().max()))


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf")])
@pytest.mark.parametrize("H,KVH,Dk,Dv,page,n,ctx,opt", [
    (6, 2, 128, 128, 64, 300, 0, {}), (2, 2, 128, 128, 16, 200, 70, dict(window=50)), (4, 1, 128, 128, 16, 150, 333, dict(window=33, keep=5)),
    (4, 2, 128, 128, 32, 129, 100, dict(block_of=48)), (8, 2, 64, 64, 16, 130, 9, dict(window=40)), (12, 1, 576, 512, 64, 77, 130, {}),
    (5, 1, 576, 512, 16, 90, 40, dict(window=30)), (4, 2, 320, 256, 16, 65, 20, dict(window=20, keep=3))])
def test_values_that_are_no_numbers_stay_with_the_rows_that_see_them(ops, H, KVH, Dk, Dv, page, n, ctx, opt, bad):
    """One column of some keys' values holds an infinity or NaN: that column is no number in every row that sees such a
    key, and every other element is the same bits as without (a weight of zero times it would be NaN)."""
    g = torch.Generator(device=DEV).manual_seed(n + Dk)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    m, window, block_of, keep = n + ctx, opt.get("window"), opt.get("block_of"), opt.get("keep", 0)
    pages = -(-m // page)
    pool_k = rnd(pages, KVH, page, Dk).bfloat16()
    pool_v = None if Dv != Dk else rnd(pages, KVH, page, Dv).bfloat16()
    step = SimpleNamespace(q_start=i32([0, n]), seq_lens=i32([m]), num_requests=1, num_decode=0, max_q_len=n, max_seq_len=m)
    q, table = rnd(n, H, Dk).bfloat16(), i32([list(range(pages))])
    if pool_v is None:
        q[:, :, :Dv] = 0                                   # (the latent column that is spoiled is also a key's: no score may see it)

    def attend():
        out = torch.full((n, H, Dv), -7.0, device=DEV).bfloat16()
        keys, ops.biased_tc_keys = ops.biased_tc_keys, 1
        try:
            ops.attention_biased(out, q, pool_k, pool_v, table, step, KVH, page, Dk ** -0.5, 0.0, None, window, chunk=block_of, keep=keep)
        finally:
            ops.biased_tc_keys = keys
        assert ops.tc_status() == 0
        return out

    clean = attend()
    i, j = torch.arange(n, device=DEV)[:, None] + ctx, torch.arange(m, device=DEV)[None, :]
    seen = j <= i
    if window:
        seen &= (j > i - window) | (j < keep)
    if block_of:
        seen &= j >= i // block_of * block_of
    spoiled = [(m - 1, 3), (ctx + n // 2, Dv - 1), (ctx + 1, Dv // 2), (max(0, ctx - 20), 17), (2, 40)]
    for at, col in spoiled:
        rows = pool_v if pool_v is not None else pool_k
        rows[at // page, KVH - 1, at % page, col] = bad
    dirty = attend()
    spoilt, per = torch.zeros_like(clean, dtype=torch.bool), H // KVH
    for at, col in spoiled:
        spoilt[:, (KVH - 1) * per:, col] |= seen[:, at, None]
    if pool_v is None:
        # (zero times the spoiled column is NaN in the score of every row that sees the key)
        hit = torch.stack([seen[:, at] for at, _ in spoiled]).any(0)
        assert bool(dirty[hit][:, (KVH - 1) * per:].isnan().all()) and torch.equal(dirty[~hit], clean[~hit])
        assert torch.equal(dirty[:, :(KVH - 1) * per], clean[:, :(KVH - 1) * per])
    else:
        # (an infinity times a weight's two terms, of which the second may be negative, is NaN too)
        assert torch.equal(~dirty.isfinite(), spoilt) and torch.equal(dirty[~spoilt], clean[~spoilt])
