"""Prompt portions of the attention with two score maps a head on tcgen05, beside single tokens and portions too short for it:
against each request alone in 64 bits.

Bounds: a weight enters the product as one bfloat16 in the kernel for few rows (2^-9 of itself, errors of both signs over many
keys), as two terms in the other; the difference of two maps is divided by its root mean square, the result is bfloat16: a few 2^-8 of an element of size 1."""

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("H,KVH,V,page,reqs", [
    (6, 2, 128, 16, [(1, 300), (200, 0), (5, 100), (65, 129)]), (12, 2, 64, 64, [(43, 0), (22, 490), (2, 7)]),
    (4, 1, 128, 48, [(1, 0), (128, 128), (4, 200)]), (2, 2, 64, 32, [(129, 0)])])
def test_two_maps_in_portions(H, KVH, V, page, reqs, shuffled):
    from turingserve_b200 import kernels
    ops = kernels.ops()
    D, G = 64, H // KVH
    assert ops.lib.ts_attention_maps_tc_supported(H, KVH, D, V, page, 1)
    g = torch.Generator(device=DEV).manual_seed(H * V + page)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    n_pages = [-(-(n + c) // page) for n, c in reqs]
    ids = torch.randperm(sum(n_pages), generator=g, device=DEV).tolist() if shuffled else list(range(sum(n_pages)))
    width = max(n_pages) + 1
    pool_k = torch.full((sum(n_pages) + 1, KVH, page, 2 * D), float("nan"), device=DEV).bfloat16()
    pool_v = torch.full((sum(n_pages) + 1, KVH, page, V), float("nan"), device=DEV).bfloat16()
    tables, ks, vs = [], [], []
    for (n, c), m in zip(reqs, n_pages):
        table = [ids.pop(0) + 1 for _ in range(m)]
        k, v, at = rnd(n + c, KVH, 2 * D).bfloat16(), rnd(n + c, KVH, V).bfloat16(), torch.arange(n + c, device=DEV)
        pages = torch.tensor(table, device=DEV)[at // page]
        pool_k[pages, :, at % page], pool_v[pages, :, at % page] = k, v
        tables.append(table + [0] * (width - m)), ks.append(k), vs.append(v)
    # (what the kernel for few rows may read behind a request's last key is zeroed by itself; the null page stays NaN)
    lens = [n for n, _ in reqs]
    starts = [sum(lens[:i]) for i in range(len(lens) + 1)]
    step = SimpleNamespace(q_start=i32(starts), seq_lens=i32([n + c for n, c in reqs]), num_requests=len(reqs),
                           num_decode=sum(n == 1 for n in lens), max_q_len=max(lens), max_seq_len=max(n + c for n, c in reqs),
                           q_lens=lens, token_request=i32([r for r, n in enumerate(lens) for _ in range(n)]))
    proj = rnd(sum(lens), H * 2 * D + 24).bfloat16()
    out = torch.full((sum(lens), H * V), float("nan"), device=DEV).bfloat16()
    lam, keys = 0.4, ops.diff_tc_keys
    ops.diff_tc_keys = 1
    try:
        ops.attention_diff(out, proj, pool_k, pool_v, i32(tables), step, H, KVH, D, V, page, 0.125, lam, 1e-6, 0.5)
    finally:
        ops.diff_tc_keys = keys
    assert ops.tc_status() == 0
    for (n, c), at, k, v in zip(reqs, starts, ks, vs):
        q = proj[at:at + n, :H * 2 * D].double().view(n, H, 2, D)
        hidden = torch.arange(n + c, device=DEV)[None, :] > torch.arange(n, device=DEV)[:, None] + c
        for h in range(H):
            maps = [torch.softmax((q[:, h, m] @ k[:, h // G, m * D:(m + 1) * D].double().T * 0.125).masked_fill(hidden, float("-inf")), -1)
                    @ v[:, h // G].double() for m in (0, 1)]
            o = maps[0] - lam * maps[1]
            want = o / torch.sqrt(o.pow(2).mean(-1, keepdim=True) + 1e-6) * 0.5
            assert torch.allclose(out[at:at + n, h * V:(h + 1) * V].double(), want, rtol=2 ** -7, atol=2 ** -7), (n, c, h)


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("H,KVH,V,page,n,ctx", [(6, 2, 128, 16, 300, 9), (2, 2, 64, 64, 129, 70)])
def test_values_that_are_no_numbers_reach_no_earlier_row(H, KVH, V, page, n, ctx, bad):
    """A value that is an infinity or NaN: heads of rows that see its key are NaN, all others the same bits as without it."""
    from turingserve_b200 import kernels
    ops = kernels.ops()
    g = torch.Generator(device=DEV).manual_seed(n + V)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV).bfloat16()
    pages = -(-(n + ctx) // page)
    pool_k, pool_v, proj = rnd(pages, KVH, page, 128), rnd(pages, KVH, page, V), rnd(n, H * 128)
    step = SimpleNamespace(q_start=i32([0, n]), seq_lens=i32([n + ctx]), num_requests=1, num_decode=0, max_q_len=n, max_seq_len=n + ctx,
                           q_lens=[n], token_request=i32([0] * n))

    def attend():
        out = torch.full((n, H * V), -7.0, device=DEV).bfloat16()
        keys, ops.diff_tc_keys = ops.diff_tc_keys, 1
        try:
            ops.attention_diff(out, proj, pool_k, pool_v, i32([list(range(pages))]), step, H, KVH, 64, V, page, 0.125, 0.4, 1e-6, 0.5)
        finally:
            ops.diff_tc_keys = keys
        assert ops.tc_status() == 0
        return out.view(n, KVH, -1)

    clean, at = attend(), ctx + n // 2
    pool_v[at // page, 0, at % page, 5] = bad
    dirty = attend()
    assert torch.equal(dirty[:n // 2], clean[:n // 2]) and torch.equal(dirty[:, 1:], clean[:, 1:])
    assert bool(dirty[n // 2:, 0].isnan().all())


@pytest.mark.parametrize("size", [0.3, 1.0, 3.0])
def test_no_further_from_64_bits_than_the_kernel_for_few_rows(monkeypatch, size):
    """The weights refer to a maximum that may lag behind the row's, so the largest is no exact 1 as in attention_diff_mma.cu:
    as one bfloat16 each they would be up to 1.6 times further off there (scores of size 3)."""
    from turingserve_b200 import kernels
    ops = kernels.ops()
    H, KVH, D, V, page, n = 4, 2, 64, 128, 16, 700
    g = torch.Generator(device=DEV).manual_seed(11)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    pages = -(-n // page)
    pool_k, pool_v = rnd(pages, KVH, page, 2 * D).bfloat16(), rnd(pages, KVH, page, V).bfloat16()
    proj = (rnd(n, H * 2 * D) * size).bfloat16()
    step = SimpleNamespace(q_start=i32([0, n]), seq_lens=i32([n]), num_requests=1, num_decode=0, max_q_len=n, max_seq_len=n,
                           q_lens=[n], token_request=i32([0] * n))
    flat = lambda pool: pool.transpose(1, 2).reshape(pages * page, KVH, -1)[:n].double()
    k, v, hidden = flat(pool_k), flat(pool_v), torch.ones(n, n, dtype=torch.bool, device=DEV).triu(1)
    want = []
    for h in range(H):
        maps = []
        for m in (0, 1):
            q = proj[:, (2 * h + m) * D:(2 * h + m + 1) * D].double()
            s = (q @ k[:, h // (H // KVH), m * D:(m + 1) * D].T * 0.125).masked_fill(hidden, float("-inf"))
            maps.append(torch.softmax(s, -1) @ v[:, h // (H // KVH)])
        o = maps[0] - 0.4 * maps[1]
        want.append(o / torch.sqrt(o.pow(2).mean(-1, keepdim=True) + 1e-6) * 0.5)
    want = torch.cat(want, 1)
    errors = []
    for keys in (1, 1 << 30):
        monkeypatch.setattr(ops, "diff_tc_keys", keys)
        out = torch.empty(n, H * V, device=DEV).bfloat16()
        ops.attention_diff(out, proj, pool_k, pool_v, i32([list(range(pages))]), step, H, KVH, D, V, page, 0.125, 0.4, 1e-6, 0.5)
        errors.append(float((out.double() - want).norm() / want.norm()))
    assert ops.tc_status() == 0 and errors[0] <= 1.001 * errors[1], errors
