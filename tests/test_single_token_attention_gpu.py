"""Attention of single tokens on clusters of blocks, against the softmax in 64 bits: context lengths around a tile (16 keys), a
block's two rounds (320), the cluster; pages of any size; 1 to 32 heads a kv head; every option of the attention with options.

Bound: an output is rounded to bfloat16 (2^-8 of it, half a step).  Weights as two bfloat16 terms carry 2^-17, exponentials and caps in 32
bits about 1e-5 at scores up to 30: 1e-4 of the mean of |v| under the weights; as one term 2^-8 of it."""

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


class Case:
    def __init__(self, lens, H, KVH, D, V, page, latent=False, seed=0, limit=0):
        g = torch.Generator(device=DEV).manual_seed(seed + sum(lens) + D + H)
        rnd = lambda *s, std=1.0: (torch.randn(*s, generator=g, device=DEV) * std).bfloat16()
        self.lens, self.H, self.KVH, self.D, self.V, self.page = lens, H, KVH, D, V, page
        width = max(1, max(-(-n // page) for n in lens))
        pages = len(lens) * width + 1
        self.k, self.v = rnd(pages, KVH, page, D), None if latent else rnd(pages, KVH, page, V)
        self.tables = (torch.randperm(pages - 1, generator=g, device=DEV)[: len(lens) * width] + 1).view(len(lens), width).int()
        self.q = rnd(len(lens), H, D, std=0.4 if latent else 1.0)
        self.step = SimpleNamespace(q_start=i32(list(range(len(lens) + 1))), seq_lens=i32(lens), num_requests=len(lens),
                                    num_decode=len(lens), max_q_len=1, max_seq_len=limit or max(lens))

    def want(self, scale, cap=0.0, slopes=None, window=None, chunk=None, sinks=None, keep=0, out_freq=None, gate=None):
        """(outputs, mean of |v| under the weights times the gate) in 64 bits."""
        outs, sizes = [], []
        for b, n in enumerate(self.lens):
            rows = lambda t: t[self.tables[b].long()].transpose(0, 1).flatten(1, 2)[:, :n].double()     # [KVH, n, .]
            k = rows(self.k)
            v = k[..., : self.V] if self.v is None else rows(self.v)
            per = self.H // self.KVH
            k, v = k.repeat_interleave(per, 0), v.repeat_interleave(per, 0)
            s = torch.einsum("hd,hnd->hn", self.q[b].double(), k) * scale
            if cap:
                s = cap * torch.tanh(s / cap)
            j, pos = torch.arange(n, device=DEV), n - 1
            if slopes is not None:
                s = s - slopes.double()[:, None] * (pos - j)
            seen = torch.ones(n, dtype=torch.bool, device=DEV)
            if window:
                seen = (pos - j < window) | (j < keep)
            if chunk:
                seen = seen & (j >= pos // chunk * chunk)
            s = s.masked_fill(~seen, float("-inf"))
            m = s.max(-1, keepdim=True).values
            if sinks is not None:
                m = torch.maximum(m, sinks.double()[:, None])
            e = torch.exp(s - m)
            total = e.sum(-1, keepdim=True)
            if sinks is not None:
                total = total + torch.exp(sinks.double()[:, None] - m)
            p = e / total
            o, w = torch.einsum("hn,hnv->hv", p, v), torch.einsum("hn,hnv->hv", p, v.abs())
            if out_freq is not None:
                a = pos * out_freq.double()
                x, y = o.chunk(2, -1)
                o = torch.cat([x * a.cos() + y * a.sin(), y * a.cos() - x * a.sin()], -1)
                w = w + w.roll(self.V // 2, -1)
            if gate is not None:
                f = torch.sigmoid(gate[b].double())[:, None]
                o, w = o * f, w * f
            outs.append(o)
            sizes.append(w)
        return torch.stack(outs), torch.stack(sizes)


def launched(ops, monkeypatch):
    """The kernel's own calls (True where it took one)."""
    calls, real = [], type(ops)._attention_single
    monkeypatch.setattr(type(ops), "_attention_single", lambda self, *a: calls.append(real(self, *a)) or calls[-1])
    return calls


PLAIN = [([1, 15, 16, 17], 0), ([33, 160, 161, 320, 321], 0), ([700, 1, 2000], 4096), ([5000], 0), ([9, 2600], 30000), ([64] * 70, 0), ([40] * 40, 0)]


@pytest.mark.parametrize("lens,limit", PLAIN)
@pytest.mark.parametrize("H,KVH,D,page", [(14, 2, 64, 16), (12, 2, 128, 16), (3, 3, 64, 24), (16, 1, 128, 8), (9, 1, 64, 64), (5, 1, 128, 1)])
def test_plain(ops, monkeypatch, lens, limit, H, KVH, D, page):
    for window in (None, 100):
        c = Case(lens, H, KVH, D, D, page, limit=limit)
        calls = launched(ops, monkeypatch)
        qkv = torch.cat([c.q.flatten(1), torch.full((len(lens), 2 * KVH * D), float("nan"), device=DEV).bfloat16()], 1)
        out = torch.full((len(lens), H * D), float("nan"), device=DEV).bfloat16()
        ops.attention(out, qkv, c.k, c.v, c.tables, c.step, H, KVH, D, page, D ** -0.5, window)
        monkeypatch.undo()
        assert calls == ([True] if len(lens) * KVH <= ops.num_sms else [])
        want, size = c.want(D ** -0.5, window=window)
        err = (out.view(want.shape).double() - want).abs()
        assert bool((err <= 2.0 ** -8 * want.abs() + (2.0 ** -8 + 1e-4) * size).all())


OPTIONS = [dict(), dict(cap=30.0, slopes=True, window=1024), dict(window=50, keep=7), dict(window=90, keep=40, sinks=True), dict(chunk=64, gate=True),
           dict(cap=5.0, sinks=True, gate=True), dict(out_freq=True, slopes=True), dict(window=16)]


@pytest.mark.parametrize("options", OPTIONS, ids=lambda o: "-".join(o) or "none")
@pytest.mark.parametrize("lens,limit", [([1, 16, 17, 63, 64, 65], 0), ([500, 321, 40], 3000), ([2100], 0), ([30, 7] * 40, 0)])
@pytest.mark.parametrize("H,KVH,D,V,page", [(12, 2, 128, 128, 64), (6, 1, 64, 64, 16), (16, 1, 128, 128, 16), (12, 1, 576, 512, 64), (28, 1, 576, 512, 16),
                                            (17, 1, 576, 512, 8)])
def test_options(ops, monkeypatch, options, lens, limit, H, KVH, D, V, page):
    latent = D == 576
    if latent and "out_freq" in options:
        pytest.skip("the pairs of latent values are not turned")
    c = Case(lens, H, KVH, D, V, page, latent=latent, limit=limit)
    o = dict(options)
    for name in ("slopes", "sinks"):
        if name in o:
            o[name] = torch.rand(H, device=DEV) * (0.2 if name == "slopes" else 2.0)
    if "out_freq" in o:
        o["out_freq"] = torch.rand(V // 2, device=DEV) * 0.01
    if "gate" in o:
        o["gate"] = torch.randn(len(lens), H + 3, device=DEV).bfloat16()[:, :H]
    calls = launched(ops, monkeypatch)
    out = torch.full((len(lens), H, V + 8), float("nan"), device=DEV).bfloat16()[:, :, :V]
    scale = 192 ** -0.5 if latent else D ** -0.5
    ops.attention_biased(out, c.q, c.k, c.v, c.tables, c.step, KVH, page, scale, o.get("cap", 0.0), o.get("slopes"), o.get("window"),
                         o.get("chunk"), o.get("sinks"), o.get("keep", 0), o.get("out_freq"), o.get("gate"))
    monkeypatch.undo()
    assert calls == [True]
    want, size = c.want(scale, **o)
    err = (out.double() - want).abs()
    assert bool((err <= 2.0 ** -8 * want.abs() + (3e-4 if "out_freq" in o else 1e-4) * size + 1e-30).all())


def test_no_key_and_infinite_values(ops):
    """A request without keys gives zeros; an infinite value of a visible key reaches its own column and no other request."""
    H, KVH, D, page = 12, 2, 128, 16
    c = Case([40, 0, 350], H, KVH, D, D, page, limit=400)
    c.v[c.tables[2, 3], 0, 2, 5] = float("inf")                    # key 50, kv head 0, column 5
    qkv = torch.cat([c.q.flatten(1), torch.zeros(3, 2 * KVH * D, device=DEV).bfloat16()], 1)
    out = torch.full((3, H * D), float("nan"), device=DEV).bfloat16()
    ops.attention(out, qkv, c.k, c.v, c.tables, c.step, H, KVH, D, page, D ** -0.5, None)
    out = out.view(3, H, D)
    assert bool((out[1] == 0).all()) and bool(out[0].isfinite().all()) and bool(out[2, 6:].isfinite().all())
    assert bool((out[2, :6, 5] == float("inf")).all()) and bool(out[2, :6, :5].isfinite().all()) and bool(out[2, :6, 6:].isfinite().all())


def test_the_new_row_is_read_after_the_kernel_before(ops):
    """The newest key and value, written by a kernel of the same chain just before, are the ones that count."""
    H, KVH, D, page = 12, 2, 128, 16
    c = Case([33, 1, 160, 700], H, KVH, D, D, page)
    x, w = torch.randn(4, 256, device=DEV).bfloat16(), (torch.randn((H + 2 * KVH) * D, 256, device=DEV) * 0.1).bfloat16()
    pos, slots = i32([n - 1 for n in c.lens]), i32([int(c.tables[b, (n - 1) // page]) * page + (n - 1) % page for b, n in enumerate(c.lens)])
    cos, sin = torch.ones(800, D // 2, device=DEV), torch.zeros(800, D // 2, device=DEV)
    for _ in range(20):
        w = w.roll(1, 0).contiguous()
        torch.cuda.synchronize()
        out = torch.empty(4, H * D, device=DEV).bfloat16()
        qkv = ops.qkv_rope(torch.empty(4, w.shape[0], device=DEV).bfloat16(), x, w, None, pos, cos, sin, H, KVH, D, D, c.k, c.v, slots, page)
        ops.attention(out, qkv, c.k, c.v, c.tables, c.step, H, KVH, D, page, D ** -0.5, None)
        c.q = qkv[:, : H * D].reshape(4, H, D).clone()
        want, size = c.want(D ** -0.5)
        assert bool(((out.view(want.shape).double() - want).abs() <= 2.0 ** -8 * want.abs() + (2.0 ** -8 + 1e-4) * size).all())


@pytest.mark.parametrize("H,KVH,D,V,page", [(12, 2, 128, 128, 16), (6, 1, 64, 64, 16), (12, 1, 576, 512, 64), (28, 1, 576, 512, 16)])
def test_unsettled_steps_wait_for_every_row_and_array(ops, monkeypatch, H, KVH, D, V, page):
    """All rows of the cache and the lengths, written by kernels of the same chain just before (behind one that runs a while), are
    the ones that count with options and with latent rows."""
    c = Case([33, 1, 160, 700], H, KVH, D, V, page, latent=D == 576)
    caches = [t for t in (c.k, c.v) if t is not None]
    sources = [t.clone() for t in caches]
    rows = torch.arange(caches[0].numel() // D, device=DEV).int()
    x, w = (torch.zeros(n, 4096, device=DEV).bfloat16() for n in (64, 16384))
    product, lens, places = torch.empty(64, 16384, device=DEV).bfloat16(), c.step.seq_lens.clone(), i32([0, 1, 2, 3])
    scale = 192 ** -0.5 if D == 576 else D ** -0.5
    want, size = c.want(scale, cap=30.0, window=500)
    calls = launched(ops, monkeypatch)
    for _ in range(20):
        for t in caches:
            t.zero_()
        c.step.seq_lens.fill_(1)
        out = torch.full((4, H, V), float("nan"), device=DEV).bfloat16()
        torch.cuda.synchronize()
        ops.linear(product, x, w)
        ops.feed_tokens(c.step.seq_lens, places, places, lens, 1 << 20)
        for t, s in zip(caches, sources):
            ops.gather_rows(t.view(-1, t.shape[-1]), s.view(-1, t.shape[-1]), rows)
        ops.attention_biased(out, c.q, c.k, c.v, c.tables, c.step, KVH, page, scale, 30.0, None, 500)
        err = (out.double() - want).abs()
        assert bool((err <= 2.0 ** -8 * want.abs() + 1e-4 * size).all())
    assert calls == [True] * 20


@pytest.mark.parametrize("splits", [1, 3])
@pytest.mark.parametrize("H,KVH,D,V,page", [(12, 2, 128, 128, 64), (16, 1, 64, 64, 16), (12, 1, 576, 512, 64), (28, 1, 576, 512, 16)])
def test_a_number_of_splits_runs_the_kernel_that_splits(ops, monkeypatch, splits, H, KVH, D, V, page):
    c = Case([1, 64, 333, 2100, 700], H, KVH, D, V, page, latent=D == 576)
    monkeypatch.setattr(ops, "biased_decode_splits", splits)
    calls, took = launched(ops, monkeypatch), []
    real = ops.lib.ts_attention_biased_mma
    monkeypatch.setattr(ops.lib, "ts_attention_biased_mma", lambda *a: took.append(a[23]) or real(*a))
    sinks, gate = torch.rand(H, device=DEV), torch.randn(5, H, device=DEV).bfloat16()
    scale = 192 ** -0.5 if D == 576 else D ** -0.5
    for window, keep in ((None, 0), (500, 40)):
        out = torch.full((5, H, V), float("nan"), device=DEV).bfloat16()
        ops.attention_biased(out, c.q, c.k, c.v, c.tables, c.step, KVH, page, scale, 20.0, None, window, None, sinks, keep, None, gate)
        want, size = c.want(scale, cap=20.0, window=window, sinks=sinks, keep=keep, gate=gate)
        assert bool(((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4 * size).all())
    assert calls == [] and took == [splits, splits]


@pytest.mark.parametrize("H,KVH,D,page,lens,cluster", [(12, 2, 128, 24, [40000, 33000], True), (14, 2, 64, 24, [50000, 7], True),
                                                       (12, 2, 128, 24, [40000], False), (28, 4, 128, 24, [34001], True)])
def test_long_contexts_on_pages_that_the_streaming_kernel_does_not_take(ops, monkeypatch, H, KVH, D, page, lens, cluster):
    c = Case(lens, H, KVH, D, D, page)
    calls = launched(ops, monkeypatch)
    qkv = torch.cat([c.q.flatten(1), torch.zeros(len(lens), 2 * KVH * D, device=DEV).bfloat16()], 1)
    out = torch.full((len(lens), H * D), float("nan"), device=DEV).bfloat16()
    ops.attention(out, qkv, c.k, c.v, c.tables, c.step, H, KVH, D, page, D ** -0.5, None)
    assert calls == ([True] if cluster else [])
    want, size = c.want(D ** -0.5)
    assert bool(((out.view(want.shape).double() - want).abs() <= 2.0 ** -8 * want.abs() + (2.0 ** -8 + 1e-4) * size).all())
