"""The few-token products whose weights pass through registers: every instance at ragged sizes (rows that are no multiple of
a tile, K of 8 to a few thousand, 1 to 16 tokens) against the product in 64 bits, and what finishes itself against the
product followed by the kernel that would.

Bound: 32-bit sums of exact products of bfloat16 values; K roundings of partial sums of at most the sum of magnitudes:
2^-24 sqrt(K) of it with chance signs, 4e-6 of an output's size for K of 5,000; 2e-5 with margin."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
PLANS = range(1, 10)


@pytest.fixture(scope="module")
def ops():
    from turingserve_b200 import kernels
    return kernels.ops()


def rnd(seed, *shape, std=1.0):
    return (torch.randn(*shape, generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV) * std).bfloat16()


@pytest.mark.parametrize("plan", PLANS)
@pytest.mark.parametrize("N,K", [(1, 8), (33, 40), (200, 72), (1001, 1000), (2400, 1536), (130, 4504), (19000, 264)])
def test_plans_against_64_bits(ops, monkeypatch, plan, N, K):
    monkeypatch.setattr(ops, "few_plan", plan)
    w, b = rnd(1, N, K, std=0.05), rnd(2, N)
    for M in (1, 7, 8, 9, 16):
        x = rnd(M, M, K)
        want = x.double() @ w.double().T
        size = (x.double().abs() @ w.double().abs().T).clamp_min(1e-3)
        out = torch.full((M, N), float("nan"), device=DEV)
        assert ops._few(out, x, w, None, M, N, K, ops.FEW_FLOAT)
        assert float(((out - want).abs() / size).max()) < 2e-5
        out = torch.full((M * N + 1,), float("nan"), device=DEV)[1:].view(M, N)         # (off the boundary of two floats)
        assert ops._few(out, x, w, b, M, N, K, ops.FEW_FLOAT)
        assert float(((out - want - b.double()).abs() / (size + b.double().abs())).max()) < 2e-5
        half = torch.full((M, N), float("nan"), device=DEV).bfloat16()
        assert ops._few(half, x, w, b, M, N, K, ops.FEW_BF16)
        assert torch.equal(half, out.bfloat16())
        old = rnd(3, M, N)
        resid = old.clone()
        assert ops._few(resid, x, w, b, M, N, K, ops.FEW_RESID)
        assert torch.equal(resid, (half.float() + old.float()).bfloat16())


@pytest.mark.parametrize("plan", PLANS)
@pytest.mark.parametrize("inter,K", [(64, 8), (448, 904), (2432, 264)])
def test_gated(ops, monkeypatch, plan, inter, K):
    monkeypatch.setattr(ops, "few_plan", plan)
    w = rnd(1, 2 * inter, K, std=0.05)
    for M in (1, 8, 13, 16):
        x, act, two, gu = rnd(M, M, K), *(torch.full((M, n), float("nan"), device=DEV).bfloat16() for n in (inter, inter, 2 * inter))
        assert ops._few(act, x, w, None, M, 2 * inter, K, ops.FEW_GATED) and ops._few(gu, x, w, None, M, 2 * inter, K, ops.FEW_BF16)
        ops.silu_mul(two, gu, 64)
        assert torch.equal(act, two)


@pytest.mark.parametrize("plan", PLANS)
@pytest.mark.parametrize("H,KVH,D,K", [(12, 2, 128, 1536), (3, 3, 64, 328), (5, 1, 64, 72)])
def test_rotation_and_cache_write(ops, monkeypatch, plan, H, KVH, D, K):
    N, page = (H + 2 * KVH) * D, 16
    monkeypatch.setattr(ops, "pair_wins", lambda *a: False)       # (the many-row kernel sums in another order)
    w, b = rnd(1, N, K, std=0.05), rnd(2, N)
    cos, sin = (torch.rand(50, D // 2, device=DEV) for _ in range(2))
    for M in (1, 8, 16):
        x, slots = rnd(M, M, K), torch.randperm(60, device=DEV)[:M].int()
        slots[M // 2] = -1
        pos, got = torch.randint(0, 50, (M,), device=DEV).int(), []
        for fused in (64, 0):
            monkeypatch.setattr(ops, "few_plan", plan)
            monkeypatch.setattr(ops, "fused_qkv_tokens", fused)
            k, v = (torch.zeros(4, KVH, page, D, device=DEV).bfloat16() for _ in range(2))
            q = torch.full((M, N), float("nan"), device=DEV).bfloat16()
            q = ops.qkv_rope(q, x, w, b, pos, cos, sin, H, KVH, D, D, k, v, slots, page)
            got.append((q.clone(), k, v))
        assert all(torch.equal(a, c) for a, c in zip(*got))


@pytest.mark.parametrize("plan", PLANS)
@pytest.mark.parametrize("N,K", [(40, 8), (130, 200), (2051, 1536), (9728, 896)])
def test_stream_and_activation(ops, monkeypatch, plan, N, K):
    """Sums into 32-bit rows and activations: the bits of product, then kernel."""
    monkeypatch.setattr(ops, "few_plan", plan)
    w, b = rnd(1, N, K, std=0.05), rnd(2, N)
    for M in (1, 8, 13, 16):
        x, half = rnd(M, M, K), torch.empty(M, N, device=DEV).bfloat16()
        assert ops._few(half, x, w, b, M, N, K, ops.FEW_BF16)
        old = rnd(3, M, N).float() * 1.1
        stream = old.clone()
        assert ops._few(stream, x, w, b, M, N, K, ops.FEW_STREAM)
        assert torch.equal(stream, old + half.float())
        for code in (1, 2, 3, 4):
            got, want, part = torch.empty_like(half), torch.empty_like(half), torch.empty(1, M, N, device=DEV)
            assert ops._few(got, x, w, b, M, N, K, ops.FEW_ACT, code) and ops._few(part, x, w, None, M, N, K, ops.FEW_FLOAT)
            ops._check(ops.lib.ts_activation_parts(want.data_ptr(), part.data_ptr(), 1, b.data_ptr(), M, N, code, 1, ops._stream()), "activation_parts")
            assert torch.equal(got, want)


def test_infinite_values_stay_with_their_token_and_row(ops, monkeypatch):
    for plan in PLANS:
        monkeypatch.setattr(ops, "few_plan", plan)
        x, w = rnd(1, 5, 200).abs(), rnd(2, 90, 200).abs()
        x[3, 77], w[40, 10] = float("inf"), float("nan")
        out = torch.empty(5, 90, device=DEV)
        assert ops._few(out, x, w, None, 5, 90, 200, ops.FEW_FLOAT)
        rows = [n for n in range(90) if n != 40]
        assert bool(out[:, 40].isnan().all()) and bool((out[3, rows] == float("inf")).all())
        assert bool(out[[0, 1, 2, 4]][:, rows].isfinite().all())


def test_sizes_left_to_tcgen05(ops):
    x, w, out = rnd(1, 3, 8968), rnd(2, 3584, 8968), torch.empty(3, 3584, device=DEV)
    assert not ops._few(out, x, w, None, 3, 3584, 8968, ops.FEW_FLOAT)
    ops.linear(out, x, w)
    assert float((out - (x.double() @ w.double().T)).abs().max()) < 2e-5 * 8968


# (which kernel is the faster one was measured with the residual add and norm, the rotation and plainly; the sizes lie on both
# sides of each line of the rule)
@pytest.mark.parametrize("M,N,K,taken", [(1, 2048, 18432, True), (16, 1536, 20480, False), (8, 256, 28416, False), (16, 1536, 16384, True), (12, 2432, 8192, False), (8, 2432, 8192, True),
                                         (8, 2816, 7168, True), (12, 2816, 7168, False), (12, 2560, 7168, True), (12, 3072, 7168, True), (1, 2816, 8192, False),
                                         (1, 4736, 5120, True), (1, 4752, 5120, False), (8, 5120, 3584, True), (1, 5120, 4352, False), (8, 5120, 5120, False), (9, 5120, 1536, True),
                                         (9, 5120, 2048, False), (1, 5632, 7168, False), (8, 6144, 6144, True), (8, 6144, 8192, False), (8, 7168, 8192, True)])
def test_which_sizes_are_left_to_tcgen05(ops, M, N, K, taken):
    x, w, out = rnd(1, M, K), rnd(2, N, K, std=0.05), torch.empty(M, N, device=DEV)
    assert ops._few(out, x, w, None, M, N, K, ops.FEW_FLOAT) == taken
    ops.linear(out, x, w)
    size = (x.double().abs() @ w.double().abs().T).clamp_min(1e-3)
    assert float(((out - x.double() @ w.double().T).abs() / size).max()) < 2e-5


# (N, K): on both sides of the rule's lines, and whether the rule takes them at up to 8 and up to 16 tokens
FRONT = [(1536, 1536, True, True), (896, 4864, True, True), (136, 200, True, True), (264, 18944, False, False), (2816, 7168, True, False),
         (5120, 1536, True, True), (5120, 2048, True, False), (5120, 5120, False, False), (7168, 2048, True, False)]


def put_off(ops, M, N, K, few, monkeypatch):
    """(a product of few tokens not launched yet, its 64-bit value, the sum of magnitudes, whether few-token calls took it)."""
    from turingserve_b200.kernels import LazyProduct
    monkeypatch.setattr(ops, "few_tokens", few)
    x, w, b = rnd(1, M, K), rnd(2, N, K, std=0.05), rnd(3, N)
    p = ops.linear(torch.full((M, N), float("nan"), device=DEV).bfloat16(), x, w, b, may_defer=True)
    assert isinstance(p, LazyProduct)
    took, real = [], type(ops)._few
    monkeypatch.setattr(type(ops), "_few", lambda self, *a: took.append(real(self, *a)) or took[-1])
    return p, x.double() @ w.double().T + b.double(), x.double().abs() @ w.double().abs().T + b.double().abs(), took


@pytest.mark.parametrize("few", [16, 0])
@pytest.mark.parametrize("M", [1, 8, 9, 16])
@pytest.mark.parametrize("N,K,to8,to16", FRONT)
@pytest.mark.parametrize("form", ["norm", "layer_norm", "row", "row_layer_norm", "sum", "row_sum"])
def test_norm_of_a_stream_that_gets_a_product(ops, monkeypatch, few, M, N, K, to8, to16, form):
    """stream += product (rounded to bfloat16) + row, then its norm: the route by size, and either kernel's result against 64 bits."""
    p, want, size, took = put_off(ops, M, N, K, few, monkeypatch)
    old = torch.randn(M, N, device=DEV) * 3
    row = torch.randn(N, device=DEV) if "row" in form else None
    weight, bias = torch.rand(N, device=DEV) + 0.5, torch.randn(N, device=DEV) if "layer_norm" in form else None
    out = None if "sum" in form else torch.full((M, N), float("nan"), device=DEV).bfloat16()
    stream = old.clone()
    ops.rmsnorm_stream(out, stream, p, None, weight, 1e-6, row=row, norm_bias=bias)
    fused = [few > 0 and (to8 if M <= 8 else to16)]
    assert any(took) == fused[0]
    total = old.double() + want + (0 if row is None else row.double())
    # (the product's rounding to bfloat16, its 32-bit sum, and two sums in 32 bits)
    assert bool(((stream - total).abs() <= 2.0 ** -8 * want.abs() + 2e-5 * size + 2.0 ** -22 * (old.double().abs() + total.abs())).all())
    if out is None:
        return
    s = stream.double()
    mean = s.mean(-1, keepdim=True) if bias is not None else 0.0
    y = (s - mean) / torch.sqrt((s - mean).pow(2).mean(-1, keepdim=True) + 1e-6) * weight.double() + (0.0 if bias is None else bias.double())
    assert bool(((out.double() - y).abs() <= 2.0 ** -8 * y.abs() + 1e-5 * (weight * 4 + 1)).all())


@pytest.mark.parametrize("few", [16, 0])
@pytest.mark.parametrize("M", [1, 8, 9, 16])
@pytest.mark.parametrize("N,K,to8,to16", FRONT)
@pytest.mark.parametrize("kind", ["gelu_tanh", "relu2", "silu", "gelu"])
def test_activation_that_gets_a_product(ops, monkeypatch, few, M, N, K, to8, to16, kind):
    p, want, size, took = put_off(ops, M, N, K, few, monkeypatch)
    ops.activation(p.out, p, kind)
    assert any(took) == (few > 0 and (to8 if M <= 8 else to16))
    act = {"gelu_tanh": lambda v: torch.nn.functional.gelu(v, approximate="tanh"), "relu2": lambda v: v.relu() ** 2,
           "silu": torch.nn.functional.silu, "gelu": torch.nn.functional.gelu}[kind]
    # what a difference of the product makes of the activation: its slope is at most 1.13, relu2's 2 |v|
    off = 2.0 ** -8 * want.abs() + 2e-5 * size
    slope = 2 * want.abs() + off if kind == "relu2" else 1.13
    y = act(want)
    assert bool(((p.out.double() - y).abs() <= 2.0 ** -8 * (y.abs() + slope * off) + slope * off + 1e-6).all())


@pytest.mark.parametrize("plan", PLANS)
def test_tokens_bias_and_residual_are_read_after_the_kernels_before(ops, monkeypatch, plan):
    """What kernels of the same chain have just written (behind one that runs a while) is what counts; the weights alone are fetched early."""
    M, N, K = 8, 2048, 1024
    monkeypatch.setattr(ops, "few_plan", plan)
    w, new = rnd(1, N, K, std=0.05), [rnd(2, M, K), rnd(3, 1, N), rnd(4, M, N)]
    long_x, long_w, long_out = (torch.zeros(*s, device=DEV).bfloat16() for s in ((64, 4096), (16384, 4096), (64, 16384)))
    rows = torch.arange(M, device=DEV).int()
    half = (new[0].double() @ w.double().T + new[1].double()).float().bfloat16().float()
    for _ in range(10):
        x, b, resid = (torch.zeros_like(t) for t in new)
        torch.cuda.synchronize()
        ops.linear(long_out, long_x, long_w)
        for to, t in zip((x, b, resid), new):
            ops.gather_rows(to, t, rows[: t.shape[0]])
        assert ops._few(resid, x, w, b.view(-1), M, N, K, ops.FEW_RESID)
        err = (resid.float() - half - new[2].float()).abs()
        assert bool((err <= 2.0 ** -7 * (half.abs() + new[2].float().abs()) + 1e-3).all())
