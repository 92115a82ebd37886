"""The experts' products on pairs of SMs over rows sorted by expert: groups of every size around a tile's 128 and 256 rows, none
among them, widths that are no multiple of a tile's, rows behind the last expert's that must stay; and the sum of choices.

Bounds: bfloat16 operands of size 1 and K^-1/2, 32-bit sums: 1e-5 of an element of size 1; bfloat16 results: 2^-8."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
GROUPS = [[300, 0, 1, 127, 128, 129, 256, 257], [0, 0, 5], [512], [1] * 40, [0, 700, 3, 0]]


@pytest.fixture(scope="module")
def ops():
    from turingserve_b200 import kernels
    return kernels.ops()


@pytest.mark.parametrize("groups", GROUPS)
@pytest.mark.parametrize("N,K", [(264, 72), (512, 200), (1536, 64), (8, 8)])
def test_products_of_sorted_rows(ops, groups, N, K):
    g = torch.Generator(device=DEV).manual_seed(N + K + len(groups))
    E, P, behind = len(groups), sum(groups), 9
    offsets = torch.tensor([sum(groups[:e]) for e in range(E + 1)], dtype=torch.int32, device=DEV)
    x = torch.randn(P + behind, K, generator=g, device=DEV).bfloat16()
    w = (torch.randn(E, N, K, generator=g, device=DEV) * K ** -0.5).bfloat16()
    assert ops.grouped_pair_takes(x, w, torch.empty(E, K, N, dtype=w.dtype, device=DEV), 1 << 20)
    want = torch.cat([x[sum(groups[:e]):sum(groups[:e + 1])].double() @ w[e].double().T for e in range(E)])
    act = {"none": lambda z: z, "gelu": torch.nn.functional.gelu, "silu": torch.nn.functional.silu, "relu2": lambda z: torch.relu(z) ** 2}
    out = torch.full((P + behind, N), 7.0, device=DEV)
    ops.grouped_pair(out, x, w, offsets)
    assert torch.allclose(out[:P].double(), want, rtol=1e-5, atol=1e-5) and bool((out[P:] == 7.0).all())
    for kind, fn in act.items():
        out = torch.full((P + behind, N), 7.0, device=DEV).bfloat16()
        ops.grouped_pair(out, x, w, offsets, kind)
        assert torch.allclose(out[:P].double(), fn(want), rtol=2 ** -6, atol=2 ** -7), kind     # (rounded before and after)
        assert bool((out[P:] == 7.0).all())
    out = torch.full((P + behind, N // 2), 7.0, device=DEV).bfloat16()
    ops.grouped_pair(out, x, w, offsets, "none", (1.5, 1.7, 1.0))
    gate, up = want[:, 0::2].clamp(max=1.5), want[:, 1::2].clamp(-1.5, 1.5)
    assert torch.allclose(out[:P].double(), gate * torch.sigmoid(1.7 * gate) * (up + 1.0), rtol=2 ** -6, atol=2 ** -6)
    assert bool((out[P:] == 7.0).all()) and ops.tc_status() == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,top,N", [(5, 2, 1536), (3, 8, 4), (7, 1, 1028), (4, 9, 64), (6, 3, 30)])
def test_sum_of_choices(ops, dtype, T, top, N):
    """Widths and choices inside and outside of what four columns a thread takes; every option at once and none."""
    g = torch.Generator(device=DEV).manual_seed(T * top + N)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    P = T * top
    y, place = rnd(P, N), torch.randperm(P, generator=g, device=DEV).int()
    weights, x, add, share = rnd(T, top), rnd(T, N).to(dtype), rnd(T, N).to(dtype), rnd(T)
    first = P * 2 // 3
    for opt in (False, True):
        out = torch.empty(T, N, dtype=dtype, device=DEV)
        extra = dict(x=x, pass_from=torch.tensor([first], dtype=torch.int32, device=DEV), add=add, share=share) if opt else {}
        ops.moe_combine(out, y, place, weights if opt else None, top, **extra)
        rows = y.double()[place.long()].view(T, top, N)
        if opt:
            rows = torch.where((place >= first).view(T, top, 1), x.double()[:, None], rows) * weights.double()[..., None]
        want = rows.sum(1) + (share.double()[:, None] * add.double() if opt else 0)
        assert torch.allclose(out.double(), want, rtol=2 ** -8 if dtype == torch.bfloat16 else 1e-5, atol=1e-4)


def test_activations_of_products_are_those_of_the_activation_kernel(ops):
    """Every bfloat16 value from -12 to 12 through the epilogue's activations: the same bits as the activation kernel gives the
    product; GELU, whose error function is one without branches there, is off the correctly rounded value no oftener than the
    32-bit error function and by no more than a rounding and 2^-15 of itself down to where the result leaves 32-bit."""
    z = torch.arange(1 << 16, dtype=torch.int32, device=DEV).to(torch.int16).view(torch.bfloat16)
    z = z[z.float().abs() <= 12].contiguous()
    P = z.numel()
    x = torch.zeros(P, 8, dtype=z.dtype, device=DEV)
    x[:, 0] = z
    w = torch.ones(1, 8, 8, dtype=z.dtype, device=DEV)
    offsets = torch.tensor([0, P], dtype=torch.int32, device=DEV)
    for kind in ("none", "gelu_tanh", "relu2", "silu", "gelu"):
        out, want = torch.empty_like(x), torch.empty_like(z)
        ops.grouped_pair(out, x, w, offsets, kind)
        assert torch.equal(out, out[:, :1].expand(P, 8))
        ops.activation(want, z, kind) if kind != "none" else want.copy_(z)
        if kind != "gelu":
            assert torch.equal(out[:, 0], want), kind
            continue
        true = 0.5 * z.double() * torch.special.erfc(-z.double() / 2 ** 0.5)
        nearest = true.float().bfloat16()
        assert int((out[:, 0] != nearest).sum()) <= int((want != nearest).sum())
        assert bool(((out[:, 0].double() - true).abs() <= (2.0 ** -8 + 2.0 ** -15) * true.abs() + 1e-37).all())
    assert ops.tc_status() == 0



def test_refused_launches_go_to_the_older_kernels(ops, monkeypatch):
    """Where the device refuses the products on pairs (at the first or at the second) the feed-forward takes the way it had."""
    from turingserve_b200.models import gugezen
    from turingserve_b200.parts.base import BuildContext, build
    mixer = {"type": "mamba2", "mixer": {"heads": 4, "vdim": 16, "state": 16, "groups": 1, "conv": 4, "norm_groups": 1}}
    mlp = {"kind": "moe", "expert": {"ff": 72}, "router": {"experts": 4, "top": 2}, "shared": {"ff": 32}}
    cfg = gugezen.make_config(width=64, vocab=64, layers=[{**mixer, "mlp": mlp}], eps=1e-6, streams=2)
    part = build("feed_forward", cfg.layers[0].feed_forward,
                 BuildContext(hidden_size=64, dtype=torch.bfloat16, device=torch.device(DEV, 0), max_positions=64))
    g = torch.Generator(device=DEV).manual_seed(3)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV) * 0.1
    w = {"router": rnd(4, 64), "shared.up": rnd(32, 64).bfloat16(), "shared.down": rnd(64, 32).bfloat16()}
    for e in range(4):
        w[f"e{e}.up"], w[f"e{e}.down"] = rnd(72, 64).bfloat16(), rnd(64, 72).bfloat16()
    part.load(w)
    real = ops.lib
    for T in (90, 700):                                    # the grouped kernels, a product an expert
        x = rnd(T, 64).mul(10).bfloat16()
        assert ops.grouped_pair_takes(x, part.w_up, part.w_down, 2 * T)
        want = ops.materialize(part.forward(x)).clone()
        for refused_from in (0, 1):
            class Lib:
                calls = 0

                def __getattr__(self, name):
                    return getattr(real, name)

                def ts_grouped_pair(self, *args):
                    Lib.calls += 1
                    return ops.UNSUPPORTED if Lib.calls > refused_from else real.ts_grouped_pair(*args)

            with monkeypatch.context() as m:
                m.setattr(ops, "lib", Lib())
                got = ops.materialize(part.forward(x))
            assert Lib.calls == refused_from + 1
            assert torch.allclose(got.double(), want.double(), rtol=2 ** -6, atol=2 ** -6 * float(want.abs().max()))
