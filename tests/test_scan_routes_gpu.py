"""The kernel that a short portion's scan goes to takes no longer than the one it would go to if its length were not known (or
one token less): device times of captured launches, the best of several, because the kernels differ by 10 to 50 % there and give
the same bits, so nothing else would show a rule that lies in the wrong place."""

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


def step_of(lens, known=True):
    return SimpleNamespace(q_start=i32([sum(lens[:k]) for k in range(len(lens) + 1)]), state_slots=i32(list(range(len(lens)))),
                           num_requests=len(lens), max_q_len=max(lens) if known else 0,
                           token_request=i32([k for k, n in enumerate(lens) for _ in range(n)]))


def device_us(*calls):
    """The least time of each call, taken in turn."""
    graphs = []
    for fn in calls:
        fn()
        torch.cuda.synchronize()
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1]):
            for _ in range(10):
                fn()
    best = [float("inf")] * len(calls)
    for _ in range(12):
        for i, g in enumerate(graphs):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(5):
                g.replay()
            b.record()
            b.synchronize()
            best[i] = min(best[i], a.elapsed_time(b) * 1e3 / 50)
    return best


@pytest.mark.parametrize("H,D,V,lens", [(6, 128, 128, [127]), (6, 128, 128, [256]), (6, 128, 128, [383] * 6), (6, 64, 64, [100]),
                                        (6, 64, 64, [1] * 8 + [300])])
def test_linear_attention_portions(ops, H, D, V, lens):
    T = sum(lens)
    proj, out = torch.randn(T, H * (2 * D + V), device=DEV).bfloat16(), torch.empty(T, H * V, device=DEV)
    state, decay = torch.zeros(len(lens), H, D, V, device=DEV), torch.full((H,), 0.9, device=DEV)
    known, unknown = device_us(*(lambda s=s: ops.lightning(out, proj, state, decay, s, H, D, V) for s in (step_of(lens), step_of(lens, False))))
    assert known < 0.96 * unknown, (known, unknown)



@pytest.mark.parametrize("H,P,N,lens", [(112, 64, 128, [64]), (112, 64, 128, [96]), (48, 64, 128, [64]), (48, 64, 64, [100]),
                                        (32, 64, 16, [1] * 8 + [100])])
def test_state_space_portions(ops, H, P, N, lens):
    G, taps, T = 2, 4, sum(lens)
    inner = H * P
    channels = inner + 2 * G * N
    ready, out = torch.rand(T, channels + 2 * H, device=DEV), torch.empty(T, inner, device=DEV)
    proj = torch.randn(T, 2 * inner + 2 * G * N + H, device=DEV).bfloat16()
    state, skip = torch.zeros(len(lens), H * N * P + 3 * channels, device=DEV), torch.ones(H, device=DEV)
    known, unknown = device_us(*(lambda s=s: ops.ssm_scan(out, ready, proj, inner, state, skip, s, H, G, N, P, taps)
                                 for s in (step_of(lens), step_of(lens, False))))
    assert known < 1.03 * unknown, (known, unknown)


@pytest.mark.parametrize("H,G,lens", [(12, 6, [64]), (12, 6, [128]), (12, 6, [1] * 32 + [64]), (28, 14, [1] * 8 + [56]), (28, 14, [512])])
def test_delta_rule_preparation(ops, H, G, lens):
    """Beside filters off their 16-byte boundary, which go to the kernel for any sizes."""
    D, V, taps, T = 128, 128, 4, sum(lens)
    C = 2 * G * D + H * V
    width = C + 2 * H + G
    ready = torch.empty_strided((T, width), (width + -width % 4, 1), dtype=torch.float32, device=DEV)
    proj, state = torch.randn(T, C + H * V + 2 * H, device=DEV).bfloat16(), torch.zeros(len(lens), H * D * V + 3 * C, device=DEV)
    step, a_log, dt = step_of(lens), torch.rand(H, device=DEV), torch.rand(H, device=DEV)
    room = torch.rand(C * taps + 4, device=DEV)
    chosen, general = device_us(*(lambda w=room[k:k + C * taps].view(C, taps): ops.delta_prepare(
        ready, proj, w, a_log, dt, state, step, H, G, D, V, taps, 1e-6) for k in (0, 1)))
    assert chosen < 1.04 * general, (chosen, general)


def test_many_short_requests_of_few_rows(ops, monkeypatch):
    """The attention with options: more single tokens than SMs, 48 heads over one kv head, 140 keys each."""
    B, H, D, page, keys = 256, 48, 128, 64, 140
    per = -(-keys // page)
    k, v = (torch.randn(B * per, 1, page, D, device=DEV).bfloat16() for _ in range(2))
    tables = torch.arange(B * per, dtype=torch.int32, device=DEV).view(B, per)
    step = SimpleNamespace(q_start=i32(list(range(B + 1))), seq_lens=i32([keys] * B), num_requests=B, num_decode=B, max_q_len=1, max_seq_len=keys)
    q, out = torch.randn(B, H, D, device=DEV).bfloat16(), torch.empty(B, H, D, device=DEV).bfloat16()

    def attend(least):
        monkeypatch.setattr(ops, "biased_tc_keys", least)
        ops.attention_biased(out, q, k, v, tables, step, 1, page, D ** -0.5, 0.0, None, None)

    chosen, other = device_us(lambda: attend(128), lambda: attend(1 << 30))
    assert chosen < 1.04 * other, (chosen, other)


@pytest.mark.parametrize("H,G,D,T", [(8, 1, 64, 8), (64, 8, 128, 8)])
def test_turned_pairs(ops, H, G, D, T):
    """Beside rows off their 16-byte boundary, which go to the kernel for any sizes."""
    pos, freq = torch.arange(T, dtype=torch.int32, device=DEV), torch.rand(D // 2, device=DEV)
    k, v = (torch.zeros(1, G, 64, D, device=DEV).bfloat16() for _ in range(2))
    room = torch.randn(T * (H + 2 * G) * D + 1, device=DEV).bfloat16()
    chosen, general = device_us(*(lambda p=room[i:i + T * (H + 2 * G) * D].view(T, -1): ops.rope_pairs_write(
        p, H * D, (H + G) * D, pos, freq, 1.0, D, k, v, pos, H, G, D, D, 64) for i in (0, 1)))
    assert chosen < 1.06 * general, (chosen, general)
