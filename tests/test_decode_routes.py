"""Which kernel the front sends single tokens to and what it tells it, on the CPU: the library is a stand-in that notes
the calls and answers as the real one would by shape."""

from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

from tests import tiny
from tests.twin_ops import TwinOps
from turingserve_b200 import kernels
from turingserve_b200.kernels import CudaOps


class Library:
    """Every ``ts_...`` call is noted and returns 0, or what ``answers`` has for it (a value or a function of the arguments)."""

    def __init__(self, **answers) -> None:
        self.calls: list[tuple] = []
        self.answers = {"ts_attention_biased_mma_supported": 1, "ts_attention_biased_mma_chunk": lambda Dk, Dv, v: min(Dv, 256),
                        "ts_attention_biased_mma_scratch_floats": 16, "ts_attention_decode_scratch_floats": 16,
                        "ts_attention_decode_tma_supported": lambda H, KVH, D, page, code: int(page % 16 == 0),
                        "ts_attention_decode_supported": 1, "ts_attention_decode_tma_blocks_per_sm": 2, **answers}

    def __getattr__(self, name):
        if not name.startswith("ts_"):
            raise AttributeError(name)

        def call(*a):
            self.calls.append((name, a))
            r = self.answers.get(name, 0)
            return r(*a) if callable(r) else r
        return call

    def launched(self) -> list[str]:
        asked = ("supported", "chunk", "floats", "per_sm", "error")
        return [n for n, _ in self.calls if not n.endswith(asked)]

    def args(self, name):
        return [a for n, a in self.calls if n == name]


def front(**answers) -> CudaOps:
    ops = CudaOps.__new__(CudaOps)
    ops.lib = Library(**answers)
    ops.num_sms, ops.launches, ops.decode_stages = 148, 0, 3
    ops.decode_kernel, ops.use_fast_attention, ops.use_tc_attention, ops.use_tma_decode = "auto", True, True, True
    ops.single_mode, ops.biased_decode_splits = 1, 0
    ops._buffers, ops._outgrown, ops._decode_slots = {}, [], {}
    ops._stream = lambda: 0
    return ops


def step_of(lens, **more):
    i32 = lambda x: torch.tensor(x, dtype=torch.int32)
    return SimpleNamespace(q_start=i32(list(range(len(lens) + 1))), seq_lens=i32(lens), num_requests=len(lens), num_decode=len(lens),
                           max_q_len=1, max_seq_len=max(lens), **more)


def biased(ops, step, H=12, KVH=2, D=128, V=128, latent=False, page=16):
    B = step.num_requests
    k = torch.zeros(B + 1, KVH, page, D).bfloat16()
    ops.attention_biased(torch.zeros(B, H, V).bfloat16(), torch.zeros(B, H, D).bfloat16(), k, None if latent else k,
                         torch.zeros(B, 4, dtype=torch.int32), step, KVH, page, 0.1, 30.0, None, None)


def plain(ops, step, H=12, KVH=2, D=128, page=16):
    B = step.num_requests
    k = torch.zeros(B + 1, KVH, page, D).bfloat16()
    ops.attention(torch.zeros(B, H * D).bfloat16(), torch.zeros(B, (H + 2 * KVH) * D).bfloat16(), k, k, torch.zeros(B, 4, dtype=torch.int32),
                  step, H, KVH, D, page, 0.1, None)


EARLY = -2                     # the argument's place in ts_attention_single


@pytest.mark.parametrize("shape", [dict(), dict(H=12, KVH=1, D=576, V=512, latent=True)], ids=["options", "latent"])
def test_options_and_latent_rows_wait_unless_the_step_is_settled(shape):
    """A step built ahead of others that still run, or by hand, may follow kernels that still write its arrays or older rows."""
    for more, early in ((dict(), 0), (dict(settled=False), 0), (dict(settled=True), 1)):
        ops = front()
        biased(ops, step_of([40, 7], **more), **shape)
        assert ops.lib.launched() == ["ts_attention_single"]
        assert [a[EARLY] for a in ops.lib.args("ts_attention_single")] == [early]


def test_the_runner_settles_its_steps_and_the_builder_does_not(tmp_path):
    from turingserve_b200.cache import CacheManager
    from turingserve_b200.engine.batch import StepEntry
    from turingserve_b200.engine.runner import ModelRunner, _StepGraph, run_needs
    from turingserve_b200.weights.loader import load_model
    kernels.use(TwinOps())
    try:
        model, cfg = load_model(tiny.make_tiny_folder("A", tmp_path), torch.float32, "cpu")
        cache = CacheManager(run_needs(model), 16, 20, 4, torch.float32, "cpu")
        runner = ModelRunner(model, cache, 64, 4, 128)
        seen, real = [], runner.forward
        runner.forward = lambda step: seen.append(step.settled) or real(step)
        rc = cache.admit("a")
        with torch.inference_mode():
            runner.step([StepEntry(rc, tiny.random_ids(5, cfg.vocab_size, 1), [4])])
        assert seen == [True]
        cache.grow(rc, 1)
        assert not runner.builder.build([StepEntry(rc, [1], [0])]).settled
        assert _StepGraph(runner, 1, 0, False)._build([StepEntry(rc, [1], [0])]).settled
    finally:
        kernels.use(None)


def test_a_fault_of_the_streaming_kernel_takes_only_that_kernel_off():
    """Single tokens stay on the kernel that has no bounded wait; what the streaming kernel took goes to the older one."""
    ops = front()
    ops.fault_reported([0, 0, 7, 0])
    ops.lib.calls.clear()
    plain(ops, step_of([40, 7]))
    assert ops.lib.launched() == ["ts_attention_single"]
    ops.lib.calls.clear()
    plain(ops, step_of([40] * 100))                    # more (request, kv head) pairs than SMs
    assert ops.lib.launched() == ["ts_attention_decode"]
    for kernel in ("tma", "cp"):
        ops = front()
        ops.decode_kernel = kernel
        ops.fault_reported([0, 0, 7, 0])
        ops.lib.calls.clear()
        plain(ops, step_of([40, 7]))
        assert ops.lib.launched() == ["ts_attention_decode"]


@pytest.mark.parametrize("shape", [dict(), dict(H=12, KVH=1, D=576, V=512, latent=True)], ids=["options", "latent"])
def test_a_number_of_splits_is_for_the_kernel_that_splits(shape):
    for splits, name in ((0, "ts_attention_single"), (1, "ts_attention_biased_mma"), (3, "ts_attention_biased_mma")):
        ops = front()
        ops._buffer = lambda *a, **k: None
        ops.biased_decode_splits = splits
        biased(ops, step_of([700, 7]), **shape)
        assert ops.lib.launched() == [name]


def test_long_contexts_that_the_streaming_kernel_does_not_take():
    """Pages that are no multiple of 16, caches that no tensor map spans: clusters, or the older kernel for a pair or two."""
    single, tma, older = "ts_attention_single", "ts_attention_decode_tma", "ts_attention_decode"
    for lens, KVH, page, answer, want in (
            ([16000] * 8, 2, 16, 0, [tma]), ([16000] * 8, 2, 24, 0, [single]), ([16000] * 8, 2, 16, CudaOps.UNSUPPORTED, [tma, single]),
            ([64000], 2, 16, 0, [tma]), ([64000], 2, 24, 0, [older]), ([64000], 2, 16, CudaOps.UNSUPPORTED, [tma, older]),
            ([64000], 4, 24, 0, [single]), ([300] * 8, 2, 24, 0, [single]),
            ([300] * 100, 2, 24, 0, [older]), ([300] * 100, 2, 16, CudaOps.UNSUPPORTED, [tma, older])):
        ops = front(ts_attention_decode_tma=answer)
        ops._buffer = lambda *a, **k: None
        plain(ops, step_of(lens), KVH=KVH, page=page)
        assert ops.lib.launched() == want, (lens, KVH, page, answer)


def test_the_front_and_the_steps_share_the_threshold(monkeypatch):
    from turingserve_b200.engine import batch
    for keys, want in ((1000, "ts_attention_single"), (120, "ts_attention_decode_tma")):
        monkeypatch.setattr(batch, "STREAMING_DECODE_KEYS", keys)
        ops = front()
        ops._buffer = lambda *a, **k: None
        plain(ops, step_of([40, 40, 40]))
        assert ops.lib.launched() == [want]
