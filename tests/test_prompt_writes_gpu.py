"""What sits between a projection and its attention, with 16-byte loads: whole-row norms, latent rows and turned pairs at the
edges of their lanes (one vector, a full turn of the warp and one more, the widest), strides wider than the row, slots of -1; rows
that start off a 16-byte boundary go to the any-size kernels and must give the same; and the router's logits of many tokens, which
are the same bits as of a few.

Bounds: 32-bit arithmetic and one rounding to bfloat16, 2^-8 of the value; angles of up to 3,000 in 32 bits, 3,000 * 2^-24 of a
rotated value of size 8 beside it."""

import pytest
import torch

from tests.twin_ops import TwinOps

pytestmark = pytest.mark.gpu
DEV = "cuda"
TOL = dict(rtol=2 ** -7, atol=2e-3)


@pytest.fixture(scope="module")
def ops():
    from turingserve_b200 import kernels
    return kernels.ops()


def rows(T, n, seed, extra=0, off=0):
    """[T, n] bfloat16 rows ``extra`` apart, starting ``off`` elements behind a 16-byte boundary."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    flat = torch.zeros(T * (n + extra) + off + 8, dtype=torch.bfloat16, device=DEV)
    view = flat[off:off + T * (n + extra)].view(T, n + extra)[:, :n]
    view.copy_(torch.randn(T, n, generator=g, device=DEV) * 2)
    return view


def slots_of(T, pages, page, seed):
    s = torch.randperm(pages * page, generator=torch.Generator().manual_seed(seed))[:T].to(torch.int32)
    if T > 2:
        s[T // 2] = -1
    return s.to(DEV)


@pytest.mark.parametrize("T", [1, 5, 130])
@pytest.mark.parametrize("H,G,D", [(1, 1, 8), (4, 1, 64), (33, 3, 8), (28, 4, 128), (32, 8, 128), (16, 2, 136)])
@pytest.mark.parametrize("extra,off", [(0, 0), (8, 0), (0, 1)])
def test_whole_row_norms(ops, T, H, G, D, extra, off):
    page, pages, n = 16, 10, (H + G) * D
    proj, other = rows(T, n, T + n, extra, off), rows(T, n, T + n)
    q_w, k_w = torch.rand(H * D, device=DEV) + 0.5, torch.rand(G * D, device=DEV) + 0.5
    pos = torch.randint(0, 3000, (T,), dtype=torch.int32, device=DEV)
    slots = slots_of(T, pages, page, T)
    caches = [torch.full((pages, G, page, D), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(4)]
    ops.qk_rownorm_write(proj, q_w, k_w, 1e-6, pos, 0.35, 5, caches[0], caches[1], slots, H, G, D, page)
    TwinOps().qk_rownorm_write(other, q_w, k_w, 1e-6, pos, 0.35, 5, caches[2], caches[3], slots, H, G, D, page)
    assert torch.allclose(proj.float(), other.float(), **TOL)
    assert torch.allclose(caches[0].float(), caches[2].float(), **TOL) and torch.equal(caches[1], caches[3])
    again = rows(T, n, T + n)
    ops.qk_rownorm_write(again, q_w, k_w, 1e-6, pos, 0.0, 1, None, None, None, H, G, D, page)
    other = rows(T, n, T + n)
    TwinOps().qk_rownorm_write(other, q_w, k_w, 1e-6, pos, 0.0, 1, None, None, None, H, G, D, page)
    assert torch.allclose(again.float(), other.float(), **TOL)


@pytest.mark.parametrize("T", [1, 5, 130])
@pytest.mark.parametrize("pairing", ["neighbours", "halves"])
@pytest.mark.parametrize("q_rank,rank,R,rot", [(8, 8, 8, 8), (264, 256, 16, 6), (768, 512, 64, 64), (2048, 2048, 72, 66), (2056, 512, 64, 64)])
@pytest.mark.parametrize("extra,off", [(0, 0), (8, 0), (0, 1)])
def test_latent_rows(ops, T, pairing, q_rank, rank, R, rot, extra, off):
    page, pages = 16, 10
    proj = rows(T, q_rank + rank + R, T + rank, extra, off)
    w, q_w = torch.rand(rank, device=DEV) + 0.5, torch.rand(q_rank, device=DEV) + 0.5
    freq = 1.0 / 50.0 ** (torch.arange(0, rot, 2, device=DEV).float() / rot)
    pos = torch.randint(0, 3000, (T,), dtype=torch.int32, device=DEV)
    slots = slots_of(T, pages, page, T)
    pools = [torch.full((pages, 1, page, rank + R), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    cqs = [torch.empty(T, q_rank, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    for o, pool, cq in ((ops, pools[0], cqs[0]), (TwinOps(), pools[1], cqs[1])):
        o.latent_kv_write(proj, q_rank, w, 1e-6, pos, freq, 1.3, rot, pool, slots, rank, R, page, pairing, cq, q_w)
    assert torch.allclose(pools[0].float(), pools[1].float(), **TOL) and torch.allclose(cqs[0].float(), cqs[1].float(), **TOL)


@pytest.mark.parametrize("T", [1, 5, 130])
@pytest.mark.parametrize("H,G,D,V,rot", [(1, 1, 8, 8, 8), (12, 2, 128, 128, 128), (28, 4, 128, 64, 64), (5, 3, 24, 16, 8), (4, 2, 64, 64, 0)])
@pytest.mark.parametrize("extra,off", [(0, 0), (8, 0), (0, 1)])
def test_turned_pairs(ops, T, H, G, D, V, rot, extra, off):
    page, pages, n = 16, 10, (H + G) * D + G * V
    proj, other = rows(T, n, T + n, extra, off), rows(T, n, T + n)
    freq = 1.0 / 50.0 ** (torch.arange(0, max(rot, 2), 2, device=DEV).float() / max(rot, 2))
    pos = torch.randint(0, 3000, (T,), dtype=torch.int32, device=DEV)
    slots = slots_of(T, pages, page, T)
    caches = [[torch.full((pages, G, page, w), 7.0, dtype=torch.bfloat16, device=DEV) for w in (D, V)] for _ in range(2)]
    for o, p, (k, v) in ((ops, proj, caches[0]), (TwinOps(), other, caches[1])):
        o.rope_pairs_write(p, H * D, (H + G) * D, pos, freq, 1.3, rot, k, v, slots, H, G, D, V, page)
    assert torch.allclose(proj.float(), other.float(), **TOL)
    assert torch.allclose(caches[0][0].float(), caches[1][0].float(), **TOL) and torch.equal(caches[0][1], caches[1][1])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("E,K,top,groups,keep,shared", [(8, 2688, 2, 1, 1, False), (7, 300, 3, 1, 1, True), (64, 72, 6, 8, 3, True), (1, 5, 1, 1, 1, False)])
@pytest.mark.parametrize("T", [515, 1789])
def test_router_of_many_tokens(ops, dtype, E, K, top, groups, keep, shared, T):
    """So many tokens (no multiple of a block's four or eight) at once and cut into pieces that one token a block takes."""
    g = torch.Generator(device=DEV).manual_seed(E)
    x = torch.randn(T, K, generator=g, device=DEV).to(dtype)
    x[7, 0] = float("nan")
    x[8, 1] = float("inf")
    wr = torch.randn(E + shared, K, generator=g, device=DEV) * K ** -0.5
    corr = torch.rand(E, generator=g, device=DEV) if groups > 1 else None

    def run(x):
        idx = torch.empty(x.shape[0], top, dtype=torch.int32, device=DEV)
        wts = torch.empty(x.shape[0], top, device=DEV)
        share = torch.empty(x.shape[0], device=DEV) if shared else None
        ops.router_topk(idx, wts, x, wr, groups == 1, True, corr, groups, keep, 1.7, share)
        return [t.view(torch.int32) for t in (idx, wts, share) if t is not None]

    for whole, pieces in zip(run(x), zip(*(run(x[a:a + 103]) for a in range(0, T, 103)))):
        assert torch.equal(whole, torch.cat(pieces))
