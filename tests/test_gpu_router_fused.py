"""Residual add + RMSNorm + router projection + top-k as one kernel through the C-ABI (B200), against the
separate kernels (b200_add_rmsnorm) and the CPU oracle of the router
(transformers Qwen3MoeTopKRouter, restated in oracle.route_ref)."""
import numpy as np
import pytest
import torch

from conftest import rel_err
import oracle

pytestmark = pytest.mark.gpu
DEV = "cuda"


def make(T, H, E, seed, with_delta=True):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(T, H, generator=g).bfloat16()
    delta = (torch.randn(T, H, generator=g) * 0.5).bfloat16() if with_delta else None
    nw = (1.0 + 0.1 * torch.randn(H, generator=g)).bfloat16()
    rw = (torch.randn(E, H, generator=g) * 0.05).bfloat16()
    return x, delta, nw, rw


@pytest.mark.parametrize("T,H,E,K", [(256, 2048, 128, 8), (1, 2048, 128, 8), (37, 4096, 128, 8), (5, 512, 16, 4),
                                     (300, 2048, 128, 8), (16, 2048, 48, 6)])
@pytest.mark.parametrize("with_delta", [True, False])
def test_fused_norm_router_topk(ops, T, H, E, K, with_delta):
    assert ops.add_rmsnorm_route_supported(H, E, K)
    x, delta, nw, rw = make(T, H, E, seed=T + H + E, with_delta=with_delta)
    xd = x.to(DEV).clone()
    h, ids, w, logits = ops.add_rmsnorm_route(xd, None if delta is None else delta.to(DEV), nw.to(DEV), 1e-6, rw.to(DEV),
                                              K, True, want_logits=True)
    # the separate kernels on the same inputs
    x2 = x.to(DEV).clone()
    h_ref = ops.add_rmsnorm(x2, None if delta is None else delta.to(DEV), nw.to(DEV), 1e-6)
    assert torch.equal(xd, x2)                       # the residual stream is exact (bf16 add)
    same = (h == h_ref).float().mean()
    assert float(same) > 0.999 and rel_err(h, h_ref) < 4e-3   # the sum of squares is taken in another order: rare 1-ulp flips
    # logits: fp32 product of the kernel's own normed rows with the bf16 router matrix
    want = h.float().cpu() @ rw.float().t()
    assert rel_err(logits, want) < 1e-4
    # routing of exactly those logits, bit-exact in ids
    rid, rwt = oracle.route_ref(logits.cpu(), K, True)
    assert torch.equal(ids.cpu(), rid)
    np.testing.assert_allclose(w.cpu().numpy(), rwt.numpy(), rtol=3e-6, atol=1e-9)


def test_rows_beyond_num_valid_get_no_expert(ops):
    T, H, E, K, n_valid = 40, 2048, 128, 8, 23
    x, delta, nw, rw = make(T, H, E, seed=1)
    nv = torch.tensor([n_valid], dtype=torch.int32, device=DEV)
    h, ids, w = ops.add_rmsnorm_route(x.to(DEV), delta.to(DEV), nw.to(DEV), 1e-6, rw.to(DEV), K, True, num_valid=nv)
    h2, ids2, w2 = ops.add_rmsnorm_route(x.to(DEV), delta.to(DEV), nw.to(DEV), 1e-6, rw.to(DEV), K, True)
    assert torch.equal(ids[:n_valid], ids2[:n_valid]) and torch.equal(w[:n_valid], w2[:n_valid])
    assert bool((ids[n_valid:] == -1).all()) and bool((w[n_valid:] == 0).all())
    assert torch.equal(h, h2)  # the norm itself is not masked: the rows are padding, their values unused


def test_repeatable_and_independent_of_the_batch_around_a_row(ops):
    """A row's result does not depend on which other rows share its cluster (graphs of different batch sizes
    must agree bit for bit)."""
    T, H, E, K = 50, 2048, 128, 8
    x, delta, nw, rw = make(T, H, E, seed=2)
    a = ops.add_rmsnorm_route(x.to(DEV), delta.to(DEV), nw.to(DEV), 1e-6, rw.to(DEV), K, True, want_logits=True)
    b = ops.add_rmsnorm_route(x[:19].contiguous().to(DEV), delta[:19].contiguous().to(DEV), nw.to(DEV), 1e-6, rw.to(DEV),
                              K, True, want_logits=True)
    for u, v in zip(a, b):
        assert torch.equal(u[:19], v)


@pytest.mark.parametrize("T,H,E", [(577, 2048, 128), (1500, 512, 16), (300, 4096, 128)])
def test_long_chunks_give_the_bits_of_short_ones(ops, T, H, E):
    """More rows than the 16-row clusters that fit the GPU at once run with 32 rows per cluster (a last cluster of one row
    included): the same sums in the same order, rows beyond num_valid without experts."""
    x, delta, nw, rw = make(T, H, E, seed=4)
    K, half = 4, (T // 32) * 16
    assert [ops.add_rmsnorm_route_rows(n, H, E) for n in (T, half, T - half)] == [32, 16, 16]

    def run(lo, hi, **kw):
        xs = x[lo:hi].contiguous().to(DEV)
        return (xs, *ops.add_rmsnorm_route(xs, delta[lo:hi].contiguous().to(DEV), nw.to(DEV), 1e-6, rw.to(DEV), K, True,
                                           want_logits=True, **kw))
    whole = run(0, T)
    for all_rows, first, rest in zip(whole, run(0, half), run(half, T)):
        assert torch.equal(all_rows, torch.cat([first, rest]))
    for n in (T - 31, T - 1, 0):
        _, h, ids, w, _ = run(0, T, num_valid=torch.tensor([n], dtype=torch.int32, device=DEV))
        assert torch.equal(h, whole[1]) and torch.equal(ids[:n], whole[2][:n]) and torch.equal(w[:n], whole[3][:n])
        assert bool((ids[n:] == -1).all()) and bool((w[n:] == 0).all())


@pytest.mark.parametrize("T,H,E", [(1024, 512, 16), (1024, 1024, 64), (513, 2048, 128), (1024, 2048, 64), (513, 4096, 64), (2048, 512, 128)])
def test_rows_that_a_wave_of_short_clusters_takes_stay_there(ops, T, H, E):
    """Clusters of 32 rows would be as many waves here, each of them longer (3-17 % more time)."""
    assert ops.add_rmsnorm_route_rows(T, H, E) == 16


def test_unsupported_shapes_are_refused(ops):
    assert not ops.add_rmsnorm_route_supported(768, 128, 8)     # hidden not a multiple of 512
    assert not ops.add_rmsnorm_route_supported(2048, 256, 8)    # more than 128 experts
    x, delta, nw, rw = make(4, 768, 16, seed=3)
    with pytest.raises(Exception, match="multiple of 512"):
        ops.add_rmsnorm_route(x.to(DEV), None, nw.to(DEV), 1e-6, rw.to(DEV), 4)


@pytest.mark.parametrize("T,H,E", [(5000, 512, 128), (5000, 2048, 64)])
def test_four_waves_of_long_clusters_in_place_of_five(ops, T, H, E):
    """On 148 SMs; the same rows in calls of one wave of short clusters: the same bits."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("wave counts of a GPU with 148 SMs")
    assert ops.add_rmsnorm_route_rows(T, H, E) == 32 and ops.add_rmsnorm_route_rows(400, H, E) == 16
    g = torch.Generator().manual_seed(T + H)
    x, delta = (torch.randn(T, H, generator=g).bfloat16().to(DEV) for _ in range(2))
    nw, rw = (1 + 0.1 * torch.randn(H, generator=g)).bfloat16().to(DEV), (torch.randn(E, H, generator=g) * 0.05).bfloat16().to(DEV)

    def run(lo, hi):
        xs = x[lo:hi].clone()
        return xs, *ops.add_rmsnorm_route(xs, delta[lo:hi], nw, 1e-6, rw, 8, want_logits=True)
    parts = [run(lo, min(T, lo + 400)) for lo in range(0, T, 400)]
    for i, whole in enumerate(run(0, T)):
        assert torch.equal(whole, torch.cat([p[i] for p in parts]))
