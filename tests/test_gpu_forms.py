"""Kernels that come in two forms: which call goes to which, and that both give the same bits."""
import pytest
import torch

from conftest import pkg

pytestmark = pytest.mark.gpu
DEV, BF = "cuda", torch.bfloat16


def randn(*shape, seed, dtype=torch.float32):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(dtype).to(DEV)


def line(form, lo=1, hi=1 << 17):
    """The smallest count from `lo` on that goes to form 1, where there is one."""
    if not form(hi):
        return None
    while lo < hi:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if form(mid) else (mid + 1, hi)
    return lo


def same_bits(call, rows, step):
    """All rows in one call, and a few at a time: `call(lo, hi)` gives tensors by row."""
    whole, parts = call(0, rows), [call(lo, min(rows, lo + step)) for lo in range(0, rows, step)]
    for i, t in enumerate(whole):
        assert torch.equal(t, torch.cat([p[i] for p in parts]))


@pytest.mark.parametrize("center", [True, False])
def test_residual_norm_goes_by_what_an_sm_holds(ops, center):
    """A CTA has a thread for eight columns, so that rows of half the width have twice as many CTAs on an SM: the form that has more
    of them has nothing to offer before they are used up."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    lines = [line(lambda n: ops.residual_norm_form(n, ld, center)) for ld in (256, 512, 1024, 2048, 4096)]
    assert all(b < a for a, b in zip(lines, lines[1:]))
    assert all((n - 1) % sms == 0 for n in lines) and lines[-1] == sms + 1  # 512 threads: one CTA per SM, and two
    assert ops.residual_norm_form(1, 4104, center) == 1  # more than 512 threads: the only form
    assert ops.residual_norm_form(1 << 17, 512, center, torch.float32) == 0


@pytest.mark.parametrize("width,ld", [(250, 256), (1024, 1024), (4090, 4096)])
def test_residual_norm_forms_give_the_same_bits(ops, width, ld):
    P = pkg("gated").Pending
    M, top = line(lambda n: ops.residual_norm_form(n, ld)) + 7, 9
    cut = (torch.arange(ld) < width).to(DEV)
    x, w, bias = randn(M, ld, seed=1) * cut, (1 + randn(ld, seed=2)) * cut, randn(ld, seed=6) * cut
    d, gate, e = (randn(M, ld, seed=s, dtype=BF) * cut for s in (3, 4, 5))
    pairs = torch.randint(-1, M, (M, top), generator=torch.Generator().manual_seed(7)).to(torch.int32).to(DEV)
    pw = torch.rand(M, top, generator=torch.Generator().manual_seed(8)).to(DEV)
    for pending in (lambda a, b: None, lambda a, b: P(dense=d[a:b], gate=gate[a:b], bias=bias),
                    lambda a, b: P(expert_rows=e, row_of_pair=pairs[a:b].contiguous(), pair_weight=pw[a:b].contiguous(), gate=gate[a:b])):
        def call(a, b):
            xs = x[a:b].clone()
            return ops.residual_norm(xs, pending(a, b), w, 1e-3, width), xs
        assert ops.residual_norm_form(M, ld) == 1 and ops.residual_norm_form(100, ld) == 0
        same_bits(call, M, 100)


def test_combine_goes_by_what_an_sm_holds(ops):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    lines = [line(lambda n: ops.moe_combine_add_rmsnorm_form(n, h)) for h in (256, 512, 1024, 2048, 4096)]
    assert all(b < a for a, b in zip(lines, lines[1:]))
    assert all((n - 1) % sms == 0 for n in lines) and lines[-1] == sms + 1  # 512 threads: one CTA per SM, and two
    assert ops.moe_combine_add_rmsnorm_form(1 << 17, 5120) == 0  # 640 threads: one CTA per SM of either form
    assert ops.moe_combine_add_rmsnorm_form(1, 8192) == 1        # 1024 threads, for which the other form has no registers


@pytest.mark.parametrize("H,K", [(256, 8), (1024, 9), (4096, 2)])
def test_combine_forms_give_the_same_bits(ops, H, K):
    T = line(lambda n: ops.moe_combine_add_rmsnorm_form(n, H)) + 7
    y, x, nw = randn(T * K, H, seed=1, dtype=BF), randn(T, H, seed=2, dtype=BF), (1 + 0.1 * randn(H, seed=3)).to(BF)
    rows = torch.randperm(T * K, generator=torch.Generator().manual_seed(4)).view(T, K).to(torch.int32)
    rows[torch.rand(T, K, generator=torch.Generator().manual_seed(5)) < 0.1] = -1
    rows, w = rows.to(DEV), torch.rand(T, K, generator=torch.Generator().manual_seed(6)).to(DEV)

    def call(a, b):
        xs = x[a:b].clone()
        return ops.moe_combine_add_rmsnorm(y, rows[a:b].contiguous(), w[a:b].contiguous(), xs, nw, 1e-6), xs
    assert ops.moe_combine_add_rmsnorm_form(T, H) == 1 and ops.moe_combine_add_rmsnorm_form(100, H) == 0
    same_bits(call, T, 100)


@pytest.mark.parametrize("parts", [1, 16])
def test_grouped_norm_goes_by_what_an_sm_holds(ops, parts):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    lines = [line(lambda n: ops.group_rmsnorm_form(n, w, w, parts)) for w in (512, 1024, 2048, 4096)]
    assert all(b < a for a, b in zip(lines, lines[1:]))
    assert all((n - 1) % sms == 0 for n in lines) and lines[-1] == sms + 1  # 512 threads: one CTA per SM, and two
    assert ops.group_rmsnorm_form(1 << 17, 3072, 3072, parts) == 0  # 384 threads: two CTAs per SM of either form
    assert ops.group_rmsnorm_form(1, 4104, 4104, 1) == 1            # more than 512 threads: the only form
    assert ops.group_rmsnorm_form(1 << 17, 512, 512, parts, torch.float32) == 0


@pytest.mark.parametrize("width,ld,groups", [(510, 512, 6), (1024, 1024, 4), (4096, 4096, 1)])
def test_grouped_norm_forms_give_the_same_bits(ops, width, ld, groups):
    M = line(lambda n: ops.group_rmsnorm_form(n, width, ld, groups)) + 7
    cut = (torch.arange(ld) < width).to(DEV)
    x, d, w = randn(M, ld, seed=1) * cut, randn(M, ld, seed=2, dtype=BF) * cut, ((1 + randn(ld, seed=3)) * cut).to(BF)

    def call(a, b):
        xs = x[a:b].clone()
        return ops.group_rmsnorm(xs, d[a:b], w, 1e-3, width, groups), xs
    assert ops.group_rmsnorm_form(M, width, ld, groups) == 1 and ops.group_rmsnorm_form(100, width, ld, groups) == 0
    same_bits(call, M, 100)


@pytest.mark.parametrize("delta", [True, False])
@pytest.mark.parametrize("dtype", [BF, torch.float32])
def test_states_wait_in_shared_memory_where_more_of_them_fit(ops, delta, dtype):
    """In registers two CTAs fit on an SM; with 64 KB of state and the vectors of the head in shared memory three or two."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for dim, vdim in ((128, 128), (100, 120), (64, 256), (256, 64)):
        assert not ops.state_step_held(2 * sms, 1, dim, vdim, delta, dtype) and ops.state_step_held(2 * sms + 1, 1, dim, vdim, delta, dtype)
    for dim, vdim in ((32, 512), (16, 1024), (12, 1024), (512, 32), (1024, 16), (128, 64), (144, 144)):
        assert not ops.state_step_held(4096, 16, dim, vdim, delta, dtype)


@pytest.mark.parametrize("T,E,K", [(1023, 128, 8), (1024, 128, 8), (1100, 256, 8), (2047, 256, 8), (2048, 256, 8), (5462, 160, 3), (16400, 1024, 1)])
def test_ranks_on_both_sides_of_the_line(ops, T, E, K):
    """Pairs of an expert in their order, experts one after the other, dropped pairs nowhere."""
    ids = torch.rand(T, E, generator=torch.Generator().manual_seed(T)).topk(K, dim=1).indices.to(torch.int32)
    ids[T // 2, 0] = -1
    p = ops.moe_permute(ids.to(DEV), E)
    flat = ids.flatten()
    order = torch.argsort(torch.where(flat < 0, E, flat), stable=True)[: int((flat >= 0).sum())]
    want = torch.full((T * K,), -1, dtype=torch.int32)
    want[order] = torch.arange(len(order), dtype=torch.int32)
    assert torch.equal(p.row_of_pair.cpu().flatten(), want)
    assert torch.equal(p.expert_offsets.cpu().diff(), torch.bincount(flat[flat >= 0], minlength=E).to(torch.int32))


FIRST_CALL_IN_A_CAPTURE = """
import importlib, sys, torch
from types import SimpleNamespace
sys.path.insert(0, {root!r})
ops = importlib.import_module("inference-server_b200.ops")
torch.manual_seed(0)
M, W = 400, 2048
r = lambda *s, dtype=torch.bfloat16: torch.randn(*s, device="cuda", dtype=dtype)
x, w, d = r(M, W, dtype=torch.float32), r(W, dtype=torch.float32), r(M, W)
y, xb, rows, pw = r(M * 2, W), r(M, W), torch.randperm(M * 2, device="cuda").to(torch.int32).view(M, 2), torch.rand(M, 2, device="cuda")
ids = torch.rand(M, 16, device="cuda").topk(2, dim=1).indices.to(torch.int32)
H, D = 4, 128
act, state, decay = r(M, 3 * H * D), r(M, 2, H, D, D, dtype=torch.float32), torch.rand(H, device="cuda")
slots, pos = torch.arange(M, device="cuda", dtype=torch.int32), torch.full((M,), 3, device="cuda", dtype=torch.int32)
sw = SimpleNamespace(heads=H, qk_heads=H, d=D, dv=D, decay=decay)
q, kp, table = r(600, 32, 128), r(40, 4, 16, 128), torch.arange(40, device="cuda", dtype=torch.int32)
def all_of_them():
    xs, xg, xc, S, o = x.clone(), x.clone(), xb.clone(), state.clone(), torch.empty(M, H, D, device="cuda")
    ops.state_step(act, sw, S, slots, pos, o)
    return [ops.residual_norm(xs, None, w, 1e-5, W), ops.group_rmsnorm(xg, d, w.bfloat16(), 1e-5, W, 4),
            ops.moe_combine_add_rmsnorm(y, rows, pw, xc, w.bfloat16(), 1e-5), ops.moe_permute(ids, 16).row_of_pair, o, S,
            ops.paged_attn_prefill(q, kp, kp, table, 0, 0.1)]
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    captured = all_of_them()
g.replay()
torch.cuda.synchronize()
assert all(torch.equal(a, b) for a, b in zip(captured, all_of_them()))
print("same")
"""


def test_the_first_call_of_a_process_may_be_captured(ops):
    """What the rules ask of the runtime they may ask while a graph is being captured."""
    import subprocess
    import sys

    from conftest import ROOT
    run = subprocess.run([sys.executable, "-c", FIRST_CALL_IN_A_CAPTURE.format(root=ROOT)], capture_output=True, text=True, timeout=240)
    assert run.returncode == 0 and run.stdout.strip().endswith("same"), run.stderr[-2000:]
