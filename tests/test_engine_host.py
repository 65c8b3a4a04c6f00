"""Host side of the engines: how long a prompt pass is and what its buffers are sized for (CPU, no kernels)."""
from types import SimpleNamespace

import pytest
import torch

from conftest import pkg

HIDDEN = 8


class HostEngine:
    """DecodeEngine with the passes played on the host: at most `room_to_run` rows fit in one."""

    def __new__(cls, q_heads=32, kv_heads=4, head_dim=128, room_to_run=1 << 30, ep_state=None):
        eng = pkg("engine")

        class Engine(eng.DecodeEngine):
            def __init__(self):
                self.cfg = SimpleNamespace(q_heads=q_heads, kv_heads=kv_heads, head_dim=head_dim, experts=16, top_k=4, hidden=512,
                                           moe_inter=256, vocab_size=64)
                self.device, self.max_pages, self.num_slots, self.keep_logits = torch.device("cpu"), 512, 0, False
                self.ep_state, self.scratch_block, self.passes = ep_state, 0, []

            def _prompt_hidden(self, token_ids, row, lo, chunk, slot):
                if len(token_ids) > room_to_run:
                    raise torch.OutOfMemoryError("rows")
                self.passes.append((lo, len(token_ids)))
                return torch.zeros(len(token_ids), HIDDEN)

            def _pick(self, h, out=None):
                return torch.zeros(h.shape[0], dtype=torch.int64)

        return Engine()


@pytest.fixture
def host_ops(monkeypatch):
    """Workspaces of one byte per row; more than `room` rows do not fit.  Notes the rows asked for."""
    ops, box = pkg("ops"), SimpleNamespace(moe=[], attn=[], room=1 << 30)

    def moe(rows, *a):
        if rows > box.room:
            raise torch.OutOfMemoryError("workspace")
        box.moe.append(rows)
        return torch.zeros(256 + rows, dtype=torch.uint8)

    def attn(rows, *a):
        box.attn.append(rows)
        return torch.zeros(256 + rows, dtype=torch.uint8)

    monkeypatch.setattr(ops, "moe_fp8_workspace", moe)
    monkeypatch.setattr(ops, "paged_attn_workspace", attn)
    return box


def run(e, n, **kw):
    e.passes.clear()
    e.prefill(list(range(n)), list(range(-(-n // 16))), **kw)
    return e.passes


def test_prompt_buffers_are_sized_by_the_prompts(host_ops):
    e = HostEngine()
    assert run(e, 10) == [(0, 10)] and run(e, 1024) == [(0, 1024)] and host_ops.moe == [1024]
    assert run(e, 1500, cached_tokens=600) == [(600, 900)] and host_ops.moe == [1024]
    e._prefill_attn_ws[0], e._prefill_moe_ws[0] = 7, 9  # recorded findings outlive the growth
    assert run(e, 2500) == [(0, 2048), (2048, 452)] and host_ops.moe == [1024, 2048]
    assert (int(e._prefill_attn_ws[0]), int(e._prefill_moe_ws[0])) == (7, 9)
    assert run(e, 10) == [(0, 10)] and host_ops.moe == [1024, 2048]
    assert run(e, 100, chunk=64) == [(0, 64), (64, 36)] and host_ops.moe == [1024, 2048, 64]
    with pytest.raises(ValueError):
        run(e, 100, chunk=-1)


@pytest.mark.parametrize("chunk,kv_heads", [(512, 4), (3000, 4), (3000, 8)])
def test_a_pass_length_set_for_the_engine_is_kept(host_ops, chunk, kv_heads):
    e = HostEngine(kv_heads=kv_heads)
    e.prompt_chunk = chunk
    assert run(e, 700) == [(lo, min(chunk, 700 - lo)) for lo in range(0, 700, chunk)]
    assert run(e, 2500) == [(lo, min(chunk, 2500 - lo)) for lo in range(0, 2500, chunk)] and host_ops.moe == [chunk]


def test_shapes_without_the_tiled_kernel_keep_short_passes(host_ops):
    """Their split partials grow with the pass (32 / 8 heads of 128)."""
    e = HostEngine(kv_heads=8)
    assert run(e, 2500) == [(0, 1024), (1024, 1024), (2048, 452)] and host_ops.attn == host_ops.moe == [1024]


def test_a_default_pass_that_does_not_fit_runs_as_shorter_ones(host_ops):
    e = HostEngine()
    host_ops.room = 1024
    want = [(0, 1024), (1024, 1024), (2048, 452)]
    assert run(e, 2500) == want and run(e, 2500) == want and host_ops.moe == [1024]
    with pytest.raises(torch.OutOfMemoryError):  # asked for
        run(e, 2500, chunk=2048)
    host_ops.room = 1 << 30
    e = HostEngine(room_to_run=1500)  # the buffers fit, the rows do not
    assert run(e, 2500) == want and run(e, 2500) == want
    with pytest.raises(torch.OutOfMemoryError):
        run(e, 2500, chunk=2048)
    e = HostEngine(room_to_run=1000)
    with pytest.raises(torch.OutOfMemoryError):
        run(e, 2500)


def test_an_expert_parallel_pass_is_never_run_twice(host_ops):
    """The other ranks have taken part in the round."""
    e = HostEngine(room_to_run=1500, ep_state=SimpleNamespace(T=2048))
    with pytest.raises(torch.OutOfMemoryError):
        run(e, 2500)
    assert e.passes == []


def test_kept_logits_have_the_rows_of_the_output_matrix(monkeypatch):
    """It may be padded beyond the vocabulary of the configuration."""
    def argmax(x, w, workspace=None, out=None, status=None, logits=None):
        assert logits.shape == (x.shape[0], w.shape[0]) and logits.dtype == torch.bfloat16
        return logits.zero_().argmax(1)

    monkeypatch.setattr(pkg("ops"), "lm_head_argmax", argmax)
    e = HostEngine()
    e.lm_head, e.vocab_size, e.argmax_ws, e.gemm_status = torch.zeros(80, HIDDEN), 64, None, None
    tokens, logits = e._pick_with_logits(torch.zeros(3, HIDDEN))
    assert tokens.shape == (3,) and logits.shape == (3, 80)


@pytest.mark.parametrize("want_first", [True, False])
def test_a_mixed_pass_leaves_the_logits_of_its_decode_rows(want_first):
    """Row i of the pass has logits of i: two rows of a chunk, three of a decode step."""
    n, B = 2, 3
    e = HostEngine()
    e.keep_logits, e.max_batch, e.last_logits = True, B, "an earlier step's"
    e.tokens, e.ctx_lens, e.next_tokens = (torch.zeros(B, dtype=t) for t in (torch.int64, torch.int32, torch.int64))
    e.block_table = torch.zeros(B, e.max_pages, dtype=torch.int32)
    rows = torch.arange(n + B).float().view(-1, 1)
    e._mixed_hidden = lambda *a: rows
    e._pick = lambda h, out=None: h[:, 0].long() if out is None else out.copy_(h[:, 0].long())
    e._logits = lambda h: h.expand(-1, 4)
    e._pick_with_logits = lambda h, out=None: (e._pick(h, out), e._logits(h))
    tokens, first, logits = e.mixed_step(B, [5, 6], [0], 0, want_first=want_first)
    assert tokens.tolist() == [2, 3, 4] and e.ctx_lens.tolist() == [1, 1, 1]
    assert torch.equal(e.last_logits, rows[n:].expand(-1, 4))
    assert first == (1 if want_first else None) and (logits.tolist() == [1.0] * 4 if want_first else logits is None)


def test_token_ids_of_any_kind_give_what_torch_makes_of_them():
    import numpy as np
    f = pkg("engine").token_tensor
    ids = [3, 0, 151935, 7]
    for given in (ids, tuple(ids), [np.int64(v) for v in ids], [np.int32(v) for v in ids], np.array(ids, dtype=np.int32), torch.tensor(ids)):
        got = f(given, "cpu")
        assert got.tolist() == ids and not got.is_floating_point()
    assert f([2 ** 40], "cpu").tolist() == [2 ** 40] and f([], "cpu").numel() == 0
    assert f([1.5], "cpu").is_floating_point()  # and what is no token id stays what it was
