"""Tiled causal prompt attention over KV pages through the C-ABI (B200) vs the CPU oracle, which is pinned on
transformers eager attention with the causal mask over the reference's own page gather
(tests/golden/attn_prefill_d64.npz, tests/test_oracle_golden.py)."""
import numpy as np
import pytest
import torch

from conftest import golden, rel_err
import oracle

pytestmark = pytest.mark.gpu
DEV = "cuda"
TOL = 1e-2  # max |err| / max |ref| for bf16 outputs


def test_golden_suffix_on_a_cached_prefix(ops):
    g = golden("attn_prefill_d64.npz")
    q, kp, vp = (torch.from_numpy(g[k]).bfloat16() for k in ("q", "k_pool", "v_pool"))
    row = torch.from_numpy(g["table_row"])
    first, scale = int(g["first_pos"]), float(g["scale"])
    status = torch.zeros(64, dtype=torch.int32, device=DEV)
    out = ops.paged_attn_prefill(q.to(DEV), kp.to(DEV), vp.to(DEV), row.to(DEV), first, scale, status)
    ops.read_status(status, "paged_attn_prefill")
    ref = oracle.paged_prefill_ref(q, kp, vp, row.tolist(), first, scale)  # same bf16 inputs
    assert rel_err(out, ref) < TOL
    assert rel_err(out, torch.from_numpy(g["out"])) < 2e-2  # and close to the fp32 run of the reference's path


def case(hq, hkv, d, first, rows, seed):
    g = torch.Generator().manual_seed(seed)
    total = first + rows
    n_pages = (total + 15) // 16
    ids = torch.randperm(n_pages + 7, generator=g)[:n_pages].to(torch.int32)
    kp = torch.randn(n_pages + 7, hkv, 16, d, generator=g).bfloat16()
    vp = torch.randn(n_pages + 7, hkv, 16, d, generator=g).bfloat16()
    q = torch.randn(rows, hq, d, generator=g).bfloat16()
    row = torch.zeros(n_pages + 3, dtype=torch.int32)
    row[:n_pages] = ids
    return q, kp, vp, row


@pytest.mark.parametrize("hq,hkv,d", [(32, 4, 128), (64, 4, 128), (8, 2, 64)])
@pytest.mark.parametrize("first,rows", [(0, 1), (0, 17), (100, 128), (37, 300), (1000, 16), (2047, 33)])
def test_chunk_shapes_and_positions(ops, hq, hkv, d, first, rows):
    q, kp, vp, row = case(hq, hkv, d, first, rows, seed=first + rows)
    status = torch.zeros(64, dtype=torch.int32, device=DEV)
    out = ops.paged_attn_prefill(q.to(DEV), kp.to(DEV), vp.to(DEV), row.to(DEV), first, d ** -0.5, status)
    ops.read_status(status, "paged_attn_prefill")
    ref = oracle.paged_prefill_ref(q, kp, vp, row.tolist(), first, d ** -0.5)
    assert rel_err(out, ref) < TOL
    # row by row too: a wrong causal edge shows in single rows long before it moves the tensor-wide maximum
    per_row = (out.float().cpu() - ref).abs().amax(dim=(1, 2)) / ref.abs().amax()
    assert float(per_row.max()) < TOL


def test_same_rows_as_the_decode_kernel_gives_them_one_by_one(ops):
    """The row of position p is decode attention at context length p + 1."""
    hq, hkv, d, first, rows = 32, 4, 128, 200, 64
    q, kp, vp, row = case(hq, hkv, d, first, rows, seed=5)
    qd, kd, vd, rd = q.to(DEV), kp.to(DEV), vp.to(DEV), row.to(DEV)
    out = ops.paged_attn_prefill(qd, kd, vd, rd, first, d ** -0.5)
    table = rd.view(1, -1).expand(rows, -1).contiguous()
    lens = torch.arange(first + 1, first + rows + 1, dtype=torch.int32, device=DEV)
    dec = ops.paged_attn_decode(qd, kd, vd, table, lens, d ** -0.5)
    assert rel_err(out, dec) < 5e-3


def test_positions_past_the_table_and_bad_pages_are_reported_not_read(ops):
    q, kp, vp, row = case(32, 4, 128, 0, 40, seed=7)
    with pytest.raises(Exception, match="do not fit"):
        ops.paged_attn_prefill(q.to(DEV), kp.to(DEV), vp.to(DEV), row.to(DEV), row.numel() * 16 - 10, 0.1)
    bad = row.clone()
    bad[1] = 10_000
    status = torch.zeros(64, dtype=torch.int32, device=DEV)
    ops.paged_attn_prefill(q.to(DEV), kp.to(DEV), vp.to(DEV), bad.to(DEV), 0, 0.1, status)
    with pytest.raises(Exception, match="block table entry"):
        ops.read_status(status, "paged_attn_prefill")


@pytest.mark.parametrize("hq,hkv,d,first,rows,chunk", [
    (32, 4, 128, 0, 1280, 0),       # TMA queries, 8 heads per kv head, several waves
    (32, 4, 128, 5000, 1008, 0),    # an odd number of tiles: the last CTA has one
    (64, 4, 128, 123, 661, 0),      # 16 heads per kv head, a last tile of five positions
    (24, 8, 128, 300, 977, 0),      # 42 positions per tile, copied queries
    (64, 4, 128, 121, 700, 128),    # chunk edges between and inside the tiles of a CTA
    (40, 8, 64, 77, 1900, 512),     # head_dim 64; tiles that see different numbers of key tiles
])
def test_two_tiles_per_cta_give_the_bits_of_one(ops, hq, hkv, d, first, rows, chunk):
    """More tiles of rows than SMs: two per CTA.  The same rows in calls of a few whole tiles each, one per CTA: the same bits."""
    q, kp, vp, row = (t.to(DEV) for t in case(hq, hkv, d, first, rows, seed=rows))
    gate = torch.randn(rows, hq, generator=torch.Generator().manual_seed(1)).to(DEV)
    status = torch.zeros(64, dtype=torch.int32, device=DEV)

    def run(lo, hi):
        return ops.paged_attn_prefill_chunked(q[lo:hi], kp, vp, row, first + lo, d ** -0.5, status, chunk, gate[lo:hi])

    tile = 128 // (hq // hkv)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert -(-rows // tile) * hkv > sms
    step = sms // hkv // 2 * tile
    whole = run(0, rows)
    pieces = torch.cat([run(lo, min(rows, lo + step)) for lo in range(0, rows, step)])
    ops.read_status(status, "paged_attn_prefill_chunked")
    assert torch.equal(whole, pieces)
    # and a few rows against decode attention, which sees a row's own chunk likewise: two results that round P and the output to bf16
    # (2^-9 each) differ by at most 4 * 2^-9 = 7.8e-3
    for p in (0, rows // 2, rows - 1):
        ws = ops.paged_attn_workspace(1, hq, d, row.numel(), 16, 1024, DEV)
        lens = torch.tensor([first + p + 1], dtype=torch.int32, device=DEV)
        dec = ops.paged_attn_decode_chunked(q[p:p + 1], kp, vp, row[None], lens, d ** -0.5, 1024, ws, chunk, gate[p:p + 1])
        assert rel_err(whole[p:p + 1], dec) < TOL


@pytest.mark.parametrize("hq,hkv,d,first,rows,chunk,pairs,short", [
    (32, 4, 128, 4000, 1500, 0, 37, False),  # a wave of CTAs with two tiles, then one of single tiles
    (32, 4, 128, 5000, 1208, 0, 37, False),  # the same with two single tiles per head
    (32, 4, 128, 1800, 1200, 0, 37, True),   # pieces by the other kernel, over up to 3000 keys
    (40, 8, 64, 1900, 1100, 0, 18, True),
])
def test_mixed_grids_and_both_kernels_give_the_same_bits(ops, hq, hkv, d, first, rows, chunk, pairs, short):
    sms, tile = torch.cuda.get_device_properties(0).multi_processor_count, 128 // (hq // hkv)
    step = sms // hkv // 2 * tile
    if sms == 148:
        assert ops.paged_attn_prefill_pairs(rows, first, hq, hkv, chunk) == (pairs, False)
        assert ops.paged_attn_prefill_pairs(step, first, hq, hkv, chunk) == (0, short)
    q, kp, vp, row = (t.to(DEV) for t in case(hq, hkv, d, first, rows, seed=rows))
    status = torch.zeros(64, dtype=torch.int32, device=DEV)

    def run(lo, hi):
        return ops.paged_attn_prefill_chunked(q[lo:hi], kp, vp, row, first + lo, d ** -0.5, status, chunk)

    whole = run(0, rows)
    assert torch.equal(whole, torch.cat([run(lo, min(rows, lo + step)) for lo in range(0, rows, step)]))
    ops.read_status(status, "paged_attn_prefill_chunked")
    # and tiles of both kinds against decode attention: the same bound as above
    for p in (0, tile, rows // 2, rows - 1):
        ws = ops.paged_attn_workspace(1, hq, d, row.numel(), 16, 1024, DEV)
        lens = torch.tensor([first + p + 1], dtype=torch.int32, device=DEV)
        dec = ops.paged_attn_decode_chunked(q[p:p + 1], kp, vp, row[None], lens, d ** -0.5, 1024, ws, chunk)
        assert rel_err(whole[p:p + 1], dec) < TOL


@pytest.mark.parametrize("hq,hkv,d,first,rows", [
    (32, 4, 128, 3056, 17),  # queries by TMA, 8 and 16 heads per kv head
    (64, 4, 128, 3100, 21),
    (24, 8, 128, 3500, 50),  # copied queries, 42 positions per tile
    (40, 8, 64, 3300, 60),   # head_dim 64, 25 positions per tile
])
def test_single_tiles_that_see_many_keys(ops, hq, hkv, d, first, rows):
    assert ops.paged_attn_prefill_pairs(rows, first, hq, hkv) == (0, False)
    q, kp, vp, row = case(hq, hkv, d, first, rows, seed=first)
    status = torch.zeros(64, dtype=torch.int32, device=DEV)
    out = ops.paged_attn_prefill_chunked(q.to(DEV), kp.to(DEV), vp.to(DEV), row.to(DEV), first, d ** -0.5, status)
    ops.read_status(status, "paged_attn_prefill_chunked")
    ref = oracle.paged_prefill_ref(q, kp, vp, row.tolist(), first, d ** -0.5)
    per_row = (out.float().cpu() - ref).abs().amax(dim=(1, 2)) / ref.abs().amax()
    assert float(per_row.max()) < TOL
