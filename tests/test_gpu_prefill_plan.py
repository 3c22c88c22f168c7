"""Sizes at which the plan kernel and the grouped GEMM of a W4A4 layer call change their split: one, two, four and eight CTAs in the
plan's cluster (1024, 2048 and 4096 pairs are the last sizes of one, two and four), runs of pairs too long for a warp's registers
(more than 65536 pairs), operand boxes streamed through the ring because a tile's records do not fit (13 boxes of 128 rows).

A token's result does not depend on the batch around it: its rows are quantised on their own, accumulated in the same K order in
whatever tile they sit, and summed in slot order. So a call must equal the same tokens in calls of at most 64 bit for bit, and calls of
that size are checked against the oracle stage by stage (test_gpu_prefill; the streamed operand here)."""
import numpy as np
import pytest
import torch

from helpers import _i32, check_prefill_call, make_layer, prefill_map
from oracle import nvfp4_oracle as O
from test_gpu_decode import inputs
from test_gpu_prefill import run_prefill, sample

pytestmark = pytest.mark.gpu

MOST = 4097


def in_parts(w, x, ids, wts, most):
    n = -(-x.shape[0] // 64)
    return torch.cat([run_prefill(w, a, b, c, most).clone() for a, b, c in zip(*(torch.tensor_split(t, n) for t in (x, ids, wts)))])


@pytest.mark.parametrize("top_k,m", [(8, 128), (8, 129), (8, 256), (8, 257), (8, 512), (8, 513), (16, 4096), (16, MOST)])
def test_plan_sizes(top_k, m):
    cfg = dict(experts=24, hidden=256, inter=64, top_k=top_k)
    w, _ = make_layer(**cfg, seed=8)
    x, ids, wts = inputs(cfg, m, 50 + m)
    ids, wts = ids.clone(), wts.clone()
    ids[m // 2, 1], wts[m // 2, 1] = -1, 0          # an empty slot
    parts = in_parts(w, x, ids, wts, MOST)
    out = run_prefill(w, x, ids, wts, MOST)
    assert torch.equal(out, parts)
    flat = ids.reshape(-1).numpy()
    order = np.argsort(np.where(flat < 0, 1 << 20, flat), kind="stable")[: (flat >= 0).sum()]
    mp, ws = prefill_map(w, MOST), w.prefill.workspace
    assert np.array_equal(_i32(ws, mp["pairs"], flat.size)[: order.size], order)
    rows = _i32(ws, mp["dst_row"], flat.size)
    row_pair = _i32(ws, mp["row_pair"], 128 * int(_i32(ws, mp["ntiles"], 1)[0]))
    assert np.array_equal(row_pair[rows[order]], order) and (row_pair >= 0).sum() == order.size and rows[flat < 0].max() == -1


# Up to 1024 pairs every block of the quantising kernel works the plan out for itself, above it is a kernel: all tables against the router's
# definition on both sides of the line, with empty slots, an id that is no expert, one expert with all pairs, up to 256 experts.
@pytest.mark.parametrize("experts,top_k,m,same", [(24, 8, 17, False), (24, 8, 128, False), (24, 8, 129, False), (24, 8, 128, True), (256, 6, 170, False),
                                                  (256, 6, 171, False), (256, 16, 64, False), (2, 1, 1000, False), (2, 2, 512, True)])
def test_tables_of_small_batches(experts, top_k, m, same):
    cfg = dict(experts=experts, hidden=128, inter=64, top_k=top_k)
    w, _ = make_layer(**cfg, seed=8)
    x, ids, wts = inputs(cfg, m, 90 + m)
    ids, wts = ids.clone(), wts.clone()
    if same:
        ids[:] = torch.arange(top_k, dtype=torch.int32)
    ids[m // 2, top_k - 1], wts[m // 2, top_k - 1] = -1, 0
    ids[m // 3, 0], wts[m // 3, 0] = experts, 0
    run_prefill(w, x, ids, wts, 1024)
    mp, ws = prefill_map(w, 1024), w.prefill.workspace
    flat = ids.reshape(-1).numpy()
    e = np.where((flat < 0) | (flat >= experts), 1 << 20, flat)
    routed = int((e < experts).sum())
    order = np.argsort(e, kind="stable")[:routed]
    cnt = np.bincount(flat[order], minlength=experts)
    off = np.concatenate([[0], np.cumsum(cnt)])
    touched = np.nonzero(cnt)[0]
    tiles = [(q, off[q] + 128 * j, off[q + 1]) for q in touched for j in range(-(-cnt[q] // 128))]
    umax, nt = min(experts, flat.size), len(tiles)
    assert int(_i32(ws, mp["ntiles"], 1)[0]) == nt
    assert np.array_equal(_i32(ws, mp["experts"], umax), np.pad(touched, (0, umax - touched.size), constant_values=-1))
    assert np.array_equal(_i32(ws, mp["offsets"], umax + 1), np.pad(off[touched], (0, umax + 1 - touched.size), constant_values=routed))
    assert np.array_equal(_i32(ws, mp["pairs"], routed), order)
    for i, name in enumerate(("tile_expert", "tile_first", "tile_end")):
        assert np.array_equal(_i32(ws, mp[name], nt), [t[i] for t in tiles]), name
    first_tile = np.concatenate([[0], np.cumsum(-(-cnt // 128))])
    rows = np.full(flat.size, -1)
    rows[order] = np.concatenate([128 * first_tile[q] + np.arange(cnt[q]) for q in touched])
    assert np.array_equal(_i32(ws, mp["dst_row"], flat.size), rows)
    row_pair = np.full(128 * nt, -1)
    row_pair[rows[order]] = order
    assert np.array_equal(_i32(ws, mp["row_pair"], 128 * nt), row_pair)


def test_workspace_holds_the_most_tiles_there_can_be():
    """Every expert ends in a tile of one row at the very number of tokens the workspace was sized for: all of its tiles are in use, and
    nothing is written behind it."""
    cfg = dict(experts=16, hidden=512, inter=128, top_k=8)
    w, _ = make_layer(**cfg, seed=4)
    m = 16 * 129 // 8
    x, _, wts = inputs(cfg, m, 3)
    ids = (torch.arange(m * 8, dtype=torch.int32) % 16).reshape(m, 8)
    nbytes = w.prefill_workspace_bytes(m)
    ws = torch.zeros(nbytes + (1 << 20), dtype=torch.uint8, device="cuda")
    ws[nbytes:] = 0x5a
    w.enable_prefill(max_tokens=m, workspace=ws)
    out = run_prefill(w, x, ids, wts, m).clone()
    mp = prefill_map(w, m)
    assert mp["max_tiles"] == 32 == int(_i32(ws, mp["ntiles"], 1)[0])
    assert bool((ws[nbytes:] == 0x5a).all())
    assert torch.equal(out, in_parts(w, x, ids, wts, 1000))


@pytest.mark.parametrize("m", [17, 40])
def test_small_call_after_a_large_one(m):
    """The tables that a large call left in the workspace index beyond a small call's tensors: nothing of them may be used."""
    cfg = dict(experts=24, hidden=1024, inter=128, top_k=8)
    w, _ = make_layer(**cfg, seed=3)
    big = [t.cuda() for t in inputs(cfg, 2000, 1)]
    x, ids, wts = (t.cuda() for t in inputs(cfg, m, 2))
    w.enable_prefill(max_tokens=2000)
    first = w.forward(x, ids, wts).clone()
    w.forward(*big)
    assert torch.equal(w.forward(x, ids, wts), first)
    w.prefill_status()
    w.prefill = None
    w.enable_mid(max_tokens=2000, min_tokens=17)
    first = w.forward(x, ids, wts).clone()
    w.forward(*big)
    assert torch.equal(w.forward(x, ids, wts), first)
    w.mid_status()


@pytest.mark.parametrize("m", [40, 150])
def test_streamed_operand_boxes(m):
    cfg = dict(experts=4, hidden=3328, inter=192, top_k=2)
    w, ow = make_layer(**cfg, seed=5)
    x, ids, wts = inputs(cfg, m, 6)
    ids = ids.clone()
    ids[:, 1] = 1 + ids[:, 1] % 3
    ids[:, 0] = 0                                   # one expert of many rows; the others' records fit
    check_prefill_call(w, ow, x, ids, wts, run_prefill(w, x, ids, wts), 512, sample_tokens=sample(ids, 8, 1), what=f"13 K boxes, {m} tokens")


# How many ring slots a CTA has depends on the number of tiles: up to one an expert, up to two, more; with a resident operand (8 boxes) and a streamed
# one (13). Rows are the same bits as in calls of at most 64 tokens, whose operand is resident and whose tiles are one an expert.
@pytest.mark.parametrize("hidden", [2048, 3328])
@pytest.mark.parametrize("rows", [(128, 100), (129, 100), (256, 200), (257, 250), (300, 400)])
def test_ring_depth(hidden, rows):
    cfg = dict(experts=2, hidden=hidden, inter=320, top_k=1)
    w, _ = make_layer(**cfg, seed=6)
    m = sum(rows)
    x, ids, wts = inputs(cfg, m, 8)
    ids = torch.repeat_interleave(torch.arange(2, dtype=torch.int32), torch.tensor(rows))[torch.randperm(m, generator=torch.Generator().manual_seed(1))][:, None].contiguous()
    assert torch.equal(run_prefill(w, x, ids, wts, 1024), in_parts(w, x, ids, wts, 1024))


# Beside a streamed operand it also goes by the tiles of an expert that has any (ten boxes: 1.5, thirteen: 3), however many experts the layer has: rows on two
# experts of sixteen, on both sides.
@pytest.mark.parametrize("hidden,rows", [(2560, (128, 200)), (2560, (200, 200)), (3328, (300, 300)), (3328, (300, 400))])
def test_ring_depth_on_few_experts(hidden, rows):
    cfg = dict(experts=16, hidden=hidden, inter=128, top_k=1)
    w, _ = make_layer(**cfg, seed=6)
    m = sum(rows)
    x, ids, wts = inputs(cfg, m, 8)
    ids = torch.repeat_interleave(torch.tensor([3, 11], dtype=torch.int32), torch.tensor(rows))[torch.randperm(m, generator=torch.Generator().manual_seed(1))][:, None].contiguous()
    assert torch.equal(run_prefill(w, x, ids, wts, 1024), in_parts(w, x, ids, wts, 1024))
    assert _i32(w.prefill.workspace, prefill_map(w, 1024)["ntiles"], 2)[1] == 2


# Rows that L2 does not hold (4100 tokens of 16 slots and 1024 columns) are added up by more threads with fewer loads each.
def test_rows_beyond_l2():
    cfg = dict(experts=24, hidden=1024, inter=64, top_k=16)
    w, _ = make_layer(**cfg, seed=7)
    x, ids, wts = inputs(cfg, 4100, 9)
    assert 4100 * 16 * 1024 * 2 > 126 << 20
    assert torch.equal(run_prefill(w, x, ids, wts, 4100), in_parts(w, x, ids, wts, 4100))


@pytest.mark.parametrize("hidden", [2560, 4096])
def test_silu_division_of_wide_layers(hidden):
    """Above nine K boxes FC1's SiLU divides with IEEE rounding. A gate of -88 shows it: 1 + exp(88) lies between 2^126 and 2^128, where
    the approximate division returns zero. The up value and the activation scale (1e28) bring the quotient (-5e-37) back into range.
    Every value of a block is the same, so its code is exact and the error is that of the E4M3 scale (2^-4) and of the output's bf16."""
    from sm120fp4_b200.vllm_backend import Weights
    inter, m = 64, 20
    q1 = torch.zeros(1, 2 * inter, hidden // 2, dtype=torch.uint8, device="cuda")
    s1 = torch.full((1, 2 * inter, hidden // 16), 0x38, dtype=torch.uint8, device="cuda")        # 1.0
    q1[:, :inter], s1[:, :inter] = 0x77, 0x7e                                                    # up: 6 x 448 everywhere
    q1[:, inter:, 0] = 0x0a                                                                      # gate: -1 at the first value
    q2 = torch.full((1, hidden, inter // 2), 0x22, dtype=torch.uint8, device="cuda")             # 1.0
    s2 = torch.full((1, hidden, inter // 16), 0x38, dtype=torch.uint8, device="cuda")
    xq = 6 * 0.171875                                                                            # what x = 1 becomes in NVFP4 (scale E4M3(1/6))
    a1, a2 = 88.0 / xq, 1e28
    w = Weights(q1, s1, torch.tensor([a1], device="cuda"), q2, s2, torch.tensor([a2], device="cuda"), 1)
    w.enable_prefill(a2_scale=1e-28, max_tokens=m)
    out = w.forward(torch.ones(m, hidden, dtype=torch.bfloat16, device="cuda"), torch.zeros(m, 1, dtype=torch.int32, device="cuda"),
                    torch.ones(m, 1, device="cuda")).double()
    want = -88.0 / (1.0 + np.exp(88.0)) * (hidden * 6 * 448 * xq * a1) * inter * a2
    assert (out / want - 1).abs().max() < 2.0 ** -4 + 2.0 ** -7, (out.flatten()[:4], want)


def test_quotient_of_wide_layers_is_ieee():
    """The division of that epilogue against IEEE division, bit for bit, for every gate there is: all 2^32 patterns of a float."""
    import sm120fp4_b200._lib as L
    n = 1 << 26
    den, out = (torch.empty(n, dtype=torch.float32, device="cuda") for _ in range(2))
    low = torch.arange(n, dtype=torch.int32, device="cuda")
    for part in range(64):
        gate = (low + (part - 32) * n).view(torch.float32)
        L.check(L.lib().b200moe_quotient_probe(L.ptr(gate), L.ptr(den), L.ptr(out), n, L.stream_ptr()), "probe")
        want = gate / den
        assert bool(((out.view(torch.int32) == want.view(torch.int32)) | (out.isnan() & want.isnan())).all()), part


# FC2's stores and the combine behind them take rows in groups of eight and columns in segments of 64: experts with one row, with whole and ragged
# groups and quadrants, up to one more than a tile; one segment pair a row (128 columns, an odd number of tokens: half a warp in the combine) and
# odd numbers of pairs of segments. Against the oracle's W4A4 arithmetic, tolerance as everywhere (2e-2 x RMS from the kernel's own codes). The
# outputs of so small a layer differ in size from token to token, up to 7 x RMS, where half a bf16 ulp may be more than that: the routing weights are
# divided by the size of the token's output, so that RMS is 1, all values are below 8 and half an ulp is at most 2^-6.
@pytest.mark.parametrize("hidden", [128, 384])
def test_rows_and_segments(hidden):
    cfg = dict(experts=16, hidden=hidden, inter=64, top_k=2)
    w, ow = make_layer(**cfg, seed=9)
    rows = [1, 7, 8, 9, 31, 32, 33, 63, 64, 65, 95, 97, 127, 129]
    first = np.repeat(np.arange(len(rows)), rows)
    m = first.size
    assert m % 2 == 1
    x, ids, wts = inputs(cfg, m, 7)
    ids = ids.clone()
    ids[:, 0], ids[:, 1] = torch.from_numpy(first.astype(np.int32)), 14 + torch.arange(m, dtype=torch.int32) % 2
    size = O.moe_reference(x.float().numpy(), ow, ids.numpy(), wts.numpy(), act_quant=True).astype(np.float64)
    wts = (wts / torch.from_numpy(np.sqrt((size ** 2).mean(axis=1, keepdims=True)))).float()
    out = run_prefill(w, x, ids, wts, 1024)
    check_prefill_call(w, ow, x, ids, wts, out, 1024, what=f"rows and segments, hidden {hidden}")
