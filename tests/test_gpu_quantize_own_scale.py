"""The one-launch quantiser (amax, scale and codes in one kernel) byte for byte against the oracle, at the sizes where its two
forms and their work units meet: one cluster up to 8192 blocks of 16 values, work units of 2048 (bf16) or 1024 (f32) blocks above."""
import numpy as np
import pytest
import torch

from oracle import nvfp4_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,k", [(1, 16), (31, 272), (64, 2048), (65, 2032), (64, 2064), (257, 1040), (1024, 2048)])
def test_single_matrix(rows, k, dtype):
    import sm120fp4_b200 as pkg
    x = (torch.randn(rows, k, generator=torch.Generator().manual_seed(rows * 7 + k)) * 3).to(dtype)
    x[rows // 2, k // 3] = 77.0
    wq, wsf, wgs = O.quantize_nvfp4(x.float().numpy(), None)
    for _ in range(2):      # the second call finds the workspace as the first left it
        q, sf, gs = pkg.quantize_nvfp4(x.cuda())
        assert np.array_equal(gs.cpu().numpy().view(np.uint32), wgs.view(np.uint32))
        assert np.array_equal(q.cpu().numpy(), wq) and np.array_equal(sf.cpu().numpy(), wsf)
    q, sw, _ = pkg.quantize_nvfp4_128x4(x.cuda(), gs)
    assert np.array_equal(q.cpu().numpy(), wq) and np.array_equal(sw.cpu().numpy(), O.to_128x4(wsf))


@pytest.mark.parametrize("swizzle", [False, True])
@pytest.mark.parametrize("groups,rows,k", [(1, 64, 64), (3, 100, 80), (5, 129, 1040), (40, 192, 512)])
def test_stacked_matrices(groups, rows, k, swizzle):
    import sm120fp4_b200 as pkg
    scale = torch.linspace(0.01, 9.0, groups)[:, None, None]
    w = (torch.randn(groups, rows, k, generator=torch.Generator().manual_seed(groups)) * scale).to(torch.bfloat16)
    q, sf, gs = pkg.quantize_nvfp4_experts(w.cuda(), swizzle=swizzle)
    for g in range(groups):
        wq, wsf, wgs = O.quantize_nvfp4(w[g].float().numpy(), None)
        assert np.array_equal(gs[g:g + 1].cpu().numpy().view(np.uint32), wgs.view(np.uint32))
        assert np.array_equal(q[g].cpu().numpy(), wq)
        assert np.array_equal(sf[g].cpu().numpy(), O.to_128x4(wsf) if swizzle else wsf)


# More than 126 MB of bf16 in groups of up to 8 MB stay in shared memory between the passes, in units of 1024 blocks of 16 values: groups
# of many units with a ragged last one, of one ragged unit, and the largest that the form takes (1.75 rounds of 148 units) beside the
# first that it does not and larger ones. The fp32 copy of the same values goes the other way, and its bytes are the same.
@pytest.mark.parametrize("groups,rows,k", [(65, 1000, 1040), (8400, 500, 16), (16, 2072, 2048), (16, 2080, 2048), (13, 2840, 2048), (13, 2848, 2048)])
def test_large_inputs_on_chip(groups, rows, k):
    import sm120fp4_b200 as pkg
    g = torch.Generator(device="cuda").manual_seed(rows)
    w = torch.empty(groups, rows, k, dtype=torch.bfloat16, device="cuda").normal_(generator=g)
    w *= torch.linspace(0.01, 9.0, groups, device="cuda")[:, None, None].to(torch.bfloat16)
    w[groups // 2] = 0
    w[1, 0, :16] = float("nan")
    for swizzle in (False, True):
        got = pkg.quantize_nvfp4_experts(w, swizzle=swizzle)
        want = pkg.quantize_nvfp4_experts(w.float(), swizzle=swizzle)
        for a, b in zip(got, want):
            assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
        again = pkg.quantize_nvfp4_experts(w, swizzle=swizzle)
        assert all(torch.equal(a.view(torch.uint8), b.view(torch.uint8)) for a, b in zip(got, again))


# More than 30 MB in all: the passes of different groups alternate (15 groups apart in bf16, 7 in fp32, the last unit of each ragged), once
# or, with twice the groups, many times; a group above 30 MB: its two passes follow one another.
@pytest.mark.parametrize("dtype,groups,rows,k", [(torch.bfloat16, 16, 1000, 1040), (torch.bfloat16, 40, 1000, 1040), (torch.float32, 12, 1000, 1040),
                                                 (torch.float32, 20, 1000, 1040), (torch.bfloat16, 2, 6400, 2048), (torch.bfloat16, 2, 8200, 2048),
                                                 (torch.float32, 3, 4100, 2048)])
def test_groups_in_alternating_order(dtype, groups, rows, k):
    import sm120fp4_b200 as pkg
    scale = torch.linspace(0.01, 9.0, groups, device="cuda")[:, None, None]
    w = (torch.randn(groups, rows, k, generator=torch.Generator(device="cuda").manual_seed(groups), device="cuda") * scale).to(dtype)
    want = [O.quantize_nvfp4(w[g].float().cpu().numpy(), None) for g in range(groups)]
    small = torch.randn(3, 100, 80, generator=torch.Generator().manual_seed(1)).to(dtype).cuda()
    for swizzle in (False, True):
        q, sf, gs = pkg.quantize_nvfp4_experts(w, swizzle=swizzle)
        pkg.quantize_nvfp4_experts(small)            # a smaller call in between, on the same workspace
        for g, (wq, wsf, wgs) in enumerate(want):
            assert np.array_equal(gs[g:g + 1].cpu().numpy().view(np.uint32), wgs.view(np.uint32))
            assert np.array_equal(q[g].cpu().numpy(), wq)
            assert np.array_equal(sf[g].cpu().numpy(), O.to_128x4(wsf) if swizzle else wsf)
    got = pkg.quantize_nvfp4_experts(small)
    for g in range(3):
        wq, wsf, wgs = O.quantize_nvfp4(small[g].float().cpu().numpy(), None)
        assert np.array_equal(got[0][g].cpu().numpy(), wq) and np.array_equal(got[1][g].cpu().numpy(), wsf)


def test_every_bf16_amax():
    """Every positive bf16 value up to 2^60 as a block's largest magnitude, in matrices whose global scale makes the block scales
    land on all of E4M3's range: the block scale's division has a form of its own for bf16 inputs."""
    import sm120fp4_b200 as pkg
    bits = torch.arange(1, (127 + 60) << 7, dtype=torch.int32).to(torch.int16)
    for top in (2.0 ** 60, 2.0 ** 20, 1.0, 2.0 ** -20):
        v = bits.view(torch.bfloat16)
        v = v[v.float() <= top]
        x = torch.zeros(v.numel(), 16, dtype=torch.bfloat16)
        x[:, 5] = v
        x = x[-(-x.shape[0] // 2):] if x.shape[0] > 1 << 16 else x
        for rows in (x, x[-8000:]):          # the large and the small form
            wq, wsf, wgs = O.quantize_nvfp4(rows.float().numpy(), None)
            q, sf, gs = pkg.quantize_nvfp4(rows.contiguous().cuda())
            assert np.array_equal(gs.cpu().numpy().view(np.uint32), wgs.view(np.uint32))
            assert np.array_equal(sf.cpu().numpy(), wsf) and np.array_equal(q.cpu().numpy(), wq), top


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows", [8, 300])
def test_nan_and_infinite_values(rows, dtype):
    """A block of NaNs, single NaNs and infinities: the same bytes as amax, scale and codes in separate launches."""
    import sm120fp4_b200 as pkg
    base = torch.randn(rows, 1040, generator=torch.Generator().manual_seed(rows)).to(dtype)
    for where, value in (((3, slice(32, 48)), "nan"), ((5, 7), "nan"), ((6, slice(16, 32, 2)), "nan"), ((0, 9), "inf"), ((0, 9), "-inf")):
        x = base.clone()
        x[where] = float(value)
        x = x.cuda()
        q, sf, gs = pkg.quantize_nvfp4(x)
        assert torch.equal(gs, pkg.quant.global_scale_for(x))
        wq, wsf, _ = pkg.quantize_nvfp4(x, gs)
        assert torch.equal(q, wq) and torch.equal(sf, wsf)
        qe, se, ge = pkg.quantize_nvfp4_experts(torch.stack([x, x]))
        assert torch.equal(ge, gs.expand(2)) and torch.equal(qe, wq.expand(2, -1, -1)) and torch.equal(se, wsf.expand(2, -1, -1))


def test_scales_beyond_two_gigabytes():
    """One row of 2^28 values: its padded 128x4 scales take 2 GB, more than the one launch indexes."""
    import sm120fp4_b200 as pkg
    k = 1 << 28
    x = torch.randn(1, k, generator=torch.Generator(device="cuda").manual_seed(1), dtype=torch.bfloat16, device="cuda")
    q, sf, gs = pkg.quantize_nvfp4(x)
    qe, se, ge = pkg.quantize_nvfp4_experts(x[None], swizzle=True)
    assert torch.equal(ge, gs) and torch.equal(qe[0], q)
    tiles = se.view(-1, 512)
    assert torch.equal(tiles[:, :4].reshape(1, -1), sf) and not tiles[:, 4:].any()


def test_more_groups_than_a_grid_holds_are_refused():
    import sm120fp4_b200 as pkg
    from sm120fp4_b200._lib import ERR_ARG, B200MoEError
    with pytest.raises(B200MoEError) as e:
        pkg.quantize_nvfp4_experts(torch.ones(65536, 1, 16, dtype=torch.bfloat16, device="cuda"))
    assert e.value.code == ERR_ARG
    q, _, _ = pkg.quantize_nvfp4_experts(torch.ones(65535, 1, 16, dtype=torch.bfloat16, device="cuda"))
    assert bool((q == 0x77).all())


def _expect(x, got):
    wq, wsf, wgs = O.quantize_nvfp4(x.float().cpu().numpy(), None)
    q, sf, gs = got
    assert np.array_equal(gs.cpu().numpy().view(np.uint32), wgs.view(np.uint32))
    assert np.array_equal(q.cpu().numpy(), wq) and np.array_equal(sf.cpu().numpy(), wsf)


def _captured(x, stream):
    import sm120fp4_b200 as pkg
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        out = pkg.quantize_nvfp4(x)
    return graph, out


def _randn(rows, k, seed):
    return torch.randn(rows, k, generator=torch.Generator().manual_seed(seed)).to(torch.bfloat16).cuda()


@pytest.mark.parametrize("polls", [0, 1])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("groups,rows,k", [(1, 257, 1040), (3, 300, 2048), (40, 192, 512), (6, 1536, 2048), (45, 1530, 1040)])
def test_blocks_that_do_not_wait(groups, rows, k, dtype, polls):
    """A block that gives up waiting for other blocks' maxima works them out itself: the same bytes, twice on one workspace."""
    import sm120fp4_b200 as pkg
    import sm120fp4_b200._lib as L
    w = torch.randn(groups, rows, k, generator=torch.Generator().manual_seed(rows)).to(dtype).cuda() * torch.arange(1, groups + 1, device="cuda").to(dtype)[:, None, None]
    want = pkg.quantize_nvfp4_experts(w)
    dt = 0 if dtype == torch.bfloat16 else 1
    ws = torch.zeros(L.lib().b200moe_quantize_own_scale_workspace_bytes(dt, groups, rows, k), dtype=torch.uint8, device="cuda")
    for _ in range(2):
        got = [torch.empty_like(t) for t in want]
        L.check(L.lib().b200moe_quantize_own_scale_probe(L.ptr(w), dt, groups, rows, k, L.ptr(got[2]), L.ptr(got[0]), L.ptr(got[1]), 0, L.ptr(ws),
                                                         ws.numel(), polls, L.stream_ptr()), "probe")
        assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("tries", [0, 1, 2, 70])
@pytest.mark.parametrize("groups,rows,k", [(45, 1530, 1040), (8400, 500, 16)])
def test_waits_inside_a_block_that_give_up(groups, rows, k, tries):
    """More than 126 MB of bf16: a warp whose wait for a copy or a maximum runs out goes on without it. The same bytes."""
    import sm120fp4_b200 as pkg
    import sm120fp4_b200._lib as L
    w = torch.randn(groups, rows, k, generator=torch.Generator(device="cuda").manual_seed(rows), device="cuda", dtype=torch.bfloat16)
    w *= torch.linspace(0.1, 9.0, groups, device="cuda")[:, None, None].to(torch.bfloat16)
    want = pkg.quantize_nvfp4_experts(w)
    h = L.lib()
    ws = torch.zeros(h.b200moe_quantize_own_scale_workspace_bytes(0, groups, rows, k), dtype=torch.uint8, device="cuda")
    for _ in range(2):
        got = [torch.empty_like(t) for t in want]
        L.check(h.b200moe_quantize_own_scale_probe(L.ptr(w), 0, groups, rows, k, L.ptr(got[2]), L.ptr(got[0]), L.ptr(got[1]), 0, L.ptr(ws), ws.numel(),
                                                   -1 - tries, L.stream_ptr()), "probe")
        assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("dtype,groups", [(torch.float32, 24), (torch.bfloat16, 48)])   # (the second stays in shared memory)
def test_two_calls_at_once(dtype, groups):
    """Two large calls on two streams share the GPU's SMs in whatever way they are scheduled."""
    import sm120fp4_b200 as pkg
    streams = [torch.cuda.Stream() for _ in range(2)]
    ws = [torch.randn(groups, 768, 2048, generator=torch.Generator(device="cuda").manual_seed(i), device="cuda", dtype=dtype) for i in range(2)]
    want = [pkg.quantize_nvfp4_experts(w) for w in ws]
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(6):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                got[i].append(pkg.quantize_nvfp4_experts(ws[i]))
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for i in range(2) for o in got[i] for a, b in zip(o, want[i]))


def test_captured_call_keeps_its_workspace():
    """A larger eager call on the stream of a captured one, and whatever it lets the allocator hand out, touch nothing that a replay uses."""
    import sm120fp4_b200 as pkg
    stream = torch.cuda.Stream()
    x = _randn(1024, 2048, 1)
    pkg.quantize_nvfp4(x)
    torch.cuda.synchronize()
    graph, out = _captured(x, stream)
    with torch.cuda.stream(stream):
        big = _randn(4096, 2048, 2)
        _expect(big, pkg.quantize_nvfp4(big))
        filled = [torch.full((4096,), 0x5a, dtype=torch.uint8, device="cuda") for _ in range(256)]
    torch.cuda.synchronize()
    for seed in (3, 4):
        x.copy_(_randn(1024, 2048, seed) * seed)
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        _expect(x, out)
    assert all(bool((t == 0x5a).all()) for t in filled)


def test_two_graphs_of_one_stream():
    """Captured on one stream before any eager call on it; the second alone, then an eager call, then each on either stream."""
    import sm120fp4_b200 as pkg
    stream, other = torch.cuda.Stream(), torch.cuda.Stream()
    xs = [_randn(1024, 2048, 5), _randn(640, 4096, 6)]
    torch.cuda.synchronize()
    (g0, out0), (g1, out1) = (_captured(x, stream) for x in xs)
    for seed in (7, 8):
        xs[1].copy_(_randn(640, 4096, seed) * seed)
        torch.cuda.synchronize()
        g1.replay()
        torch.cuda.synchronize()
        _expect(xs[1], out1)
    with torch.cuda.stream(stream):
        e = _randn(300, 2048, 9)
        _expect(e, pkg.quantize_nvfp4(e))
    torch.cuda.synchronize()
    for g, s in ((g0, stream), (g1, other), (g0, other)):
        with torch.cuda.stream(s):
            g.replay()
        torch.cuda.synchronize()
    _expect(xs[0], out0)
    _expect(xs[1], out1)
