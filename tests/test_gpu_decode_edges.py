"""Sizes at which the decode call changes its way: hidden sizes above 3072 (mma.sync kernel), x expanded by every worker itself up to
256 blocks of 16 values and eight tokens, and the same boundaries for tensors in page-locked host memory."""
import numpy as np
import pytest
import torch

from helpers import check_layer_output, decode_map, make_layer
from oracle import nvfp4_oracle as O
from test_gpu_decode import inputs, run

pytestmark = pytest.mark.gpu

_layers = {}


def edge_layer(hidden, inter=192):
    cfg = dict(experts=16, hidden=hidden, inter=inter, top_k=4)
    if (hidden, inter) not in _layers:
        _layers.clear()
        _layers[hidden, inter] = make_layer(**cfg, seed=9)
    return cfg, *_layers[hidden, inter]


def bare_forward(w, x, ids, wts):
    """The decode call of a second handle on the same weights that has not been prepacked; None where it refuses the shape."""
    import ctypes as C
    from sm120fp4_b200 import _lib
    h, bare = _lib.lib(), C.c_void_p()
    _lib.check(h.b200moe_layer_create(C.byref(bare), w.E, w.H, w.I, w.k, _lib.ptr(w.q1), _lib.ptr(w.s1), _lib.ptr(w.alpha1), _lib.ptr(w.q2),
                                      _lib.ptr(w.s2), _lib.ptr(w.alpha2)), "create")
    ws = torch.zeros_like(w.workspace)
    x, ids, wts = x.cuda(), ids.cuda(), wts.cuda()
    out = torch.empty_like(x)
    rc = h.b200moe_decode_forward(bare, _lib.ptr(x), _lib.ptr(ids), _lib.ptr(wts), x.shape[0], _lib.ptr(out), _lib.ptr(ws), ws.numel(), _lib.stream_ptr())
    torch.cuda.synchronize()
    h.b200moe_layer_destroy(bare)
    if rc == -2:
        return None
    _lib.check(rc, "decode")
    return out


# 512: 8 tokens are the last, 256 blocks; 4096: one token is; 2048 x 2; 3200 = 12.5 K boxes
@pytest.mark.parametrize("hidden,m", [(512, 8), (512, 9), (2048, 2), (2048, 3), (3072, 1), (3072, 16), (3200, 1), (3200, 8), (3200, 9), (3200, 16),
                                      (4096, 1), (4096, 2), (4096, 8), (4096, 9), (4096, 16)])
def test_hidden_sizes_and_batches(hidden, m):
    cfg, w, ow = edge_layer(hidden)
    x, ids, wts = inputs(cfg, m, 40 + m)
    out = run(w, x, ids, wts).clone()
    check_layer_output(out, O.moe_reference(x.float().numpy(), ow, ids.numpy(), wts.numpy()), f"hidden {hidden}, {m} tokens")
    pinned = [t.pin_memory() for t in (x, ids, wts)]
    host = torch.empty_like(x).pin_memory()
    for _ in range(2):
        host.zero_()
        torch.cuda.synchronize()
        w.forward_host(*pinned, host)
        torch.cuda.synchronize()
        assert torch.equal(host, out.cpu())
    w.status()


# Activations far beyond what the tcgen05 kernel's fixed activation scale holds (336 by default): the layers above 3072 compute with
# f16 activations, whatever the batch size.
@pytest.mark.parametrize("hidden,m", [(3200, 2), (4096, 1), (4096, 8), (4096, 9)])
def test_wide_layers_hold_large_activations(hidden, m):
    cfg, w, ow = edge_layer(hidden)
    x, ids, wts = inputs(cfg, m, 70 + m)
    x = (x.float() * 20).to(torch.bfloat16)
    out = run(w, x, ids, wts)
    w.status()
    check_layer_output(out, O.moe_reference(x.float().numpy(), ow, ids.numpy(), wts.numpy()), f"hidden {hidden}, {m} tokens, x * 20")


# A row's scale comes from its finite values: NaNs are passed over, also where they fill a block of 16 or every second value of one
# (two values are compared at a time). Expanded by the workers (1 and 2 tokens of 2048) and by the kernel ahead of them (9).
@pytest.mark.parametrize("which", [slice(32, 48), slice(32, 48, 2), slice(33, 48, 2)])
@pytest.mark.parametrize("m", [1, 2, 9])
def test_nan_values_do_not_set_the_row_scale(m, which):
    cfg, w, _ = edge_layer(2048)
    x, ids, wts = inputs(cfg, m, 90 + m)
    x = x.clone()
    x[0, which] = float("nan")
    run(w, x, ids, wts)
    amax = x[0].float()[~x[0].isnan()].abs().max().numpy()
    at = decode_map(w)["xscale"]
    got = w.workspace[at:at + 4].view(torch.float32).cpu().numpy()[0]
    assert got == np.float32(1) / (np.float32(2688) / amax)


# Wide layers decode from the tile records, under set_decode_impl("mma") and without a prepack from the checkpoint layout: the same tiles
# in the same order, so the same bits. Intermediate sizes with a whole and a part 128-row scale run and K box.
@pytest.mark.parametrize("hidden,inter", [(3200, 64), (3328, 192), (4096, 320), (6144, 192)])
def test_tile_records_and_checkpoint_layout_agree(hidden, inter):
    cfg, w, _ = edge_layer(hidden, inter)
    for m in (1, 8, 9, 16) if hidden <= 5376 else (1, 8):
        x, ids, wts = inputs(cfg, m, 50 + m)
        out = run(w, x, ids, wts).clone()
        assert torch.equal(out, bare_forward(w, x, ids, wts)), m
        w.set_decode_impl("mma")
        try:
            assert torch.equal(out, run(w, x, ids, wts)), m
        finally:
            w.set_decode_impl("auto")


@pytest.mark.parametrize("hidden,ms", [(3200, (1, 8, 9, 16)), (4096, (1, 8, 9, 16)), (7168, (1, 8))])
def test_wide_layers_decode_from_the_records_alone(hidden, ms):
    import sm120fp4_b200._lib as L
    cfg = dict(experts=16, hidden=hidden, inter=192, top_k=4)
    w, _ = make_layer(**cfg, seed=13)
    batches = [inputs(cfg, m, 80 + m) for m in ms]
    want = [run(w, *b).clone() for b in batches]
    w.release_checkpoint_layout()
    for b, o in zip(batches, want):
        assert torch.equal(run(w, *b), o)
        pinned = [t.pin_memory() for t in b]
        host = torch.empty_like(b[0]).pin_memory()
        w.forward_host(*pinned, host)
        torch.cuda.synchronize()
        assert torch.equal(host, o.cpu())
    x, ids, wts = (t.cuda() for t in batches[0])
    act = torch.zeros(ms[0] * w.k, w.I, dtype=torch.bfloat16, device="cuda")
    for refused in (lambda: w.set_decode_impl("mma"), lambda: w.fc1(x, ids, wts, act), lambda: w.fc2(act, ids, wts, torch.empty_like(x))):
        with pytest.raises(L.B200MoEError):
            refused()


@pytest.mark.parametrize("hidden", [640, 3200])
def test_weights_changed_in_place(hidden):
    """The halves and the mma.sync kernel by request compute with the weights as they are at the call; the layer call follows a new prepack."""
    from sm120fp4_b200 import _lib
    from sm120fp4_b200.vllm_backend import Weights
    cfg = dict(experts=16, hidden=hidden, inter=192, top_k=4)
    w, _ = make_layer(**cfg, seed=12)
    w.q1.copy_(w.q1.roll(1, 0))
    w.q2.copy_(w.q2.roll(1, 0))
    fresh = Weights(w.q1.clone(), w.s1, w.alpha1, w.q2.clone(), w.s2, w.alpha2, w.k, scale_layout="128x4")
    for m in (3, 12):
        x, ids, wts = (t.cuda() for t in inputs(cfg, m, 5))
        act = [torch.zeros(m * w.k, w.I, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
        out = [torch.empty_like(x) for _ in range(2)]
        for i, layer in enumerate((w, fresh)):
            layer.fc1(x, ids, wts, act[i])
            layer.fc2(act[0], ids, wts, out[i])
        assert torch.equal(*act) and torch.equal(*out)
        for layer in (w, fresh):
            layer.set_decode_impl("mma")
        assert torch.equal(w.forward(x, ids, wts), fresh.forward(x, ids, wts))
        for layer in (w, fresh):
            layer.set_decode_impl("auto")
    _lib.check(_lib.lib().b200moe_layer_prepack(w._h, _lib.ptr(w.prepack), w.prepack.numel(), _lib.stream_ptr()), "prepack")
    assert torch.equal(w.forward(x, ids, wts), fresh.forward(x, ids, wts))
    w.status()


# Up to 8 tokens a block has three workers while its ring has two stages for each (hidden sizes up to 6656, 5888 from the checkpoint layout),
# then two; the largest hidden sizes leave them one stage each: 11264, and 11008 from the checkpoint layout. Above 8 tokens x takes twice the
# room: 5632 and 5376.
@pytest.mark.parametrize("hidden,ms", [(5376, (1, 9, 16)), (5504, (16,)), (5632, (9, 16)), (6144, (1, 8)), (7168, (1, 8)), (10496, (1, 8)), (11008, (1, 8)), (11264, (1, 8))])
def test_widest_layers(hidden, ms):
    cfg, w, ow = edge_layer(hidden, 128)
    for m in ms:
        x, ids, wts = inputs(cfg, m, 20 + m)
        check_layer_output(run(w, x, ids, wts), O.moe_reference(x.float().numpy(), ow, ids.numpy(), wts.numpy()), f"hidden {hidden}, {m} tokens")
        bare = bare_forward(w, x, ids, wts)
        if hidden > (11008 if m <= 8 else 5376):
            assert bare is None
        else:
            assert torch.equal(bare, w.forward(x.cuda(), ids.cuda(), wts.cuda()))


@pytest.mark.parametrize("hidden,m", [(11392, 1), (11392, 8), (5760, 9)])
def test_hidden_sizes_beyond_the_kernel_are_refused(hidden, m):
    import sm120fp4_b200._lib as L
    cfg, w, _ = edge_layer(hidden, 64)
    x, ids, wts = inputs(cfg, m, 3)
    with pytest.raises(L.B200MoEError):
        w.forward(x.cuda(), ids.cuda(), wts.cuda())
    w.status()


# Where K is cut and in which order partial sums are added follows from the shares of the tile list alone, not from how many workers deal
# with it: up to 8 tokens three workers a block have the bits of two, which run batches above 8 (here with a ninth token of empty slots).
# Few tiles a block (chains over all three workers) up to about 50.
@pytest.mark.parametrize("hidden,inter", [(3200, 64), (3328, 192), (4096, 320), (4096, 832)])
def test_sums_do_not_depend_on_the_number_of_workers(hidden, inter):
    cfg, w, _ = edge_layer(hidden, inter)
    for m in (1, 2, 5, 8):
        x, ids, wts = inputs(cfg, m, 30 + m)
        pad = 9 - m
        more = run(w, torch.cat([x, torch.zeros(pad, hidden, dtype=x.dtype)]), torch.cat([ids, torch.full((pad, cfg["top_k"]), -1, dtype=ids.dtype)]),
                   torch.cat([wts, torch.zeros(pad, cfg["top_k"])])).clone()
        assert torch.equal(run(w, x, ids, wts), more[:m]), m
    w.status()


# Calls of a wide layer overlap their launches: a chain of them, each on the output of the one before, gives what the calls give one by one.
def test_chained_wide_calls():
    cfg, w, _ = edge_layer(3200)
    for m in (2, 9):
        x, ids, wts = (t.cuda() for t in inputs(cfg, m, 60 + m))
        want = []
        y = x
        for _ in range(6):
            y = w.forward(y, ids, wts)
            torch.cuda.synchronize()
            want.append(y.clone())
            y = (y.float() / y.float().abs().amax()).to(torch.bfloat16)
        ys = [x]
        outs = []
        for _ in range(6):
            outs.append(w.forward(ys[-1], ids, wts))
            ys.append((outs[-1].float() / outs[-1].float().abs().amax()).to(torch.bfloat16))
        for _ in range(20):
            back_to_back = [w.forward(v, ids, wts) for v in ys[:6]]
        torch.cuda.synchronize()
        for a, b, c in zip(want, outs, back_to_back):
            assert torch.equal(a, b) and torch.equal(a, c)
    w.status()
