"""GPU parity of the W4A16 mid-batch path (17 tokens up to a few hundred in one call) against the oracle's W4A16 arithmetic
(sm120fp4/kernels/bench_moe_baseline.py:53-74) and against the 16-token slices it replaces."""
import pytest
import torch

from helpers import check_layer_output, make_layer
from oracle import nvfp4_oracle as O
from test_gpu_decode import inputs, layer

pytestmark = pytest.mark.gpu


def run_mid(w, x, ids, wts, max_tokens=256):
    if w.mid is None or w.mid.max_tokens < max_tokens:
        w.enable_mid(max_tokens=max_tokens)
    out = w.forward(x.cuda(), ids.cuda(), wts.cuda())
    w.mid_status()
    return out


@pytest.mark.parametrize("name,m", [("tiny", 33), ("tiny", 40), ("tiny", 130), ("mid", 33), ("mid", 64), ("mid", 255), ("odd", 100), ("gemma", 48)])
def test_mid_batches_match_the_w4a16_oracle(name, m):
    cfg, w, ow = layer(name)
    x, ids, wts = inputs(cfg, m, 700 + m)
    out = run_mid(w, x, ids, wts)
    err, rel = check_layer_output(out, O.moe_reference(x.float().numpy(), ow, ids.numpy(), wts.numpy()), f"mid {name} m={m}")
    print(f"mid {name} m={m}: max-abs/rms {err:.2e} normwise {rel:.2e}")


def test_mid_is_deterministic_row_independent_and_close_to_the_slices():
    cfg, w, ow = layer("mid")
    x, ids, wts = inputs(cfg, 96, 31)
    slices = w.forward(x.cuda(), ids.cuda(), wts.cuda()).clone()        # without the mid path: slices of 16
    a = run_mid(w, x, ids, wts).clone()
    for _ in range(3):
        assert torch.equal(run_mid(w, x, ids, wts), a)
    perm = torch.randperm(96, generator=torch.Generator().manual_seed(5))
    b = run_mid(w, x[perm], ids[perm], wts[perm])
    assert torch.equal(b, a[perm.cuda()])                                # a token's output does not depend on its neighbours
    rms = float(a.float().pow(2).mean().sqrt())
    assert float((a.float() - slices.float()).abs().max()) <= 2e-2 * rms  # same arithmetic up to summation order and bf16 rounding
    # masked slots (expert-parallel shards) and a fully masked row
    masked = ids.clone()
    masked[:, 1] = -1
    masked[0, :] = -1
    wz = wts.clone()
    wz[masked < 0] = 0
    out = run_mid(w, x, masked, wz)
    check_layer_output(out, O.moe_reference(x.float().numpy(), ow, ids.numpy(), wz.numpy()), "mid masked")
    assert float(out[0].float().abs().max()) == 0.0


# Up to 1024 pairs, and hidden sizes up to 2048, there is no plan kernel: the same tokens in a batch beyond that give the same bits.
@pytest.mark.parametrize("hidden,m,more", [(256, 128, 129), (256, 33, 200), (2048, 100, 140), (2304, 100, 140)])
def test_mid_batches_on_both_sides_of_the_plan_kernel(hidden, m, more):
    cfg = dict(experts=24, hidden=hidden, inter=128, top_k=8)
    w, _ = make_layer(**cfg, seed=6)
    x, ids, wts = inputs(cfg, more, 60 + m)
    ids, wts = ids.clone(), wts.clone()
    ids[m // 2, 1], wts[m // 2, 1] = -1, 0
    whole = run_mid(w, x, ids, wts).clone()
    assert torch.equal(run_mid(w, x[:m], ids[:m], wts[:m]), whole[:m])


# The last kernel takes eight slots at a time above four slots where it has one to two blocks an SM (a token of 2048 columns is a block), else four: numbers of slots
# that are no multiple of either, on both sides of both ends (the same bits; the form for four is what the tests above hold to the oracle).
@pytest.mark.parametrize("top_k", [3, 5, 8, 9, 16])
def test_mid_batches_on_both_sides_of_the_combine(top_k):
    cfg = dict(experts=24, hidden=2048, inter=64, top_k=top_k)
    w, _ = make_layer(**cfg, seed=6)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    x, ids, wts = inputs(cfg, 2 * sms + 1, 80 + top_k)
    ids, wts = ids.clone(), wts.clone()
    ids[50, top_k - 1], wts[50, top_k - 1] = -1, 0
    whole = run_mid(w, x, ids, wts, 512).clone()
    for m in (2 * sms, sms + 1, sms):
        assert torch.equal(run_mid(w, x[:m], ids[:m], wts[:m], 512), whole[:m])


def test_qwen_shape_mid_batches():
    cfg, w, ow = layer("qwen")
    for m in (40, 128):
        x, ids, wts = inputs(cfg, m, 8100 + m)
        out = run_mid(w, x, ids, wts)
        check_layer_output(out, O.moe_reference(x.float().numpy(), ow, ids.numpy(), wts.numpy()), f"mid qwen m={m}")


# Outputs (bf16 bits) that move by one step when the order of roundings in a term sum changes - FC1 rounds a term's product before it
# adds it, FC2 does not - as this path has computed them from its first form on.
@pytest.mark.parametrize("m,want", [(40, {(1, 238): -17320, (1, 426): 15468, (1, 440): -18272, (1, 498): -17332, (6, 166): 14253}),
                                    (90, {(7, 11): 14738, (7, 133): 15404, (7, 157): -17462, (7, 354): -17398, (7, 482): -17682, (8, 86): -17929})])
def test_mid_roundings_are_pinned(m, want):
    cfg = dict(experts=12, hidden=512, inter=640, top_k=4)
    w, _ = make_layer(**cfg, seed=1)
    bits = run_mid(w, *inputs(cfg, m, 900 + m)).cpu().view(torch.int16)
    assert {at: int(bits[at]) for at in want} == want
