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
