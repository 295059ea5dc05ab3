"""Weights off a 16-byte boundary: pointer tables only promise the block struct's two bytes (q4_k.hpp:45-52 of the reference)."""
import copy

import pytest
import torch

from sager_b200 import lib, ops, synth
from sager_b200.layer import MoeLayerRunner, PrefillLayer
from tests.util import DEV, f16_close, make_q4k, make_x16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [2, 4, 6, 8, 12])
@pytest.mark.parametrize("H,F", [(512, 256), (1024, 512)])
def test_weights_at_every_alignment_give_the_same_bits(H, F, shift):
    """Experts on 2-, 4- and 8-byte boundaries are copied by other instructions than aligned ones: the same layer, in the chunk
    (whole and ragged row tiles) and in every decode kernel."""
    E, K = 12, 4
    w = synth.MoeWeights(H, F, E, DEV, seed=95, std=0.05)
    v = copy.copy(w)
    v.__dict__.pop("_tables", None)
    big = torch.empty(w.blob.numel() + 16, dtype=torch.uint8, device=DEV)
    v.blob = big[shift:shift + w.blob.numel()].view(w.blob.shape)
    v.blob.copy_(w.blob)
    got = []
    for m in (w, v):
        outs = []
        for n in (70, 200):
            x16 = synth.normal_fp16((n, H), 96 + n, DEV)
            x = x16.clone()
            PrefillLayer(n, H, F, E, K, DEV).run(n, x16, x, m, m.table())
            outs.append(x)
        for n, kernel in ((1, None), (3, None), (4, None), (2, "items"), (9, "rows"), (40, "rows")):
            x16 = synth.normal_fp16((n, H), 97 + n, DEV)
            x = x16.clone()
            r = MoeLayerRunner(n, H, F, E, K, DEV)
            r.run(r.args(n, x16, m.router, m.table(), m.shared_ptrs(), x_f16=x), kernel=kernel)
            torch.cuda.synchronize()
            outs.append(x)
        got.append(outs)
    assert all(torch.equal(a.view(torch.int16), b.view(torch.int16)) for a, b in zip(*got))
    assert lib().raw("sgr_status")(0) == 0


@pytest.mark.parametrize("shift", [0, 2, 4, 8])
def test_ragged_row_tiles_at_every_alignment(oracle, shift):
    n_rows, k = 200, 768
    w_np, w_dev = make_q4k(n_rows, k, 61)
    big = torch.empty(w_dev.numel() + 16, dtype=torch.uint8, device=DEV)
    big[shift:shift + w_dev.numel()] = w_dev.reshape(-1)
    tab = torch.tensor([big.data_ptr() + shift], dtype=torch.int64, device=DEV)
    x_np, x_dev = make_x16(21, k, 62)
    xq = torch.zeros(21, k // 256 * 276, dtype=torch.uint8, device=DEV)
    ops.quantize_q8_k(x_dev, xq, 21 * k)
    y = torch.zeros(21, n_rows, dtype=torch.float16, device=DEV)
    ops.moe_grouped_gemm_i8(tab, torch.tensor([0, 21], dtype=torch.int32, device=DEV), xq, y, n_rows, k, 1)
    for r in (0, 20):
        assert f16_close(y[r].cpu().numpy(), oracle.gemv(w_np, xq.cpu().numpy()[r], n_rows, k)), r
