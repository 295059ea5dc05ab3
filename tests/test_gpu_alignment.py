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


class Scattered:
    """The weights of `w`, every matrix at an offset of its own from a 16-byte boundary (shared expert included)."""

    def __init__(self, w, offset_of):
        self.router, E = w.router, w.n_expert
        addr = []
        self.keep = []
        for e in range(E + 1):
            for m in range(3):
                src = w.matrix(e, m)
                buf = torch.empty(src.numel() + 16, dtype=torch.uint8, device=DEV)
                o = offset_of(e, m)
                buf[o:o + src.numel()] = src
                self.keep.append(buf)
                addr.append(buf.data_ptr() + o)
        self.tab = torch.tensor(addr[:3 * E], dtype=torch.int64).view(E, 3).t().contiguous().to(DEV)
        self.sh = addr[3 * E:]

    def table(self):
        return self.tab

    def shared_ptrs(self):
        return self.sh


# (gate, up, down): the narrower boundary on either side, in down alone, and whole experts on a 16-byte boundary in between, so
# that a ring slot is filled by the TMA unit and by the warp's own stores in turn
MIXED = [(0, 2, 0), (0, 0, 0), (2, 0, 4), (4, 2, 8), (0, 0, 2), (2, 8, 6), (0, 0, 0), (8, 4, 0), (4, 0, 2), (12, 6, 0), (0, 0, 0)]


@pytest.mark.parametrize("turn", [0, 4, 7])
@pytest.mark.parametrize("H,F", [(512, 256), (1024, 512)])
def test_every_matrix_at_an_alignment_of_its_own(H, F, turn):
    """A table promises each pointer by itself: gate, up and down of an expert on different boundaries, aligned experts among
    them, in both forms of the chunk and in every decode kernel."""
    E, K = 12, 4
    w = synth.MoeWeights(H, F, E, DEV, seed=95, std=0.05)
    v = Scattered(w, lambda e, m: MIXED[(e + turn) % len(MIXED)][m])
    assert {p % 16 for p in v.tab.flatten().tolist()} == {0, 2, 4, 6, 8, 12}
    got = []
    for m in (w, v):
        outs = []
        for n in (70, 200):                     # row-streaming GEMM, tcgen05 GEMM
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
