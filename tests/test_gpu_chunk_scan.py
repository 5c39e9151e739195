"""The recurrences' scan by chunks of sixteen tokens (prompts of 256 tokens and more; with more than 64 key channels of 144 to 208, the gated delta rule above
128 channels of 320)."""
from __future__ import annotations

import pytest
import torch

import bizulix_util as bu
import maferax_util as mu
import pamasun_util as pu
import virusun_util as vu

pytestmark = pytest.mark.gpu
TOL = pu.TOL[torch.float32]


def layers_of(dim):
    """One layer of every form: removal per channel, decay per channel, gated delta rule over shared keys, mLSTM with its unit column, decay per head."""
    return [(pu.config([pu.delta(heads=3, dim=dim, ff=0, rank=5)], vocab=61, width=48), pu.engine_and_oracle),
            (mu.config([mu.gla(heads=2, dim=dim, vdim=11)], vocab=61, width=48), mu.engine_and_oracle),
            (vu.config([vu.delta(heads=4, kv_heads=2, dim=dim, vdim=9, conv=3)], vocab=61, width=48), vu.engine_and_oracle),
            (vu.config([vu.par(b=vu.right(heads=2, dim=dim, vdim=8))], vocab=61, width=48), vu.engine_and_oracle),
            (bu.config([bu.ret(heads=2, dim=dim + dim % 2, vdim=12)], vocab=61, width=48), bu.engine_and_oracle)]


@pytest.mark.parametrize("form", range(5))
@pytest.mark.parametrize("dim", [5, 32, 33, 64, 96, 200])
def test_scan_by_chunks(dim, form):
    """Padded key channels, last chunks of any size, a sequence shorter than a chunk and a single token beside long ones; then a second long portion on the
    state left behind, then a short one that the four-token scan takes on; against the oracles."""
    cfg, make = layers_of(dim)[form]
    lens, second, third = ((273, 256, 19, 1), (257, 3, 260, 31), (20, 1, 5, 33)) if dim <= 128 else ((337, 320, 19, 1), (321, 3, 324, 31), (20, 1, 5, 33))
    model, orc, _ = make(cfg, seed=4, max_tokens=4096, max_seqs=4, page_size=16, max_step_tokens=704)
    toks = [pu.tokens(a + b + c, 61, a) for a, b, c in zip(lens, second, third)]
    want = [orc.forward(t) for t in toks]
    seqs, at = [model.open_sequence() for _ in lens], [0] * 4
    for part in (lens, second, third):
        got = model.forward([(s, t[a:a + n], list(range(n))) for s, t, a, n in zip(seqs, toks, at, part)]).clone()
        row = 0
        for i, n in enumerate(part):
            if at[i] + n > 1:
                lo = 1 if at[i] == 0 and n > 1 else 0                # the first row's spread says nothing about the scan
                assert pu.rel_err(got[row + lo:row + n], want[i][at[i] + lo:at[i] + n]) < TOL
            row += n
            at[i] += n
    for s in seqs:
        model.close_sequence(s)
    model.check_device_errors()


@pytest.mark.parametrize("n", [150, 161, 225])
def test_two_blocks_of_columns_per_block(n):
    """More blocks of columns than SMs above 64 channels: two per block of threads, the last one alone (13 blocks of columns of 12 heads)."""
    for cfg, make in ((pu.config([pu.delta(heads=12, dim=104, ff=0, rank=5)], vocab=61, width=48), pu.engine_and_oracle),
                      (mu.config([mu.gla(heads=12, dim=96, vdim=100)], vocab=61, width=48), mu.engine_and_oracle)):
        model, orc, _ = make(cfg, seed=6, max_step_tokens=256)
        toks = pu.tokens(n, 61, n)
        seq = model.open_sequence()
        got = model.forward([(seq, toks, list(range(n)))]).clone()
        model.close_sequence(seq)
        assert pu.rel_err(got, orc.forward(toks)) < TOL


@pytest.mark.parametrize("form", range(4))
def test_tokens_take_nothing_from_later_ones_of_their_chunk(form):
    """A token that is not finite leaves the logits of every earlier one as they are, whatever its place in the chunk."""
    bad = 60
    cfg, make = layers_of(16)[form]
    model, _, _ = make(cfg, seed=5, edit=spoil, max_step_tokens=512)
    toks = [t % bad for t in pu.tokens(290, 61, 1)]

    def logits(row):
        seq = model.open_sequence()
        out = model.forward([(seq, row, list(range(len(row))))]).clone()
        model.close_sequence(seq)
        return out

    want = logits(toks)
    for at in range(256, 273):
        got = logits(toks[:at] + [bad] + toks[at + 1:])
        assert torch.equal(got[:at], want[:at])
        assert not bool(got[at:].isfinite().any())


def spoil(w):
    w["embed"][60] = float("nan")


def test_both_forms_on_either_side_of_the_rule():
    """Sixteen channels take chunks while a step has few blocks of columns: one sequence by chunks, four together four tokens at a time, alike beyond rounding."""
    for form in (1, 2, 3):
        cfg, make = layers_of(16)[form]
        wide = {"heads": 12, "vdim": 16}
        layer = cfg["layers"][0]["mixer"]
        (layer["right"] if "right" in layer else layer).update(wide, **({"kv_heads": 12} if "kv_heads" in layer else {}))
        model, orc, _ = make(cfg, seed=8, max_tokens=8192, max_seqs=16, page_size=16, max_step_tokens=16 * 264)
        toks = pu.tokens(264, 61, form)
        want = orc.forward(toks)
        for many in (1, 16):
            seqs = [model.open_sequence() for _ in range(many)]
            got = model.forward([(s, toks, list(range(264)) if s is seqs[-1] else []) for s in seqs]).clone()
            assert pu.rel_err(got[1:], want[1:]) < TOL
            for s in seqs:
                model.close_sequence(s)
        model.check_device_errors()


@pytest.mark.parametrize("make", [lambda n: vu.engine_and_oracle(vu.config([vu.delta(heads=4, kv_heads=2, dim=128, vdim=128)], vocab=61, width=48), seed=4, max_step_tokens=n),
                                  lambda n: vu.engine_and_oracle(vu.config([vu.par(b=vu.right(heads=4, dim=128, vdim=128))], vocab=61, width=48), seed=4, max_step_tokens=n)])
def test_no_room_for_records_that_no_step_makes(make):
    """The gated delta rule's and the mLSTM's scan of shorter prompts has none: an engine for 192 tokens a step keeps none, one for 224 does."""
    size = {n: make(n)[0]._workspace.numel() for n in (160, 192, 224, 256)}
    assert size[224] - size[192] > 2 * (size[192] - size[160])
    assert size[256] - size[224] < size[224] - size[192]
