"""Few-token attention with two states per range (first and second halves of 64 keys): the same bits with one warp per query row and with two, and nothing that
is not a number gets lost where the two are joined."""
from __future__ import annotations

import pytest
import torch

import pamasun_util as pu
import sunutar_util as su
import virusun_util as vu

pytestmark = pytest.mark.gpu
BAD = 60
# heads over their own keys: a sequence alone leaves every block an SM to itself, four together do not
LAYERS = {
    "sink-penalty": lambda: (pu.config([pu.attn(heads=12, kv_heads=12, dim=64, vdim=64, scale=0.125, ff=0)], vocab=61, width=48), pu.engine_and_oracle),
    "odd": lambda: (pu.config([pu.attn(heads=12, kv_heads=12, dim=9, vdim=7, ff=0)], vocab=61, width=48), pu.engine_and_oracle),
    "window": lambda: (su.config([su.layer(su.left(heads=12, kv_heads=12, dim=24, vdim=20, window=77))], vocab=61, width=48), su.engine_and_oracle),
    "two-maps": lambda: (vu.config([vu.att(heads=12, kv_heads=12, dim=32, vdim=40)], vocab=61, width=48), vu.engine_and_oracle),
}
MANY = 16


def spoil(w):
    w["embed"][BAD] = float("nan")


def decoded(model, rows, portions):
    """Logits of the last token of every row, the rows in front of it brought in `portions`, all sequences in one step."""
    seqs, at = [model.open_sequence() for _ in rows], 0
    for n in portions + [1]:
        got = model.forward([(s, r[at:at + n], [n - 1]) for s, r in zip(seqs, rows)])[:, :BAD].clone()
        at += n
    for s in seqs:
        model.close_sequence(s)
    return got


KEYS = (32, 33, 34, 63, 64, 65, 95, 96, 97, 130)


# (the layer beside the window's adds in another order in front of a hundred tokens or so, depending on the step)
@pytest.mark.parametrize("name,n", [(name, n) for name in LAYERS for n in ((101, 110, 111, 128, 135) if name == "window" else KEYS)])
def test_decoding_does_not_depend_on_the_other_sequences(name, n):
    """A sequence's `n`-th token decoded alone and beside fifteen others: the number of keys around half a round and a round."""
    cfg, make = LAYERS[name]()
    model, orc, _ = make(cfg, seed=12, edit=spoil, max_tokens=8192, max_seqs=MANY, page_size=16, max_step_tokens=MANY * 136)
    rows = [[t % BAD for t in pu.tokens(n, 61, 10 * i + n)] for i in range(MANY)]
    together = decoded(model, rows, [n - 1])
    for i in (0, 7, MANY - 1):
        assert torch.equal(decoded(model, rows[i:i + 1], [n - 1])[0], together[i])
    want = [orc.forward(r) for r in rows[:3]]
    for i, w in enumerate(want):
        assert pu.rel_err(torch.cat([together[i:i + 1].cpu().double(), w[:-1, :BAD].double()]), w[[-1] + list(range(n - 1)), :BAD].double()) < pu.TOL[torch.float32]
    model.check_device_errors()


@pytest.mark.parametrize("name", ["sink-penalty", "odd", "two-maps"])
@pytest.mark.parametrize("lo,hi", [(32, 64), (0, 32), (40, 41), (0, 64)])
def test_keys_that_are_not_numbers_show(name, lo, hi):
    """All keys of a range's second half (or its first, or a single one, or both halves) are not numbers, those of the next range and the decoded token are."""
    cfg, make = LAYERS[name]()
    model, _, _ = make(cfg, seed=12, edit=spoil, max_tokens=8192, max_seqs=MANY, page_size=16, max_step_tokens=MANY * 136)
    rows = [[BAD if lo <= j < hi else t % BAD for j, t in enumerate(pu.tokens(80, 61, 3 * i))] for i in range(MANY)]
    alone, together = decoded(model, rows[:1], [79]), decoded(model, rows, [79])
    assert not bool(alone.isfinite().any()) and not bool(together.isfinite().any())
