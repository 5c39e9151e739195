"""Residual, embedding and final norms on rows held in registers: widths around a piece, a warp's and a block's row, on both sides of the rows that give each a warp."""
from __future__ import annotations

import pytest
import torch

import maferax_util as mu
from pamasun_util import TOL, attn, config, delta, engine_and_oracle, rel_err, tokens

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [4, 124, 128, 132, 764, 768, 772, 1532, 1536, 1540, 2044, 2048, 2052, 50])
@pytest.mark.parametrize("rows", [1, 511, 512, 515])
def test_norms_of_rows(width, rows):
    """A sequence's whole prompt, every position's logits; widths beyond 2048 or not of whole 16-byte pieces take the general kernels."""
    cfg = config([attn(heads=1, kv_heads=1, dim=8, vdim=8, ff=16)], vocab=33, width=width)
    model, orc, _ = engine_and_oracle(cfg, seed=9, max_step_tokens=520)
    toks = tokens(rows, 33, rows)
    seq = model.open_sequence()
    got = model.forward([(seq, toks, list(range(rows)))]).clone()
    model.close_sequence(seq)
    keep = slice(None) if rows < 8 else slice(2, None)
    assert rel_err(got[keep], orc.forward(toks)[keep]) < TOL[torch.float32]


@pytest.mark.parametrize("vdim", [64, 128, 60, 132])
def test_ends_of_recurrences(vdim):
    """Rows of 64 and 128 columns as 16-byte pieces, others element by element; both gates and norm weights."""
    for cfg, make in ((config([delta(heads=3, dim=vdim, ff=0, rank=5)], vocab=61, width=48), engine_and_oracle),
                      (mu.config([mu.gla(heads=3, dim=16, vdim=vdim)], vocab=61, width=48), mu.engine_and_oracle)):
        model, orc, _ = make(cfg, seed=10, max_step_tokens=256)
        toks = tokens(37, 61, vdim)
        seq = model.open_sequence()
        got = model.forward([(seq, toks, list(range(37)))]).clone()
        model.close_sequence(seq)
        assert rel_err(got, orc.forward(toks)) < TOL[torch.float32]


@pytest.mark.parametrize("width", [4, 128, 132, 764, 768, 1540, 2048])
def test_a_row_does_not_depend_on_the_number_of_rows(width):
    """A sequence alone, whose rows have a block each, and beside another, where they have a warp each: the same bits."""
    cfg = config([attn(heads=1, kv_heads=1, dim=8, vdim=8, ff=16)], vocab=33, width=width)
    model, _, _ = engine_and_oracle(cfg, seed=9, max_step_tokens=520)
    toks, other = tokens(300, 33, width), tokens(215, 33, 1)
    seqs = [model.open_sequence() for _ in range(3)]
    alone = model.forward([(seqs[0], toks, list(range(300)))]).clone()
    both = model.forward([(seqs[1], toks, list(range(300))), (seqs[2], other, list(range(215)))]).clone()      # all rows through the final norm as well
    assert torch.equal(alone, both[:300])
    for s in seqs:
        model.close_sequence(s)


@pytest.mark.parametrize("dim,vdim", [(4, 4), (60, 64), (64, 60), (68, 4), (128, 124), (132, 8), (6, 8), (8, 6), (62, 64)])
def test_preparation_of_attention_rows(dim, vdim):
    """Heads of whole 16-byte pieces up to 128 elements, sixteen and thirty-two pieces a unit, and those that are not: a prompt, then tokens behind it."""
    cfg = config([attn(heads=3, kv_heads=1, dim=dim, vdim=vdim, ff=0)], vocab=61, width=48)
    model, orc, _ = engine_and_oracle(cfg, seed=15)
    toks = tokens(26, 61, dim)
    seq, at, got = model.open_sequence(), 0, []
    for n in (21, 3, 1, 1):
        got.append(model.forward([(seq, toks[at:at + n], list(range(n)))]).clone())
        at += n
    model.close_sequence(seq)
    assert rel_err(torch.cat(got), orc.forward(toks)) < TOL[torch.float32]
    model.check_device_errors()
