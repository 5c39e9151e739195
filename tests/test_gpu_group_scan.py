"""The gated delta rule's scan of four tokens at a time on heads that fill its tiles: nothing is cleared there but the tokens that a last group lacks."""
from __future__ import annotations

import pytest
import torch

import virusun_util as vu
from pamasun_util import tokens

pytestmark = pytest.mark.gpu
BAD = 60


def spoil(w):
    w["embed"][BAD] = float("nan")


@pytest.mark.parametrize("dim,poison,lens", [(64, 128, (33, 34, 35, 61, 63, 32, 30, 1)), (128, 64, (33, 34, 35, 61, 63, 32, 30, 1)), (256, 48, (17, 18, 19, 30, 31, 16, 13, 1))])
def test_missing_tokens_of_a_last_group(dim, poison, lens):
    """The last group lies in either half of the double buffer.  In front of the sequences under test, the same launch runs more blocks than the SMs hold at once
    over tokens that are not a number, so that shared memory holds those where nothing was written; then two decoded tokens on the state left behind."""
    cfg = vu.config([vu.delta(heads=2, kv_heads=1, dim=dim, vdim=dim, conv=4)], vocab=61, width=48)
    whole = 64 if dim <= 128 else 32                      # both halves full
    model, orc, _ = vu.engine_and_oracle(cfg, seed=11, edit=spoil, max_seqs=poison + len(lens), max_step_tokens=8960, max_tokens=20000)
    toks = [[t % BAD for t in tokens(n + 2, 61, n)] for n in lens]
    want = [orc.forward(t) for t in toks]
    bad = [model.open_sequence() for _ in range(poison)]
    seqs = [model.open_sequence() for _ in lens]
    parts = [(s, [BAD] * whole, []) for s in bad] + [(s, t[:n], list(range(n))) for s, t, n in zip(seqs, toks, lens)]
    at = [0] * len(lens)
    for new in (parts, *[[(s, [t[n + k]], [0]) for s, t, n in zip(seqs, toks, lens)] for k in range(2)]):
        got = model.forward(new).cpu()
        row = 0
        for i, n in enumerate(lens if new is parts else [1] * len(lens)):
            # a row of its own spread says little: the sequence's rows so far go with it
            assert vu.rel_err(torch.cat([got[row:row + n, :BAD].double(), want[i][:, :BAD].double()]),
                              torch.cat([want[i][at[i]:at[i] + n, :BAD].double(), want[i][:, :BAD].double()])) < vu.TOL[torch.float32]
            row += n
            at[i] += n
    for s in bad + seqs:
        model.close_sequence(s)
    model.check_device_errors()
