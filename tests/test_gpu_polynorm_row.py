"""One token's PolyNorm feed-forward, whose activation rides in the down-projection's prologue, against two tokens' (two kernels) and the
float64 oracle: rows of a few pieces and of 2048 elements and more (16 warps), outputs of whole and ragged blocks of 8 and 16 columns,
a row too long for shared memory (two kernels again)."""
import pytest
import torch

from pamasun_util import TOL, attn, config, engine_and_oracle, rel_err, tokens

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,ff", [(64, 8), (72, 40), (64, 1000), (96, 2048), (72, 2056), (64, 4608), (2376, 64), (64, 24312), (64, 24576)])
def test_one_row_against_two(width, ff):
    cfg = config([attn(ff=ff)], vocab=61, width=width)
    model, orc, _ = engine_and_oracle(cfg, seed=3, dtype=torch.bfloat16)
    a, b = tokens(1, 61, seed=1), tokens(1, 61, seed=2)

    def step(rows):
        seqs = [model.open_sequence() for _ in rows]
        out = model.forward([(q, t, [0]) for q, t in zip(seqs, rows)]).clone()
        for q in seqs:
            model.close_sequence(q)
        return out

    alone, both = step([a]), step([a, b])
    model.check_device_errors()
    want = orc.forward(a)
    assert rel_err(alone, want) < TOL[torch.bfloat16]
    # the same roundings but for the order of PolyNorm's sums: a bf16 activation in some thousand moves by one place (2^-8 of it)
    assert rel_err(alone, both[:1]) < 2.0 ** -8


@pytest.mark.parametrize("width,ff", [(64, 48), (64, 1000), (64, 2040), (96, 2048), (72, 4104), (64, 24312)])
def test_one_row_has_the_bits_it_has_beside_another(width, ff):
    """The sums of PolyNorm are taken in the same order whichever kernel takes the row: 8 warps of the down-projection (up to 2040
    elements) or 16, or a kernel of its own."""
    cfg = config([attn(ff=ff)], vocab=61, width=width)
    model, _, _ = engine_and_oracle(cfg, seed=3, dtype=torch.bfloat16)
    rows = [tokens(1, 61, seed=s) for s in range(1, 9)]
    for i in range(0, 8, 2):
        seqs = [model.open_sequence() for _ in range(2)]
        both = model.forward([(q, t, [0]) for q, t in zip(seqs, rows[i:i + 2])]).clone()
        for q in seqs:
            model.close_sequence(q)
        for j in range(2):
            seq = model.open_sequence()
            alone = model.forward([(seq, rows[i + j], [0])]).clone()
            model.close_sequence(seq)
            assert torch.equal(alone, both[j:j + 1])
    model.check_device_errors()
