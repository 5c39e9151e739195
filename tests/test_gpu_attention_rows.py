"""Float32 prompts' attention: 16 (a warp has four rows) or 4 neighbouring rows of a sequence and head per block, 32 keys at a time in shared memory."""
from __future__ import annotations

import pytest
import torch

import maferax_util as mu
import pamasun_util as pu
import sunutar_util as su
import virusun_util as vu

pytestmark = pytest.mark.gpu
BAD = 60

# twelve heads: from 193 tokens on there are enough blocks of 16 rows for every SM
LAYERS = {
    "sink-penalty": lambda: (pu.config([pu.attn(heads=12, kv_heads=4, dim=64, vdim=64, scale=0.125, ff=0)], vocab=61, width=48), pu.engine_and_oracle),
    "odd": lambda: (pu.config([pu.attn(heads=12, kv_heads=3, dim=9, vdim=7, ff=0)], vocab=61, width=48), pu.engine_and_oracle),
    "wide-values": lambda: (pu.config([pu.attn(heads=12, kv_heads=12, dim=20, vdim=300, ff=0)], vocab=61, width=48), pu.engine_and_oracle),
    "no-room": lambda: (pu.config([pu.attn(heads=12, kv_heads=2, dim=400, vdim=500, scale=0.05, ff=0)], vocab=61, width=48), pu.engine_and_oracle),
    "window": lambda: (su.config([su.layer(su.left(heads=12, kv_heads=4, dim=24, vdim=20, window=37))], vocab=61, width=48), su.engine_and_oracle),
    "two-maps": lambda: (vu.config([vu.att(heads=12, kv_heads=4, dim=32, vdim=40)], vocab=61, width=48), vu.engine_and_oracle),
    "latent": lambda: (mu.config([mu.latent(heads=12, dim=16, rot_dim=8, vdim=12, q_rank=24, kv_rank=40)], vocab=61, width=48), mu.engine_and_oracle),
}


def spoil(w):
    w["embed"][BAD] = float("nan")


@pytest.mark.parametrize("name", LAYERS)
def test_rows_of_prompts(name):
    """Last blocks and last tiles of any size, sequences of a few rows beside long ones, a second portion behind cached keys; both block heights."""
    cfg, make = LAYERS[name]()
    model, orc, _ = make(cfg, seed=7, max_tokens=2048, max_seqs=4, page_size=16, max_step_tokens=512)
    for lens, second in (((211, 9, 33, 1), (10, 21, 65, 9)), ((9, 17), (12, 31))):
        toks = [pu.tokens(a + b, 61, a) for a, b in zip(lens, second)]
        want = [orc.forward(t) for t in toks]
        seqs, at = [model.open_sequence() for _ in lens], [0] * len(lens)
        for part in (lens, second):
            got = model.forward([(s, t[a:a + n], list(range(n))) for s, t, a, n in zip(seqs, toks, at, part)]).clone()
            row = 0
            for i, n in enumerate(part):
                assert pu.rel_err(torch.cat([got[row:row + n].cpu().double(), want[i][-1:].double()]), torch.cat([want[i][at[i]:at[i] + n].double(), want[i][-1:].double()])) < pu.TOL[torch.float32]
                row += n
                at[i] += n
        for s in seqs:
            model.close_sequence(s)
    model.check_device_errors()


@pytest.mark.parametrize("name", ["sink-penalty", "window", "two-maps", "latent"])
def test_rows_take_nothing_from_keys_they_do_not_see(name):
    """A token that is not finite leaves the logits of every earlier one of its block as they are."""
    cfg, make = LAYERS[name]()
    model, _, _ = make(cfg, seed=8, edit=spoil, max_step_tokens=256)
    toks = [t % BAD for t in pu.tokens(200, 61, 3)]

    def logits(row):
        seq = model.open_sequence()
        out = model.forward([(seq, row, list(range(len(row))))])[:, :BAD].clone()      # (a tied head has that token's column)
        model.close_sequence(seq)
        return out

    want = logits(toks)
    for at in range(160, 178):
        got = logits(toks[:at] + [BAD] + toks[at + 1:])
        assert torch.equal(got[:at], want[:at])
        assert not bool(got[at].isfinite().any())


@pytest.mark.parametrize("window", [20, 32, 37])
@pytest.mark.parametrize("sizes", [(231,), (110, 121), (103, 130)])
def test_window_rows_do_not_depend_on_their_block(sizes, window):
    """A row's bits are those of blocks of 16 rows and of blocks of 4 (a prompt beside three others, and alone): what its block's first row sees does not matter."""
    cfg = su.config([su.layer(su.left(heads=12, kv_heads=4, dim=24, vdim=20, window=window))], vocab=61, width=48)
    model, orc, _ = su.engine_and_oracle(cfg, seed=13, max_tokens=4096, max_seqs=4, page_size=16, max_step_tokens=1024)
    toks, beside = pu.tokens(sum(sizes), 61, window), pu.tokens(sum(sizes), 61, 1)

    def logits(others):
        seqs, at, out = [model.open_sequence() for _ in range(1 + others)], 0, []
        for n in sizes:
            out.append(model.forward([(seqs[0], toks[at:at + n], list(range(n)))] + [(s, beside[at:at + n], []) for s in seqs[1:]]).clone())
            at += n
        for s in seqs:
            model.close_sequence(s)
        return torch.cat(out)

    alone = logits(0)
    assert pu.rel_err(alone, orc.forward(toks)) < pu.TOL[torch.float32]
    assert torch.equal(logits(3), alone)
    model.check_device_errors()


@pytest.mark.parametrize("dim,vdim", [(20, 300), (130, 130), (136, 144), (160, 20)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32], ids=["bf16", "f32"])
def test_wide_heads_of_whole_pieces_and_others(dim, vdim, dtype):
    """Both kernels of prompts' attention without a tensor-core form, on either side of their rule: whole 16-byte pieces or not, few blocks and many."""
    cfg = pu.config([pu.attn(heads=12, kv_heads=2, dim=dim, vdim=vdim, scale=dim ** -0.5, ff=0)], vocab=61, width=48)
    model, orc, _ = pu.engine_and_oracle(cfg, seed=14, dtype=dtype, max_tokens=4096, max_seqs=4, page_size=16, max_step_tokens=1024)
    for lens in ((9,), (181, 33), (250, 240, 230, 210)):
        toks = [pu.tokens(n, 61, n) for n in lens]
        seqs = [model.open_sequence() for _ in lens]
        got = model.forward([(s, t, list(range(n))) for s, t, n in zip(seqs, toks, lens)]).cpu()
        assert pu.rel_err(got, torch.cat([orc.forward(t) for t in toks])) < pu.TOL[dtype]
        for s in seqs:
            model.close_sequence(s)
    model.check_device_errors()
