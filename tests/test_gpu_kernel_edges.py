"""Kernels at the sizes where their tiles end: edges, remainders, the smallest and largest of a dispatch's range."""
from __future__ import annotations

import pytest
import torch

from pamasun_util import TOL, attn, config, delta, engine_and_oracle, rel_err, tokens

pytestmark = pytest.mark.gpu


def product_bound(a, w):
    """|error| of an fp32 sum of K products, any order, each addition off by at most 2^-23 of the sum of absolute products."""
    return (a.double().abs() @ w.double().abs().T) * (a.shape[1] * 2.0 ** -23)


FEW_ROWS = ((1, 1, 8), (1, 16, 24), (7, 17, 40), (8, 771, 2040), (9, 15, 2048), (16, 33, 2056), (17, 64, 264), (31, 50, 4104), (32, 8, 1528), (33, 48, 64),
            (2, 8192, 1536), (5, 2369, 4096), (8, 2367, 264), (13, 2368, 72), (25, 2400, 2072))


@pytest.mark.parametrize("M,N,K", FEW_ROWS)
def test_products_of_few_rows(M, N, K):
    """At most 32 rows; blocks of 8 weight rows (16 from 2368 columns on), K shared by 8 or 16 warps in steps of 32."""
    model, _, _ = engine_and_oracle(config([attn(ff=0)]), seed=9, dtype=torch.bfloat16)
    g = torch.Generator(device="cuda").manual_seed(M * 31 + K)
    a, w = (torch.randn(r, K, device="cuda", generator=g).bfloat16() for r in (M, N))
    err = (model.linear(a, w).double() - a.double() @ w.double().T).abs()
    assert bool((err <= product_bound(a, w)).all())


MANY_ROWS = ((257, 96, 64), (257, 4800, 72), (383, 97, 128), (384, 9600, 200), (512, 255, 72), (640, 257, 1000), (1025, 770, 520), (2048, 2049, 264),
             (300, 6400, 4608))


@pytest.mark.parametrize("M,N,K", MANY_ROWS)
def test_products_of_many_rows(M, N, K):
    """tcgen05 tiles of 64 to 256 columns: ragged rows, columns and last K stage, one tile per SM and several."""
    model, _, _ = engine_and_oracle(config([attn(ff=0)]), seed=9, dtype=torch.bfloat16)
    g = torch.Generator(device="cuda").manual_seed(M * 31 + K)
    a, w = (torch.randn(r, K, device="cuda", generator=g).bfloat16() for r in (M, N))
    err = (model.linear(a, w).double() - a.double() @ w.double().T).abs()
    assert bool((err <= product_bound(a, w)).all())


@pytest.mark.parametrize("M,N,K", [(3, 768, 4608), (5, 2400, 4096), (20, 768, 4608), (300, 768, 768), (300, 768, 4608), (1024, 4608, 1024), (600, 2049, 1000)])
def test_products_of_positive_values_lose_no_more_than_their_chains(M, N, K):
    """An MMA drops up to the last place (2^-23) of the sum it adds to, always downwards where all products are positive.  Few rows: every MMA
    starts from zero, so 2^-23 of the result.  Many rows: four chains of K / 64 MMAs whose sum grows evenly, so half of K / 64 places, and one for
    the four parts."""
    model, _, _ = engine_and_oracle(config([attn(ff=0)]), seed=9, dtype=torch.bfloat16)
    g = torch.Generator(device="cuda").manual_seed(M * 31 + K)
    a, w = (torch.rand(r, K, device="cuda", generator=g).bfloat16() for r in (M, N))
    want = a.double() @ w.double().T
    places = 1.0 if M <= 32 else 0.5 * -(-K // 64) + 1.0
    assert float(((model.linear(a, w).double() - want) / want).pow(2).mean().sqrt()) < places * 2.0 ** -23


@pytest.mark.parametrize("dtype,M", [(torch.bfloat16, 3), (torch.bfloat16, 40), (torch.bfloat16, 300), (torch.float32, 3), (torch.float32, 300)])
def test_a_product_waits_for_the_kernel_that_makes_its_weights(dtype, M):
    """linear()'s weights may come from the kernel just in front, and the products read weights before they wait for that kernel: every
    launch of the call depends on its predecessor as a whole (nothing is run here: the dependencies are read from the recorded graph)."""
    import ctypes

    model, _, _ = engine_and_oracle(config([attn(ff=0)]), seed=9, dtype=dtype)
    a, src = torch.randn(M, 256, device="cuda").to(dtype), torch.randn(128, 256, device="cuda")
    model.linear(a, src.to(dtype))
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        model.linear(a, (src * 2).to(dtype))
    edges = ctypes.CDLL("libcuda.so.1").cuGraphGetEdges_v2
    handle, n = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t()
    assert edges(handle, None, None, None, ctypes.byref(n)) == 0 and n.value > 0
    nodes, data = (ctypes.c_void_p * n.value), (ctypes.c_ubyte * (8 * n.value))()       # per edge: outgoing port, incoming port, type, 5 reserved
    assert edges(handle, nodes(), nodes(), data, ctypes.byref(n)) == 0
    assert list(data[2::8]) == [0] * n.value                                             # the plain dependency


F32_TILES = ((1, 1, 4), (16, 65, 36), (17, 64, 128), (64, 63, 132), (65, 130, 260), (300, 768, 1028), (31, 70, 2048), (512, 4700, 20), (640, 3841, 52))


@pytest.mark.parametrize("M,N,K", F32_TILES)
def test_float32_products(M, N, K):
    """16- and 64-row tiles, steps of 16 k with a ragged last one, K shared by 1 to 8 thread blocks."""
    model, _, _ = engine_and_oracle(config([attn(ff=0)]), seed=9)
    g = torch.Generator(device="cuda").manual_seed(M * 31 + K)
    a, w = (torch.randn(r, K, device="cuda", generator=g) for r in (M, N))
    err = (model.linear(a, w).double() - a.double() @ w.double().T).abs()
    assert bool((err <= product_bound(a, w)).all())


@pytest.mark.parametrize("N,K", [(768, 768), (4608, 768), (96, 4608), (2400, 1028), (70, 70)])
def test_float32_rows_do_not_depend_on_their_number(N, K):
    """A float32 row's product has the same bits whatever the number of rows beside it."""
    model, _, _ = engine_and_oracle(config([attn(ff=0)]), seed=9)
    g = torch.Generator(device="cuda").manual_seed(N + K)
    a, w = (torch.randn(r, K, device="cuda", generator=g) for r in (1300, N))
    whole = model.linear(a, w)
    for M in (1, 16, 17, 64, 65, 300, 700):
        assert torch.equal(model.linear(a[:M], w), whole[:M]), M


@pytest.mark.parametrize("n", [127, 128, 129, 135, 136])
def test_decay_preparation_over_groups_of_tokens(n):
    """128 tokens and more: eight tokens per block share the decay's second matrix; odd ranks, a last group of any size."""
    cfg = config([delta(heads=3, dim=24, ff=0, rank=5)], vocab=61, width=48)
    model, orc, _ = engine_and_oracle(cfg, seed=3, max_step_tokens=256)
    toks = tokens(n, 61, n)
    seq = model.open_sequence()
    got = model.forward([(seq, toks, list(range(n)))]).clone()
    model.close_sequence(seq)
    assert rel_err(got, orc.forward(toks)) < TOL[torch.float32]


@pytest.mark.parametrize("dim", [5, 32, 33, 64, 96, 200])
def test_four_token_scan_of_prompts(dim):
    """Every form of the recurrence, padded key channels, groups and chunks that end anywhere: sequences of 16 to 67 tokens beside a
    single token, continued by a second portion of 34 each, against the oracles."""
    import maferax_util as mu
    import virusun_util as vu

    lens = (67, 16, 19, 1)
    cases = [(config([delta(heads=3, dim=dim, ff=0, rank=5)], vocab=61, width=48), engine_and_oracle),
             (mu.config([mu.gla(heads=2, dim=dim, vdim=11)], vocab=61, width=48), mu.engine_and_oracle),
             (vu.config([vu.delta(heads=4, kv_heads=2, dim=dim, vdim=9, conv=3)], vocab=61, width=48), vu.engine_and_oracle),
             (vu.config([vu.par(b=vu.right(heads=2, dim=dim, vdim=8))], vocab=61, width=48), vu.engine_and_oracle)]
    for cfg, make in cases:
        model, orc, _ = make(cfg, seed=4, max_tokens=2048, max_seqs=4, page_size=16, max_step_tokens=256)
        toks = [tokens(n + 34, 61, n) for n in lens]
        want = [orc.forward(t) for t in toks]
        seqs = [model.open_sequence() for _ in lens]
        first = model.forward([(s, t[:n], list(range(n))) for s, t, n in zip(seqs, toks, lens)]).clone()
        then = model.forward([(s, t[n:], list(range(34))) for s, t, n in zip(seqs, toks, lens)]).clone()
        for s in seqs:
            model.close_sequence(s)
        at = 0
        for i, n in enumerate(lens):
            if n > 1:
                assert rel_err(first[at:at + n], want[i][:n]) < TOL[torch.float32]
            assert rel_err(then[34 * i:34 * i + 34], want[i][n:]) < TOL[torch.float32]
            at += n


def test_tokens_take_nothing_from_later_ones_in_the_four_token_scan():
    """A token that is not finite leaves the logits of every earlier one as they are, whatever its place among the scan's four."""
    import maferax_util as mu

    bad = 60
    cases = [(config([delta(heads=3, dim=16, ff=0, rank=5)], vocab=61, width=48), engine_and_oracle),
             (mu.config([mu.gla(heads=2, dim=16, vdim=11)], vocab=61, width=48), mu.engine_and_oracle)]

    def spoil(w):
        w["embed"][bad] = float("nan")

    for cfg, make in cases:
        model, _, _ = make(cfg, seed=5, edit=spoil, max_step_tokens=256)
        toks = [t % bad for t in tokens(43, 61, 1)]

        def logits(row):
            seq = model.open_sequence()
            out = model.forward([(seq, row, list(range(len(row))))]).clone()
            model.close_sequence(seq)
            return out

        want = logits(toks)
        for at in range(35, 42):
            got = logits(toks[:at] + [bad] + toks[at + 1:])
            assert torch.equal(got[:at], want[:at])
            assert not bool(got[at:].isfinite().any())


@pytest.mark.parametrize("streams,frames", [(1, 11), (3, 5), (8, 3), (11, 2), (12, 9), (17, 6)])
def test_codec_runs_of_frames_equal_single_steps(streams, frames):
    """decode() takes up to 8 frames of few streams, 4 of many, at once: bit for bit what decode_step returns frame by frame."""
    from smoltts_b200.mimi import MimiModel
    from smoltts_b200.synth import make_mimi_state_dict

    m = MimiModel(max_streams=streams, max_frames=16)
    m.load_state_dict(make_mimi_state_dict(3))
    codes = torch.randint(0, 2048, (streams, 8, frames), generator=torch.Generator().manual_seed(frames))
    whole = m.decode(codes)
    caches = [m.make_cache() for _ in range(streams)]
    steps = torch.cat([m.decode_step(codes[:, :, t:t + 1], caches).clone() for t in range(frames)], -1)
    assert torch.equal(whole, steps)
    assert not m.overflowed()


ATTENTION_FORMS = {"sink-64-64": ("pamasun", lambda u: u.attn(heads=4, kv_heads=2, dim=64, vdim=64, ff=0)),
                   "sink-40-72": ("pamasun", lambda u: u.attn(heads=2, kv_heads=1, dim=40, vdim=72, ff=0)),
                   "sink-104-8": ("pamasun", lambda u: u.attn(heads=3, kv_heads=3, dim=104, vdim=8, ff=0)),
                   "latent-48": ("maferax", lambda u: u.latent(heads=3, dim=16, rot_dim=8, vdim=16, q_rank=24, kv_rank=40)),
                   "latent-96": ("maferax", lambda u: u.latent(heads=3, dim=16, rot_dim=16, vdim=16, q_rank=24, kv_rank=80)),
                   "latent-160": ("maferax", lambda u: u.latent(heads=2, dim=32, rot_dim=32, vdim=32, q_rank=24, kv_rank=128)),
                   "maps-64-128": ("virusun", lambda u: u.att(heads=2, kv_heads=1, dim=64, vdim=128)),
                   "maps-24-40": ("virusun", lambda u: u.att(heads=4, kv_heads=2, dim=24, vdim=40)),
                   "many-maps-64-128": ("virusun", lambda u: u.att(heads=10, kv_heads=2, dim=64, vdim=128)),
                   "many-maps-24-40": ("virusun", lambda u: u.att(heads=10, kv_heads=5, dim=24, vdim=40)),
                   "rotated-32-16": ("virusun", lambda u: u.par(u.left(heads=4, kv_heads=2, dim=32, vdim=16))),
                   "window-48-16": ("sunutar", lambda u: u.layer(u.left(dim=48, vdim=16, window=100))),
                   "capped-24-24": ("bizulix", lambda u: u.att(dim=24, vdim=24))}


@pytest.mark.parametrize("page_size", [16, 64])
@pytest.mark.parametrize("form", ATTENTION_FORMS)
def test_prompt_attention_of_128_row_tiles(form, page_size):
    """bf16 prompts that end at and around the tiles' 128 rows and the steps' 64 keys, beside a sequence of three tokens, continued by a
    second portion: as close to the oracle as the same prompts in portions of at most 8 tokens, which the few-token kernel takes.  The two
    differ in the order of fp32 sums, so at most by one bf16 rounding (2^-8) of what each writes."""
    import importlib

    name, layer = ATTENTION_FORMS[form]
    u = importlib.import_module(f"{name}_util")
    cfg = u.config([layer(u)], vocab=61, width=48)
    model, orc, _ = u.engine_and_oracle(cfg, seed=6, dtype=torch.bfloat16, max_tokens=2048, max_seqs=5, page_size=page_size, max_step_tokens=640)
    lens, more = (193, 128, 129, 65, 3), 66
    toks = [tokens(n + more, 61, n) for n in lens]
    want = [orc.forward(t) for t in toks]

    def rows(portions):
        seqs, out = [model.open_sequence() for _ in lens], [[] for _ in lens]
        for step in portions:
            got = model.forward([(s, t[a:b], list(range(b - a))) for s, t, (a, b) in zip(seqs, toks, step) if b > a]).clone()
            at = 0
            for o, (a, b) in zip(out, step):
                o.append(got[at:at + b - a])
                at += b - a
        for s in seqs:
            model.close_sequence(s)
        return [torch.cat(o) for o in out]

    whole = rows([[(0, n) for n in lens], [(n, n + more) for n in lens]])
    pieces = rows([[(min(a, n + more), min(a + 8, n + more)) for n in lens] for a in range(0, max(lens) + more, 8)])
    for w, p, o in zip(whole, pieces, want):
        assert rel_err(w, o) < TOL[torch.bfloat16]
        assert rel_err(w, o) < 1.5 * rel_err(p, o) + 2.0 ** -8
    model.check_device_errors()


@pytest.mark.parametrize("form", ["narrow", "wide", "latent"])
def test_many_short_prompts_beside_each_other(form):
    """More (sequence, head) pairs than SMs with a few tokens each are taken by the 64-row kernel, each of them alone by the 128-row one: both as
    close to the oracle as one bf16 rounding (2^-8) of what they write."""
    import maferax_util as mu

    cfg, u = {"narrow": (config([attn(heads=12, kv_heads=4, dim=64, vdim=64, ff=0)], vocab=61, width=48), None),
              "wide": (config([attn(heads=12, kv_heads=4, dim=72, vdim=128, ff=0)], vocab=61, width=48), None),
              "latent": (mu.config([mu.latent(heads=12, dim=16, rot_dim=8, vdim=16, q_rank=24, kv_rank=40)], vocab=61, width=48), mu)}[form]
    lens = [9 + i % 8 for i in range(14)]
    model, orc, _ = (u.engine_and_oracle if u else engine_and_oracle)(cfg, seed=8, dtype=torch.bfloat16, max_tokens=2048, max_seqs=16, page_size=64, max_step_tokens=256)
    toks = [tokens(n, 61, n + i) for i, n in enumerate(lens)]

    def run(group):
        seqs = [model.open_sequence() for _ in group]
        got = model.forward([(s, t, list(range(len(t)))) for s, t in zip(seqs, group)]).clone()
        for s in seqs:
            model.close_sequence(s)
        return got.split([len(t) for t in group])

    for t, together, alone in zip(toks, run(toks), [run([t])[0] for t in toks]):
        want = orc.forward(t)
        assert rel_err(together, want) < TOL[torch.bfloat16]
        assert rel_err(together, want) < 1.5 * rel_err(alone, want) + 2.0 ** -8
