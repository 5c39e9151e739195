"""The batched decode (csrc/rows_phases.cuh, csrc/tile_phases.cuh) and the prompt kernel (csrc/prompt_phases.cuh) at the sizes where they can go wrong:
batches around the row groups, widths whose chains are long or cut unevenly, ragged heads, 16 depth positions, every group size of
the attention, contexts around its splits, both page sizes.  The yardstick is the CUDA-core variant on the same inputs (itself held to
the oracle): the two differ by the rounding of bf16 activations only, so their logits by a few bf16 ulps; bits that must not depend on
the batch are compared as bits."""
import pytest
import torch

from smoltts_b200.config import named_config
from smoltts_b200.model import RQTransformer, make_prompt_cache
from smoltts_b200.synth import byte_prompt, prompt_grid, state_dict_shapes

pytestmark = pytest.mark.gpu

CONFIGS = {
    # w2 rows of 1600: 25 MMAs per chain, no K slices; 4 query heads per kv head
    "long_chains": dict(base="smoltts_byte_tiny", dim=256, fast_dim=256, n_head=4, fast_n_head=4, n_local_heads=1, fast_n_local_heads=1, intermediate_size=1600, fast_intermediate_size=1600),
    # two K slices in wo, heads that are not whole tiles, one kv head per query head
    "ragged_heads": dict(base="smoltts_byte_tiny", dim=384, fast_dim=384, n_head=6, fast_n_head=6, n_local_heads=6, fast_n_local_heads=6, intermediate_size=640, fast_intermediate_size=640,
                         vocab_size=2370, codebook_size=2050),
    # positions 8 to 15 of the depth transformer
    "deep": dict(base="smoltts_byte_tiny", num_codebooks=16),
    "70m": dict(base="smoltts_byte_70m", n_layer=2, n_fast_layer=2),
}


def _model(name, max_batch, max_seq_len, page_size=32):
    over = dict(CONFIGS[name])
    cfg = named_config(over.pop("base"), **over)
    g = torch.Generator(device="cuda").manual_seed(5)
    w = {k: (1.0 + 0.05 * torch.randn(*s, generator=g, device="cuda") if k.endswith("norm.weight") else torch.randn(*s, generator=g, device="cuda") * cfg.initializer_range).to(torch.bfloat16)
         for k, s in state_dict_shapes(cfg).items()}
    model = RQTransformer(cfg, max_batch=max_batch, max_seq_len=max_seq_len, page_size=page_size)
    model.load_state_dict(w)
    return cfg, model


def _frame(cfg, model, lens, rows, min_batch, frames=1):
    """One forced frame of the sequences `rows` behind caches of the given lengths; (token logits, depth logits, cached pages)."""
    g = torch.Generator(device="cuda").manual_seed(11)
    n = len(lens)
    codes = torch.randint(0, min(cfg.codebook_size, 1000), (2, n, cfg.n_rows), generator=g, device="cuda", dtype=torch.int32)
    kv = torch.randn(n, max(lens), cfg.n_layer, 2, cfg.n_local_heads, 64, generator=g, device="cuda", dtype=torch.bfloat16)
    batch = model.new_batch(len(rows), max_positions=model.max_seq_len, max_frames=frames)
    try:
        ps, pages = model.page_size, batch.block_table.long()
        pad = torch.zeros(len(rows), pages.shape[1] * ps - max(lens), *kv.shape[2:], dtype=kv.dtype, device="cuda")
        model.kv_view()[pages] = torch.cat([kv[rows], pad], 1).view(len(rows), -1, ps, *kv.shape[2:]).permute(0, 1, 3, 4, 5, 2, 6)
        force = codes[1][rows].contiguous()
        model.set_force(force)
        batch.tokens.copy_(codes[0][rows])
        batch.seq_len.copy_(torch.tensor([lens[r] for r in rows], dtype=torch.int32, device="cuda"))
        batch.host_len = [lens[r] for r in rows]
        model.set_option("tc_min_batch", min_batch)
        model.set_option("ll_max_batch", 0)
        model.decode_frames(batch, model.sampling(ignore_stop=True), frames)
        torch.cuda.synchronize()
        return model.debug_buffer("token_logits", len(rows)).clone(), model.debug_buffer("depth_logits", len(rows)).clone(), model.kv_view()[pages].clone()
    finally:
        model.set_force(None)
        model.set_option("tc_min_batch", 9)
        model.set_option("ll_max_batch", 8)
        batch.release()


def _close(a, b, what):
    scale = b.float().pow(2).mean().sqrt()
    d = (a.float() - b.float())
    # two bf16 executions of a few layers: each rounding is 2^-9 of its value (rms 0.29 ulps), some thirty of them in a row
    assert torch.isfinite(a).all() and d.pow(2).mean().sqrt() < 0.03 * scale and d.abs().max() < 0.25 * scale, (what, (d.pow(2).mean().sqrt() / scale).item(), (d.abs().max() / scale).item())


@pytest.mark.parametrize("name,page_size", [("long_chains", 32), ("ragged_heads", 16), ("deep", 32), ("70m", 16)])
@pytest.mark.parametrize("batch", [9, 17, 33, 65])
def test_batched_decode_at_the_edges_of_its_row_groups(name, page_size, batch):
    cfg, model = _model(name, 65, 200, page_size)
    lens = [1 + (37 * b) % 170 for b in range(batch)]
    every = list(range(batch))
    tl, dl, kv = _frame(cfg, model, lens, every, 9)
    assert model.get_option("tc_ready") == 1
    tl0, dl0, kv0 = _frame(cfg, model, lens, every, 0)
    _close(tl, tl0, "token logits")
    _close(dl, dl0, "depth logits")
    _close(kv, kv0, "keys and values")
    some = every[-9:]                       # the smallest batch: the same bits
    ts, ds, ks = _frame(cfg, model, lens, some, 9)
    assert torch.equal(ts, tl[some]) and torch.equal(ds, dl[some]) and torch.equal(ks.view(torch.int16), kv[some].view(torch.int16))


@pytest.mark.parametrize("name,longest,batch", [("70m", 127, 10), ("70m", 128, 10), ("70m", 129, 40), ("long_chains", 1030, 40), ("70m", 2300, 150), ("deep", 2300, 300),
                                                ("70m", 40, 145), ("ragged_heads", 200, 160), ("long_chains", 100, 290)])
def test_batch_attention_around_its_splits(name, longest, batch):
    """Contexts below, at and above a split; more splits than a unit has warps (states through global memory); many units.  Wide
    batches take the tiles of 128 rows: the bits stay those of nine sequences."""
    cfg, model = _model(name, batch, longest + 4)
    lens = [max(1, longest - (b * 131) % longest) for b in range(batch)]
    tl, dl, _ = _frame(cfg, model, lens, list(range(batch)), 9)
    tl0, dl0, _ = _frame(cfg, model, lens, list(range(batch)), 0)
    _close(tl, tl0, "token logits")
    _close(dl, dl0, "depth logits")
    ts, ds, _ = _frame(cfg, model, lens, list(range(9)), 9)
    assert torch.equal(ts, tl[:9]) and torch.equal(ds, dl[:9])


@pytest.mark.parametrize("name,page_size", [("long_chains", 32), ("ragged_heads", 16), ("70m", 32)])
@pytest.mark.parametrize("n,tile", [(9, 0), (10, 0), (16, 0), (65, 0), (130, 0), (130, 50), (301, 0)])
def test_prompt_logits_equal_those_of_its_last_position_alone(name, page_size, n, tile):
    """forward_generate of a prompt against the prefill of all but its last position and that position by itself: the same bits in
    logits, hidden state and cache."""
    cfg, model = _model(name, 1, 320, page_size)
    prompt = prompt_grid(byte_prompt(max(1, n - 12), seed=n)[-n:], cfg)[None].to(device="cuda", dtype=torch.int32)
    n = prompt.shape[2]
    model.set_option("prefill_tile", tile)
    cache = make_prompt_cache(model)
    logits, hidden = model.forward_generate(prompt, cache)
    pages = torch.tensor(cache.batch.pages, device="cuda")
    assert int(cache.batch.seq_len[0]) == n and cache.batch.host_len == [n] and torch.equal(cache.batch.tokens[0], prompt[0, :, -1])
    kv = model.kv_view()[pages].clone()
    cache.batch.release()
    model.kv_view().zero_()
    cache = make_prompt_cache(model)
    model.prefill(cache.batch, prompt, torch.tensor([n], dtype=torch.int32, device="cuda"))
    model.slow_step(cache.batch, advance=True)
    torch.cuda.synchronize()
    assert torch.equal(logits, model.debug_buffer("token_logits", 1)) and torch.equal(hidden.view(torch.int16), model.debug_buffer("x", 1).view(torch.int16))
    kv0 = model.kv_view()[torch.tensor(cache.batch.pages, device="cuda")]
    flat = lambda t: t.permute(1, 2, 3, 0, 4, 5).flatten(3, 4)[..., :n, :].contiguous().view(torch.int16)  # noqa: E731
    assert torch.equal(flat(kv), flat(kv0))
    cache.batch.release()


def _depth_attention(q, kv, depth_pos):
    """Attention of one depth position as the CUDA-core kernels add it up: q [B, Hq, 64], kv [B, 2, depth, Hkv, 64] bf16.  A product of
    two bf16 numbers is exact in fp32, so an fp32 sum of products is a chain of FMAs."""
    B, Hq, _ = q.shape
    G = Hq // kv.shape[3]
    q, kv = q.float(), kv.float().repeat_interleave(G, dim=3)
    part = torch.zeros(B, Hq, depth_pos + 1, 4, device=q.device)
    qd, kd = q.view(B, Hq, 1, 4, 16), kv[:, 0, :depth_pos + 1].transpose(1, 2).reshape(B, Hq, depth_pos + 1, 4, 16)
    for e in range(16):
        part = part + qd[..., e] * kd[..., e]
    score = ((part[..., 0] + part[..., 1]) + (part[..., 2] + part[..., 3])) * 0.125
    p = torch.exp(score - score.amax(-1, keepdim=True))
    row = torch.zeros(B, Hq, 16, device=q.device)
    row[..., :depth_pos + 1] = p
    row = row[..., :8] + row[..., 8:]
    for _ in range(3):
        row = row[..., 0::2] + row[..., 1::2]
    p = p.to(torch.bfloat16).float()
    o = torch.zeros(B, Hq, 64, device=q.device)
    for j in range(depth_pos + 1):
        o = o + p[..., j, None] * kv[:, 1, j]
    return (o * (1.0 / row)).to(torch.bfloat16)


@pytest.mark.parametrize("name", ["long_chains", "ragged_heads", "deep", "70m"])    # 4, 1, 2 and 3 query heads per kv head
@pytest.mark.parametrize("batch", [9, 40, 150])
def test_depth_attention_adds_up_as_the_cuda_core_kernels_do(name, batch):
    cfg, model = _model(name, batch, 64)
    _frame(cfg, model, [1 + b % 50 for b in range(batch)], list(range(batch)), 9)
    Hq, Hkv, last = cfg.fast_n_head, cfg.fast_n_local_heads, cfg.max_fast_seqlen - 1
    q = model.debug_buffer("q", batch).view(batch, Hq, 64)
    kv = model.debug_buffer("fkv", batch).view(batch, cfg.n_fast_layer, 2, -1, Hkv, 64)[:, -1]
    got = model.debug_buffer("attn", batch).view(batch, Hq, 64)
    assert torch.equal(got.view(torch.int16), _depth_attention(q, kv, last).view(torch.int16))


@pytest.mark.parametrize("what", ["frames of 12", "frames of 160", "prompt"])
def test_phase_recorder_covers_the_launch_once(what):
    """Work and waits are disjoint and belong to their own phases: together they are what the launch takes, and no phase in it is empty."""
    n = 160 if what.endswith("160") else 12 if what.startswith("frames") else 1
    cfg, model = _model("70m", n, 200)
    batch = model.new_batch(n, max_positions=190, max_frames=4)
    prompt = prompt_grid(byte_prompt(88, seed=1), cfg)[None].to(device="cuda", dtype=torch.int32)
    model.set_option("ll_max_batch", 0)
    frames = 4

    def run():
        batch.seq_len.zero_()
        batch.step.zero_()
        batch.host_len = [0] * n
        if what == "prompt":
            model.forward_generate(prompt, type("Cache", (), {"batch": batch}))
        else:
            model.decode_frames(batch, model.sampling(ignore_stop=True), frames)

    run()
    prof = model.set_profile(True)
    run()
    torch.cuda.synchronize()
    prof.zero_()
    begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    begin.record()
    run()
    end.record()
    torch.cuda.synchronize()
    ns = prof[:1024].view(512, 2).cpu()
    model.set_profile(False)
    last = 5 * cfg.n_layer if what == "prompt" else model.phase_count - 1
    first = [i for i in range(last + 1)]
    assert (ns >= 0).all() and (ns[first, 0] > 0).all() and (ns[first[:-1], 1] > 0).all() and ns[last + 1:].sum() == 0
    wall = begin.elapsed_time(end) * 1e6
    # CTA 0's clock against events around the call's launches and copies: what is recorded twice or not at all would be a third of it
    assert 0.6 * wall < ns.sum().item() < 1.02 * wall, (ns.sum().item(), wall)
    # waits of many barriers, not of one
    assert ns[:, 1].max() < 0.25 * ns[:, 1].sum()


KERNEL = {"groups": 3, "tiles": 4, "prompt": 5}     # SMOL_KERNEL_*


@pytest.mark.parametrize("name,batch", [("70m", 9), ("ragged_heads", 40), ("deep", 33), ("long_chains", 130)])
@pytest.mark.parametrize("mode", [0, 1])
def test_groups_and_tiles_give_the_same_bits(name, batch, mode):
    cfg, model = _model(name, batch, 300)
    model.set_option("mode", mode)
    lens = [1 + (37 * b) % 280 for b in range(batch)]
    out = {}
    for kernel, rows in (("groups", 100000), ("tiles", 0)):
        model.set_option("tc_group_rows", rows)
        out[kernel] = _frame(cfg, model, lens, list(range(batch)), 9, frames=2)[:2]
        assert model.get_option("last_kernel") == KERNEL[kernel]
    assert all(torch.equal(a, b) for a, b in zip(out["groups"], out["tiles"]))


@pytest.mark.parametrize("name", ["long_chains", "70m"])
@pytest.mark.parametrize("batch,rows", [(9, 100000), (33, 100000), (65, 100000), (65, 0), (160, 0)])
def test_small_grids_give_the_bits_of_the_whole_one(name, batch, rows):
    """Fewer CTAs than tile blocks: a CTA walks several blocks of a phase, in groups of rows and on tiles."""
    cfg, model = _model(name, batch, 150)
    model.set_option("tc_group_rows", rows)
    lens = [1 + (37 * b) % 130 for b in range(batch)]
    want = _frame(cfg, model, lens, list(range(batch)), 9)
    for n_ctas in (40, 7):
        model.set_option("n_ctas", n_ctas)
        got = _frame(cfg, model, lens, list(range(batch)), 9)
        assert model.get_option("n_ctas") == n_ctas and model.get_option("last_kernel") == KERNEL["groups" if rows else "tiles"]
        assert all(torch.equal(a.view(torch.int16 if a.dtype == torch.bfloat16 else a.dtype), b.view(torch.int16 if b.dtype == torch.bfloat16 else b.dtype))
                   for a, b in zip(got, want))
    model.set_option("n_ctas", 0)


@pytest.mark.parametrize("seqs,n,kernel", [(1, 129, "tiles"), (1, 130, "prompt"), (3, 40, "tiles"), (2, 200, "prompt"), (9, 2, "tiles")])
def test_prefills_have_the_same_bits_in_either_kernel(seqs, n, kernel):
    """A prefill against the same one cut into tiles of 100 positions: on either side of the line between the kernels."""
    cfg, model = _model("70m", seqs, 260)
    prompts = torch.stack([prompt_grid(byte_prompt(max(1, n - 12), seed=s)[-n:], cfg)[:, -n:] for s in range(seqs)]).to(device="cuda", dtype=torch.int32).contiguous()
    n = prompts.shape[2]
    lens = torch.tensor([n - (s % 3 if n > 8 else 0) for s in range(seqs)], dtype=torch.int32, device="cuda")
    out = []
    for tile in (0, 100):
        model.set_option("prefill_tile", tile)
        model.kv_view().zero_()
        batch = model.new_batch(seqs, max_positions=250)
        model.prefill(batch, prompts, lens)
        if tile == 0:
            assert model.get_option("last_kernel") == KERNEL[kernel]
        out.append((model.kv_view()[batch.block_table.long()].clone().view(torch.int16), batch.tokens.clone(), batch.seq_len.clone()))
        batch.release()
    model.set_option("prefill_tile", 0)
    assert all(torch.equal(a, b) for a, b in zip(*out))


def _prompt_logits(model, cache, prompt):
    import ctypes

    from smoltts_b200 import _capi

    _capi.check(model.lib.smol_prompt_logits(model._h, ctypes.byref(cache.batch.c), ctypes.c_void_p(prompt.data_ptr()), prompt.shape[2], model._stream()))
    torch.cuda.synchronize()
    return model.debug_buffer("token_logits", 1).clone()


def test_prompt_iterations_stay_within_the_workspace_and_the_callers_cap():
    """A tc_min_batch above the workspace's 1024 rows, and caps below tc_min_batch: the iterations follow the workspace and the cap, the
    logits stay; forward_generate then leaves the prompt to prefill and step."""
    cfg, model = _model("70m", 1, 1400)
    prompt = prompt_grid(byte_prompt(1288, seed=4), cfg)[None].to(device="cuda", dtype=torch.int32)
    cache = make_prompt_cache(model)
    want, _ = model.forward_generate(prompt, cache)
    assert model.get_option("last_kernel") == KERNEL["prompt"]
    cache.batch.release()
    for options in (dict(tc_min_batch=1200), dict(prefill_tile=5), dict(prefill_tile=1)):
        for name, value in options.items():
            model.set_option(name, value)
        cache = make_prompt_cache(model)
        assert torch.equal(_prompt_logits(model, cache, prompt), want) and int(cache.batch.seq_len[0]) == 1300
        cache.batch.release()
        assert model.get_option("prompt_min_rows") == 0
        model.set_option("tc_min_batch", 9)
        model.set_option("prefill_tile", 0)
    model.set_option("tc_min_batch", 1200)
    cache = make_prompt_cache(model)
    logits, _ = model.forward_generate(prompt, cache)
    assert model.get_option("last_kernel") == 1 and cache.batch.host_len == [1300]      # CUDA cores
    _close(logits, want, "token logits")
    cache.batch.release()
    model.set_option("tc_min_batch", 9)


@pytest.mark.parametrize("what", ["frames", "prompt"])
def test_a_wait_that_runs_out_ends_the_launch_and_the_next_call_reports_it(what):
    """One block waits for something that nothing completes: the launch ends by itself, without a CUDA error; the next call says so, and the
    call after that works, with the bits of one that never failed."""
    from smoltts_b200 import _capi

    cfg, model = _model("70m", 12, 200)
    lens = [1 + (37 * b) % 170 for b in range(12)]
    prompt = prompt_grid(byte_prompt(88, seed=1), cfg)[None].to(device="cuda", dtype=torch.int32)

    def run():
        if what == "frames":
            return _frame(cfg, model, lens, list(range(12)), 9, frames=3)[:2]
        cache = make_prompt_cache(model)
        out = tuple(t.clone() for t in model.forward_generate(prompt, cache))
        torch.cuda.synchronize()
        cache.batch.release()
        return out

    want = run()
    model.set_option("wait_ms", 20)
    model.set_option("wait_probe", 1)
    run()
    assert model.get_option("device_status") == 1
    with pytest.raises(_capi.SmolError) as e:
        run()
    assert e.value.code == _capi.SMOL_ERR_TIMEOUT and model.get_option("device_status") == 0
    model.set_option("wait_ms", 2000)
    assert all(torch.equal(a, b) for a, b in zip(run(), want))


def _prompt_against_prefill_and_step(cfg, model, n, cached=0):
    """forward_generate of n columns (behind `cached` positions) against the prefill of all but the last and that one alone: bits."""
    grid = prompt_grid(byte_prompt(max(1, n + cached - 12), seed=n)[-(n + cached):], cfg)[None].to(device="cuda", dtype=torch.int32)
    grid = torch.cat([grid, grid], 2)[:, :, :n + cached].contiguous()
    before, prompt = grid[:, :, :cached + 1].contiguous(), grid[:, :, cached:].contiguous()
    out = []
    for one_pass in (True, False):
        model.kv_view().zero_()
        cache = make_prompt_cache(model)
        if cached:
            model.prefill(cache.batch, before, torch.tensor([cached + 1], dtype=torch.int32, device="cuda"))
        if one_pass:
            logits, hidden = model.forward_generate(prompt, cache)
            assert model.get_option("last_kernel") == KERNEL["prompt"]
        else:
            model.prefill(cache.batch, prompt, torch.tensor([n], dtype=torch.int32, device="cuda"))
            model.slow_step(cache.batch, advance=True)
            logits, hidden = model.debug_buffer("token_logits", 1).clone(), model.debug_buffer("x", 1).clone()
        assert int(cache.batch.seq_len[0]) == n + cached and cache.batch.host_len == [n + cached]
        kv = model.kv_view()[torch.tensor(cache.batch.pages, device="cuda")].permute(1, 2, 3, 0, 4, 5).flatten(3, 4)[..., :n + cached, :]
        out.append((logits, hidden.view(torch.int16), kv.contiguous().view(torch.int16)))
        cache.batch.release()
    assert all(torch.equal(a, b) for a, b in zip(*out))


@pytest.mark.parametrize("name,page_size", [("long_chains", 32), ("70m", 16)])
@pytest.mark.parametrize("n,cached", [(10, 1), (17, 31), (130, 300), (1024, 0), (1025, 0), (1100, 3), (1990, 0)])
def test_prompt_logits_behind_a_cache_and_over_several_iterations(name, page_size, n, cached):
    """On top of what the sequence holds; a last iteration of a single row (1025 positions); the last position's attention over up to 32
    splits of 64 positions, and over longer ones."""
    cfg, model = _model(name, 1, 2040, page_size)
    _prompt_against_prefill_and_step(cfg, model, n, cached)


def test_a_prompt_alone_sets_the_variant_up():
    cfg, model = _model("70m", 1, 64)
    assert model.get_option("tc_ready") == 0 and model.get_option("last_kernel") == 0
    cache = make_prompt_cache(model)
    model.forward_generate(prompt_grid(byte_prompt(20, seed=1), cfg)[None].to(device="cuda", dtype=torch.int32), cache)
    assert model.get_option("tc_ready") == 1


def test_the_longest_program_fits_beside_the_tiles():
    """498 of at most 512 phases: their table lies in shared memory beside the weight tiles."""
    over = dict(base="smoltts_byte_tiny", n_layer=64, n_fast_layer=5)
    CONFIGS["long_program"] = over
    cfg, model = _model("long_program", 12, 64)
    assert model.phase_count == 5 * 64 + 2 + 8 * (4 * 5 + 2) == 498
    lens = [1 + b for b in range(12)]
    out = [_frame(cfg, model, lens, list(range(12)), 9)[:2]]
    assert model.get_option("last_kernel") == KERNEL["groups"]
    model.set_option("tc_group_rows", 0)
    out.append(_frame(cfg, model, lens, list(range(12)), 9)[:2])
    assert all(torch.equal(a, b) for a, b in zip(*out))
