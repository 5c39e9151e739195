"""Oracle parity at the sizes BASELINE.json's configurations run at (150m), through the C-ABI:

  * the tensor-core variant at bs=64 and bs=256: two teacher-forced frames for every row of the
    batch against the CPU oracle (bf16) and its fp32 twin, under the calibrated bars of test_gpu_decode.py
    (our error against the fp32 logits <= 1.3x rms / 1.6x max of the bf16 oracle's own error; argmax = fp32 argmax
    wherever its margin exceeds TAU);
  * long contexts: prefill of 2100 and 4300 positions (> 128 KV pages, RoPE rows beyond 4096, up to 9
    attention blocks of 512 positions), then two teacher-forced frames, at bs=1 (data-flow kernel) and as rows of a
    ragged batch of 32 (tensor-core variant, batch attention), against the CPU oracle's bf16 logits.

The oracle runs on the box's host cores inside the test (results cached per prompt), sized to finish in about a minute.
"""
import numpy as np
import pytest
import torch

from gpu_util import model_and_oracle, np_rms
from smoltts_b200.generate import pack_prompts
from smoltts_b200.synth import teacher_grid

pytestmark = pytest.mark.gpu

SIZE = "smoltts_byte_150m"
TAU = 0.15
N_FRAMES = 2
_ORACLE = {}


def _gpu_teacher_forced(model, grids, n_frames=N_FRAMES):
    """grids: list of [R, S_b] int64.  Row b: its first S_b - n_frames columns are the prompt (prefill), the following
    n_frames columns are forced.  Returns (token logits [B, n, V], depth logits [B, n, Nf, C]) as numpy."""
    B = len(grids)
    dev = model.device
    prompts = [g[:, : g.shape[1] - n_frames] for g in grids]
    padded, lens = pack_prompts(model, prompts)
    batch = model.new_batch(B, max_positions=max(int(g.shape[1]) for g in grids) + 2, max_frames=n_frames)
    tok, cb = [], []
    try:
        model.prefill(batch, padded, lens)
        s = model.sampling(ignore_stop=True)
        for f in range(n_frames):
            force = torch.stack([g[:, g.shape[1] - n_frames + f] for g in grids]).to(device=dev, dtype=torch.int32).contiguous()
            model.set_force(force)
            model.decode_frames(batch, s, 1)
            torch.cuda.synchronize()
            tok.append(model.debug_buffer("token_logits", B).cpu().clone())
            cb.append(model.debug_buffer("depth_logits", B).cpu().clone())
        assert batch.seq_len.tolist() == [int(g.shape[1]) - 1 for g in grids]
    finally:
        model.set_force(None)
        batch.release()
    return torch.stack(tok, 1).numpy(), torch.stack(cb, 1).numpy()


def _oracle_teacher_forced(orc, grid, n_frames=N_FRAMES):
    """grid [B, R, S] -> the same two tensors from the CPU oracle (float32 numpy)."""
    S = grid.shape[2]
    P = S - n_frames
    with torch.no_grad():
        tl, cbd = orc.teacher_forced(grid, stepwise_from=P - 1, fast_positions=list(range(P - 1, P - 1 + n_frames)))
    tok = tl[:, P - 1:P - 1 + n_frames].float().numpy()
    cb = torch.stack([cbd[t] for t in range(P - 1, P - 1 + n_frames)], 1).float().numpy()
    return tok, cb


def _margins(x):
    top2 = np.sort(x, axis=-1)[..., -2:]
    return x.argmax(-1), top2[..., 1] - top2[..., 0]


@pytest.mark.timeout(900)
@pytest.mark.parametrize("B", [64, 256])
def test_tensor_core_batches_vs_oracle_150m(B):
    from oracle.dualar_oracle import DualAROracle

    cfg, sd, model, orc = model_and_oracle(SIZE, max_batch=256, max_seq_len=256)
    assert B >= model.get_option("tc_min_batch") > 0
    grid = teacher_grid(cfg, n_text=14, n_audio=4 + N_FRAMES, batch=B, seed=300 + B, zero_code_at=2)   # [B, R, 20]
    tok, cb = _gpu_teacher_forced(model, [grid[b] for b in range(B)])
    assert model.get_option("tc_ready") == 1, "the tensor-core variant did not run"
    rbf_t, rbf_c = _oracle_teacher_forced(orc, grid)
    orc32 = DualAROracle(cfg, sd, dtype=torch.float32, max_seq_len=256)
    rf_t, rf_c = _oracle_teacher_forced(orc32, grid)
    for name, ours, rbf, rf in (("token", tok, rbf_t, rf_t), ("codebook", cb, rbf_c, rf_c)):
        e_ours, e_ref = np_rms(ours, rf), np_rms(rbf, rf)
        m_ours, m_ref = np.abs(ours - rf).max(), np.abs(rbf - rf).max()
        print(f"150m bs={B} {name}: rms vs fp32 ours {e_ours:.4f} oracle-bf16 {e_ref:.4f}; max ours {m_ours:.4f} oracle {m_ref:.4f}; "
              f"ours vs oracle-bf16: max {np.abs(ours - rbf).max():.4f}, bit-exact {(ours == rbf).mean():.3f}")
        assert e_ours <= 1.3 * e_ref + 1e-3, f"{name}: rms error {e_ours} vs the bf16 oracle's own {e_ref}"
        assert m_ours <= 1.6 * m_ref + 1e-2, f"{name}: max error {m_ours} vs the bf16 oracle's own {m_ref}"
        # argmax against the fp32 oracle: a flip needs two logit errors that add up to the margin, so bf16 executions (the
        # oracle's own included: its logits are off by up to m_ref) flip decisions up to margins of about that size.  Bar: no
        # flip beyond twice TAU, and not more flips beyond TAU than the bf16 oracle itself has (plus 0.5 % of the decisions).
        am, mg = _margins(rf)
        bad = (ours.argmax(-1) != am) & (mg > TAU)
        bad_ref = (rbf.argmax(-1) != am) & (mg > TAU)
        print(f"150m bs={B} {name}: argmax flips against fp32 beyond margin {TAU}: ours {int(bad.sum())}, bf16 oracle {int(bad_ref.sum())} of {am.size}"
              f" (largest margin ours {float(mg[bad].max()) if bad.any() else 0:.3f}, oracle {float(mg[bad_ref].max()) if bad_ref.any() else 0:.3f})")
        assert not ((ours.argmax(-1) != am) & (mg > 2 * TAU)).any(), f"{name}: argmax differs from the fp32 oracle at margins {mg[bad][:8]}"
        assert int(bad.sum()) <= int(bad_ref.sum()) + max(2, am.size // 200), f"{name}: {int(bad.sum())} flips beyond {TAU} (bf16 oracle: {int(bad_ref.sum())})"


def _long_grid(cfg, total, seed):
    return teacher_grid(cfg, n_text=200, n_audio=total - 200, batch=1, seed=seed)[0]      # [R, total]


def _oracle_long(cfg, sd, orc, total, seed):
    key = (total, seed)
    if key not in _ORACLE:
        _ORACLE[key] = _oracle_teacher_forced(orc, _long_grid(cfg, total, seed)[None])
    return _ORACLE[key]


def _check_long(name, ours_t, ours_c, want_t, want_c):
    for what, ours, want, rms_bar in (("token", ours_t, want_t, 0.05), ("codebook", ours_c, want_c, 0.08)):
        e, m = np_rms(ours, want), np.abs(ours - want).max()
        print(f"{name} {what}: rms vs oracle-bf16 {e:.4f} (bar {rms_bar}), max {m:.4f}, bit-exact {(ours == want).mean():.3f}")
        # two bf16 executions of the reference itself differ by rms 0.035 / 0.056 from fp32 (tests/test_gpu_decode.py):
        # the distance between two of them is bounded by sqrt(2) x that
        assert e <= rms_bar, f"{name} {what}: rms {e}"
        assert m <= 0.45, f"{name} {what}: max {m}"
        am, mg = _margins(want)
        bad = (ours.argmax(-1) != am) & (mg > TAU)
        assert not bad.any(), f"{name} {what}: argmax differs from the oracle at margins {mg[bad]}"


@pytest.mark.timeout(1200)
@pytest.mark.parametrize("total", [2100, 4300])
def test_long_context_bs1_dataflow_vs_oracle_150m(total):
    """bs=1: prefill through the tensor-core tiles (128 prompt positions per iteration), the two frames on the data-flow
    kernel, across 66 / 135 KV pages and 5 / 9 attention blocks."""
    cfg, sd, model, orc = model_and_oracle(SIZE, max_batch=32, max_seq_len=4352)
    g = _long_grid(cfg, total, seed=500 + total)
    tok, cb = _gpu_teacher_forced(model, [g])
    assert model.get_option("ll_ready") == 1, "the data-flow kernel did not run"
    want_t, want_c = _oracle_long(cfg, sd, orc, total, 500 + total)
    _check_long(f"150m bs=1 context {total}", tok, cb, want_t, want_c)


@pytest.mark.timeout(1200)
def test_long_context_bs32_tensor_core_vs_oracle_150m():
    """A ragged batch of 32 on the tensor-core variant: rows 0 and 31 carry the 4300- and 2100-position probes (same prompts as
    the bs=1 test, so the oracle's results are shared), the other rows random contexts of 40..3000 positions."""
    cfg, sd, model, orc = model_and_oracle(SIZE, max_batch=32, max_seq_len=4352)
    gen = torch.Generator().manual_seed(77)
    grids = []
    for b in range(32):
        if b == 0:
            grids.append(_long_grid(cfg, 4300, seed=500 + 4300))
        elif b == 31:
            grids.append(_long_grid(cfg, 2100, seed=500 + 2100))
        else:
            n = int(torch.randint(40, 3000, (1,), generator=gen))
            grids.append(teacher_grid(cfg, n_text=min(200, n - 8), n_audio=n - min(200, n - 8), batch=1, seed=900 + b)[0])
    tok, cb = _gpu_teacher_forced(model, grids)
    assert model.get_option("tc_ready") == 1
    for row, total in ((0, 4300), (31, 2100)):
        want_t, want_c = _oracle_long(cfg, sd, orc, total, 500 + total)
        _check_long(f"150m bs=32 row {row} context {total}", tok[row:row + 1], cb[row:row + 1], want_t, want_c)
