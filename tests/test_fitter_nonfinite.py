"""The fitters on tmp_data that holds NaN, infinities and values that overflow
on the way, at each launch shape, and CholeskyQR2 against the 256-thread form
of the fused pipeline, whose weights it has bit for bit."""
import numpy as np
import pytest

import bmfr_b200 as B
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

SHAPES = [(64, 48), (416, 352), (704, 640), (1280, 720)]   # one block per SM, two, four, seven


def _draw(rng, blocks):
    """tmp_data with finite values, and a copy whose even blocks hold others."""
    t = np.empty((blocks, 13, 1024), np.float32)
    t[:, 0] = 1.0
    n = rng.standard_normal((blocks, 3, 1024))
    t[:, 1:4] = n / np.linalg.norm(n, axis=1, keepdims=True)
    t[:, 4:7] = rng.uniform(-4, 4, (blocks, 3, 1)) + rng.standard_normal((blocks, 3, 1024))
    t[:, 7:10] = t[:, 4:7] ** 2
    t[:, 10:13] = rng.lognormal(-1.0, 1.5, (blocks, 3, 1024))
    plain = t.astype(np.float16)
    mixed = plain.copy()
    for b in range(0, blocks, 2):
        kind, column = rng.integers(0, 6), rng.integers(0, 13)
        if kind == 0:      # anywhere
            mixed[b, column, rng.integers(0, 1024, 3)] = rng.choice([np.nan, np.inf, -np.inf])
        elif kind == 1:    # in the first rows, which are R's and the right-hand side's
            mixed[b, column, rng.integers(0, 12)] = rng.choice([np.nan, np.inf, -np.inf])
        elif kind == 2:
            mixed[b, column] = np.nan
        elif kind == 3:
            mixed[b, column] = rng.choice([np.inf, -np.inf], 1024)
        elif kind == 4:    # what the accumulation makes of infinities: later columns overflow
            mixed[b, rng.integers(1, 13, 4), rng.integers(0, 1024, 4)] = rng.choice([65504.0, -65504.0], 4)
        else:              # the same in the first rows
            mixed[b, rng.integers(1, 4, 2), rng.integers(0, 12, 2)] = rng.choice([65504.0, -65504.0], 2)
    return plain, mixed


@pytest.mark.parametrize("W,H", SHAPES)
def test_reference_arithmetic_matches_oracle(cuda, W, H):
    import torch
    plan, o = B.Plan(W, H), Oracle(W, H)
    _, mixed = _draw(np.random.default_rng(W), o.blocks)
    want_w, want_mm = np.zeros(o.blocks * 30, np.float32), np.zeros(o.blocks * 12, np.float32)
    o.fitter(want_w, want_mm, mixed.reshape(-1).copy(), 5)
    w, mm = torch.empty(o.blocks * 30, device=cuda), torch.empty(o.blocks * 12, device=cuda)
    B.fitter(plan, w, mm, torch.from_numpy(mixed.reshape(-1)).to(cuda), 5)
    np.testing.assert_array_equal(mm.cpu().numpy(), want_mm)
    np.testing.assert_array_equal(w.cpu().numpy(), want_w)
    plan.close()


@pytest.mark.parametrize("W,H", SHAPES)
def test_cholesky_qr2_keeps_blocks_apart(cuda, W, H):
    """Bounds as the oracle's, and the finite blocks' weights as without the others."""
    import torch
    plan, o = B.Plan(W, H, fp32_qr=B.QR_CHOLESKY2), Oracle(W, H)
    draws = _draw(np.random.default_rng(W), o.blocks)
    want_w, want_mm = np.zeros(o.blocks * 30, np.float32), np.zeros(o.blocks * 12, np.float32)
    o.fitter(want_w, want_mm, draws[1].reshape(-1).copy(), 5)
    got = []
    for tmp in draws:
        w, mm = torch.empty(o.blocks, 30, device=cuda), torch.empty(o.blocks * 12, device=cuda)
        B.fitter(plan, w, mm, torch.from_numpy(tmp.reshape(-1)).to(cuda), 5)
        got.append(w)
    np.testing.assert_array_equal(mm.cpu().numpy(), want_mm)
    assert torch.isfinite(got[0]).all()
    assert torch.equal(got[0][1::2], got[1][1::2])
    plan.close()


@pytest.mark.parametrize("W,H", [
    (64, 48), (416, 352), (704, 640),
    (2080, 1440),   # 3036 blocks: six rounds
    (2464, 1440),   # 3588: seven, groups brought together
])
def test_cholesky_qr2_equals_the_256_thread_form(cuda, W, H):
    sc = B.Scene(7, W, H, 8)
    frames = [sc.render(f) for f in range(2)]
    got = []
    for pipeline in (B.PIPELINE_STAGED, B.PIPELINE_FUSED):
        plan = B.Plan(W, H, fp32_qr=B.QR_CHOLESKY2, half_history=1, pipeline=pipeline)
        for f, d in enumerate(frames):
            plan.upload_frame(d["albedo"], d["normals"], d["positions"], d["noisy"])
            plan.denoise_frame(sc.prev_camera(f), sc.pixel_offset(f))
        got.append(plan.download_result())
        plan.close()
    np.testing.assert_array_equal(got[0], got[1])
