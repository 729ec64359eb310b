"""The reference-arithmetic and CholeskyQR2 fitters at every launch shape they take.

The number of 32x32 blocks per SM decides how many teams share a block and
how many blocks share an SM, so the sizes here lie on both sides of each
line, with one and with several blocks per group.  tmp_data is drawn, not
rendered: columns of mixed ranges, constant columns, a first column that is
not the constant feature, black and +-65504 colours, and infinities.  Weights
and min/max values must equal the oracle's.
"""
import numpy as np
import pytest

import bmfr_b200 as B
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def _draw(rng, blocks, special=True):
    t = np.empty((blocks, 13, 1024), np.float32)
    t[:, 0] = 1.0
    n = rng.standard_normal((blocks, 3, 1024))
    t[:, 1:4] = n / np.linalg.norm(n, axis=1, keepdims=True)
    scale = np.exp2(rng.uniform(-12, 7, (blocks, 3, 1)))
    t[:, 4:7] = rng.uniform(-4, 4, (blocks, 3, 1)) + scale * rng.standard_normal((blocks, 3, 1024))
    t[:, 7:10] = t[:, 4:7] ** 2
    t[:, 10:13] = rng.lognormal(-1.0, 1.5, (blocks, 3, 1024))
    kind = rng.integers(0, 12 if special else 2, blocks)
    t[kind == 0, 5] = 0.0                     # a plane: no range
    t[kind == 0, 8] = 0.0
    t[kind == 1, 10:13] = 0.0                 # black
    t[kind == 2, 0] = rng.uniform(0.5, 2.0, (int((kind == 2).sum()), 1024))   # not the constant feature
    t[kind == 3, 11] = 65504.0
    t[kind == 4, 4:10] = -65504.0
    t = np.clip(t, -65504, 65504).astype(np.float16)
    t[kind == 5, 12, 17] = np.inf
    t[kind == 6, 6, 1000] = -np.inf
    return t


# The precision form's stated errors against the FP64 fit: mean 1e-4, at most 2e-2.
@pytest.mark.parametrize("W,H", [
    (64, 48),       # 9 blocks: one per SM
    (384, 320),     # 143
    (416, 352),     # 168: up to three per SM
    (672, 608),     # 440
    (704, 640),     # 483: four groups per SM
    (1600, 1024),   # 1683: three blocks each
    (1856, 1280),   # 2419: five
    (2080, 1440),   # 3036: six
    (2464, 1440),   # 3588: seven, groups brought together, most idle in the last
    (2592, 1440),   # 3772: seven
])
def test_cholesky_qr2_shapes_match_fp64(cuda, W, H):
    import torch
    plan = B.Plan(W, H, fp32_qr=B.QR_CHOLESKY2)
    blocks = plan.sizes.blocks
    tmp = _draw(np.random.default_rng(W * 5 + H), blocks, special=False)
    dev = torch.from_numpy(tmp.reshape(-1)).to(cuda)
    w, mm, mm64 = (torch.empty(blocks, n, device=cuda) for n in (30, 12, 12))
    w64 = torch.empty(blocks, 30, device=cuda, dtype=torch.float64)
    B.fitter(plan, w, mm, dev, 5)
    B.fitter_fp64(plan, w64, mm64, dev, 5)
    assert torch.equal(mm, mm64)
    err = (w.double() - w64).norm(dim=1) / w64.norm(dim=1).clamp(min=1e-3)
    assert err.mean() < 1e-4 and err.max() < 2e-2, (err.mean().item(), err.max().item())
    plan.check_device()
    plan.close()


@pytest.mark.parametrize("W,H,noise", [
    (64, 48, 1e-2),       # 9 blocks: one per SM
    (384, 320, 1e-2),     # 143
    (416, 352, 1e-2),     # 168: up to three per SM
    (672, 608, 1e-2),     # 440
    (704, 640, 1e-2),     # 483: six groups per SM, some idle
    (928, 928, 1e-2),     # 900: a second block for some groups
    (1056, 960, 1e-2),    # 1054
    (1280, 720, 1e-2),    # 984: seven per SM
    (1600, 1024, 1e-2),   # 1683: two blocks per group
    (1760, 1056, 1e-2),   # 1904: seven groups, two rounds
    (64, 48, 0.0),
    (64, 48, 1.5),        # noise beyond the fast two-sum
])
def test_fitter_shapes_match_oracle(cuda, W, H, noise):
    import torch
    o = Oracle(W, H, noise_amount=noise)
    plan = B.Plan(W, H, noise_amount=noise)
    tmp = _draw(np.random.default_rng(W * 7 + H), o.blocks)
    want_w, want_mm = np.zeros(o.blocks * 30, np.float32), np.zeros(o.blocks * 12, np.float32)
    o.fitter(want_w, want_mm, tmp.reshape(-1).copy(), 5)
    dev = torch.from_numpy(tmp.reshape(-1)).to(cuda)
    w, mm = torch.empty(o.blocks * 30, device=cuda), torch.empty(o.blocks * 12, device=cuda)
    B.fitter(plan, w, mm, dev, 5)
    np.testing.assert_array_equal(mm.cpu().numpy(), want_mm)
    np.testing.assert_array_equal(w.cpu().numpy(), want_w)
    plan.check_device()
    plan.close()


@pytest.mark.parametrize("noise", [1e-2, 1.5])
def test_float_tmp_data_matches_oracle(cuda, noise):
    """First columns that are and are not the constant feature, noise on both sides of 1."""
    import torch
    W, H = 320, 200
    o = Oracle(W, H, use_half=False, noise_amount=noise)
    plan = B.Plan(W, H, use_half_precision_in_tmp_data=0, noise_amount=noise)
    tmp = np.nan_to_num(_draw(np.random.default_rng(3), o.blocks).astype(np.float32), posinf=1.0, neginf=-1.0)
    want_w, want_mm = np.zeros(o.blocks * 30, np.float32), np.zeros(o.blocks * 12, np.float32)
    o.fitter(want_w, want_mm, tmp.reshape(-1).copy(), 5)
    w, mm = torch.empty(o.blocks * 30, device=cuda), torch.empty(o.blocks * 12, device=cuda)
    B.fitter(plan, w, mm, torch.from_numpy(tmp.reshape(-1)).to(cuda), 5)
    np.testing.assert_array_equal(mm.cpu().numpy(), want_mm)
    np.testing.assert_array_equal(w.cpu().numpy(), want_w)
    plan.close()


def test_fused_pipeline_with_large_noise_matches_staged(cuda):
    W, H = 96, 80
    sc = B.Scene(5, W, H, 8)
    got = []
    for pipeline in (B.PIPELINE_STAGED, B.PIPELINE_FUSED):
        plan = B.Plan(W, H, noise_amount=1.5, pipeline=pipeline)
        for f in range(3):
            d = sc.render(f)
            plan.upload_frame(d["albedo"], d["normals"], d["positions"], d["noisy"])
            plan.denoise_frame(sc.prev_camera(f), sc.pixel_offset(f))
        got.append(plan.download_result())
        plan.close()
    np.testing.assert_array_equal(got[0], got[1])
