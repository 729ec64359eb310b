"""The per-pixel stages on values of every size.

Where a divisor serves several quotients, they come from its reciprocal when
everything lies within 2^+-60 and from true divisions otherwise; the values
here lie on both sides, with zeros, infinities and NaN among them.  Results
must equal the oracle's.
"""
import numpy as np
import pytest

import bmfr_b200 as B
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def _any_size(rng, shape, low=-70, high=70):
    v = np.exp2(rng.uniform(low, high, shape)) * rng.choice([-1.0, 1.0], shape)
    kind = rng.integers(0, 400, shape)
    v[kind == 0], v[kind == 1], v[kind == 2], v[kind == 3] = 0.0, np.inf, -np.inf, np.nan
    return v.astype(np.float32)


@pytest.mark.parametrize("W,H,frame", [(63, 47, 3), (256, 96, 9)])
def test_pixel_stages_match_oracle_on_any_size(cuda, W, H, frame):
    import torch
    rng = np.random.default_rng(W + frame)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    plan, o = B.Plan(W, H), Oracle(W, H)
    img, px = (H, W, 3), W * H
    # History positions over the whole image and past its edges, some exact.
    pix = np.stack(np.meshgrid(np.arange(W), np.arange(H)), -1) + rng.uniform(-3, 3, (H, W, 2))
    pix[rng.integers(0, 4, (H, W)) == 0] = np.round(pix)[rng.integers(0, 4, (H, W)) == 0][:1]
    pix = pix.astype(np.float32)
    inside = (pix[..., 0] >= 0) & (pix[..., 0] < W - 1) & (pix[..., 1] >= 0) & (pix[..., 1] < H - 1)
    accept = np.where(inside, rng.integers(0, 16, (H, W)), 0).astype(np.uint8)
    spp = rng.integers(1, 256, (H, W)).astype(np.uint8)

    # weighted sum: ranges on both sides of 1 and of 2^60
    weights = rng.standard_normal((o.blocks, 10, 3)).astype(np.float32)
    mm = np.sort(_any_size(rng, (o.blocks, 6, 2), -8, 66), -1)
    normals, positions = _any_size(rng, img, -10, 2), _any_size(rng, img, -30, 33)
    want, got = np.zeros(img, np.float32), torch.zeros(img, device=cuda)
    o.weighted_sum(weights, mm, want, normals, positions, frame)
    B.weighted_sum(plan, t(weights), t(mm), got, t(normals), t(positions), None, frame)
    np.testing.assert_array_equal(got.cpu().numpy(), want)

    # filtered accumulation
    filt, albedo, before = _any_size(rng, img), rng.uniform(0, 1, img).astype(np.float32), _any_size(rng, img)
    want, mapped = np.zeros(img, np.float32), np.zeros(img, np.float32)
    got, tm = torch.zeros(img, device=cuda), torch.zeros(img, device=cuda)
    o.accumulate_filtered_data(filt, pix, accept, albedo, mapped, spp, before, want, frame)
    B.accumulate_filtered_data(plan, t(filt), t(pix), t(accept), t(albedo), tm, t(spp), t(before), got, frame)
    np.testing.assert_array_equal(got.cpu().numpy(), want)

    # taa: colours below 2^60 in the frame, any size in the history
    new = _any_size(rng, img, -20, 20)
    want, got = np.zeros(img, np.float32), torch.zeros(img, device=cuda)
    o.taa(pix, new, want, before, frame)
    B.taa(plan, t(pix), t(new), got, t(before), frame)
    np.testing.assert_array_equal(got.cpu().numpy(), want)
    plan.close()
