"""The per-pixel stages far from ordinary magnitudes, against the oracle:
values down to the subnormals and up to overflow, black pixels over fading
histories, NaN and infinities, history positions on whole pixels and beyond
the image.  Every output but the tone map (pow) must equal the oracle's.
"""
import numpy as np
import pytest

import bmfr_b200 as B
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def _sized(rng, shape, low, high, special=0.005):
    """Magnitudes 2^low..2^high of either sign, a few zeros, infinities and NaN."""
    v = np.exp2(rng.uniform(low, high, shape)) * rng.choice([-1.0, 1.0], shape)
    v[rng.random(shape) < special] = 0.0
    v[rng.random(shape) < special / 4] = np.inf
    v[rng.random(shape) < special / 4] = np.nan
    return v.astype(np.float32)


def _positions(rng, W, H):
    """History positions over the image and past its edges, a third of them on whole pixels."""
    pix = np.stack(np.meshgrid(np.arange(W), np.arange(H)), -1) + rng.uniform(-3, 3, (H, W, 2))
    whole = rng.integers(0, 3, (H, W)) == 0
    pix[whole] = np.round(pix[whole])
    pix[:4][whole[:4], 0] = W - 1   # the last column and row among them
    pix[-4:][whole[-4:], 1] = H - 1
    inside = whole & (pix >= 0).all(-1) & (pix[..., 0] < W) & (pix[..., 1] < H)
    assert len(np.unique(pix[inside], axis=0)) > W * H // 8
    return pix.astype(np.float32)


def _accept(rng, pix):
    """Accept bits, only for taps inside the image."""
    H, W, _ = pix.shape
    fx, fy = np.floor(pix[..., 0]), np.floor(pix[..., 1])
    bits = np.zeros((H, W), np.uint8)
    for b, (dx, dy) in enumerate(((0, 0), (1, 0), (0, 1), (1, 1))):
        inside = (fx + dx >= 0) & (fx + dx < W) & (fy + dy >= 0) & (fy + dy < H)
        bits |= (inside & (rng.random((H, W)) < 0.8)).astype(np.uint8) << b
    return bits


def _black(rng, img):
    """Half of the pixels black, so that the history alone makes their colour."""
    img[rng.integers(0, 2, img.shape[:2]) == 0] = 0.0
    return img


RANGES = [(-149, -60), (-70, 70), (50, 127.9)]


@pytest.mark.parametrize("low,high", RANGES)
@pytest.mark.parametrize("W,H,scale,half", [(64, 64, 1.0, True), (63, 47, 2.0 ** -64, True), (64, 64, 2.0 ** 64, False)])
def test_accumulate_noisy_data(cuda, W, H, scale, half, low, high):
    import torch
    rng = np.random.default_rng(W + int(high))
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    plan = B.Plan(W, H, position_limit_squared=1e30, normal_limit_squared=1e30,
                  use_half_precision_in_tmp_data=int(half))
    o = Oracle(W, H, 1e30, 1e30, use_half=half)
    # A camera that maps world x, y to history positions: exactly at 64 x 64.
    cam = np.zeros((4, 4), np.float32)
    cam[0, 0], cam[1, 1], cam[3, 0], cam[3, 1], cam[3, 3] = 2.0 / W, 2.0 / H, -1.0, -1.0, 1.0
    cam *= np.float32(scale)
    pos = np.concatenate([_positions(rng, W, H), _sized(rng, (H, W, 1), -20, 6)], -1)
    pos[rng.random((H, W)) < 0.01, 0] = 1e12      # beyond every integer
    pos[rng.random((H, W)) < 0.01, 1] = np.nan
    prev_p, nrm, prev_n = pos.copy(), _sized(rng, (H, W, 3), -4, 0), _sized(rng, (H, W, 3), -4, 0)
    prev_p[rng.random((H, W)) < 0.1] = np.nan     # rejected taps
    noisy, before = _black(rng, _sized(rng, (H, W, 3), low, high)), _sized(rng, (H, W, 3), low, high)
    spp = rng.integers(0, 256, (H, W)).astype(np.uint8)
    want = dict(pix=np.zeros((H, W, 2), np.float32), accept=np.zeros((H, W), np.uint8), colour=noisy.copy(),
                spp=np.zeros((H, W), np.uint8), tmp=o.new_tmp())
    got = {k: t(v) for k, v in want.items()}
    offset = np.array([0.0, 1.0], np.float32)
    o.accumulate_noisy_data(want["pix"], want["accept"], nrm, prev_n, pos, prev_p, want["colour"], before, spp,
                            want["spp"], want["tmp"], cam, offset, 5)
    B.accumulate_noisy_data(plan, got["pix"], got["accept"], t(nrm), t(prev_n), t(pos), t(prev_p), got["colour"],
                            t(before), t(spp), got["spp"], got["tmp"], cam, offset, 5)
    assert len(np.unique(want["accept"])) == 16
    for k, v in want.items():
        np.testing.assert_array_equal(got[k].cpu().numpy(), v, err_msg=k)
    plan.close()


@pytest.mark.parametrize("low,high", RANGES)
@pytest.mark.parametrize("W,H", [(63, 47), (256, 96)])
def test_accumulate_filtered_data(cuda, W, H, low, high):
    import torch
    rng = np.random.default_rng(W + int(high))
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    plan, o = B.Plan(W, H), Oracle(W, H)
    pix = _positions(rng, W, H)
    accept, spp = _accept(rng, pix), rng.integers(0, 256, (H, W)).astype(np.uint8)
    filt, before = _black(rng, _sized(rng, (H, W, 3), low, high)), _sized(rng, (H, W, 3), low, high)
    albedo = rng.uniform(0, 1, (H, W, 3)).astype(np.float32)
    want, mapped = np.zeros((H, W, 3), np.float32), np.zeros((H, W, 3), np.float32)
    got, tm = t(want), t(mapped)
    o.accumulate_filtered_data(filt, pix, accept, albedo, mapped, spp, before, want, 7)
    B.accumulate_filtered_data(plan, t(filt), t(pix), t(accept), t(albedo), tm, t(spp), t(before), got, 7)
    np.testing.assert_array_equal(got.cpu().numpy(), want)
    plan.close()


@pytest.mark.parametrize("W,H", [(63, 47), (256, 96)])
def test_weighted_sum_of_small_differences(cuda, W, H):
    """One scaled feature per block counts, a little above its minimum: the quotient by its range alone."""
    import torch
    rng = np.random.default_rng(W)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    plan, o = B.Plan(W, H), Oracle(W, H)
    weights = np.zeros((o.blocks, 10, 3), np.float32)
    weights[np.arange(o.blocks), rng.integers(4, 7, o.blocks)] = _sized(rng, (o.blocks, 3), 0, 20, 0.0)
    mm = np.zeros((o.blocks, 6, 2), np.float32)
    mm[..., 0] = _sized(rng, (o.blocks, 6), -130, -90)
    mm[..., 1] = np.exp2(rng.uniform(-1, 70, (o.blocks, 6)))
    positions, normals = _sized(rng, (H, W, 3), -140, -90), _sized(rng, (H, W, 3), -4, 0, 0.0)
    want = np.zeros((H, W, 3), np.float32)
    got = t(want)
    o.weighted_sum(weights, mm, want, normals, positions, 3)
    B.weighted_sum(plan, t(weights), t(mm), got, t(normals), t(positions), None, 3)
    np.testing.assert_array_equal(got.cpu().numpy(), want)
    plan.close()


def _taa(cuda, W, H, pix, new, before):
    import torch
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    plan, o = B.Plan(W, H), Oracle(W, H)
    want = np.zeros((H, W, 3), np.float32)
    got = t(want)
    o.taa(pix, new, want, before, 4)
    B.taa(plan, t(pix), t(new), got, t(before), 4)
    np.testing.assert_array_equal(got.cpu().numpy(), want)
    plan.close()


@pytest.mark.parametrize("low,high", [(-149, -120), (118, 127.99)])
@pytest.mark.parametrize("W,H", [(63, 47), (256, 96)])
def test_taa_at_the_ends_of_the_range(cuda, W, H, low, high):
    """Fading histories, products by 2 that overflow, products by 1/4 that round."""
    rng = np.random.default_rng([W, int(abs(high))])
    _taa(cuda, W, H, _positions(rng, W, H), _sized(rng, (H, W, 3), low, high), _sized(rng, (H, W, 3), low, high))


@pytest.mark.parametrize("W,H", [(63, 47), (256, 96)])
def test_taa_cross_without_a_number(cuda, W, H):
    """A cross without a number has the bounds +inf and -inf, whatever its
    box's corners hold: numbers, infinities, NaN.  One NaN channel makes the
    cross NaN and leaves the pixel's others to be seen."""
    rng = np.random.default_rng(W)
    new, before = _sized(rng, (H, W, 3), -3, 3, 0.0), _sized(rng, (H, W, 3), -3, 3, 0.05)
    for y in range(1, H - 1, 3):
        for x in range(1, W - 1, 3):
            ch = rng.integers(0, 3)
            new[y, x - 1:x + 2, ch], new[y - 1:y + 2, x, ch] = np.nan, np.nan
            for dy, dx in ((-1, -1), (-1, 1), (1, -1), (1, 1)):
                new[y + dy, x + dx] = rng.choice([0.5, 2.0, np.inf, -np.inf, np.nan])
    _taa(cuda, W, H, _positions(rng, W, H), new, before)
