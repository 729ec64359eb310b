"""Frames whose inputs hold infinities: binary16 columns overflow inside the fit
(tests/test_fitter_nonfinite.py holds the staged pipeline's fitter to the oracle
there), and the fused pipeline must give the staged one's results."""
import numpy as np
import pytest

import bmfr_b200 as B

pytestmark = pytest.mark.gpu


def test_fused_pipeline_equals_staged(cuda):
    W, H = 333, 211
    got = []
    for pipeline in (B.PIPELINE_STAGED, B.PIPELINE_FUSED):
        rng = np.random.default_rng(W)
        sc, plan, results = B.Scene(5, W, H, 8), B.Plan(W, H, pipeline=pipeline), []
        for f in range(5):
            d = {k: v.astype(np.float32) for k, v in sc.render(f).items()}
            for k in ("noisy", "normals", "positions"):
                kind = rng.random(d[k].shape)
                for lo, v in ((0.0, np.nan), (2e-4, np.inf), (4e-4, -np.inf)):
                    d[k][(kind >= lo) & (kind < lo + 2e-4)] = v
            plan.upload_frame(d["albedo"], d["normals"], d["positions"], d["noisy"])
            plan.denoise_frame(sc.prev_camera(f), sc.pixel_offset(f))
            results.append(plan.download_result())
        got.append(results)
        plan.close()
    for f in range(5):
        np.testing.assert_array_equal(got[0][f], got[1][f], err_msg=f"frame {f}")
