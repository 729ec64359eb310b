"""Plans on streams of their own, at sizes whose fitters share an SM with
another stream's, give the frames that they give one after another."""
import numpy as np
import pytest

import bmfr_b200 as B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("qr", [B.QR_REFERENCE, B.QR_CHOLESKY2])
@pytest.mark.parametrize("W,H", [(64, 48), (320, 240), (400, 340), (640, 360)])   # 9, 99, 168, 273 blocks
def test_frames_equal_those_run_alone(cuda, W, H, qr):
    import torch
    plans, frames = 6, 4
    scenes = [B.Scene(20 + i, W, H, 8) for i in range(plans)]
    names = ("albedo", "normals", "positions", "noisy")
    inputs = [[{k: torch.from_numpy(np.ascontiguousarray(d[k])).to(cuda) for k in names}
               for d in (sc.render(f) for f in range(frames))] for sc in scenes]

    def run(streams):
        ps = [B.Plan(W, H, fp32_qr=qr) for _ in range(plans)]
        out = [torch.empty(frames, H, W, 3, device=cuda) for _ in range(plans)]
        torch.cuda.synchronize()
        for f in range(frames):
            for i, p in enumerate(ps):
                d, prev = inputs[i][f], inputs[i][f - 1] if f else None
                p.denoise_frame_io(d["albedo"], d["normals"], d["positions"], d["noisy"],
                                   prev and prev["normals"], prev and prev["positions"], scenes[i].prev_camera(f),
                                   scenes[i].pixel_offset(f), result=out[i][f], stream=streams[i])
        torch.cuda.synchronize()
        for p in ps:
            p.check_device()
            p.close()
        return out

    one = torch.cuda.Stream()
    for a, b in zip(run([one] * plans), run([torch.cuda.Stream() for _ in range(plans)])):
        assert torch.equal(a, b)
