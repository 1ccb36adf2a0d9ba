"""Pose evaluation at the sizes where a launch changes shape: one request, a CTA's last request
alone, skeletons of one bone, of a warp's width and one more, and of the most bones; device arrays
that are only 4-byte aligned.  Against the oracle's restatement of sft_pose_update, with the bound
of test_gpu_pose.py (device and host acosf / sinf / cosf round differently in the slerp)."""
import numpy as np
import pytest
import torch

from oracle_lib import oracle_pose, pose_blob
from sofren2_gb300 import runtime, scenes

pytestmark = pytest.mark.gpu

TOL = 2e-5


@pytest.mark.parametrize("bones,n,shift", [(1, 1, 0), (6, 33, 1), (32, 17, 0), (33, 5, 3), (22, 1231, 0), (128, 9, 2)])
def test_pose_sizes_match_oracle(renderer, bones, n, shift):
    rig = scenes.pose_rig(6200 + bones, n_bones=max(bones, 6))
    if bones < 6:      # the generator's animations name bones up to 5
        rig["bones"] = rig["bones"][:bones]
    req = [(a, t) for a, t in scenes.pose_requests(rig, n + n // 2 + 4, seed=bones) if 0 <= a < len(rig["anims"])][:n]
    ref = oracle_pose(pose_blob(rig, req), bones, n)
    sk = renderer.skeleton_upload(rig)
    rec = np.zeros(n, runtime.POSE_REQUEST_DTYPE)
    rec["skeleton"], rec["animation"], rec["time"] = sk, [a for a, _ in req], [t for _, t in req]
    d_req = torch.from_numpy(rec.view(np.uint8).copy()).cuda()
    d_off = torch.arange(0, n * bones, bones, dtype=torch.int32, device="cuda")
    flat = [torch.zeros(n * bones * 16 + 4, dtype=torch.float32, device="cuda") for _ in range(2)]
    renderer.pose_eval_device(d_req.data_ptr(), d_off.data_ptr(), n, flat[0].data_ptr() + 4 * shift, flat[1].data_ptr() + 4 * shift)
    torch.cuda.synchronize()
    for k, f in enumerate(flat):
        got = f.cpu().numpy()
        assert not got[:shift].any() and not got[shift + n * bones * 16:].any(), "written outside the outputs"
        got = got[shift:shift + n * bones * 16].reshape(n, bones, 16)
        exp = ref[:, k].reshape(n, bones, 16)
        scale = np.abs(exp).max(axis=2, keepdims=True) + 1e-6
        assert (np.abs(got - exp) / scale).max() <= TOL
