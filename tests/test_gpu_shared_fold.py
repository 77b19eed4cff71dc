"""Dense reduced system with cameras that many images share: the entries
between two slots of more than 32 images each are folded from the list of
image pairs. Cameras used by 32 (one short of the list), 33 and many images,
one and several at once, held parameters and images without observations,
against the oracle (FP64, same iterations; cost and parameters 1e-6, the
bars of the other dense parity tests)."""
import numpy as np
import pytest

from sfmtory_gb300 import abi, native, scenes

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


@pytest.mark.parametrize("images_per_camera", [(32, 32), (33, 33), (40, 1, 35, 33, 8), (120,)],
                         ids=["short_of_the_list", "just_listed", "mixed", "one"])
@pytest.mark.parametrize("precision", [abi.PRECISION_FP64, abi.PRECISION_MIXED], ids=["fp64", "mixed"])
def test_shared_slots_match_oracle(oracle_lib, images_per_camera, precision):
    nI, nC = sum(images_per_camera), len(images_per_camera)
    p = scenes.shared_radial(seed=nI, scale=(nI / 2000.0) ** 2, n_cameras=1)
    nI = p.num_images
    cam = np.repeat(np.arange(nC), images_per_camera)[:nI].astype(np.int32)
    mask = np.repeat(p.fixed_camera_params, nC, 0)
    keep = p.obs_image != nI // 2  # an image without observations
    p = p.copy(camera_of_image=cam, camera_model=np.repeat(p.camera_model, nC),
               camera_params=np.repeat(p.camera_params, nC, 0), fixed_cameras=np.zeros(nC, bool),
               fixed_camera_params=mask, obs_image=p.obs_image[keep], obs_point=p.obs_point[keep],
               obs_xy=p.obs_xy[keep])
    p.fixed_poses[nI // 2] = True
    kw = dict(robust_loss=abi.LOSS_NONE, max_iterations=30)
    g = native.bundle_adjust_arrays(p, solver=abi.SOLVER_DENSE, precision=precision, **kw)
    r = oracle_lib.bundle_adjust(p, **kw)
    bar = 1e-6 if precision == abi.PRECISION_FP64 else 1e-5  # mixed: the FP32 loop stops on its own rounding
    assert abs(g.final_cost - r.final_cost) <= bar * r.final_cost, (g.final_cost, r.final_cost)
    if precision == abi.PRECISION_FP64:
        assert g.iterations_run == r.iterations_run
        for a, b in ((g.poses, r.poses), (g.points, r.points), (g.camera_params, r.camera_params)):
            assert _rel(a, b) <= 1e-6
