"""The FP64 total cost and the mean error of a host problem: every loss, one
camera model and several, observations in any order, one to many blocks of
them, none at all, and indices out of range (found on the device, reported
with the status and words of the host's check).

Bar: 1e-10 against the oracle. A residual of about a pixel out of coordinates
of about 1e3 carries 1e3 roundings of 1.1e-16 at most ten times over, 1e-12
relative; the sums of at most 3e4 non-negative terms add less."""
import ctypes as C

import numpy as np
import pytest

from sfmtory_gb300 import abi, native, scenes

ALL = (abi.PINHOLE, abi.SIMPLE_PINHOLE, abi.SIMPLE_RADIAL, abi.RADIAL, abi.OPENCV)


def _problem(images, points, models, order, seed=5):
    rng = np.random.default_rng(seed)
    p = scenes.local_window(rng, images, points, views=4.0, models=models)
    n = len(p.obs_image)
    at = {"sorted": np.arange(n), "reversed": np.arange(n)[::-1], "shuffled": rng.permutation(n)}[order]
    p.obs_image, p.obs_point, p.obs_xy = p.obs_image[at].copy(), p.obs_point[at].copy(), p.obs_xy[at].copy()
    return p


@pytest.mark.gpu
@pytest.mark.parametrize("order", ["sorted", "reversed", "shuffled"])
@pytest.mark.parametrize("models", [(abi.OPENCV,), ALL], ids=["one-model", "all-models"])
@pytest.mark.parametrize("images,points", [(2, 1), (3, 64), (9, 900), (20, 7000)])
def test_cost_and_mean_error_match_oracle(oracle_lib, images, points, models, order):
    p = _problem(images, points, models, order)
    for loss in (abi.LOSS_NONE, abi.LOSS_HUBER, abi.LOSS_CAUCHY):
        g, r = native.total_cost(p, robust_loss=loss), oracle_lib.total_cost(p, robust_loss=loss)
        assert abs(g - r) <= 1e-10 * r
    g, r = native.mean_reprojection_error_arrays(p), oracle_lib.mean_reprojection_error(p)
    assert abs(g - r) <= 1e-10 * r


@pytest.mark.gpu
def test_no_observations():
    p = _problem(3, 10, (abi.PINHOLE,), "sorted")
    p.obs_image, p.obs_point, p.obs_xy = p.obs_image[:0], p.obs_point[:0], p.obs_xy[:0]
    assert native.total_cost(p) == 0.0
    assert native.mean_reprojection_error_arrays(p) == 0.0


def _status(p, mode):
    """Status and message of the C entry, called without the binding's own checks."""
    L = native.load()
    packed = native.PackedProblem(p)
    out = C.c_double()
    st = (L.sfmba_mean_reprojection_error(C.byref(packed.struct), C.byref(out)) if mode else
          L.sfmba_total_cost(C.byref(packed.struct), C.byref(native.default_options()), C.byref(out)))
    return st, L.sfmba_last_error().decode()


# Runs with and without a GPU: a wrong index is reported before a missing device.
def _check_rejected(mode, field, value):
    p = _problem(4, 50, (abi.PINHOLE,), "sorted")
    getattr(p, field)[1] = value
    st, msg = _status(p, mode)
    assert st == 1
    name = {"camera_model": "camera 1 has an unknown model id"}.get(field, f"{field}[1] out of range")
    assert name in msg


BAD = [("obs_image", -1), ("obs_image", 4), ("obs_point", -1), ("obs_point", 50), ("camera_of_image", 4),
       ("camera_of_image", -1), ("camera_model", 99)]


@pytest.mark.parametrize("mode", [0, 1], ids=["cost", "mean"])
@pytest.mark.parametrize("field,value", BAD)
def test_rejected_without_device_work(mode, field, value):
    _check_rejected(mode, field, value)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [0, 1], ids=["cost", "mean"])
@pytest.mark.parametrize("field,value", BAD)
def test_rejected_on_the_device(mode, field, value):
    _check_rejected(mode, field, value)
    p = _problem(4, 50, (abi.PINHOLE,), "sorted")
    assert native.total_cost(p) > 0.0  # the context is usable afterwards
