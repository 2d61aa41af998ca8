"""Cameras whose vectors are not float64 arrays: subclasses may give lists,
tuples, integer or float32 arrays.  The view matrix is numpy's look-at of the
vectors as they are given (float32 vectors compute in float32)."""

import numpy as np
import pytest

from pyvr_gb300 import Camera
from pyvr_gb300.renderer import camera_uniforms

POSITION, UP = (2.0, -1.0, 3.0), (0.0, 0.0, 1.0)


class _Fixed(Camera):
    vectors = None

    def get_camera_vectors(self):
        return self.vectors


def _look_at(target, position, up):
    fwd = target - position
    fwd = fwd / np.linalg.norm(fwd)
    right = np.cross(fwd, up)
    right = right / np.linalg.norm(right)
    up_c = np.cross(right, fwd)
    m = np.eye(4)
    m[:3, 0], m[:3, 1], m[:3, 2] = right, up_c, -fwd
    m[3, :3] = -np.dot(right, position), -np.dot(up_c, position), np.dot(fwd, position)
    return m.astype(np.float32)


@pytest.mark.parametrize("make", [list, tuple, lambda v: np.array(v, np.int64), lambda v: np.array(v, np.float32),
                                  lambda v: np.array(v, np.float64)])
def test_vectors_of_other_types(make):
    cam = _Fixed()
    cam.vectors = make(POSITION), make(UP)
    want = _look_at(cam.target, *cam.vectors)
    assert np.array_equal(cam.get_view_matrix(), want)
    view, _, pos = camera_uniforms(cam, 40, 30)
    assert np.array_equal(view, want) and np.array_equal(pos, np.array(POSITION, np.float32))
