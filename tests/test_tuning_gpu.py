"""What a launch tuning says and does: the one a launcher reports is the one it
runs."""

import ctypes

import pytest

from pyvr_gb300 import _native

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_reported_default_is_what_runs():
    # as many persistent blocks as fit, which is blocks_per_sm 0: setting the
    # reported tuning again changes nothing
    from pyvr_gb300.batch import BatchRenderer, Tuning
    br = BatchRenderer(capacity=1, slots=1)
    t = _native.PvrTuning()
    _native.check(_native.load().pvr_batch_get_tuning(br.handle, ctypes.byref(t)))
    br.close()
    default = Tuning()
    assert (t.tile_w, t.tile_h, t.steps_per_iter, t.blocks_per_sm) == (
        default.tile_w, default.tile_h, default.steps_per_iter, default.blocks_per_sm) == (16, 16, 1, 0)
