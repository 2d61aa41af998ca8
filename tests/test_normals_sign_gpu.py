"""Signs of zero in float16 normals: a gradient of -0 (a difference of zeros of
either sign, or half of the smallest negative half) gives the component -0, as
numpy's division does."""

import numpy as np
import pytest

from pyvr_gb300 import Volume, compute_normal_volume

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("records", ["float", "half_normals"])
@pytest.mark.parametrize("brick", [2, 3, 4])
def test_negative_zero_components(records, brick):
    from pyvr_gb300.batch import DeviceVolume, get_compact_records, set_compact_records
    tiny = 2.0 ** -24
    values = np.array([0.0, -0.0, tiny, 2 * tiny, -tiny, 0.5, 1.0], np.float16)
    data = values[np.random.default_rng(brick).integers(0, len(values), (37, 37, 37))]
    with np.errstate(all="ignore"):
        want = compute_normal_volume(data).astype(np.float32)
    prev = get_compact_records()
    set_compact_records(records)
    try:
        dv = DeviceVolume(Volume(data=data), normals="device", brick_log2=brick)
    finally:
        set_compact_records(prev)
    got = dv.read_normals()
    dv.close()
    number = ~np.isnan(want)
    assert (np.signbit(want) & (want == 0.0)).sum() > 100
    assert np.array_equal(np.isnan(got), ~number)
    assert np.array_equal(got[number].view(np.uint32), want[number].view(np.uint32))
