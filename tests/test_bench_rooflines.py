"""The flux line of bench.py: the launch that ran is the one that is reported,
with its own faces (CPU; the times are made up)."""
import pytest

import bench


def prof(**ms):
    p = {n: (0., 0) for n in ("k_flux_x", "k_flux_y", "k_flux_z", "k_flux_all", "k_flux_fix")}
    p.update({n: (v, 2) for n, v in ms.items()})
    return p


def test_one_launch_a_direction():
    name, ms, faces = bench.flux_launch(prof(k_flux_x=2., k_flux_y=3., k_flux_z=3., k_flux_fix=9.), 192, 96, 64)
    assert (name, ms, faces) == ("k_flux_x", 1., 193 * 98 * 66)


@pytest.mark.parametrize("shape, faces", [((128, 128, 1), 129 * 130 + 130 * 129), ((40, 1, 1), 41),
                                          ((24, 16, 8), 25 * 18 * 10 + 26 * 17 * 10 + 26 * 18 * 9)])
def test_one_launch_for_all_directions(shape, faces):
    assert bench.flux_launch(prof(k_flux_all=4., k_flux_fix=1.), *shape) == ("k_flux_all", 2., faces)


def test_traffic_belongs_to_the_captured_launch():
    a = bench.flux_roofline(prof(k_flux_x=2.), 192, 96, 64, 6500., "measured", 18.)
    assert a["kernel"] == "k_flux_x" and a["traffic"] > a["algorithmic_bytes_per_launch"] and a["traffic_source"]
    b = bench.flux_roofline(prof(k_flux_x=2.), 96, 96, 64, 6500., "measured", 18.)
    assert b["traffic"] is None and b["traffic_source"] is None
    assert b["fp64"]["achieved_tflops"] == pytest.approx(bench.FLUX_FP64_PER_FACE * 97 * 98 * 66 / 1e-3 / 1e12)
