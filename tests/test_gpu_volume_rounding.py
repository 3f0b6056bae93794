"""Submerged volumes are rounded once: a sixth of the faces' sum."""
import numpy as np
import pytest

from stonefish_gb300 import scenarios
from stonefish_gb300.hydro import transform
from tests.helpers import io_dict

pytestmark = pytest.mark.gpu


def test_volume_is_the_rounded_sixth(hctx):
    """Tetrahedra under water with two legs of 1 m and one of a / 64 m: the
    faces' sum a / 64 is exact in FP32, its sixth is not in FP64."""
    faces = np.array([[0, 2, 1], [0, 1, 3], [0, 3, 2], [1, 2, 3]], dtype=np.uint32)
    ocean, st = scenarios.flat_ocean(), scenarios.settings()
    T = transform(np.eye(3), np.array([0.0, 0.0, 2.0]))
    sums = []
    for a in range(1, 129):
        xyz = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, a / 64.0]], dtype=np.float32)
        io = io_dict()
        hctx.surface_forces(st, hctx.upload_mesh(xyz, faces), ocean, T, T, np.zeros(3), np.zeros(3), io)
        assert io["Vsub"][0] == (a / 64.0) / 6.0, a
        sums.append(a / 64.0)
    assert sum(v / 6.0 != v * (1.0 / 6.0) for v in sums) > 30
