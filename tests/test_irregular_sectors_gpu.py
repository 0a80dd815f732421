"""The plain form builds sectors only for the grains that its corrector
corrects: none of a grain whose motion was irregular (src/box.cpp:428-447),
whatever its junctions."""
import numpy as np
import pytest

from gragles2d_b200 import gg
from gragles2d_b200 import microstructure as ms

pytestmark = pytest.mark.gpu


def _crowded(nn=96, side=24, tooth=3, arm=20):
    """A square grain (5) between 28 others of 3 x 3 pixels, all within a sector
    radius of the next, so that it has more junctions than a sector's list
    holds (24), and four outer grains; arms one pixel wide, gone after a step,
    halve its contour, which makes its motion irregular."""
    y, x = np.mgrid[0:nn, 0:nn]
    labels = 1 + (x > y) + 2 * (x + y >= nn)
    a, b, mid = (nn - side) // 2, (nn + side) // 2, nn // 2
    labels[a:b, a:b] = 5
    gid = 6
    for k in range(a, b, tooth):
        if k <= mid < k + tooth:
            continue
        for block in ((slice(k, k + tooth), slice(a - tooth, a)), (slice(k, k + tooth), slice(b, b + tooth)),
                      (slice(a - tooth, a), slice(k, k + tooth)), (slice(b, b + tooth), slice(k, k + tooth))):
            labels[block] = gid
            gid += 1
    labels[mid + 1, a - arm:b + arm] = 5
    labels[a - arm:b + arm, mid + 1] = 5
    n = gid - 1
    rng = np.random.Generator(np.random.PCG64(5))
    euler = ms.quaternion_to_bunge(ms.shoemake_quaternions(rng, n))
    return ms.Microstructure(labels.astype(ms.voronoi(2, 8, 1).labels.dtype), rng.random((n, 2)), euler)


@pytest.mark.parametrize("stages", [False, True])
def test_irregular_grain_with_crowded_junctions(tmp_path, stages):
    xml = ms.make_case(str(tmp_path), "ring", _crowded(), IsIsotropicNetwork=0)
    h = gg.GrainHandler(gg.Settings(xml, precision=gg.PRECISION_PLAIN), device=0)
    try:
        h.load_voxel_files()
        h.distanceInitialisation()
        h.find_neighbors()
        for _ in range(2):
            if stages:
                for stage in (h.convolution, h.updateSecondOrderNeighbors, h.comparison_box, h.level_set,
                              h.redistancing):
                    stage()
            else:
                h.step(1)
            if h.loop == 1:
                core = h.grain_stats()[4]
                assert core.state == 1 and core.motion_regular == 0
        assert h.status() == 0
    finally:
        h.close()
