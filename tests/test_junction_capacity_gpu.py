"""A grain with more junctions than its list holds (48) is a capacity error,
whichever lanes of the level set's warp found the ones too many."""
import numpy as np
import pytest

from gragles2d_b200 import gg
from gragles2d_b200 import microstructure as ms

pytestmark = pytest.mark.gpu


def _alternating(blocks, nn=96, tooth=3):
    """A square grain (2) whose sides are lined by blocks of 3 x 3 pixels that
    belong to two grains in turn: about 4 x blocks junctions, 3 neighbours."""
    labels = np.ones((nn, nn), int)
    a = (nn - tooth * blocks) // 2
    b = a + tooth * blocks
    labels[a:b, a:b] = 2
    for k in range(blocks):
        at = slice(a + tooth * k, a + tooth * (k + 1))
        labels[at, a - tooth:a] = labels[a - tooth:a, at] = 3 + k % 2
        labels[at, b:b + tooth] = labels[b:b + tooth, at] = 4 - k % 2
    rng = np.random.Generator(np.random.PCG64(5))
    euler = ms.quaternion_to_bunge(ms.shoemake_quaternions(rng, 4))
    return ms.Microstructure(labels.astype(ms.voronoi(2, 8, 1).labels.dtype), rng.random((4, 2)), euler)


def _step(directory, precision, blocks):
    xml = ms.make_case(str(directory), "ring", _alternating(blocks), IsIsotropicNetwork=1)
    h = gg.GrainHandler(gg.Settings(xml, precision=precision), device=0)
    try:
        h.load_voxel_files()
        h.distanceInitialisation()
        h.find_neighbors()
        h.step(1)
        return h.status()
    finally:
        h.close()


@pytest.mark.parametrize("blocks", [12, 14, 16])  # 52, 60 and 68 junctions
@pytest.mark.parametrize("precision", [gg.PRECISION_PLAIN, gg.PRECISION_BATCHED])
def test_more_junctions_than_the_list_holds(tmp_path, precision, blocks):
    with pytest.raises(gg.GGError, match="status 0x8") as e:
        _step(tmp_path, precision, blocks)
    assert e.value.code == 5


def test_as_many_junctions_as_fit(tmp_path):
    """36 junctions; in the plain form, as the batched one builds sectors of them, whose lists are shorter."""
    assert _step(tmp_path, gg.PRECISION_PLAIN, 8) == 0
