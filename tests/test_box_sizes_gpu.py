"""Every stage of the isotropic step over the range of box sizes, against the
C restatement: networks of a few grains whose boxes reach from a few cells to
more than 200, among them boxes that span the whole domain.  The plain form
must match bit for bit (fields, IDLocal, contours, boxes, areas) on every
step; the batched form's areas must stay within FP32's reach of the plain
form's.

A few steps move an area by far less than a cell, and FP32 rounds the field
by about 1e-7 h, a contour of P cells' length by at most 1e-7 P cells; grains
here have areas above P / 4 cells, so 1e-5 relative leaves a factor of 25.
"""
import os

import numpy as np
import pytest

from gragles2d_b200 import dumpfile, gg
from gragles2d_b200 import microstructure as ms
from test_oracle_port import _restate_step

pytestmark = pytest.mark.gpu

# (grains, grid): box edges about 14-32 (the whole domain), 30-60, 60-100, 100-150, above 150
CASES = [(1, 9), (2, 18), (40, 200), (9, 160), (5, 190), (4, 260)]


def _run(tmp_path, grains, grid, precision, steps, isotropic=1, gamma=1.0):
    xml = ms.make_case(str(tmp_path), f"v{grains}_{grid}", ms.voronoi(grains, grid, 7), IsIsotropicNetwork=isotropic)
    settings = gg.Settings(xml, precision=precision)
    settings.p.gamma_hagb *= gamma
    h = gg.GrainHandler(settings, device=0)
    try:
        h.load_voxel_files()
        h.distanceInitialisation()
        h.find_neighbors()
        p = os.path.join(str(tmp_path), f"{precision}.dump")
        h.dump(p, 0)
        for k in range(steps):
            h.step(1)
            h.dump(p, k + 1, append=True)
        assert h.status() == 0
        return dumpfile.read(p), h.areas()
    finally:
        h.close()


@pytest.mark.parametrize("grains,grid", CASES)
def test_plain_steps_match_the_restatement(tmp_path, grains, grid):
    d, _ = _run(tmp_path, grains, grid, gg.PRECISION_PLAIN, 3)
    for r0, r1 in zip(d.records, d.records[1:]):
        checked, skipped = _restate_step(d, r0, r1)
        assert checked == sum(1 for g in r0.grains.values() if g.state == 1) and skipped == 0


@pytest.mark.parametrize("isotropic", [1, 0])
@pytest.mark.parametrize("grains,grid", CASES)
def test_batched_areas_follow_the_plain_ones(tmp_path, grains, grid, isotropic):
    """Anisotropic (Read-Shockley) networks put the corrector's two searches for
    the nearest contour vertex side by side: the plain form's by tiles, the
    batched form's by cells, on contours up to some 600 points."""
    _, plain = _run(tmp_path, grains, grid, gg.PRECISION_PLAIN, 3, isotropic)
    _, batched = _run(tmp_path, grains, grid, gg.PRECISION_BATCHED, 3, isotropic)
    np.testing.assert_allclose(batched, plain, rtol=1e-5)


@pytest.mark.parametrize("grains,grid", CASES)
def test_batched_corrector_of_the_whole_band(tmp_path, grains, grid):
    """With a relative high-angle energy above 1 no pixel takes the convolved
    value as it is: the whole band of 2 delta around each boundary is projected,
    also far from it and over whole tiles, by the batched form's queues."""
    _, plain = _run(tmp_path, grains, grid, gg.PRECISION_PLAIN, 3, 0, 1.01)
    _, batched = _run(tmp_path, grains, grid, gg.PRECISION_BATCHED, 3, 0, 1.01)
    np.testing.assert_allclose(batched, plain, rtol=1e-5)
