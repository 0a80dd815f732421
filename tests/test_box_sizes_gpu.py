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
import torch

from gragles2d_b200 import dumpfile, gg
from gragles2d_b200 import microstructure as ms
from test_oracle_port import _restate_step, port

pytestmark = pytest.mark.gpu

# (grains, grid): box edges about 14-32 (the whole domain), 30-60, 60-100, 100-150, above 150
CASES = [(1, 9), (2, 18), (40, 200), (9, 160), (5, 190), (4, 260)]


def _run(tmp_path, grains, grid, precision, steps, isotropic=1, gamma=1.0, micro=None):
    xml = ms.make_case(str(tmp_path), f"v{grains}_{grid}", micro or ms.voronoi(grains, grid, 7),
                       IsIsotropicNetwork=isotropic)
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


def _shapes(name, nn):
    """Labels of grains whose contours are no single ring met by every row twice."""
    y, x = np.mgrid[0:nn, 0:nn]
    if name == "comb":  # two grains with interlocking teeth: one long contour each
        labels = np.where((x // 12) % 2 == 0, 1, 2)
        labels[:12], labels[-12:] = 1, 2
    elif name == "islands":  # a grain with holes, and islands of others in it
        labels = np.ones((nn, nn), int)
        labels[:, nn - nn // 4:] = 2
        labels[10:22, 8:20] = 3
        labels[30:45, 10:28] = 4
        labels[34:40, 15:22] = 5
    else:  # blocks that meet at corners: saddles
        labels = np.where((x // 8 + y // 8) % 2 == 0, 1, 2 + (x // 8) % 2)
    return labels


@pytest.mark.parametrize("name,nn", [("comb", 60), ("comb", 90), ("islands", 60), ("blocks", 48)])
def test_contours_of_winding_grains(tmp_path, name, nn):
    """The level set walks a contour in pieces from starts in several rows:
    long contours between two starts, other contours in the box, and saddles
    must give the reference's points in its order (bit for bit), from the first
    contours on."""
    labels = _shapes(name, nn)
    n = int(labels.max())
    rng = np.random.Generator(np.random.PCG64(3))
    euler = ms.quaternion_to_bunge(ms.shoemake_quaternions(rng, n))
    micro = ms.Microstructure(labels.astype(ms.voronoi(2, 8, 1).labels.dtype), rng.random((n, 2)), euler)
    d, _ = _run(tmp_path, n, nn, gg.PRECISION_PLAIN, 2, micro=micro)
    first = d.records[0]
    for gid, g in first.grains.items():
        if g.state == 1:
            assert g.id_box == g.box
            pts, _ = port.contour(g.phi, g.box, g.idlocal, gid)
            np.testing.assert_array_equal(pts, g.contour[:, :2], err_msg=f"contour of grain {gid}")
    checked = sum(_restate_step(d, r0, r1)[0] for r0, r1 in zip(d.records, d.records[1:]))
    assert checked >= 2


@pytest.mark.parametrize("n", [4, 17, 31, 32, 33, 64, 127])
def test_static_box_convolution_at_the_edges_of_its_kernels(n):
    """Boxes up to 32 cells take one CTA, larger ones three kernels.  Four direct
    sums of at most n terms round by 2 n 2^-53 of their largest partial sum each,
    in all below 1e-12 of the field's maximum at n = 128."""
    nn, dt = 800, 3.125e-6
    x = np.random.default_rng(n).standard_normal((n, n))
    i2 = np.arange(n // 2 + 1)
    j2 = np.minimum(np.arange(n), n - np.arange(n))
    g = np.exp(-np.sqrt(2 / np.pi) * (i2[None, :] ** 2 + j2[:, None] ** 2) * 4.0 * dt * nn ** 2 / n ** 2 * np.pi ** 2)
    ref = np.fft.irfft2(np.fft.rfft2(x) * g, s=(n, n))
    src = torch.tensor(x, device="cuda")
    out = torch.full((n, n), float("nan"), dtype=torch.float64, device="cuda")
    gg.convolve_box_static(src.data_ptr(), out.data_ptr(), n, dt, nn)
    np.testing.assert_allclose(out.cpu().numpy(), ref, rtol=0, atol=1e-12 * np.abs(x).max())
    gg.convolve_box_static(src.data_ptr(), src.data_ptr(), n, dt, nn)  # in place
    assert torch.equal(src, out)
