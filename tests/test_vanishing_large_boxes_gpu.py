"""Grains that vanish while their boxes are large.  A lamella a few cells wide
between two grains keeps its length until it is gone, so its box still has an
edge of 100 cells and more in the step it vanishes in: it belongs to the level
set's kernel for large boxes in that step and in the next, which deletes it.
In the reference a grain without a contour stays for one step and is deleted
by the next level set (src/grainhdl.cpp:830-848); in between its neighbours
still see it, so their motion is regular.
"""
import os

import numpy as np
import pytest

from gragles2d_b200 import dumpfile, gg
from gragles2d_b200 import microstructure as ms
from test_oracle_port import _restate_step, port

pytestmark = pytest.mark.gpu

NN, LENGTH, STEPS = 200, 120, 8
LARGE = 97  # the longest box edge of the level set's kernel for ordinary boxes
FORMS = [gg.PRECISION_PLAIN, gg.PRECISION_BATCHED]


def _lamellae():
    """Lamellae of 1 to 4 cells' width, each between two slabs, in a Voronoi
    network (24 points per grain, so that they take 1 to 6 steps to vanish)."""
    labels = ms.voronoi(60, NN, 3).labels.astype(int)
    x0, x1, y, top = (NN - LENGTH) // 2, (NN + LENGTH) // 2, 12, 60
    for width in (1, 2, 3, 4):
        lower = y + 14 + width
        labels[y:lower] = top + 1
        labels[lower:lower + 14] = top + 2
        labels[y + 14:lower, x1:] = top + 2
        labels[y + 14:lower, x0:x1] = top + 3
        y, top = lower + 24, top + 3
    ids, labels = np.unique(labels, return_inverse=True)
    rng = np.random.Generator(np.random.PCG64(3))
    n = len(ids)
    euler = ms.quaternion_to_bunge(ms.shoemake_quaternions(rng, n))
    lamellae = [int(np.searchsorted(ids, 60 + 3 * k)) + 1 for k in (1, 2, 3, 4)]
    micro = ms.Microstructure((labels.reshape(NN, NN) + 1).astype(ms.voronoi(2, 8, 1).labels.dtype),
                              rng.random((n, 2)), euler)
    return micro, lamellae


def _run(directory, precision, isotropic, read, **params):
    """Runs the network; read(handler, step) is called after the set-up and after every step."""
    micro, lamellae = _lamellae()
    xml = ms.make_case(str(directory), "lamellae", micro, IsIsotropicNetwork=isotropic, **params)
    h = gg.GrainHandler(gg.Settings(xml, precision=precision), device=0)
    try:
        h.load_voxel_files()
        h.distanceInitialisation()
        h.find_neighbors()
        read(h, 0)
        for k in range(STEPS):
            h.step(1)
            read(h, k + 1)
        assert h.status() == 0
        return lamellae
    finally:
        h.close()


def _dumped(directory, precision, isotropic, **params):
    path = os.path.join(str(directory), "run.dump")
    lamellae = _run(directory, precision, isotropic, lambda h, k: h.dump(path, k, append=k > 0), **params)
    return dumpfile.read(path), lamellae


def _check_lifetimes(d, lamellae):
    """Every grain that is gone had vanished for exactly one step, and the
    neighbours of a vanished lamella moved regularly, with the energies of all
    their contour points known, unless their own contour shrank too fast (such
    grains keep the energies of new points, -1)."""
    large = 0
    for gid in d.records[0].grains:
        states = [r.grains[gid].state for r in d.records]
        after = states[states.index(2):] if 2 in states else []
        assert states == [1] * (len(states) - len(after)) + [2] * bool(after) + [0] * (len(after) - bool(after)), gid
        if gid not in lamellae or not after:
            continue
        k = states.index(2)
        before, now = d.records[k - 1].grains, d.records[k].grains
        edge = before[gid].box[1] - before[gid].box[0]
        large += edge > LARGE
        for q in [e[0] for e in before[gid].neighbours]:
            if q == 0 or now[q].state != 1:
                continue
            _, flagged = port.motion_regular(len(before[q].contour), len(now[q].contour), before[q].volume,
                                             port.area(now[q].contour[:, :2], d.h), d.dt)
            assert now[q].regular == int(not flagged), (gid, q)
            assert flagged or (now[q].contour[:-1, 2] >= 0).all(), (gid, q)
    assert large >= 3


@pytest.mark.parametrize("isotropic", [1, 0])
def test_plain_lamellae(tmp_path, isotropic):
    d, lamellae = _dumped(tmp_path, gg.PRECISION_PLAIN, isotropic)
    _check_lifetimes(d, lamellae)
    if not isotropic:
        return
    b = (d.ngridpoints - d.nn) // 2
    for r0, r1 in zip(d.records, d.records[1:]):
        for gid, g1 in r1.grains.items():
            if g1.state == 2:  # a dump has no IDLocal of a vanished grain: the restatement's in its place
                g0 = r0.grains[gid]
                conv = {k: port.convolve(r0.grains[k].phi, d.dt, d.nn) for k in [gid, *g1.cmp]}
                members = [(k, r0.grains[k].box, conv[k]) for k in g1.cmp]
                g1.idlocal = port.compare(g0.box, conv[gid], members, g0.id_box, g0.idlocal, d.ngridpoints, b, d.h,
                                          d.delta)[1]
        _restate_step(d, r0, r1)


@pytest.mark.parametrize("isotropic", [1, 0])
def test_batched_lamellae(tmp_path, isotropic):
    d, lamellae = _dumped(tmp_path, gg.PRECISION_BATCHED, isotropic)
    _check_lifetimes(d, lamellae)


@pytest.mark.parametrize("isotropic", [1, 0])
def test_batched_runs_are_equal(tmp_path, isotropic):
    """The level set's two kernels run side by side: what they do must not
    depend on which one is ahead."""
    def once():
        seen = []
        _run(tmp_path, gg.PRECISION_BATCHED, isotropic, lambda h, k: seen.append(bytes(h.grain_stats())))
        return seen
    first = once()
    for _ in range(19):
        assert once() == first


@pytest.mark.parametrize("precision", FORMS)
def test_boxes_that_keep_their_size(tmp_path, precision):
    """DecoupleGrains: no box shrinks, so every grain above 83 cells vanishes in a large one."""
    d, lamellae = _dumped(tmp_path, precision, 1, DecoupleGrains=1)
    _check_lifetimes(d, lamellae)


@pytest.mark.parametrize("precision", FORMS)
def test_through_grid_coarsening(tmp_path, precision):
    """The coarser grid's contours come from the same kernels: a grain that
    vanishes there, or had vanished before, is deleted by the next level set,
    once (its state is then 0 without a 2 in between)."""
    dims = []
    path = os.path.join(str(tmp_path), "run.dump")

    def read(h, k):
        dims.append(h.dims().ngridpoints)
        h.dump(path, k, append=k > 0)

    _run(tmp_path, precision, 0, read, GridCoarsement=1, GridCoarsementGradient=0.95)
    assert dims[-1] < dims[0]
    d = dumpfile.read(path)
    for gid in d.records[0].grains:
        states = [r.grains[gid].state for r in d.records]
        assert states == sorted(states, key=(1, 2, 0).index) and states.count(2) <= 1, gid
