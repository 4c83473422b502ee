"""The forms that a step and the network choose by size against the general ones, at the edges of their ranges."""
import copy
import ctypes

import numpy as np
import pytest

import alebgk4paper_b200 as ab
from alebgk4paper_b200 import _abi

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("Nx,Nv", [(3, 4), (7, 5), (9, 8), (12, 10), (17, 6)])
def test_fp64_march_equals_gather(gpu, Nx, Nv):
    """Tiles and segments with remainders, an odd row length, a lattice smaller than a tile.  Both sum the same
    80 products in another order: eps64 times the stencil's sum of |c| (at most 5) times sqrt(80), each step."""
    c = ab.Case("cavity3d", Nx, Nv, -1.0, 2)
    a, b = ab.Solver(c, precision=64), ab.Solver(c, precision=64, transport=1)
    assert a.counters()["transport_kernel"] == 2 and b.counters()["transport_kernel"] == 1
    a.cudaStep(3), b.cudaStep(3)
    (ga, ma), (gb, mb) = a.cudaDownloadFull(), b.cudaDownloadFull()
    assert _rel(ga, gb) < 3 * 5 * 9 * 1.2e-16
    assert _rel(ma[:, 0], mb[:, 0]) < 3 * 5 * 9 * 1.2e-16


@pytest.mark.parametrize("Nx,Nv,marches", [(6, 8, True), (8, 10, False), (9, 12, False), (10, 12, False), (11, 12, True),
                                           (12, 10, True), (14, 8, True)])
def test_fp64_lattices_march_where_it_is_faster(gpu, Nx, Nv, marches):
    """Small lattices with long rows are gathered (bitwise the plain gather); FP32 ones march as they always did."""
    c = ab.Case("cavity3d", Nx, Nv, -1.0, 2)
    s, f = ab.Solver(c, precision=64), ab.Solver(c, precision=32)
    assert (s.counters()["transport_kernel"], f.counters()["transport_kernel"]) == (2 if marches else 1, 2)
    if not marches:
        p = ab.Solver(c, precision=64, transport=1)
        s.cudaStep(3), p.cudaStep(3)
        np.testing.assert_array_equal(s.cudaDownloadFull()[0], p.cudaDownloadFull()[0])
        p.close()
    s.close(), f.close()


def test_required_march_is_refused_in_fp64(gpu):
    """Transport 2 is the FP32 march: an FP64 context is refused by what it asks for, a cloud that is no lattice by what
    it is."""
    for name, precision, says in (("cavity3d", 64, "transport 0"), ("cavity3d-cube", 32, "complete 3-D lattice")):
        with pytest.raises(ab.AlebgkError, match=says):
            ab.Solver(ab.Case(name, 12, 4, -1.0, 2, fixed_body=True), precision=precision, transport=2)


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("name,Nx,Nv", [("cavity3d-cube", 12, 5), ("cavity3d-cube", 17, 6), ("cavity3d-sphere", 21, 4),
                                        ("cavity3d-cube", 24, 8)])
def test_gather_by_tiles_equals_plain_gather(gpu, name, Nx, Nv, precision):
    """Odd rows (one velocity a lane), partial chunks, lattices with partial tiles, wall layers in strips and
    remainders, bodies in the middle: every particle sums its slots in the same order, so the states are
    the same bits."""
    c = ab.Case(name, Nx, Nv, -1.0, 2, fixed_body=True)
    a, b = ab.Solver(c, precision=precision), ab.Solver(c, precision=precision, transport=1)
    a.set_gather_tiles(True)
    assert min(a.gather_counts()) > 0 and b.gather_counts() == (0, 0, c.N)
    a.cudaStep(3), b.cudaStep(3)
    (ga, ma), (gb, mb) = a.cudaDownloadFull(), b.cudaDownloadFull()
    np.testing.assert_array_equal(ga, gb)
    np.testing.assert_array_equal(ma, mb)


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("name,Nx,Nv,tiled", [("cavity3d-cube", 12, 6, False), ("cavity3d-cube", 8, 16, False),
                                              ("cavity3d-cube", 24, 6, True), ("cavity3d-sphere", 24, 4, True)])
def test_tiles_are_taken_where_they_pay(gpu, name, Nx, Nv, tiled, precision):
    """Not where one wave of the plain gather holds the cloud, or few particles are in tiles and strips.  Asked for
    between steps, the same bits."""
    c = ab.Case(name, Nx, Nv, -1.0, 2, fixed_body=True)
    s, p = ab.Solver(c, precision=precision), ab.Solver(c, precision=precision, transport=1)
    assert (s.gather_counts()[0] > 0) == tiled
    for always in (False, True, False):
        s.set_gather_tiles(always)
        assert (sum(s.gather_counts()[:2]) > 0) == (tiled or always)
        s.cudaStep(2), p.cudaStep(2)
    np.testing.assert_array_equal(s.cudaDownloadFull()[0], p.cudaDownloadFull()[0])
    s.close(), p.close()


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("cells", [2.75, 3.0, 5.0])
def test_gather_by_tiles_equals_plain_gather_at_a_large_step(gpu, cells, precision):
    """Steps of more cells than the support reaches (2.5): nodes whose foot point has no neighbour keep the particle's
    own value.  Bitwise, as at an ordinary step; the fastest node along an axis moves `cells` cells."""
    c = ab.Case("cavity3d-cube", 17, 6, -1.0, 2, fixed_body=True)
    c.dt = cells * c.params["dx"] / max(abs(c.params["vmin"]), c.params["vmin"] + (c.Nv - 1) * c.params["dv"])
    out = []
    for transport in (0, 1):
        cfg = c.config(precision, 0, transport)
        cfg.limiter = 0
        s = ab.Solver(c, config=cfg)
        s.set_gather_tiles(True)
        assert transport == 1 or s.gather_counts()[0] > 0
        s.cudaStep(1)
        out.append(s.cudaDownloadFull())
        s.close()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])


def test_gather_beyond_524280_particles(gpu):
    """The gather as its own kernel above 65 535 blocks of eight particles, against the march (the FP32 sums in
    another order: as far apart as test_lattice_march_matches_gather allows)."""
    c = ab.LatticeCase("cavity3d", 82, 4)
    assert c.N > 8 * 65535
    out = []
    for transport in (1, 2):
        cfg = c.config(32, 0, transport)
        cfg.limiter = 0
        s = ab.Solver(c, config=cfg)
        s.cudaStep(1)
        s.sync()
        out.append(s.cudaDownloadFull()[0])
        s.close()
    assert _rel(out[0], out[1]) < 1e-5


def _own_cloud(xyz, h, Nv, wall_first=False, box=(0, 0, 0), reach=2.5):
    """A case of these positions at spacing h: neighbours within reach h (over the box's edges where it has a length), the
    density varying from particle to particle.  With wall_first particle 0 is a wall particle.  Returns the box's
    lengths at the case's scale too."""
    from scipy.spatial import cKDTree
    c = copy.copy(ab.Case("cavity3d", 6, Nv, -1.0, 2))
    N = len(xyz)
    scale = c.params["radius"] / (2.5 * h)
    near = cKDTree(xyz, boxsize=box).query_ball_point(xyz, reach * h)
    c.N, c.xyz, c.meshv = N, np.ascontiguousarray(xyz * scale), np.zeros((N, 3))
    c.nnb, c.nbr = np.zeros(N, np.int32), np.zeros((N, _abi.MAX_NEIGH), np.int32)
    for i, js in enumerate(near):
        js = [j for j in js if j != i]
        c.nnb[i] = len(js)
        c.nbr[i, :len(js)] = js
    c.boundary, c.body_id = np.zeros(N, np.int32), np.full(N, -1, np.int32)
    c.wall = np.tile(c.wall[0], (N, 1))
    c.boundary[0] = int(wall_first)
    f = 1.0 + 0.01 * np.cos(np.arange(N))[:, None]
    c.g, c.macro = c.g[:1] * f, np.tile(c.macro[0], (N, 1))
    c.macro[:, 0] *= f[:, 0]
    return c, [scale * b for b in box]


def _assert_auto_equals_plain(c, precision, box=(0, 0, 0), tiles=True):
    out = []
    for transport, always in ((0, False), (0, True), (1, True)):
        cfg = c.config(precision, 0, transport)
        for a in range(3):
            cfg.periodic[a], cfg.L[a] = int(box[a] > 0), box[a]
        s = ab.Solver(c, config=cfg)
        assert s.counters()["transport_kernel"] == 1
        s.set_gather_tiles(always)
        n = s.gather_counts()
        assert 8 * n[0] + 4 * n[1] + n[2] == c.N
        assert not always or (n[0] > 0) == (tiles and transport == 0), n
        s.cudaStep(2)
        out.append(s.cudaDownloadFull())
        s.close()
    for g, m in out[1:]:
        np.testing.assert_array_equal(g, out[0][0])
        np.testing.assert_array_equal(m, out[0][1])


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("n", [13, 33])
def test_tiles_of_a_lattice_that_does_not_hold_the_first_particle(gpu, n, precision):
    """Cell centres and one wall point, half a cell off them in every axis: the particles' distances from it are k + 1/2
    cells to an ulp, to either side.  At n = 33 columns rounded from there give 4 437 tiles over the 18 792
    particles of 2 349.  Every particle is in one tile, one strip or neither."""
    ax = (np.arange(n) + 0.5) / n
    z, y, x = np.meshgrid(ax, ax, ax, indexing="ij")
    xyz = np.concatenate([np.zeros((1, 3)), np.column_stack([x.ravel(), y.ravel(), z.ravel()])])
    c, _ = _own_cloud(xyz, 1.0 / n, 4, True)
    _assert_auto_equals_plain(c, precision)


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("n,roll", [(13, 0), (13, 2), (14, 3)])
def test_tiles_of_a_periodic_lattice(gpu, n, roll, precision):
    """Stencils that reach over the box's edges, of one class with those that do not: no tile reaches over an edge, and
    with an odd number of rows none overlaps another.  Rolled, the class's first particle lies inside."""
    ax = np.roll((np.arange(n) + 0.5) / n, -roll)
    z, y, x = np.meshgrid(ax, ax, ax, indexing="ij")
    c, box = _own_cloud(np.column_stack([x.ravel(), y.ravel(), z.ravel()]), 1.0 / n, 4, box=(1, 1, 1))
    _assert_auto_equals_plain(c, precision, box, tiles=roll > 0)


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("shape", [(7, 6, 3), (3, 6, 7), (7, 3, 3)])
def test_lattice_of_three_periodic_planes_is_gathered(gpu, shape, precision):
    """In an axis of three periodic planes the neighbour over the edge is two planes back: particles of one class, whose
    offsets differ from member to member (lists of the 26 next neighbours, whose offsets all lie in the march's
    template)."""
    axes = [(np.arange(k) + 0.5) / 10 for k in shape]
    z, y, x = np.meshgrid(axes[2], axes[1], axes[0], indexing="ij")
    c, box = _own_cloud(np.column_stack([x.ravel(), y.ravel(), z.ravel()]), 0.1, 4,
                        box=[0.3 if k == 3 else 0 for k in shape], reach=1.8)
    _assert_auto_equals_plain(c, precision, box, tiles=False)


@pytest.mark.parametrize("precision", [32, 64])
def test_lattice_with_a_neighbour_listed_twice_is_gathered(gpu, precision):
    """Both entries count, as in any other cloud."""
    c = ab.Case("cavity3d", 9, 4, -1.0, 2)
    i = int(np.nonzero(c.boundary == 0)[0][100])
    c.nbr[i, c.nnb[i]] = c.nbr[i, 7]
    c.nnb[i] += 1
    _assert_auto_equals_plain(c, precision)


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("Nx,Nv", [(6, 7), (6, 9), (7, 12), (5, 14), (5, 16), (4, 20), (4, 27)])
def test_row_groups_equal_general_particle_kernel(gpu, Nx, Nv, precision):
    """Groups of four, two and one rows, the last group of a kind partly filled, rows below and above one round of
    the block, rows with the FP64 collision.  FP32: three roundings a value and step in the collision."""
    c = ab.Case("cavity3d", Nx, Nv, -1.0, 2)
    c.g *= 1.0 + 0.01 * np.cos(np.arange(c.N))[:, None]
    c.macro[:, 0] = c.g.sum(1) * c.params["dv"] ** 3
    a = ab.Solver(c, precision=precision, transport=1)
    b = ab.Solver(c, precision=precision, transport=1, particle=1)
    # (registers hold Nv 12 and FP32's 14; shorter FP32 rows stream)
    form = 3 if Nv == 12 or (Nv, precision) == (14, 32) else (2 if (precision, Nv < 14) == (32, True) else 4)
    assert (a.counters()["particle_kernel"], b.counters()["particle_kernel"]) == (form, 1)
    a.cudaStep(2), b.cudaStep(2)
    (ga, ma), (gb, mb) = a.cudaDownloadFull(), b.cudaDownloadFull()
    tol = 1e-13 if precision == 64 else 2 * 5 * 3 * 6e-8
    assert _rel(ga, gb) < tol
    assert _rel(ma[:, 0], mb[:, 0]) < tol and _rel(ma[:, 4], mb[:, 4]) < tol
    ca, cb = a.counters(), b.counters()
    assert ca["transport_flags"] == cb["transport_flags"]
    assert ca["positivity_fixes"] == cb["positivity_fixes"]


@pytest.mark.parametrize("Nx,Nv,precision,form", [(6, 7, 64, 4), (6, 14, 64, 4), (5, 20, 64, 4), (6, 16, 32, 4),
                                                  (5, 28, 32, 4), (8, 6, 64, 3), (6, 12, 64, 3), (6, 12, 32, 3),
                                                  (6, 14, 32, 3), (8, 6, 64, 2)])
def test_row_forms_repair_negative_rows_like_the_oracle(gpu, Nx, Nv, precision, form):
    """Negative nodes planted so that many interior and wall rows come out mixed-sign, MOOD off so that the repaired rows
    are collided: groups of four, two and one rows (the moments of the kept part are a pass of their own), register
    rows, and the streamed form where it is asked for.  Tolerances of the other repair tests."""
    from oracle.oracle import Oracle
    c = ab.Case("cavity3d", Nx, Nv, -1.0, 2)
    inner, wall = np.nonzero(c.boundary == 0)[0], np.nonzero(c.boundary)[0]
    c.g[inner[::2], ::9] *= -2
    c.g[wall[::7], ::4] *= -0.3
    cfg = c.config(precision, 0, 1, 2 if form == 2 else 0)
    cfg.limiter = 0
    s = ab.Solver(c, config=cfg)
    assert s.counters()["particle_kernel"] == form
    # (in FP32 a node of the tail may round below zero: the general kernel repairs the same rows)
    cfg.particle = 1
    k = ab.Solver(c, config=cfg)
    o = Oracle.from_case(c, limiter=0)
    s.cudaStep(1), k.cudaStep(1)
    want = o.step(1)["positivity_fixes"]
    assert s.counters()["positivity_fixes"] == k.counters()["positivity_fixes"] > len(inner) // 2
    assert precision == 32 or k.counters()["positivity_fixes"] == want
    g, m = s.cudaDownloadFull()
    tg, tm = (1e-10, 1e-10) if precision == 64 else (3e-4, 5e-5)
    assert np.abs(g - o.g).max() <= tg * np.abs(o.g).max()
    for q in (0, 4):
        assert np.abs(m[:, q] - o.macro[:, q]).max() <= tm * np.abs(o.macro[:, q]).max(), q
    s.close()


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("name,Nx,Nv", [("cavity2d", 9, 6), ("cavity2d", 64, 6), ("cavity2d", 65, 6),
                                        ("cavity3d", 16, 4), ("cavity3d", 17, 4), ("cavity3d", 27, 4)])
def test_merged_end_of_step_equals_separate_launches(gpu, name, Nx, Nv, precision):
    """Clouds of a few blocks and of many: bitwise the chain of single kernels (timed steps).  (What the merged kernels
    do when they have rows to finish is in the two tests below.)"""
    c = ab.Case(name, Nx, Nv, -1.0, 2)
    a, b = ab.Solver(c, precision=precision), ab.Solver(c, precision=precision)
    if name == "cavity2d":
        a.set_launch(256, 0), b.set_launch(256, 0)
    a.cudaStep(4)
    ms = (ctypes.c_float * _abi.NSTAGES)()
    ab._check(b.lib.alebgk_profile_steps(b.ctx, 4, ms), b.ctx)
    (ga, ma), (gb, mb) = a.cudaDownloadFull(), b.cudaDownloadFull()
    np.testing.assert_array_equal(ga, gb)
    np.testing.assert_array_equal(ma, mb)
    ca, cb = a.counters(), b.counters()
    for k in ("mass_before", "mass_after_transport", "mass_scale", "mass_end", "transport_flags"):
        assert ca[k] == cb[k], k


def _merged_and_separate_steps(c, precision, limiter, steps):
    """The state and counters after steps of the merged chain; bitwise those of the single kernels."""
    cfg = c.config(precision)
    cfg.limiter = limiter
    a, b = ab.Solver(c, config=cfg), ab.Solver(c, config=cfg)
    if c.dim == 2:
        a.set_launch(256, 0), b.set_launch(256, 0)
    a.cudaStep(steps)
    ms = (ctypes.c_float * _abi.NSTAGES)()
    ab._check(b.lib.alebgk_profile_steps(b.ctx, steps, ms), b.ctx)
    (ga, ma), (gb, mb), ca = a.cudaDownloadFull(), b.cudaDownloadFull(), a.counters()
    np.testing.assert_array_equal(ga, gb)
    np.testing.assert_array_equal(ma, mb)
    assert ca == b.counters()
    a.close(), b.close()
    return ga, ma, ca


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("limiter", [0, 2])
@pytest.mark.parametrize("name,Nx,Nv,radius", [("cavity2d", 16, 8, 1.5), ("cavity2d", 16, 8, 99.0),
                                               ("cavity3d", 12, 6, 2.1), ("cavity3d", 12, 6, 5.0)])
def test_merged_end_of_step_finishes_rows_without_mass(gpu, name, Nx, Nv, radius, limiter, precision):
    """A ball of empty rows, of which a few or many come out of the first transport without positive mass: finished like
    by the single kernels, and like by the oracle."""
    from oracle.oracle import Oracle
    from test_mls_tables import _tables
    c = ab.Case(name, Nx, Nv, -1.0, 2)
    inner = np.nonzero(c.boundary == 0)[0]
    c.g[np.linalg.norm(c.xyz - c.xyz[inner[len(inner) // 2]], axis=1) < radius * c.params["dx"]] = 0
    cls, nslot, slots, coef, V = _tables(c)
    empty = sum(not (coef[cls[i], :nslot[i]] * c.g[slots[i, :nslot[i]], :V]).sum() > 0 for i in inner)
    assert 1 <= empty <= 8 if radius < 3 else empty > 8
    g, m, _ = _merged_and_separate_steps(c, precision, limiter, 1)
    if precision == 64:
        o = Oracle.from_case(c, limiter=limiter)
        o.step(1)
        assert np.abs(g - o.g).max() <= 1e-10 * np.abs(o.g).max()
        assert np.abs(m[:, 0] - o.macro[:, 0]).max() <= 1e-10 * np.abs(o.macro[:, 0]).max()
    _merged_and_separate_steps(c, precision, limiter, 3)


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("name,Nx,Nv", [("cavity2d", 12, 8), ("cavity2d", 65, 6), ("cavity3d", 12, 6),
                                        ("cavity3d", 27, 4)])
def test_merged_end_of_step_after_a_failed_moodcheck(gpu, name, Nx, Nv, precision):
    """The second collision and the end mass by its last block: like the single kernels."""
    c = ab.Case(name, Nx, Nv, -1.0, 2)
    i = int(np.nonzero(c.boundary == 0)[0][20])
    c.g[i] = -50.0 * np.abs(c.g[i])
    assert _merged_and_separate_steps(c, precision, 2, 1)[2]["mood_fail"] == 1
    _merged_and_separate_steps(c, precision, 2, 3)


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("Nx,Nv", [(5, 6), (12, 15), (34, 6), (35, 6), (42, 8), (43, 8), (20, 28)])
def test_small_2d_form_equals_plain_form(gpu, Nx, Nv, precision):
    """Up to eight (FP64) and twelve (FP32) particles an SM and above: bitwise the plain fused form."""
    c = ab.Case("cavity2d", Nx, Nv, -1.0, 2)
    a, b = ab.Solver(c, precision=precision), ab.Solver(c, precision=precision)
    b.set_launch(0, 8)
    a.cudaStep(4), b.cudaStep(4)
    (ga, ma), (gb, mb) = a.cudaDownloadFull(), b.cudaDownloadFull()
    np.testing.assert_array_equal(ga, gb)
    np.testing.assert_array_equal(ma, mb)
    assert a.counters() == b.counters()


def test_forward_rows_do_not_depend_on_the_call(gpu):
    """One to three tiles in flight a block, full and ragged last tiles: a point's outputs are the same bits."""
    from alebgk4paper_b200 import warmstart as ws
    rng = np.random.default_rng(3)
    net = ws.WarmStartNet(ws.init_params(1))
    q = rng.uniform(0, 1, (3 * 148 * 128 + 300, 4)).astype(np.float32)
    full = net.forward(q).cpu().numpy()
    assert np.isfinite(full).all()
    for n in (1, 127, 128, 129, 148 * 128, 148 * 128 + 1, 2 * 148 * 128 + 77, len(q) - 1):
        np.testing.assert_array_equal(net.forward(q[:n]).cpu().numpy(), full[:n])
    net.close()
