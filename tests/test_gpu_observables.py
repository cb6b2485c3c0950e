"""GPU tests of the coordination-number and VTK observables: the device cell-grid count
against the reference's fixtures (exact ties included) and against the oracle's all-pairs count
on larger states, in both forms; the engine's VTK files against the reference's."""
import glob
import os

import numpy as np
import pytest

from vedo_gb300 import scenes
from vedo_gb300.scene import Boundary, Scene

from test_observables import mask_granular, vtk_array

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FIXTURES = sorted(glob.glob(os.path.join(ROOT, "tests", "golden", "observables", "*.npz")))


def _name(p):
    return os.path.splitext(os.path.basename(p))[0]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("path", FIXTURES, ids=[_name(p) for p in FIXTURES])
def test_device_coordination_matches_reference(path, precision, engine_lib, port_lib, tmp_path):
    from oracle import PortWorld
    g = np.load(path)
    sc = Scene.from_ido(g["ido"].tobytes())
    e = engine_lib.GpuEngine(sc, precision=precision)
    below, touching, avg = e.coordination(g["box"])
    assert avg == float(g["average"])
    ref = vtk_array(g["coord_vtk"].tobytes().decode(), "CoordinateNumber")
    spheres = np.array([sc.models[m].shape == 1 for m in sc.model_index])
    np.testing.assert_array_equal(below[spheres].astype(float), ref)
    pb, pt, _ = PortWorld(sc).coordination(g["box"])
    np.testing.assert_array_equal(below, pb)
    np.testing.assert_array_equal(touching, pt)
    # the engine's files equal the reference's (granular temperatures aside)
    e.write_vtk(str(tmp_path / "c.vtu"), with_coordination=True)
    e.write_vtk(str(tmp_path / "w.vtu"))
    assert mask_granular((tmp_path / "c.vtu").read_text()) == mask_granular(g["coord_vtk"].tobytes().decode())
    assert mask_granular((tmp_path / "w.vtu").read_text()) == mask_granular(g["world_vtk"].tobytes().decode())
    e.close()


def _scene_at(sc, st):
    out = Scene(sc.sp, sc.models, sc.iact_models, sc.model_index, st["position"], st["velocity"],
                sc.orientation_x, sc.orientation_z, st["angular_velocity"])
    return out


@pytest.mark.parametrize("precision", [0, 1])
def test_device_coordination_equals_oracle_on_a_settling_box(precision, engine_lib, port_lib):
    """A 5,832-sphere box after 1,500 steps of colliding (hundreds of overlapping pairs, walls
    present): the device counts equal the oracle's all-pairs counts on the same state, and so does
    a box average."""
    from oracle import PortWorld
    sc = scenes.lsd_box(n_side=18, spacing=2.02e-3, vel_sigma=0.3)
    e = engine_lib.GpuEngine(sc, up_iact=20, precision=precision)
    e.run(1500)
    st = e.state(("position", "velocity", "angular_velocity"))
    box = (-0.01, 0.01, -0.01, 0.01, 0.0, 0.02)
    below, touching, avg = e.coordination(box)
    pb, pt, pavg = PortWorld(_scene_at(sc, st)).coordination(box)
    np.testing.assert_array_equal(below, pb)
    np.testing.assert_array_equal(touching, pt)
    assert avg == pavg
    assert below.sum() > 500                                # hundreds of overlapping pairs
    e.close()


def test_device_coordination_of_a_dense_lattice(engine_lib, port_lib):
    """A 27,000-sphere FCC lattice whose neighbours overlap by a hair: 12 contacts per interior
    sphere, counted exactly (equal to the oracle), at the grid's largest cell occupancy."""
    from oracle import PortWorld
    sc = scenes.dense_pack(n=27000)
    e = engine_lib.GpuEngine(sc, precision=1)
    below, touching, _ = e.coordination()
    pb, pt, _ = PortWorld(sc).coordination((0, 0, 0, 0, 0, 0))
    np.testing.assert_array_equal(below, pb)
    np.testing.assert_array_equal(touching, pt)
    assert below.max() == 12
    e.close()


def test_coordination_needs_a_single_scene(engine_lib):
    b = engine_lib.BatchEngine([scenes.cluster(n=27, seed=1), scenes.cluster(n=27, seed=2)])
    with pytest.raises(engine_lib.EngineError) as ex:
        b.coordination()
    assert ex.value.code == 1
    b.close()


@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 1500])
@pytest.mark.parametrize("far", [0.0, 1.0, 1e4])
def test_device_coordination_where_each_of_its_tests_decides(n, far, engine_lib, port_lib):
    """Polydisperse touching spheres (exact ties among them), some pulled apart or together by one
    part in 1e6 to 1e12, with one sphere `far` metres away: the wider the scene, the fewer pairs the
    FP32 and the double-float test may decide.  Every count equals the oracle's."""
    from oracle import PortWorld
    rng = np.random.default_rng(n)
    sc = scenes.cluster(n=n, seed=n, polydisperse=True, walls="none")
    r = np.array([sc.models[m].attrs[0] for m in sc.model_index])
    x = np.zeros((n, 3))
    for i in range(1, n):                      # three touching chains side by side
        row, prev = i % 3, i - 3
        d = (r[i] + r[prev]) * (1.0 + rng.choice([0.0, 1e-12, -1e-12, 1e-9, -1e-9, 1e-6, -1e-6])) if prev >= 0 else 0.0
        x[i] = [(x[prev, 0] + d) if prev >= 0 else 0.0, 1.9e-3 * row, 1e-4 * row]
    if far and n > 2:
        x[n // 2, 2] += far
    sc.position[:] = x
    e = engine_lib.GpuEngine(sc)
    box = (x[:, 0].min(), x[:, 0].mean() + 1e-4, -1.0, 1.0, -1.0, 1.0)
    below, touching, avg = e.coordination(box)
    pb, pt, pavg = PortWorld(sc).coordination(box)
    np.testing.assert_array_equal(below, pb)
    np.testing.assert_array_equal(touching, pt)
    assert avg == pavg or (np.isnan(avg) and np.isnan(pavg))
    e.close()


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("away", [0.0, 1e3, 1e4])
def test_contact_activity_far_from_the_origin(away, periodic, engine_lib):
    """4,096 sphere pairs whose surfaces are 1e-12 to 2e-8 of the radius sum apart or into each other, in
    a scene `away` metres from the origin (to 5e6 radius sums), some of them across a periodic face: the
    contact activity and the contact count of both forms are the reference's FP64 decision,
    (r + r) - |x_b - x_a| > 0."""
    rng = np.random.default_rng(11)
    n, r = 8192, 1e-3
    sc = scenes.cluster(n=n, seed=3, walls="none", radius=r)
    a = np.stack(np.meshgrid(*(np.arange(16),) * 3, indexing="ij"), -1).reshape(-1, 3) * 6e-3
    u = rng.normal(size=a.shape)
    u /= np.linalg.norm(u, axis=1)[:, None]
    gap = rng.choice([-1.0, 1.0], size=len(a)) * 10.0 ** rng.uniform(-12.0, np.log10(2e-8), size=len(a))
    b = a + (2.0 * r * (1.0 + gap))[:, None] * u
    at = away * np.array([1.0, -0.7, 0.4])
    side = 16 * 6e-3
    if periodic:                               # the faces go through the pairs of one lattice plane
        sc.sp.pbc = Boundary(switch=(True, True, True), lower=tuple(at - 1e-4), upper=tuple(at - 1e-4 + side))
    x = np.stack([a + at, b + at], 1).reshape(n, 3)
    if periodic:
        lo, hi = np.array(sc.sp.pbc.lower), np.array(sc.sp.pbc.upper)
        x = np.where(x < lo, x + (hi - lo), x)
        x = np.where(x >= hi, x - (hi - lo), x)
    sc.position[:] = x
    sc.velocity[:] = 0.0
    d = x[1::2] - x[0::2]                      # the higher index is the master
    if periodic:
        L = hi - lo
        d = np.where(d >= 0.5 * L, d - L, d)
        d = np.where(d < -0.5 * L, d + L, d)
    truth = (r + r) - np.sqrt(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]) > 0.0
    assert 1000 < truth.sum() < 3000
    for kw in ({"consultant": "leap"} if periodic else {}, {"precision": 1}):
        e = engine_lib.GpuEngine(sc, **kw)
        it = e.interactions()
        first, on = it["first"].astype(int), it["active"] == 1
        pair = (it["second"] == first + 1) & (first % 2 == 0)
        wrong = on != (pair & truth[first // 2])
        assert not wrong.any(), (kw, int(wrong.sum()))
        if "precision" in kw or not periodic:  # (the reference's Leap list is not complete across the faces)
            assert len(set(first[pair].tolist())) == len(truth)
            assert e.observables()[9] == truth.sum()
        e.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [1, 255, 257, 8192, 8193, 155649])
def test_observables_at_the_reductions_sizes(n, precision, engine_lib, port_lib):
    """One partial sum, 2, 32, 33 and as many as there are blocks at most, a thread
    over one object and more: the energies, extreme speeds and dispersions against the oracle's serial
    sums, to their rounding (n half-ulps)."""
    from oracle import PortWorld
    sc = scenes.cluster(n=n, seed=n, walls="none", polydisperse=True)
    e = engine_lib.GpuEngine(sc, precision=precision)
    np.testing.assert_allclose(e.observables()[:9], PortWorld(sc).energy(), rtol=1e-13 + 1.2e-16 * n, atol=1e-40)
    e.close()
