"""Sizes at which the engine's kernels change their split of the work.

* The contact kernels give a warp 1, 2, 4, ... 32 particles, by the particle
  count: both sides of each boundary, every step path, bit for bit against the
  oracle.
* The renderer works in tiles of 16 x 16 pixels and groups of 32 spheres: images
  and particle counts around their multiples, wide ones (the image plane has no
  height), tall ones (rows repeat), and an eye among the spheres, pixel for pixel
  against the renderer that tests every sphere.
* One launch per step, with re-sorts inside it, against the oracle.
* The Darcy iteration keeps one, two or four cells per thread in registers and
  leaves out those that cannot change: both sides of each of its limits, and of
  the largest grid it takes.
"""
import numpy
import pytest

from sphere_b200 import binfile, configs

import oracle as O
from test_gpu_dem_parity import compare

pytestmark = pytest.mark.gpu


def pressed(n, seed=61, model=2):
    """n spheres of a cubic lattice, in contact, under a loaded top wall."""
    side = max(3, int(numpy.ceil(n ** (1.0 / 3.0))))
    d = configs.settling_lattice(n=n, seed=seed, nx=side, ny=side, nz=side, spacing=0.0195, contactmodel=model)
    configs.add_top_wall(d, 20e3)
    d.w_x[0] -= 0.002
    d.gamma_n = 30.0
    d.gamma_t = 10.0
    return d


# a B200 holds 148 x 24 = 3552 warps of these kernels: one particle per warp up
# to 3552, two up to 7104, ... 16 up to 56832, then 32
@pytest.mark.parametrize("n,model", [(1, 2), (31, 1), (33, 2), (3552, 2), (3553, 1), (7104, 1), (7105, 2),
                                     (14208, 2), (14209, 2), (28416, 2), (28417, 1), (56832, 1), (56833, 2)])
def test_particles_per_warp(tmp_path, n, model):
    from sphere_b200.engine import Engine
    d = pressed(n, model=model)
    path = str(tmp_path / "edge.bin")
    binfile.write_bin(d, path)
    orc = O.Oracle(path)
    engines = {k: Engine(path, step_kernel=k) for k in ("stages", "stages_fused", "persistent")}
    for steps in (1, 4):
        assert orc.step(steps) == 0, orc.error()
        for k, e in engines.items():
            assert e.step(steps) == 0
            bad = compare(e, orc)
            assert not bad, (k, n, bad)
    for e in engines.values():
        e.close()


@pytest.mark.parametrize("n,w,h,scale", [(1, 16, 16, 1.0), (32, 17, 15, 1.0), (33, 1, 33, 1.0), (300, 40, 16, 1.0),
                                         (300, 15, 47, 1.0), (300, 48, 48, 12.0)])
def test_render_tiles(n, w, h, scale):
    import render_oracle as R
    from sphere_b200.engine import Engine
    d = configs.settling_lattice(n=n, seed=103, nx=7, ny=7, nz=7, spacing=0.0195)
    d.radius = d.radius * scale       # 12: spheres around the eye and behind it
    with Engine(d, precision="faithful") as e:
        x, vel = e.get("x"), e.get("vel")
        for method, max_val in ((0, 1.0), (2, 0.02)):
            img = e.render(method=method, max_val=max_val, width=w, height=h)
            val = R.method_values(method, x, vel, e.get("angvel"), e.get("xyzsum"), e.get("angpos"), e.get("p"))
            ref = R.render(x, vel, d.L, w, h, method=method, val=val, max_val=max_val)
            assert (ref[:, :, :3] != 255).any() or w < 16 or n == 1
            assert numpy.array_equal(img[:, :, :3], ref[:, :, :3]), (n, w, h, method)


# the one-launch step leaves one of its 888 blocks to the walls: 3548 warps for the
# particles; beyond 32 in each it takes three launches
@pytest.mark.parametrize("n,model", [(3548, 2), (3549, 1), (7096, 2), (7097, 2), (14192, 1), (14193, 2),
                                     (28384, 2), (28385, 1), (56768, 2), (56769, 2), (113536, 1), (113537, 2)])
def test_particles_per_warp_of_one_launch_steps(tmp_path, n, model):
    from sphere_b200.engine import Engine
    d = pressed(n, model=model)
    path = str(tmp_path / "edge.bin")
    binfile.write_bin(d, path)
    orc = O.Oracle(path)
    with Engine(path, step_kernel="stages_fused") as e:
        for steps in (1, 4):
            assert orc.step(steps) == 0, orc.error()
            assert e.step(steps) == 0
            bad = compare(e, orc)
            assert not bad, (n, bad)


# a tile stages spheres 256 at a time and traces them when more than 256 are
# there: every tile of these images meets hundreds to thousands
@pytest.mark.parametrize("n,scale", [(257, 12.0), (600, 12.0), (3000, 1.0), (3000, 5.0)])
def test_render_tiles_with_many_spheres(n, scale):
    import render_oracle as R
    from sphere_b200.engine import Engine
    d = configs.settling_lattice(n=n, seed=104, nx=15, ny=15, nz=15, spacing=0.0195)
    d.radius = d.radius * scale
    with Engine(d, precision="faithful") as e:
        x, vel = e.get("x"), e.get("vel")
        for w, h in ((16, 16), (33, 33)):
            val = R.method_values(2, x, vel, e.get("angvel"), e.get("xyzsum"), e.get("angpos"), e.get("p"))
            ref = R.render(x, vel, d.L, w, h, method=2, val=val, max_val=0.02)
            assert (ref[:, :, :3] != 255).any()
            for _ in range(5):
                img = e.render(method=2, max_val=0.02, width=w, height=h)
                assert numpy.array_equal(img[:, :, :3], ref[:, :, :3]), (n, w, h)


# a lid of cells that stay as they are, and none; one cell per thread of the
# solver's 148 x 256 threads, and four
@pytest.mark.parametrize("grid,lid", [((8, 8, 9), 2), ((33, 35, 32), 0), ((40, 40, 60), 3), ((40, 40, 80), 0)])
def test_darcy_cells_per_thread(tmp_path, grid, lid):
    from sphere_b200.engine import Engine
    from test_gpu_darcy import RTOL
    d = configs.settling_lattice(n=300, seed=51, nx=7, ny=7, nz=7, spacing=0.0195, steps=40)
    d.num = numpy.array(grid, dtype=numpy.uint32)
    d.L = numpy.array(grid) * 0.024
    configs.add_top_wall(d, 10e3)
    d.w_x[0] = (grid[2] - lid) * 0.024 + 0.001
    d.wmode[0] = 1
    # viscous enough for the porosity 0.9 of the empty cells
    configs.init_fluid_darcy(d, mu=2e-3, k_c=3.5e-13, tolerance=1e-7, maxiter=400, bottom_no_flow=True)
    path = str(tmp_path / "d.bin")
    binfile.write_bin(d, path)
    orc = O.Oracle(path, fluid=True)
    with Engine(path, fluid=True, precision="faithful") as e:
        for _ in range(3):
            assert e.step(1) >= 0
            assert orc.step(1) == 0, orc.error()
            assert int(e.get("darcy_iters")[0]) == int(orc.get("darcy_nijac_last")[0])
            for f in ("darcy_p", "darcy_v", "darcy_phi"):
                a, b = numpy.ravel(e.get(f)), numpy.ravel(orc.get(f))
                assert numpy.abs(a - b).max() <= RTOL * max(numpy.abs(b).max(), 1e-300), f


# layers of 1184 = 148 x 8 cells, the top one fixed: a block of the solver takes 256
# changing cells with one per thread, 512 with two, 1024 with four; beyond 148 x
# 1024 cells in all k_jacobi runs.  Pressures that differ in every cell
@pytest.mark.parametrize("nz,per_thread", [(33, 1), (34, 2), (65, 2), (66, 4), (128, 4), (129, None)])
def test_darcy_cells_per_thread_limits(tmp_path, nz, per_thread):
    import torch
    from sphere_b200.engine import Engine
    from test_gpu_darcy import RTOL
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if sms != 148:
        pytest.skip("the limits are those of 148 SMs")
    grid = (37, 32, nz)
    cells, active = 1184 * nz, 1184 * (nz - 1)
    chunk = (-(-active // sms) + 31) // 32 * 32
    assert per_thread == (None if cells > sms * 1024 else 1 if chunk <= 256 else 2 if chunk <= 512 else 4)
    d = configs.settling_lattice(n=300, seed=51, nx=7, ny=7, nz=7, spacing=0.0195, steps=40)
    d.num = numpy.array(grid, dtype=numpy.uint32)
    d.L = numpy.array(grid) * 0.024
    configs.init_fluid_darcy(d, mu=2e-3, k_c=3.5e-13, tolerance=1e-7, maxiter=45, bottom_no_flow=True)
    d.p_f[:, :, :-1] = numpy.random.default_rng(nz).uniform(1e3, 2e3, size=d.p_f[:, :, :-1].shape)
    path = str(tmp_path / "d.bin")
    binfile.write_bin(d, path)
    orc = O.Oracle(path, fluid=True)
    with Engine(path, fluid=True, precision="faithful") as e:
        for _ in range(2):
            assert e.step(1) >= 0
            assert orc.step(1) == 0, orc.error()
            assert int(e.get("darcy_iters")[0]) == int(orc.get("darcy_nijac_last")[0]) > 30
            for f in ("darcy_p", "darcy_v"):
                a, b = numpy.ravel(e.get(f)), numpy.ravel(orc.get(f))
                assert numpy.abs(a - b).max() <= RTOL * numpy.abs(b).max(), f


def crowded_cells():
    """Some 200 spheres in reach of each of 4 x 4 x 5 fluid cells."""
    d = configs.settling_lattice(n=1700, seed=52, nx=12, ny=12, nz=12, spacing=0.0195, steps=40)
    d.num = numpy.array([4, 4, 5], dtype=numpy.uint32)
    d.L = numpy.array([0.234, 0.234, 0.29])
    return d


# the porosity kernels queue the spheres of a cell and evaluate them 32 at a time:
# queues that run over several times.  Bound: about 220 additions of positive
# terms below the cell's volume, 1.1e-16 each, and the last bits of pow
def test_darcy_porosity_of_crowded_cells(tmp_path):
    from sphere_b200.engine import Engine
    d = crowded_cells()
    configs.init_fluid_darcy(d, mu=2e-3, k_c=3.5e-13, tolerance=1e-5, maxiter=50, bottom_no_flow=True)
    path = str(tmp_path / "d.bin")
    binfile.write_bin(d, path)
    orc = O.Oracle(path, fluid=True)
    with Engine(path, fluid=True, precision="faithful") as e:
        for _ in range(3):
            assert e.step(1) >= 0
            assert orc.step(1) == 0, orc.error()
            phi = numpy.ravel(orc.get("darcy_phi"))
            assert (phi < 0.6).sum() > 40
            assert numpy.abs(numpy.ravel(e.get("darcy_phi")) - phi).max() <= 1e-13


def test_ns_porosity_of_crowded_cells():
    from sphere_b200.engine import Engine
    d = crowded_cells()
    configs.init_fluid_ns(d, mu=8.9e-4, hydrostatic=True, tolerance=1e-6, maxiter=50)
    nx, ny, nz = (int(v) for v in d.num)
    cell = d.L / d.num
    R = cell.min()
    volume = 4.0 / 3.0 * 3.14159265358979 * R ** 3
    ref = numpy.empty((nz, ny, nx))
    for z in range(nz):
        for y in range(ny):
            for x in range(nx):
                X = numpy.array([x, y, z]) * cell + 0.5 * cell
                solid = 0.0
                for sx in (-1, 0, 1):
                    for sy in (-1, 0, 1):
                        dist = X - d.x + numpy.array([sx, sy, 0]) * d.L
                        r = d.radius
                        # vector lengths are single precision
                        l = numpy.sqrt((dist ** 2).sum(axis=1).astype(numpy.float32)).astype(numpy.float64)
                        part = (R - r < l) & (l < R + r)
                        lens = numpy.pi * (R + r - l) ** 2 * (l * l + 2 * l * r - 3 * r * r + 2 * l * R + 6 * r * R -
                                                              3 * R * R) / (12.0 * l)
                        solid += lens[part].sum() + (4.0 / 3.0 * numpy.pi * r ** 3)[l <= R - r].sum()
                ref[z, y, x] = min(1.0, max(0.0, (volume - solid) / volume))
    assert (ref < 0.6).sum() > 40
    with Engine(d, fluid=True, precision="faithful") as e:
        assert e.step(1) >= 0
        phi = numpy.ravel(e.get("darcy_phi"))
        # single-precision lengths: a last-bit difference of one of them shows
        assert numpy.abs(phi - numpy.ravel(ref)).max() <= 1e-7


# one launch per step: re-sorts inside it, the walls one launch behind, calls of
# one odd length replayed from a graph on either view
@pytest.mark.parametrize("n,model", [(400, 2), (5000, 1)])
def test_one_launch_steps_with_resorts(tmp_path, n, model):
    from sphere_b200.engine import Engine
    d = pressed(n, model=model)
    d.vel = numpy.random.default_rng(7).uniform(-20.0, 20.0, size=(n, 3))   # some sphere changes cell on most steps
    path = str(tmp_path / "resort.bin")
    binfile.write_bin(d, path)
    orc = O.Oracle(path)
    with Engine(path, step_kernel="stages_fused") as e:
        for steps in (3, 5, 5, 5, 5, 40):
            assert orc.step(steps) == 0, orc.error()
            assert e.step(steps) == 0
            bad = compare(e, orc)
            assert not bad, (steps, bad)
        assert e.info().resorts > 5


# graphs that cannot be instantiated: calls of an odd length step one by one from
# the buffer that holds the state
@pytest.mark.parametrize("kernel,steps", [("stages_fused", (3, 5, 5, 5, 5, 6, 6)), ("auto", (5, 5, 5, 5, 5, 150)),
                                          ("stages", (5, 5, 5))])
def test_steps_without_graphs(tmp_path, kernel, steps):
    from sphere_b200.engine import Engine
    d = pressed(400)
    path = str(tmp_path / "nograph.bin")
    binfile.write_bin(d, path)
    orc = O.Oracle(path)
    with Engine(path, step_kernel=kernel, inject_timeout="graph") as e:
        for n in steps:
            assert orc.step(n) == 0, orc.error()
            assert e.step(n) == 0
            bad = compare(e, orc)
            assert not bad, (n, bad)


# rows set by the caller that name a partner twice: the first of its slots is the
# one that takes this step's periodic shift, whatever slot it had before; with
# velocities so that particles change places in the sort meanwhile
@pytest.mark.parametrize("kernel", ["stages", "stages_fused", "persistent"])
def test_rows_with_a_partner_twice(tmp_path, kernel):
    from sphere_b200.engine import Engine
    d = pressed(400)
    d.vel = numpy.random.default_rng(7).uniform(-20.0, 20.0, size=(d.np, 3))
    path = str(tmp_path / "twice.bin")
    binfile.write_bin(d, path)
    orc = O.Oracle(path)
    with Engine(path, step_kernel=kernel) as e:
        assert orc.step(5) == 0 and e.step(5) == 0
        rows = e.get("contacts").reshape(d.np, -1)
        shift = e.get("distmod").reshape(d.np, -1, 4)
        assert (numpy.abs(shift[:, -1, :2]).sum(axis=1) > 0).sum() > 10
        rows[:, 0] = rows[:, -1]
        orc.set("contacts", rows)
        e.set("contacts", rows)
        before = e.info().resorts
        for steps in (1, 4, 25):
            assert orc.step(steps) == 0, orc.error()
            assert e.step(steps) == 0
            bad = compare(e, orc)
            assert not bad, (steps, bad)
        assert e.info().resorts > before + 3


def test_reported_step_path():
    from sphere_b200.engine import Engine
    d = pressed(400)
    shape = lambda i: (i.step_path, i.step_threads > 0, i.step_grid > 0, i.tuned)  # noqa: E731
    for kernel, path in (("stages", 0), ("persistent", 1), ("stages_fused", 2)):
        with Engine(d, step_kernel=kernel) as e:
            e.step(5)
            assert shape(e.info())[:3] == (path, path == 1, path == 1)
    with Engine(d) as e:
        e.step(5)                      # too short to tune on
        assert shape(e.info()) == (2, False, False, 0)
        e.step(400)
        path, threads, grid, tuned = shape(e.info())
        assert tuned == 1 and threads == grid == (path == 1)


# more neighbours than a list holds (48): the particle scans the cells instead
@pytest.mark.parametrize("model", [1, 2])
def test_full_neighbour_list(tmp_path, model):
    from sphere_b200.engine import Engine
    m, R, r = 60, 0.05, 0.01
    d = configs.settling_lattice(n=m + 1, seed=9, nx=4, ny=4, nz=4, contactmodel=model)
    k = numpy.arange(m) + 0.5
    phi, th = numpy.arccos(1.0 - 2.0 * k / m), numpy.pi * (1.0 + 5.0 ** 0.5) * k
    shell = numpy.column_stack([numpy.cos(th) * numpy.sin(phi), numpy.sin(th) * numpy.sin(phi), numpy.cos(phi)])
    d.x = 0.2 + numpy.vstack([numpy.zeros((1, 3)), (R + r - 1e-5) * shell])
    d.radius = numpy.concatenate([[R], numpy.full(m, r)])
    d.gamma_n = d.gamma_t = 20.0
    configs.grid_for(d, L=[0.4, 0.4, 0.4], dx=0.13)
    path = str(tmp_path / "full.bin")
    binfile.write_bin(d, path)
    orc = O.Oracle(path, nc=64)
    engines = {s: Engine(path, capacity=64, step_kernel=s) for s in ("stages", "stages_fused", "persistent")}
    for steps in (1, 6):
        assert orc.step(steps) == 0, orc.error()
        for s, e in engines.items():
            assert e.step(steps) == 0
            bad = compare(e, orc)
            assert not bad, (s, bad)
    if model == 2:
        assert (orc.get("contacts").reshape(m + 1, 64)[0] != m + 1).sum() > 48
    for e in engines.values():
        e.close()
