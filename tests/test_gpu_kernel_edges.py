"""Sizes at which the engine's kernels change their split of the work.

* The contact kernels give a warp 1, 2, 4, ... 32 particles, by the particle
  count: both sides of each boundary, every step path, bit for bit against the
  oracle.
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
@pytest.mark.parametrize("n,model", [(1, 2), (31, 1), (33, 2), (3552, 2), (3553, 1), (7105, 2), (14209, 2),
                                     (28417, 1), (56833, 2)])
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
