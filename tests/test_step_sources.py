"""Sources and receivers in the outermost four cells of a grid, where no cell
is updated: whole steps and the sweeps give the same bits.  Depths at which a
warp of the whole-step kernels begins with the first such column among them."""
import numpy as np
import pytest

from tests.test_gpu_parity import _batch_inputs
from tests.test_step_ways import engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stage,nx,nz,pml,nshots,way", [
    (2, 230, 30, 11, 1, "burst"),  # pairs, columns 48 .. 51 outside: a warp's first
    (1, 300, 46, 11, 1, "burst"),  # plain, second strip's columns 64 .. 67
    (1, 230, 41, 8, 1, "burst"),
    (2, 300, 94, 11, 6, "march"),  # pairs, columns 112 .. 115
    (1, 300, 78, 11, 7, "march"),  # plain, columns 96 .. 99
])
@pytest.mark.parametrize("kind", ["stress", "vz"])
def test_sources_and_receivers_outside_the_update_region(stage, nx, nz, pml, nshots, way, kind):
    import sfwi_gb300 as sg
    nt = 30
    _, model, shots = _batch_inputs(stage, nshots=nshots, allnx=nx, allnz=nz, pml=pml, nt=nt)
    model["sou"] = np.random.default_rng(1).standard_normal(nt).astype(np.float32)
    n, w = nz + 2 * pml, shots[0]["nx"] + 2 * pml
    for isx, isz, igz in ((w // 2, n - 4, n - 5), (w // 2, n - 2, n - 4), (w // 3, 1, 4), (2, n - 3, 3), (w - 2, n // 2, n - 1)):
        out = []
        for sweeps in (False, True):
            fd = engine(stage, nx, nz, pml, nt, model, sweeps)
            if kind == "vz":
                fd.set_source(sg.SOURCE_VZ_FORCE)
            for d in shots:
                fd.enqueue_shot(d["nx"], isx, isz, igz, d["ngx_left"], d["delta_left"], 0, d["gc"], d["obs_z"],
                                d["obs_x"])
            _, per = fd.run()
            assert sweeps or fd.debug_steps()[0] == way
            out.append([per] + list(fd.read_gradients_f64()) +
                       [v for k, d in enumerate(shots) for v in fd.read_records(k, d["ntr"]).values()])
            fd.close()
        assert all(np.array_equal(x, y) for x, y in zip(*out)), (isx, isz, igz)
