"""The reverse steps of the Born adjoint (csrc/sfwi_adjoint.cu) at sizes where a
thread's column pair, a block's rows or the strips of damped cells end: odd
heights, windows of other than whole blocks, several shots, one time step.
<L m, d> = <m, L^T d> holds to the rounding of FP32 fields: each side is a sum of
nt steps of terms with relative errors of about 6e-8 that grow at most
linearly over the steps, so 60 steps stay below 1e-5."""
import numpy as np
import pytest

from tests.test_gpu_parity import _batch_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz,pml,nshots,nt", [
    (33, 25, 8, 1, 60), (40, 32, 8, 2, 60), (63, 47, 11, 3, 60), (65, 30, 20, 2, 60), (150, 83, 11, 5, 60),
    (31, 25, 8, 1, 1), (31, 25, 8, 1, 2),
])
def test_reverse_steps_are_the_transpose(nx, nz, pml, nshots, nt):
    import sfwi_gb300 as sg
    cfg, model, shots = _batch_inputs(2, nshots=nshots, allnx=nx, allnz=nz, pml=pml, nt=max(nt, 30))
    sou = np.ascontiguousarray(model["sou"][:nt])
    sou[0] = 1.0  # the wave starts at once
    fd = sg.FD2DGPU_ELASTIC(sou, cfg["dx"], cfg["dx"], cfg["dt"], nx + 2 * pml, nz + 2 * pml, nx, nz, 1, pml, nt, 4,
                            shots[0]["ntr"], stage=2)
    fd.GPUbufferVPVS(model["vp"], model["vs"], None)
    rng = np.random.default_rng(7)
    dvp, dvs = (rng.standard_normal((nx, nz)).astype(np.float32) for _ in range(2))
    fd.GPUbufferM(dvp, dvs)

    def queue(rec):
        for k, d in enumerate(shots):
            z, x = rec[k] if rec else (None, None)
            fd.enqueue_shot(d["nx"], d["isx"], pml + 2, pml, d["ngx_left"], d["delta_left"], 0, d["gc"], z, x)

    queue(None)
    fd.run_forward()
    syn = [fd.read_records(k, d["ntr"]) for k, d in enumerate(shots)]
    data = [(rng.standard_normal((d["ntr"], nt)).astype(np.float32), rng.standard_normal((d["ntr"], nt)).astype(np.float32))
            for d in shots]
    left = [np.vdot(s["syn_z"].astype(np.float64), z) + np.vdot(s["syn_x"].astype(np.float64), x)
            for s, (z, x) in zip(syn, data)]
    size = sum(np.linalg.norm(s["syn_z"]) * np.linalg.norm(z) + np.linalg.norm(s["syn_x"]) * np.linalg.norm(x)
               for s, (z, x) in zip(syn, data))
    queue(data)
    ip, is_ = fd.born_adjoint()
    fd.close()
    right = np.vdot(dvp.astype(np.float64), ip) + np.vdot(dvs.astype(np.float64), is_)
    assert nt < 3 or size > 0
    assert abs(sum(left) - right) <= 1e-5 * size


@pytest.mark.parametrize("scale", [2.0 ** -60, 2.0 ** -40, 2.0 ** 40])
def test_reverse_steps_keep_any_units(scale):
    """source and records in other units (a power of two): the image scales by
    both.  Images are FP64 sums of FP32 fields, which a power of two scales without
    rounding while they are normal numbers (down to about 2^-126)."""
    import sfwi_gb300 as sg
    cfg, model, shots = _batch_inputs(2, nshots=2, allnx=64, allnz=30, pml=8, nt=120)
    pml, nx, nz, nt = cfg["pml"], cfg["allnx"], cfg["allnz"], cfg["nt"]
    rng = np.random.default_rng(3)
    data = [tuple(rng.standard_normal((d["ntr"], nt)).astype(np.float32) for _ in range(2)) for d in shots]
    out = []
    for f in (1.0, scale):
        fd = sg.FD2DGPU_ELASTIC((f * model["sou"]).astype(np.float32), cfg["dx"], cfg["dx"], cfg["dt"], nx + 2 * pml,
                                nz + 2 * pml, nx, nz, 1, pml, nt, 4, shots[0]["ntr"], stage=2)
        fd.GPUbufferVPVS(model["vp"], model["vs"], None)
        fd.GPUbufferM(model["dvp"], model["dvs"])
        for d, (z, x) in zip(shots, data):
            fd.enqueue_shot(d["nx"], d["isx"], pml + 2, pml, d["ngx_left"], d["delta_left"], 0, d["gc"],
                            np.float32(f) * z, np.float32(f) * x)
        out.append(np.concatenate(fd.born_adjoint()))
        fd.close()
    a, b = out[0], out[1] / scale ** 2
    assert np.abs(a).max() > 0 and np.linalg.norm(a - b) <= 1e-6 * np.linalg.norm(a)
