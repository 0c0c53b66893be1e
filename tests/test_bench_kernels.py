"""The kernels that a benchmark record names are those that the timed passes ran."""
import bench


def test_a_direction_of_whole_steps_names_no_sweeps():
    sweeps = {"k_fwd_v<born>": 1.0, "k_fwd_s<born>": 2.0, "k_bwd_s": 3.0, "k_bwd_v": 4.0}
    f = bench.step_kernels
    assert f(sweeps, ("sweeps", "sweeps"), True, None, 5.0, 6.0) == sweeps
    assert f(sweeps, ("march", "sweeps"), True, None, 5.0, 6.0) == {"k_bwd_s": 3.0, "k_bwd_v": 4.0,
                                                                    "k_march_fwd<born>": 5.0}
    assert f(sweeps, ("sweeps", "march"), True, None, 5.0, 6.0) == {"k_fwd_v<born>": 1.0, "k_fwd_s<born>": 2.0,
                                                                    "k_march_bwd": 6.0}
    assert f(sweeps, ("burst", "burst"), False, "f16", 5.0, 6.0) == {"k_burst_fwd": 5.0, "k_burst_bwd<f16>": 6.0}
    for k in f(sweeps, ("march", "march"), True, "f32", 5.0, 6.0):
        assert k in bench.KERNEL_BYTES
