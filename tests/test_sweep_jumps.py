"""Extra sweeps that pass by quiet layers in the middle of a block and go on
above them (some hundred times in each of these solves): near-tie events on a
checkerboard, whose corrections die out here and there.  GPU, both precisions
and column blocks: the field of the rounds alone, bit for bit, however many
extra sweeps."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [6, 7])
@pytest.mark.parametrize("prec", [0, 1])
def test_jumps_bitwise(gpu_lib, prec, shape):
    import fm3dt
    from fm3dt import synth
    h = synth.section_header(128, 94, 75, 12, 14, 14)
    params = np.array([synth.planewave_params(h, 32.0 + 3 * k, 90.0 * (k % 4) + (-1) ** k * (4.0 + 0.3 * k))
                       for k in range(12)])
    n = len(params)
    with fm3dt.Solver(h, precision=prec, max_events=n) as s:
        s.set_velocity(synth.velocity_model(h, "checker", 3))
        s.set_tuning(0, 0, 0, 0)
        assert s.solve_planewave(params)["converged"] == 1
        ref = np.concatenate([s.get_times(e) for e in range(n)])
        s.set_tuning(0, 0, 0, 1)
        s.set_sweep_shape(shape)
        for sweeps in (2, 6):
            s.set_schedule(tie_sweeps=sweeps, tie_ratio=0.2)
            assert s.solve_planewave(params)["converged"] == 1
            run, skipped = s.tie_sweep_items()
            assert len(run) == sweeps and run[1] > 0 and skipped[1] > 0
            assert np.array_equal(np.concatenate([s.get_times(e) for e in range(n)]), ref)
