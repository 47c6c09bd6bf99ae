"""Height segments of the streaming sweep: any number asked for gives the
field of the rounds alone, bit for bit, also where the segments' common length
would leave the last of them empty (22 layers in 9 segments of 3 fill 8; in 16
segments of 2 fill 11)."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("segments", [1, 5, 9, 16, 21, 127])
def test_uneven_segments_bitwise(gpu_lib, prec, segments):
    import fm3dt
    from fm3dt import synth
    w = synth.config(1, scale=22, nev=6)
    # oblique events, and near ties (whose extra sweeps are one launch each)
    baz = [40.0, 140.0, 230.0, 94.5, 184.0, 355.0]
    params = np.array([synth.planewave_params(w.header, 40.0 + 7 * k, b) for k, b in enumerate(baz)])
    with fm3dt.Solver(w.header, precision=prec, max_events=6) as s:
        s.set_velocity(w.velv)
        s.set_tuning(0, 0, 0, 0)
        s.solve_planewave(params)
        ref = np.concatenate([s.get_times(e) for e in range(6)])
        s.set_tuning(0, 0, 0, 1)
        s.set_sweep_segments(segments, segments)
        assert s.solve_planewave(params)["converged"] == 1
        got = np.concatenate([s.get_times(e) for e in range(6)])
    assert np.array_equal(got, ref)
