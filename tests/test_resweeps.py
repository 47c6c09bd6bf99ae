"""A number of re-sweeps that the caller sets is kept to in double precision
too: as many as with a round cap (which leaves the rounds as they come), and
the default's choice where none is set.  GPU: boundary frames along an axis of
a checkerboard, which stay above the threshold for several re-sweeps; the same
field, bit for bit."""
import numpy as np
import pytest


@pytest.mark.gpu
def test_resweeps_are_the_callers(gpu_lib, orc):
    import fm3dt
    from fm3dt import synth
    from test_ordered_rounds import _header
    w = synth.config(1, scale=24, nev=1)
    h = _header(w.header, (64, 65, 67))
    g = orc.grid_from_header(h.nv, h.vorig, h.vstep, h.nn, h.norig, h.nstep, h.earth)
    i = (np.indices((h.nv[2] + 2, h.nv[1] + 2, h.nv[0] + 2)) // 3).sum(0) % 2
    velv = w.velv * np.where(i, 1.05, 0.95).reshape(-1)
    nev = 12
    frames = np.stack([orc.planewave_frame(g, orc.planewave_params(g, 40.0 + e, 90.0 * (e % 4) + 6.0 + 0.3 * e))
                       .reshape(h.nn[1:]) for e in range(nev)])
    sweeps, fields = {}, []
    for cap in (0, 1000000):
        for resweeps in (-1, 0, 1, 3, 5):
            with fm3dt.Solver(h, fom=1, max_events=nev, precision=fm3dt.FP64) as s:
                s.set_tuning(0, max_rounds=cap)
                s.set_schedule(tie_sweeps=0, resweeps=resweeps)
                s.set_velocity(velv)
                sweeps[cap, resweeps] = s.solve(frames)["sweep_launches"] - 1      # (the main sweep)
                fields.append(np.stack([s.get_times(e) for e in range(nev)]))
    assert sweeps[0, -1] == 2 and sweeps[1000000, -1] > 2
    for resweeps in (0, 1, 3, 5):
        assert sweeps[0, resweeps] == sweeps[1000000, resweeps]
    assert sweeps[0, 1] == 1 and sweeps[0, 3] == 3
    assert all(np.array_equal(fields[0], f) for f in fields)
