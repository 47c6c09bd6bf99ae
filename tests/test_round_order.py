"""The field does not depend on the schedule: the rounds alone (whose passes
take a tile's changed nodes from a list, or a column a thread where they are
many), and the sweeps, certification and rounds together, for every tile shape,
on grids that are no multiple of any tile or column block, with boundary nodes
that have no time.

GPU, through the C ABI: double precision against the CPU oracle's fixed point to
1e-9 s (the bound of the other checks against it); in both precisions the same
field for all tile shapes and both schedules, bit for bit."""
import numpy as np
import pytest

# fewer layers and columns than a tile, a node more or less than one, several
GRIDS = [(9, 11, 34), (33, 17, 31), (35, 41, 65)]
BAZ = (45.0, 131.0, 204.0, 278.0, 352.0)         # two of them near an axis


@pytest.mark.gpu
@pytest.mark.parametrize("holes", [0.0, 0.03])
@pytest.mark.parametrize("nn", GRIDS)
def test_schedules(gpu_lib, orc, nn, holes):
    import fm3dt
    from fm3dt import synth
    w = synth.config(1, scale=24, nev=1)
    c = w.header
    step = tuple(d * (m - 1) / (n - 1) for d, m, n in zip(c.nstep, c.nn, nn))
    h = synth.Header(c.nv, c.vorig, c.vstep, nn, c.norig, step, c.earth)
    g = orc.grid_from_header(h.nv, h.vorig, h.vstep, h.nn, h.norig, h.nstep, h.earth)
    veln, _ = orc.gridder(g, w.velv)
    frames = np.stack([orc.planewave_frame(g, orc.planewave_params(g, 50.0, b)).reshape(nn[1:]) for b in BAZ])
    frames[np.random.default_rng(5).uniform(size=frames.shape) < holes] = 0.0
    for prec in (fm3dt.FP64, fm3dt.FP32_OFFSET):
        want = None
        for shape in range(6):
            for sweep in (0, 1):
                with fm3dt.Solver(h, fom=1, max_events=len(BAZ), precision=prec) as s:
                    s.set_tuning(shape, sweep=sweep)
                    s.set_velocity(w.velv)
                    s.solve(frames)
                    got = np.stack([s.get_times(e) for e in range(len(BAZ))])
                if want is None:
                    want = got
                    if prec == fm3dt.FP64:
                        for e, f in enumerate(frames):
                            ref, _ = orc.fixed_point(g, veln, f)
                            assert np.max(np.abs(got[e].ravel() - np.asarray(ref).ravel())) < 1e-9
                assert np.array_equal(want, got), (shape, sweep, prec)
