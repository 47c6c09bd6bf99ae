"""Rounds in the order of time give the field of the rounds as they come (which a
caller's round cap asks for), bit for bit.

GPU: point sources (ordered from the first round), near a face and inside, with
and without the refined source grid, for every tile shape, on odd grids and on
one whose layers are far closer than its columns; boundary frames in double
precision along an axis of a checkerboard whose re-sweeps leave many tiles."""
import numpy as np
import pytest

from test_point import _src


def _header(c, nn, depth=1.0):
    from fm3dt import synth
    step = tuple(d * (m - 1) / (n - 1) for d, m, n in zip(c.nstep, c.nn, nn))
    return synth.Header(c.nv, c.vorig, c.vstep, nn, c.norig, (step[0] * depth,) + step[1:], c.earth)


@pytest.mark.gpu
@pytest.mark.parametrize("nn,refine,depth", [((33, 29, 37), 0, 1.0), ((33, 29, 37), 3, 1.0), ((64, 33, 65), 0, 0.1)])
def test_point_order(gpu_lib, orc, nn, refine, depth):
    import fm3dt
    from fm3dt import synth
    w = synth.config(1, scale=24, nev=1)
    h = _header(w.header, nn, depth)
    src = np.stack([_src(orc, h, 0, 9.4, 10.6, 6.0 * depth), _src(orc, h, 0, 21.3, 3.2, 90.0 * depth)])
    # (with layers that close, single precision ends in a cycle of last bits
    # whatever the order of the rounds)
    for prec in (fm3dt.FP64, fm3dt.FP32_OFFSET) if depth == 1.0 else (fm3dt.FP64,):
        want = None
        for shape in range(6):
            for cap in (0, 1000000):
                with fm3dt.Solver(h, fom=1, max_events=2, precision=prec) as s:
                    s.set_tuning(shape, max_rounds=cap)
                    s.set_velocity(w.velv)
                    s.solve_point(src, refine, 3)
                    got = np.stack([s.get_times(e) for e in range(2)])
                want = got if want is None else want
                assert np.all(np.isfinite(got))
                assert np.array_equal(want, got), (shape, cap, prec)


@pytest.mark.gpu
@pytest.mark.parametrize("nev", [12, 40])
def test_frames_order(gpu_lib, orc, nev):
    """Double precision, every event near an axis or most of them off the axes."""
    import fm3dt
    from fm3dt import synth
    w = synth.config(1, scale=24, nev=1)
    h = _header(w.header, (64, 65, 67))
    g = orc.grid_from_header(h.nv, h.vorig, h.vstep, h.nn, h.norig, h.nstep, h.earth)
    i = (np.indices((h.nv[2] + 2, h.nv[1] + 2, h.nv[0] + 2)) // 3).sum(0) % 2
    velv = w.velv * np.where(i, 1.05, 0.95).reshape(-1)
    baz = [90.0 * (e % 4) + (6.0 + 0.3 * e if e < 12 else 20.0 + 1.7 * (e - 12)) for e in range(nev)]
    frames = np.stack([orc.planewave_frame(g, orc.planewave_params(g, 40.0 + e, b)).reshape(h.nn[1:])
                       for e, b in enumerate(baz)])
    got, rounds = [], []
    for cap in (0, 1000000):
        with fm3dt.Solver(h, fom=1, max_events=nev, precision=fm3dt.FP64) as s:
            s.set_tuning(0, max_rounds=cap)
            s.set_schedule(tie_sweeps=0)
            s.set_velocity(velv)
            s.solve(frames)
            got.append(np.stack([s.get_times(e) for e in range(nev)]))
            rounds.append(len(s.round_trace()[0]))
    # (rounds in the order of time are more, and smaller)
    assert rounds[0] > rounds[1]
    assert np.array_equal(*got)
