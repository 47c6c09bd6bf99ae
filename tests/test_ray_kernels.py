"""Rays and Frechet rows do not depend on how many rays a call traces: few rays
share a warp (two or eight of them), many run one a thread.  The same receivers
in calls of every kind give the same end points, columns and values, bit for
bit, on velocity nodes coarser than the grid (few crossings) and finer (a
crossing or more in every step)."""
import numpy as np
import pytest


def _rows(out, nev, nrc, take):
    """(end point, columns, values) of receivers 0..take-1 of every event."""
    row_ptr, cols, vals, ends = out
    got = []
    for e in range(nev):
        for i in range(take):
            q = e * nrc + i
            s = slice(row_ptr[q], row_ptr[q + 1])
            got.append((ends[q].tobytes(), cols[s].tobytes(), vals[s].tobytes()))
    return got


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("nv", [(7, 8, 8), (40, 44, 44)])
def test_rays_bitwise_for_any_count(gpu_lib, prec, nv):
    import fm3dt
    from fm3dt import synth
    h = synth.section_header(24, 20, 22, *nv)
    velv = synth.velocity_model(h, "gauss", 11)
    nev = 7
    params = np.array([synth.planewave_params(h, 35.0 + 8 * k, 20.0 + 51 * k) for k in range(nev)])
    el, lat, lon = synth.receivers(h, 3700, 5)
    rcx, rcz = fm3dt.latlon_to_rad(lat, lon)
    with fm3dt.Solver(h, precision=prec, max_events=nev) as s:
        s.set_velocity(velv)
        s.solve_planewave(params)
        # 7 (an odd last warp), 287, 1799 / 1806 and 5999 / 6006 (either side of a
        # rule's line), 12,600 and 25,900 rays
        calls = [1, 41, 257, 258, 857, 858, 1800, 3700]
        ref = None
        for nrc in calls:
            cap = nev * nrc * 700 + 1024
            got = s.rays_frechet(el[:nrc], rcx[:nrc], rcz[:nrc], cap=cap)
            rows = _rows(got, nev, nrc, min(nrc, 41))
            if nrc == 1:
                first = rows
                continue
            if ref is None:
                ref = rows
                assert [r for k, r in enumerate(ref) if k % 41 == 0] == first
                assert any(len(r[1]) for r in ref)
            assert rows == ref, f"{nev * nrc} rays"
