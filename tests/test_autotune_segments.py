"""The autotuner times no height segments on a solver that takes none (no GPU)."""
import pytest

from test_autotune import _Timed


class _Whole(_Timed):
    takes_sweep_segments = False

    def set_sweep_segments(self, seg, tie_seg):
        raise AssertionError("segments set on a solver that takes none")


def test_no_segments_are_timed_where_none_are_taken(gpu_lib):
    import fm3dt
    from fm3dt import autotune
    assert fm3dt.Solver.takes_sweep_segments is False
    s = _Whole(lambda ts: (3, 16), (2, 0.1), 0)
    *_, ms, sched, seg = autotune.autotune(s, 0, 64, repeats=1)
    assert seg == 0 and sched[0] == 2 and ms == pytest.approx(100.0)
    # 8 sweep shapes, 12 tile settings, 8 schedules, the tile settings again
    assert s.solves == 2 * (8 + 12 + 8 + 12)
