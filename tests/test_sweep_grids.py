"""The sweeps against the rounds alone, bit for bit, on grids with partial
column blocks and boundary nodes without a time.  GPU, both precisions and
column blocks:

* batches whose blocks outnumber the resident warps (the main sweep's form that
  passes values layer by layer), most events swept once, some near ties;
* heights about the sweeps' rings (16 and 32 rows) and the limits of the chunk
  masks (32 chunks of 4, then 8 layers), near ties and not."""
import numpy as np
import pytest


def _compare(nn, nev, prec, shape, holes, delta):
    import fm3dt
    from fm3dt import synth
    h = synth.section_header(*nn, 10, 9, 11)
    # (4.2 to 5.4 degrees off an axis near ties, the others 10 and more)
    baz = [90.0 * (e % 4) + (4.2 + 0.05 * (e % 24) if e % 6 == 0 else 10.0 + 70.0 * e / nev) for e in range(nev)]
    params = [synth.planewave_params(h, delta + 50.0 * e / nev, b) for e, b in enumerate(baz)]
    frames = synth.planewave_frames(h, params).reshape(nev, *nn[1:])
    frames[np.random.default_rng(7).uniform(size=frames.shape) < holes] = 0.0
    with fm3dt.Solver(h, precision=prec, max_events=nev) as s:
        s.set_velocity(synth.velocity_model(h, "checker", 3))
        s.set_sweep_shape(shape)
        got = []
        for sweep in (0, 1):
            s.set_tuning(0, sweep=sweep)
            assert s.solve(frames)["converged"] == 1
            got.append(np.stack([s.get_times(e) for e in range(nev)]))
    assert np.array_equal(*got)


@pytest.mark.gpu
@pytest.mark.parametrize("holes", [0.0, 0.03])
@pytest.mark.parametrize("shape", [6, 7])
@pytest.mark.parametrize("prec", [0, 1])
def test_large_batch(gpu_lib, prec, shape, holes):
    import torch
    nn, nev = (19, 22, 37), 320
    sx, sz = ((4, 8), (2, 16))[shape - 6]
    # (five of six events are swept once, at most 32 one-warp blocks a multiprocessor)
    blocks = -(-nn[1] // sx) * -(-nn[2] // sz) * (nev * 5 // 6)
    assert blocks > 32 * torch.cuda.get_device_properties(0).multi_processor_count
    _compare(nn, nev, prec, shape, holes, 32.0)


@pytest.mark.gpu
@pytest.mark.parametrize("nnr", [3, 15, 16, 17, 31, 32, 33, 127, 128, 129, 256, 257])
@pytest.mark.parametrize("prec", [0, 1])
def test_heights(gpu_lib, prec, nnr):
    for shape in (6, 7):
        _compare((nnr, 21, 35), 12, prec, shape, 0.0, 32.0)
