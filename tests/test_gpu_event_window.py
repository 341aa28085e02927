"""The event loop's resident window against the full per-event scan
(event_scan=1), which evaluates every frontier row at every event: identical
states (NaN extents included), grains and event counts."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
DECKS = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "decks")

# one voxel of beam travel and several hundred captures per step: more frontier
# rows than a window holds, windows opened again within a step, rows of captures
# two and more generations deep, negative-time events
WIDE = """dx 2.5e-6
nX %d %d %d
bmV 1.0
bmP 200.0
bmDelT 2.5e-6
r 2e-3
lT 30e-6
bpH 12.5e-6
tL 1609
tS 1531.5
meltparam 10e-6 %g %g 20e-6
bhatch 40e-6
mu 4e-4
lrate 4e-4
patternID 2
outint 1000000
offset 0.0 0.0 0.0
gridsize 1.2e-4 1.0e-4
gridtheta %g
dendritegrowth2 %g 2.0
%s
"""


def _run(deck, steps, **kw):
    from amcafe_gb300 import Simulation

    with Simulation(deck, **kw) as sim:
        sim.InitializeVoxels()
        sim.begin()
        sim.run(steps)
        st = sim.state()
        st["ctheta"] = sim.ctheta()
        s = sim.stats()
    return st, s


def _same(deck, steps):
    a, sa = _run(deck, steps)
    b, sb = _run(deck, steps, event_scan=1)
    for k in a:
        assert np.array_equal(a[k], b[k], equal_nan=a[k].dtype.kind == "f"), k
    for k in ("events", "nucleations", "negative_dt", "max_rows", "sum_rows"):
        assert sa[k] == sb[k], k
    return sa


@pytest.mark.parametrize("deck,steps", [("layers_rot.in", 90), ("odd_dims.in", 12), ("track_easm60.in", 0),
                                        ("track_ros.in", 0)])
def test_window_equals_full_scan(deck, steps):
    _same(os.path.join(DECKS, deck), steps)


@pytest.mark.parametrize("nx,ny,nz,rear,half,turn,growth,extra,steps", [
    (48, 40, 17, 40e-6, 40e-6, 0.0, 1e-5, "", 40),
    (47, 41, 19, 40e-6, 40e-6, 0.6, 1e-4, "", 24),   # six voxels of growth a step: captures many generations deep
    (45, 33, 18, 30e-6, 30e-6, 0.0, 1e-5, "rosenthal 0.35 20.0 5e-6", 60),
])
def test_wide_fronts(tmp_path, nx, ny, nz, rear, half, turn, growth, extra, steps):
    path = tmp_path / "wide.in"
    path.write_text(WIDE % (nx, ny, nz, rear, half, turn, growth, extra))
    s = _same(str(path), steps)
    assert s["events"] > 0


# a track's developed front: over a thousand rows, most of them outside the window
FRONT = """dx 2.5e-6
nX 256 128 64
bmV 1.0
bmP 200.0
bmDelT %g
r 2e-4
lT %g
bpH %g
tL 1609
tS 1531.5
meltparam 16.31e-6 425.5e-6 55.11e-6 55.11e-6
bhatch 100e-6
mu 1.25e-4
lrate 1.25e-4
patternID 2
outint 1000000
offset 0.0 0.0 0.0
gridsize 6.4e-4 3.2e-4
gridtheta 0.0
dendritegrowth2 1e-5 2.0
%s
"""


def _uploaded(path, spin, steps, extent=None):
    """`steps` steps from a developed state whose mushy cells are in part overdue (and half
    of them set to `extent`), by the window and by the full scan: same results. Returns the
    window's counts over these steps."""
    from amcafe_gb300 import Simulation

    out = []
    for scan in (0, 1):
        with Simulation(str(path), event_scan=scan) as sim:
            sim.InitializeVoxels()
            sim.begin()
            sim.run(spin)
            st, cth, s0 = sim.state(), sim.ctheta(), dict(sim.stats(), **sim.event_paths())
            m = np.flatnonzero(st["vState"] == 2)
            u = np.random.default_rng(3).random(m.size)
            if extent is not None:
                st["extents"][m[u < 0.5]] = extent
            st["extents"][m[u > 0.97]] += 3e-6
            sim.upload_state(st["gID"], st["vState"], st["extents"], st["centroid"], cth)
            sim.run(steps)
            s1 = dict(sim.stats(), **sim.event_paths())
            out.append((dict(sim.state(), ctheta=sim.ctheta()), {k: s1[k] - s0[k] for k in s1}, s1["max_rows"]))
    (a, sa, rows), (b, sb, _) = out
    for k in ("events", "nucleations", "negative_dt", "sum_rows"):
        assert sa[k] == sb[k], k
    for k in a:
        assert np.array_equal(a[k], b[k], equal_nan=a[k].dtype.kind == "f"), k
    return dict(sa, max_rows=rows)


@pytest.mark.parametrize("value", [-0.0, -1e-7])
@pytest.mark.parametrize("field,spin", [((5e-6, 30e-6, 100e-6, "seed 7"), 40),
                                        ((5e-6, 50e-6, 10e-6, "rosenthal 0.35 20.0 5e-6"), 60)])
def test_uploaded_extents_with_a_sign(tmp_path, value, field, spin):
    """Half of the mushy cells' extents -0.0 or below zero beside some that are
    overdue: the negative events that these bring clamp the others at zero."""
    path = tmp_path / "front.in"
    path.write_text(FRONT % field)
    s = _uploaded(path, spin, 4, value)
    assert s["negative_dt"] > 0


@pytest.mark.parametrize("dt", [5e-6, 1e-5, 2e-5])
def test_every_part_of_the_window_runs(tmp_path, dt):
    """A front on which the loop takes all its parts: bounds in place of records (more than
    512 rows), windows (more than 640 rows) opened again within a step, records made
    then, rows kept outside, rows set up in the loop, negative events."""
    path = tmp_path / "front.in"
    path.write_text(FRONT % (dt, 30e-6, 100e-6, "seed 7"))
    s = _uploaded(path, int(2e-4 / dt), 6)
    assert s["max_rows"] > 640 and s["full_scan_steps"] == 0
    assert s["row_evaluations"] > s["steps"] == 6  # windows opened
    for k in ("records_late", "rows_outside", "rows_filled", "negative_dt"):
        assert s[k] > 0, k


@pytest.mark.parametrize("deck,steps", [("layers_rot.in", 40), ("track_easm60.in", 0), ("track_ros.in", 0)])
def test_no_step_falls_back_to_the_full_scan(deck, steps):
    """Neither with one growth velocity nor with per-cell ones; with event_scan=1 every step with events does."""
    from amcafe_gb300 import Simulation

    seen = []
    for scan in (0, 1):
        with Simulation(os.path.join(DECKS, deck), event_scan=scan) as sim:
            sim.InitializeVoxels()
            sim.begin()
            sim.run(steps)
            seen.append((sim.event_paths()["full_scan_steps"], sim.stats()))
    assert seen[0][0] == 0 and seen[0][1]["events"] > 0
    assert 0 < seen[1][0] <= seen[1][1]["steps"]


@pytest.mark.parametrize("field", [(5e-6, 30e-6, 100e-6, "seed 7"), (5e-6, 50e-6, 10e-6, "rosenthal 0.35 20.0 5e-6")])
def test_nucleations_leave_extents_below_zero(tmp_path, field):
    """Fifteen of sixteen events nucleate: uploaded extents below zero stay as they
    are until the first capture grows them."""
    path = tmp_path / "front.in"
    path.write_text((FRONT % field).replace("r 2e-4", "r 6e-2"))
    for steps in (1, 3):
        s = _uploaded(path, 50, steps, -1e-7)
        assert s["nucleations"] > 0
