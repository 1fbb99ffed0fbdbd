"""Events of a type that the format does not define (outside 0 .. 4) evolve by their duration and amplitude and do
nothing else, whatever the number: no spoiler, no readout, no start of a pulse's propagator. Held to the float64 C
oracle (1e-10 absolute in Z in float64, the kernels' tolerance; 1e-8 mixed and 1e-3 in float32, as the tests of those
precisions) over tables with and without trains of shaped pulses, in every entry point."""
import numpy as np
import pytest

from test_pulse_propagators import OFFSETS, _close, _jvp, _row, _simulate, _table, _voxels

TYPES = [5, 7, 8, 9, 10, 11, 12, 15, 1000003, -1, -5, -6]


def _renamed(ev, where, t):
    typ = ev.type.copy()
    typ[where] = t
    return ev._replace(type=typ)


def _train():
    ev = _table([_row(f, pulses=9, samples=12, gap=((0, 0.004),)) for f in OFFSETS])
    delays = (ev.type == 0) & (ev.dt > 0)
    delays[:, -3:] = False
    return ev, delays


def _plain():
    rows = [[(0, 0.3, 0.0, 0.0, 0.0), (1, 0.02, 40.0, 0.3, f), (0, 0.01, 0.0, 0.0, 0.0), (1, 0.03, 60.0, -0.4, f),
             (0, 0.02, 0.0, 0.0, 0.0), (3, 0.0, 0.0, 0.0, 0.0)] for f in OFFSETS]
    ev = _table(rows)
    return ev, (ev.type == 0) | (ev.type == 1)


@pytest.mark.gpu
@pytest.mark.parametrize("table", [_train, _plain], ids=["train", "plain"])
@pytest.mark.parametrize("precision", [0, 1, 2], ids=["f64", "f32", "mixed"])
def test_undefined_types_only_evolve(cuda, table, precision):
    nc = 2
    P, M0 = _voxels(2, nc, seed=31)
    ev, where = table()
    for t in TYPES:
        other = _renamed(ev, where, t)
        for entry in ("bmc_simulate", "bmc_simulate_noalloc"):
            z = _simulate(cuda, P, M0, other, nc, precision, entry=entry)
            _close(z, P, M0, other, nc, (1e-10, 1e-3, 1e-8)[precision])


@pytest.mark.gpu
def test_undefined_types_only_evolve_with_tangents(cuda):
    """Tangents against the same table with delays in their place."""
    nc = 1
    P, M0 = _voxels(2, nc, seed=33)
    seeds = np.stack([P[3], P[4]])
    ev, where = _train()
    z0, j0 = _jvp(cuda, P, M0, ev, nc, [3, 4], seeds)
    for t in TYPES:
        z, j = _jvp(cuda, P, M0, _renamed(ev, where, t), nc, [3, 4], seeds)
        assert np.abs(z - z0).max() < 1e-11 and np.abs(j - j0).max() <= 1e-9 * np.abs(j0).max()


def test_the_oracle_only_evolves_undefined_types():
    nc = 2
    P, M0 = _voxels(1, nc, seed=31)
    import bmc_oracle as O
    ev, where = _train()
    want = O.c_simulate_z(P, ev, M0, nc, 6)
    for t in TYPES:
        np.testing.assert_array_equal(O.c_simulate_z(P, _renamed(ev, where, t), M0, nc, 6), want)
