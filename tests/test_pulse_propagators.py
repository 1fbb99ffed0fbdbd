"""Shaped pulses as propagators (csrc/bmc_train.cuh) and the launches of few chains.

A pulse that a row repeats is propagated once per chain and applied at every repeat. The results are held to
the float64 C oracle, which integrates every event (1e-10 absolute in Z, the tolerance of the float64 path; measured
~1e-12), over the forms a row can have: pool counts, sample counts around the least that qualifies, phases, gaps with
and without spoilers, pulses that differ, amplitudes beyond the interpolation's bound, readouts between the pulses.
Bit for bit: a row stacked with others gives what it gives alone, one voxel of a batch what it gives alone (its nodes
as chains of their own or in a loop), bmc_simulate_noalloc what bmc_simulate gives."""
import ctypes as C

import numpy as np
import pytest

import bmc_oracle as O

GAMMA = 267.5153


def _table(rows):
    """Events from lists of (type, dt, amp, phase, freq) per row, front-padded to the longest."""
    width = max(len(r) for r in rows)
    a = np.array([[(0, 0.0, 0.0, 0.0, 0.0)] * (width - len(r)) + r for r in rows], np.float64)
    typ = a[:, :, 0].astype(np.int32)
    return O.Events(typ, *[np.ascontiguousarray(a[:, :, j]) for j in range(1, 5)], np.where(typ == 3, 0, -1).astype(np.int32))


def _row(freq_hz, pulses=6, samples=20, tp=0.02, b1=1.5, phase=0.0, phase_step=0.0, gap=((0, 0.003),), gap_step=0.0,
         odd_pulse=None, adc_after=None, skew=0.05, tail=((4, 0.0), (0, 0.5))):
    t = (np.arange(samples) + 0.5) / samples
    amp = b1 * GAMMA / (2 * np.pi) * np.exp(-((t - 0.5) ** 2) / 0.06) * (1 + skew * t)
    r = [(0, 0.4, 0.0, 0.0, 0.0)]
    for j in range(pulses):
        scale = 0.5 if odd_pulse == j else 1.0
        r += [(1, tp / samples, a * scale, phase + phase_step * j, freq_hz) for a in amp]
        r += [(ty, dt + gap_step * j, 0.0, 0.0, 0.0) for ty, dt in gap]
        if adc_after == j:
            r += [(3, 0.0, 0.0, 0.0, 0.0)]
    return r + [(ty, dt, 0.0, 0.0, 0.0) for ty, dt in tail] + [(3, 0.0, 0.0, 0.0, 0.0)]


def _voxels(n, nc, seed=3, mt=True):
    import bench
    P, M0 = bench.voxel_params(n, nc, seed=seed)
    if not mt:
        P[3 + 5 * nc:8 + 5 * nc] = 0.0
        P[7 + 5 * nc] = 1.0
        M0[:, -1] = 0.0
    P[12 + 5 * nc] = np.random.default_rng(seed).uniform(0.9, 1.1, n)       # rel_b1
    return np.ascontiguousarray(P), M0


def _simulate(torch, P, M0, ev, nc, precision=0, spread=None, entry="bmc_simulate", mz=None):
    from bmc_b200 import _lib
    from bmc_b200.simulation import DeviceEvents, problem
    n, rows = P.shape[1], ev.dt.shape[0]
    mz = 2 * (1 + nc) if mz is None else mz
    dev = DeviceEvents(ev)
    dP, dM = torch.as_tensor(P).cuda(), torch.as_tensor(np.ascontiguousarray(M0)).cuda()
    out = torch.full((n, rows) if mz >= 0 else (n, rows, M0.shape[1]), float("nan"), dtype=torch.float64, device="cuda")
    sp = None
    if spread is not None:
        u, w, sigma = spread
        sp, keep = _lib.spread_struct(u, w, torch.full((n,), sigma, dtype=torch.float64, device="cuda"))
    _lib.check(getattr(_lib.lib(), entry)(problem(n, rows, ev.dt.shape[1], nc, mz, precision), C.c_void_p(dP.data_ptr()),
                                          dev.struct, C.c_void_p(dM.data_ptr()), sp, C.c_void_p(out.data_ptr()),
                                          _lib.stream_handle()))
    return out.cpu().numpy()


def _counted(torch, P, M0, ev, nc):
    """Z of the counting call, which integrates every event."""
    from bmc_b200 import _lib
    from bmc_b200.simulation import DeviceEvents, problem
    n, rows = P.shape[1], ev.dt.shape[0]
    dev, dP, dM = DeviceEvents(ev), torch.as_tensor(P).cuda(), torch.as_tensor(np.ascontiguousarray(M0)).cuda()
    out, work = torch.empty((n, rows), dtype=torch.float64, device="cuda"), torch.zeros(5, dtype=torch.int64, device="cuda")
    _lib.check(_lib.lib().bmc_simulate_counted(problem(n, rows, ev.dt.shape[1], nc, 2 * (1 + nc), _lib.F64), _lib.ptr(dP),
                                               dev.struct, _lib.ptr(dM), None, _lib.ptr(out), _lib.ptr(work),
                                               _lib.stream_handle()))
    return out.cpu().numpy()


OFFSETS = np.array([-900.0, -447.2, -30.0, 0.0, 127.7, 447.2, 1200.0])


def _close(z, P, M0, ev, nc, tol=1e-10):
    want = O.c_simulate_z(P, ev, M0, nc, 2 * (1 + nc))
    err = np.abs(z - want).max()
    print(f"max |dZ| {err:.2e}")
    assert err < tol


@pytest.mark.gpu
@pytest.mark.parametrize("nc", range(6))
@pytest.mark.parametrize("samples", [8, 33])
@pytest.mark.parametrize("skew", [0.05, 0.0], ids=["skewed", "mirrored"])
def test_pool_counts_match_the_oracle(cuda, nc, samples, skew):
    P, M0 = _voxels(3, nc, mt=nc != 1)
    for pulses in (9, 16):                                 # (five pools: from 14 pulses of 8 samples on)
        ev = _table([_row(f, pulses=pulses, samples=samples, skew=skew) for f in OFFSETS])
        _close(_simulate(cuda, P, M0, ev, nc), P, M0, ev, nc)


# when a propagator is formed: uses x samples >= FIXED + SAMPLE x samples for a mirrored pulse without a gap (train_cost)
FIXED, SAMPLE = [110, 44, 78, 77, 88, 150], [1.4, 0.42, 1.0, 0.95, 0.75, 2.2]


@pytest.mark.gpu
@pytest.mark.parametrize("nc", range(6))
@pytest.mark.parametrize("samples", [8, 30])
def test_few_pulses_are_integrated_event_by_event(cuda, nc, samples):
    """One use below the line the events are integrated as the counting call does, bit for bit; at the line the propagator
    gives the same to 1e-11 in other roundings."""
    P, M0 = _voxels(3, nc, seed=47)
    need = int(np.ceil((FIXED[nc] + SAMPLE[nc] * samples) / samples))
    for uses in (need - 1, need):
        rows = []
        for f in OFFSETS:
            t = (np.arange(samples) + 0.5) / samples
            amp = 60.0 * np.exp(-((t - 0.5) ** 2) / 0.06)
            amp = 0.5 * (amp + amp[::-1])
            rows.append([(1, 5e-4, a, 0.3 * j, f) for j in range(uses) for a in amp] + [(3, 0.0, 0.0, 0.0, 0.0)])
        ev = _table(rows)
        z = _simulate(cuda, P, M0, ev, nc)
        _close(z, P, M0, ev, nc)
        c = _counted(cuda, P, M0, ev, nc)
        assert np.abs(z - c).max() < 1e-11
        assert np.array_equal(z, c) == (uses < need), (uses, need)


@pytest.mark.gpu
@pytest.mark.parametrize("nc", [1, 4])
def test_mirrored_pulses_need_the_pools_fractions(cuda, nc):
    """Tiny, zero and negative fractions, with and without exchange: chains without the balance take the whole pulse."""
    P, M0 = _voxels(6, nc, seed=29)
    P[3 + nc:3 + 2 * nc, 1:6] = np.array([1e-7, 1e-18, 1e-25, 0.0, -1e-4])[None]
    M0[:, 2 * nc + 3:3 * nc + 3] = P[3 + nc:3 + 2 * nc].T
    P[3:3 + nc, 4] = 0.0
    ev = _table([_row(f, samples=24, skew=0.0) for f in OFFSETS])
    _close(_simulate(cuda, P, M0, ev, nc), P, M0, ev, nc)


FORMS = {
    "phases": dict(phase=0.7, phase_step=-2.1),
    "one_phase": dict(phase=1.1),
    "spoiled": dict(gap=((4, 0.0009), (0, 0.003))),
    "zero_length_spoiler": dict(gap=((0, 0.002), (4, 0.0))),
    "own_delays": dict(gap=((4, 0.0009), (0, 0.01)), gap_step=1e-4, phase_step=0.9),
    "no_gap": dict(gap=(), phase_step=0.3),
    "long_gap": dict(gap=tuple((0, 0.0004 * (j + 1)) for j in range(6))),
    "one_differs": dict(odd_pulse=1),
    "middle_differs": dict(odd_pulse=2, pulses=5),
    "readout_between": dict(adc_after=2),
    "few": dict(pulses=3),
    "short_pulses": dict(samples=7),
    "strong": dict(b1=8.0, tp=0.02),
    "beyond_the_bound": dict(b1=30.0, tp=0.02),
    "negative_lobes": dict(skew=-4.0),
    "mirrored": dict(skew=0.0, samples=21),
    "mirrored_even": dict(skew=0.0, samples=40, phase=0.4, phase_step=1.0),
    "mirrored_strong": dict(skew=0.0, samples=9, b1=8.0, tp=0.01),
    "mirrored_strong_8": dict(skew=0.0, samples=9, b1=8.0, tp=0.01, pulses=8),
    "own_delays_9": dict(gap=((4, 0.0009), (0, 0.01)), gap_step=1e-4, phase_step=0.9, pulses=9),
    "samples_1100": dict(samples=1100, tp=0.05, pulses=4),
}


@pytest.mark.gpu
@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("precision", [0, 2], ids=["f64", "mixed"])
def test_forms_of_a_train_match_the_oracle(cuda, form, precision):
    nc = 2
    P, M0 = _voxels(2, nc, seed=5)
    ev = _table([_row(f, **FORMS[form]) for f in OFFSETS])
    # mixed precision: where a row keeps the event-by-event path, the float32 tail's error (the mixed tests' bound); 30 uT in 1 ms
    # samples: 120 events of at most 3 sub-steps, each rounding terms of up to three times the state to 2^-24
    tol = 1e-10 if precision == 0 else (120 * 3 * 3 * 2.0 ** -24 if form == "beyond_the_bound" else 1e-8)
    _close(_simulate(cuda, P, M0, ev, nc, precision), P, M0, ev, nc, tol)


@pytest.mark.gpu
def test_rows_of_several_forms_are_each_their_own(cuda):
    """Stacked rows of different trains, lengths and forms, two voxels: bit for bit what each row gives alone."""
    nc = 4
    P, M0 = _voxels(2, nc, seed=7)
    rows = [_row(f, **FORMS[k]) for f, k in zip(np.resize(OFFSETS, len(FORMS) - 1), [k for k in FORMS if k != "samples_1100"])]
    rows += [[(1, 1.5, 60.0, 0.0, 200.0), (3, 0.0, 0.0, 0.0, 0.0)], _row(300.0, pulses=12, samples=64)]
    z = _simulate(cuda, P, M0, _table(rows), nc)
    for i, r in enumerate(rows):
        ev = _table([r])
        np.testing.assert_array_equal(z[:, i], _simulate(cuda, P, M0, ev, nc)[:, 0])
        _close(z[:, i:i + 1], P, M0, ev, nc)


@pytest.mark.gpu
@pytest.mark.parametrize("mz", [6, -1])
def test_spread_nodes_as_chains_and_in_a_loop(cuda, mz):
    """A spread over few chains runs its nodes as chains of their own, over many in a loop: the same bits; and the
    mean over the nodes is the oracle's weighted mean of the shifted voxels."""
    nc = 2
    u, w = np.polynomial.hermite_e.hermegauss(5)
    w = w / w.sum()
    sigma = 9.0
    for kw in (dict(), FORMS["own_delays"]):
        ev = _table([_row(f, **kw) for f in OFFSETS])
        P, M0 = _voxels(4100, nc, seed=9)                  # 28,700 chains: the loop
        many = _simulate(cuda, P, M0, ev, nc, spread=(u, w, sigma), mz=mz)
        few = _simulate(cuda, np.ascontiguousarray(P[:, :3]), M0[:3], ev, nc, spread=(u, w, sigma), mz=mz)
        np.testing.assert_array_equal(many[:3], few)
        z = few if mz >= 0 else few[:, :, 6]
        want = 0.0
        for uj, wj in zip(u, w):
            Q = P[:, :3].copy()
            Q[11 + 5 * nc] += sigma * uj / (Q[9 + 5 * nc] * Q[10 + 5 * nc] / (2 * np.pi))
            want = want + wj * O.c_simulate_z(Q, ev, M0[:3], nc, 6)
        assert np.abs(z - want).max() < 1e-10


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 2], ids=["f64", "mixed"])
def test_noalloc_gives_the_same_bits(cuda, precision):
    nc = 3
    P, M0 = _voxels(40, nc, seed=11)
    ev = _table([_row(f, **k) for f, k in zip(OFFSETS, (FORMS["phases"], {}, FORMS["own_delays"], FORMS["few"], {}, {}, {}))])
    u, w = np.array([-1.0, 0.3, 1.2]), np.array([0.25, 0.45, 0.3])
    for spread in (None, (u, w, 6.0)):
        z = _simulate(cuda, P, M0, ev, nc, precision, spread)
        assert np.all(np.isfinite(z))
        np.testing.assert_array_equal(z, _simulate(cuda, P, M0, ev, nc, precision, spread, "bmc_simulate_noalloc"))


def _jvp(torch, P, M0, ev, nc, rows, seeds, dm0=None, spread=None, counted=False):
    from bmc_b200 import _lib
    from bmc_b200.simulation import DeviceEvents, problem
    n, no, T = P.shape[1], ev.dt.shape[0], len(rows)
    dev = DeviceEvents(ev)
    up = lambda a: torch.as_tensor(np.ascontiguousarray(a)).cuda()
    dP, dM, dS = up(P), up(M0), up(seeds)
    dD = None if dm0 is None else up(dm0)
    z = torch.empty((n, no), dtype=torch.float64, device="cuda")
    j = torch.empty((T, n, no), dtype=torch.float64, device="cuda")
    tg = _lib.Tangents()
    tg.n_tangents = T
    for i, r in enumerate(rows):
        tg.field_row[i] = r
    tg.d_seed, tg.d_dm0 = dS.data_ptr(), None if dD is None else dD.data_ptr()
    sp = None
    if spread is not None:
        u, w, sigma = spread
        sp, keep = _lib.spread_struct(u, w, torch.full((n,), sigma, dtype=torch.float64, device="cuda"))
    args = [problem(n, no, ev.dt.shape[1], nc, 2 * (1 + nc), _lib.F64), _lib.ptr(dP), dev.struct, _lib.ptr(dM), sp, tg,
            _lib.ptr(z), _lib.ptr(j)]
    work = torch.zeros(5, dtype=torch.int64, device="cuda")
    _lib.check(_lib.lib().bmc_simulate_jvp_counted(*args, _lib.ptr(work), _lib.stream_handle()) if counted else
               _lib.lib().bmc_simulate_jvp(*args, _lib.stream_handle()))
    return z.cpu().numpy(), j.cpu().numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("nc", [0, 1, 2, 4, 5])
@pytest.mark.parametrize("form", ["plain", "phases", "spoiled", "own_delays", "own_delays_9", "few", "strong", "readout_between"])
def test_tangents_match_the_event_by_event_path(cuda, nc, form):
    """Every kind of tangent (rates, fractions, shifts, B0, B1, MT, the start state, the spread's width) through the
    propagators against forward mode over every event (the counting call): 1e-9 of each tangent's largest value."""
    P, M0 = _voxels(3, nc, seed=17)
    ev = _table([_row(f, **FORMS.get(form, {})) for f in OFFSETS])
    mt = 3 + 5 * nc
    rows = [0, 1, mt + 7, mt + 8, mt + 9, mt + 4, mt + 1, -1]     # r1w, r2w, gamma, b0_inhom, rel_b1, mt_r2, mt_f, dm0 only
    if nc:
        rows[:1] = [3]                                         # k of the first pool
        rows[6] = 3 + nc                                       # f of the first pool
    rng = np.random.default_rng(1)
    seeds = np.abs(P[np.maximum(rows, 0)]) * rng.uniform(0.5, 1.5, (8, 3)) + 1e-3
    dm0 = rng.uniform(-0.2, 0.2, (8,) + M0.shape) * (np.arange(8) >= 6)[:, None, None]
    z, j = _jvp(cuda, P, M0, ev, nc, rows, seeds, dm0)
    zc, jc = _jvp(cuda, P, M0, ev, nc, rows, seeds, dm0, counted=True)
    assert np.abs(z - zc).max() < 1e-11
    for t in range(8):
        scale = np.abs(jc[t]).max()
        err = np.abs(j[t] - jc[t]).max()
        print(f"tangent {rows[t]}: {err:.1e} of {scale:.1e}")
        assert err <= 1e-9 * scale + 1e-13


@pytest.mark.gpu
def test_spread_tangents_as_chains_and_in_a_loop(cuda):
    nc = 1
    u, w = np.polynomial.hermite_e.hermegauss(4)
    spread = (u, w / w.sum(), 8.0)
    rows = [3, 4, -2]
    for kw in ({}, FORMS["own_delays"]):
        ev = _table([_row(f, **kw) for f in OFFSETS])
        P, M0 = _voxels(4100, nc, seed=19)
        seeds = np.stack([P[3], P[4], np.ones(4100)])
        z, j = _jvp(cuda, P, M0, ev, nc, rows, seeds, spread=spread)
        P3, M3, s3 = np.ascontiguousarray(P[:, :3]), M0[:3], np.ascontiguousarray(seeds[:, :3])
        z3, j3 = _jvp(cuda, P3, M3, ev, nc, rows, s3, spread=spread)
        np.testing.assert_array_equal(z[:3], z3)
        np.testing.assert_array_equal(j[:, :3], j3)
        zc, jc = _jvp(cuda, P3, M3, ev, nc, rows, s3, spread=spread, counted=True)
        assert np.abs(z3 - zc).max() < 1e-11 and np.abs(j3 - jc).max() <= 1e-9 * np.abs(jc).max()


@pytest.mark.gpu
def test_non_finite_and_extreme_parameters_stay_with_their_voxel(cuda):
    nc = 1
    P, M0 = _voxels(4, nc, seed=13, mt=False)
    P[3, 1] = np.nan                                       # k of voxel 1
    P[1, 2] = 1e70                                         # R2 of voxel 2: more squarings than the cap
    ev = _table([_row(f) for f in OFFSETS])
    z = _simulate(cuda, P, M0, ev, nc)
    assert np.all(np.isnan(z[1])) and np.all(np.isnan(z[2]))
    keep = [0, 3]
    _close(z[keep], np.ascontiguousarray(P[:, keep]), M0[keep], ev, nc)


MIXED_ROWS = [("phases", {}), ("plain", {}), ("beyond_the_bound", {}), ("own_delays", {}), ("blocks", {}), ("mirrored_even", {}),
              ("few", dict(pulses=1))]


def _mixed_table():
    """Rows with a train, without one (pulses of samples of their own; a repeated block), and with one that chains refuse."""
    rows = []
    for f, (k, kw) in zip(OFFSETS, MIXED_ROWS):
        if k == "plain":
            rows.append([(1, 0.001 * (1 + 0.1 * j), 30.0 + j, 0.2 * j, f) for j in range(9)] + [(4, 0.0, 0.0, 0.0, 0.0),
                        (0, 0.5, 0.0, 0.0, 0.0), (3, 0.0, 0.0, 0.0, 0.0)])
        elif k == "blocks":
            rows.append([(1, 0.05, 40.0, 0.0, f), (0, 0.005, 0.0, 0.0, 0.0)] * 10 + [(3, 0.0, 0.0, 0.0, 0.0)])
        else:
            rows.append(_row(f, **{**dict(samples=12, pulses=16), **FORMS.get(k, {}), **kw}))
    return _table(rows)


def _tiled(a, n):
    return np.ascontiguousarray(np.resize(a.T, (n, a.shape[0])).T)


# more chains than one chunk of propagators holds (of bmc_simulate 170,496 with two pools, 37,888 with five; with tangents
# 37,888 from four pools on, 113,664 with one; of bmc_simulate_noalloc 10,656 with five) and than one window of flags
# (4,194,304), an odd rest each
@pytest.mark.gpu
@pytest.mark.parametrize("nc,n,entry,nodes", [
    (5, 8203, "bmc_simulate", 1), (5, 2003, "bmc_simulate_noalloc", 1), (5, 2003, "bmc_simulate_noalloc", 3),
    (5, 3001, "bmc_simulate", 3), (2, 24999, "bmc_simulate", 2), (0, 600701, "bmc_simulate", 1),
    (0, 600701, "bmc_simulate_noalloc", 1)])
def test_chunks_of_propagators_give_the_bits_of_one(cuda, nc, n, entry, nodes):
    """A batch of 61 voxels over and over: every voxel gives what the 61 give, which is the oracle's result."""
    P, M0 = _voxels(61, nc, seed=37)
    ev = _mixed_table()
    spread = None if nodes == 1 else (np.linspace(-1.0, 1.3, nodes), np.arange(1, nodes + 1) / (nodes * (nodes + 1) / 2), 7.0)
    one = _simulate(cuda, P, M0, ev, nc, spread=spread)
    many = _simulate(cuda, _tiled(P, n), np.resize(M0, (n, M0.shape[1])), ev, nc, spread=spread, entry=entry)
    np.testing.assert_array_equal(many, np.resize(one, many.shape))
    if nodes == 1:
        _close(one[:2], np.ascontiguousarray(P[:, :2]), M0[:2], ev, nc)


@pytest.mark.gpu
@pytest.mark.parametrize("nc,n,T,nodes", [(4, 5501, 3, 1), (1, 17003, 3, 1), (4, 5501, 1, 2), (5, 2801, 1, 3)])
def test_chunks_of_propagators_with_tangents_give_the_bits_of_one(cuda, nc, n, T, nodes):
    P, M0 = _voxels(59, nc, seed=41)
    ev = _mixed_table()
    spread = None if nodes == 1 else (np.linspace(-1.0, 1.3, nodes), np.arange(1, nodes + 1) / (nodes * (nodes + 1) / 2), 7.0)
    rows = [3, 3 + nc, 1][:T]
    seeds = P[rows] * 1.0
    z1, j1 = _jvp(cuda, P, M0, ev, nc, rows, seeds, spread=spread)
    z, j = _jvp(cuda, _tiled(P, n), np.resize(M0, (n, M0.shape[1])), ev, nc, rows, _tiled(seeds, n), spread=spread)
    np.testing.assert_array_equal(z, np.resize(z1, z.shape))
    for t in range(T):
        np.testing.assert_array_equal(j[t], np.resize(j1[t], j[t].shape))
    zc, jc = _jvp(cuda, P, M0, ev, nc, rows, seeds, spread=spread, counted=True)
    assert np.abs(z1 - zc).max() < 1e-11
    for t in range(T):
        assert np.abs(j1[t] - jc[t]).max() <= 1e-9 * np.abs(jc[t]).max()


@pytest.mark.gpu
def test_a_call_without_room_for_propagators_runs_without(cuda):
    """Scratch for speed is not needed: a captured call whose stream's workspace holds the call but not the propagators
    (here: left by a counting call, which forms none) is accepted and integrates event by event."""
    torch = cuda
    from bmc_b200 import _lib
    from bmc_b200.simulation import DeviceEvents, problem
    nc, n = 4, 3000
    P, M0 = _voxels(n, nc, seed=43)
    ev = _table([_row(f, pulses=14, samples=12) for f in OFFSETS])
    rows = ev.dt.shape[0]
    dev, dP, dM = DeviceEvents(ev), torch.as_tensor(P).cuda(), torch.as_tensor(M0).cuda()
    pr = problem(n, rows, ev.dt.shape[1], nc, 2 * (1 + nc), _lib.F64)
    z = torch.zeros((n, rows), dtype=torch.float64, device="cuda")
    want = _simulate(torch, P, M0, ev, nc)
    _simulate(torch, P, M0, ev, nc, entry="bmc_simulate_noalloc")        # every kernel loaded before the capture
    L = _lib.lib()
    stream = torch.cuda.Stream()
    work = torch.zeros(5, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    call = lambda f, *extra: _lib.check(f(pr, _lib.ptr(dP), dev.struct, _lib.ptr(dM), None, _lib.ptr(z), *extra,
                                          _lib.stream_handle()))
    with torch.cuda.stream(stream):
        call(L.bmc_simulate_counted, _lib.ptr(work))
        stream.synchronize()
        z.zero_()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            call(L.bmc_simulate)
        g.replay()
        stream.synchronize()
    assert np.abs(z.cpu().numpy() - want).max() < 1e-10
    del g


def _bound(n, theta, x):
    from math import factorial as f
    return 2.0 / 4 ** n * sum(theta ** (2 * j) / f(2 * j) * x ** (n - j) / f(n - j) for j in range(n + 1))


@pytest.mark.parametrize("n", [4, 6])
def test_interpolation_error_is_within_its_bound(n):
    """E(w) = exp([A(w) C; 0 0] h) through n Chebyshev nodes in u = (w / w_max)^2, its odd entries over w: within the
    bound the kernel chooses n by (in the balanced norm; plus rounding, a few units of 2^-53 per entry), at the largest
    w_max that n is taken for and at four times that, on generators of the benchmark's ranges."""
    from scipy.linalg import expm
    import bench
    tol = 2e-15
    lo, hi = 1e-3, 4.0
    for _ in range(60):                                    # the largest theta = w_max h that meets the tolerance
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if _bound(n, mid, 0.0) <= tol else (lo, mid)
    nc, h = 4, 2.5e-4
    z0 = 2 * (nc + 1)
    c = np.sin(np.pi / 4 * (2 * np.arange(n) + 1) / n) ** 2
    rng = np.random.default_rng(0)
    P, _ = bench.voxel_params(6, nc, seed=1)
    for v in range(6):
        for scale in (1.0, 4.0):
            wmax = lo / h * scale
            # build the generator from the oracle's matrix at two amplitudes: A(w) = A0 + w B + w^2 G
            A0, B, G = _generator(P[:, v], nc, freq=rng.uniform(-1200, 1200))
            E = lambda w: expm((A0 + w * B + w * w * G) * h)
            odd = np.zeros(A0.shape, bool)
            zi = np.arange(A0.shape[0]) >= z0
            odd[zi[:, None] != zi[None, :]] = True
            Eq = np.array([np.where(odd, E(wmax * np.sqrt(u)) / np.sqrt(u), E(wmax * np.sqrt(u))) for u in c])
            for rho in (0.0, 0.013, 0.4, -0.77, 1.0):
                u = rho * rho
                l = np.array([np.prod([(u - c[j]) / (c[q] - c[j]) for j in range(n) if j != q]) for q in range(n)])
                got = np.tensordot(l, Eq, 1)
                got = np.where(odd, rho * got, got)
                err = np.abs(got - E(wmax * rho))[:z0 + nc + 2].max()
                x = wmax ** 2 * abs(G.min()) * h
                assert err <= _bound(n, lo * scale, x) + 2e-14


def _generator(p, nc, freq):
    """(A0, B, G) of [A C; 0 0] = A0 + w B + w^2 G for one voxel's params column, phase 0, no MT lineshape change."""
    N = 3 * nc + 4
    A0, B, G = (np.zeros((N + 1, N + 1)) for _ in range(3))
    k, f, dw, r1, r2 = (p[3 + j * nc:3 + (j + 1) * nc] for j in range(5))
    mk, mf, _, mr1, _, _, b0, gam, inh, _ = p[3 + 5 * nc:]
    off = 2 * np.pi * freq - gam * b0 * inh
    for j in range(nc + 1):
        x, y, z = j, nc + 1 + j, 2 * nc + 2 + j
        d = off if j == 0 else off - dw[j - 1] * gam * b0
        R2 = p[1] + (k * f).sum() if j == 0 else r2[j - 1] + k[j - 1]
        R1 = p[0] + (k * f).sum() + mk * mf if j == 0 else r1[j - 1] + k[j - 1]
        A0[x, x] = A0[y, y] = -R2
        A0[z, z] = -R1
        A0[x, y], A0[y, x] = d, -d
        B[y, z], B[z, y] = 1.0, -1.0
        if j:
            for q in (x, y, z):
                A0[q - j, q], A0[q, q - j] = k[j - 1], k[j - 1] * f[j - 1]
            A0[z, N] = r1[j - 1] * f[j - 1]
    A0[2 * nc + 2, N - 1], A0[N - 1, 2 * nc + 2] = mk, mk * mf
    A0[2 * nc + 2, N], A0[N - 1, N] = p[0], mr1 * mf
    A0[N - 1, N - 1] = -(mr1 + mk)
    G[N - 1, N - 1] = -1e-5
    return A0, B, G
