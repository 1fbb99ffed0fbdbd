"""Events of at most one CEST pool exponentiated by the chain's own thread (csrc/bmc_sym.cuh): forward passes against
the float64 C oracle (1e-10 absolute, the float64 path's tolerance), all tangents of single-event rows against forward
mode (1e-9 of each tangent's largest value, the adjoint tests' bound), over what the turned and scaled form has to get
right -- RF phases, transverse start states, fractions that are zero, tiny or negative, start magnetisations far from
the fractions, other readout entries -- the last four of which it has to leave to the general path."""
import numpy as np
import pytest

import bmc_oracle as O
from test_pulse_propagators import GAMMA, _jvp, _simulate, _table, _voxels

pytestmark = pytest.mark.gpu
OFFSETS = np.array([-800.0, -130.0, 0.0, 3.0, 447.2])

CASES = {
    "plain": {},
    "phase": dict(phase=1.3),
    "transverse_start": dict(phase=-2.0, transverse=0.3),
    "zero_fraction": dict(f=0.0, m=0.0),
    "zero_fraction_with_magnetisation": dict(f=0.0, m=0.02),
    "tiny_fraction": dict(f=1e-13, m=0.01),
    "small_fraction": dict(f=1e-7, m=0.001),
    "negative_fraction": dict(f=-1e-4, m=0.0),
    "negative_amplitude": dict(amp=-1.0, phase=0.4),
    "short": dict(dt=0.02),
    "long": dict(dt=20.0),
    "weak_rf": dict(amp=1e-4),
    "two_blocks": dict(blocks=2),
}


def _case(nc, mt=True, f=None, m=None, transverse=0.0, phase=0.0, amp=1.0, dt=2.0, blocks=1):
    P, M0 = _voxels(3, nc, seed=23, mt=mt)
    if nc and f is not None:
        P[4, 1] = f
        M0[1, 5] = m
    if transverse:
        M0[:, :2 * (nc + 1)] = transverse * np.random.default_rng(2).standard_normal((3, 2 * (nc + 1)))
    rows = [[(1, dt / blocks, amp * 1.5 * GAMMA / (2 * np.pi), phase + 0.3 * j, x) for j in range(blocks)]
            + [(3, 0.0, 0.0, 0.0, 0.0)] for x in OFFSETS]
    return P, M0, _table(rows)


@pytest.mark.parametrize("nc", [0, 1])
@pytest.mark.parametrize("mt", [False, True], ids=["no_mt", "mt"])
@pytest.mark.parametrize("case", list(CASES))
def test_forward_matches_the_oracle(cuda, nc, mt, case):
    P, M0, ev = _case(nc, mt, **CASES[case])
    want = O.c_simulate_z(P, ev, M0, nc, 2 * (1 + nc))
    err = np.abs(_simulate(cuda, P, M0, ev, nc) - want).max()
    print(f"{err:.1e}")
    assert err < 1e-10


@pytest.mark.parametrize("nc", [0, 1])
@pytest.mark.parametrize("mt", [False, True], ids=["no_mt", "mt"])
@pytest.mark.parametrize("case", [c for c in CASES if c != "two_blocks"])
@pytest.mark.parametrize("spread", [False, True], ids=["one", "spread"])
def test_tangents_match_forward_mode(cuda, nc, mt, case, spread):
    from bmc_b200 import _lib
    P, M0, ev = _case(nc, mt, **CASES[case])
    r = 3 + 5 * nc
    rows = [0, 1, r + 8, r + 9, r, r + 1, r + 4, -2 if spread else -1]     # r1w, r2w, b0_inhom, rel_b1, mt_k, mt_f, mt_r2
    if nc:
        rows[:2], rows[6] = [3, 4], 5                                      # k, f, and the shift of the pool
    rng = np.random.default_rng(3)
    seeds = np.abs(P[np.maximum(rows, 0)]) * rng.uniform(0.5, 1.5, (8, 3)) + 1e-3
    dm0 = rng.uniform(-0.2, 0.2, (8,) + M0.shape) * (np.arange(8) >= 6)[:, None, None]
    u, w = np.array([-1.2, 0.1, 0.9]), np.array([0.3, 0.4, 0.3])
    sp = (u, w, 7.0) if spread else None
    z, j = _jvp(cuda, P, M0, ev, nc, rows, seeds, dm0, sp)
    L = _lib.lib()
    _lib.check(L.bmc_set_tangent_mode(_lib.TANGENTS_FORWARD))
    try:
        zf, jf = _jvp(cuda, P, M0, ev, nc, rows, seeds, dm0, sp)
    finally:
        _lib.check(L.bmc_set_tangent_mode(_lib.TANGENTS_AUTO))
    assert np.abs(z - zf).max() < 1e-11
    for t in range(8):
        scale, err = np.abs(jf[t]).max(), np.abs(j[t] - jf[t]).max()
        print(f"tangent {rows[t]}: {err:.1e} of {scale:.1e}")
        assert err <= 1e-9 * scale + 1e-12


def test_other_readouts_keep_the_group_kernel(cuda):
    """A readout entry that is not water's z: the general path's tangents (forward mode's values)."""
    import torch
    from bmc_b200 import _lib
    from bmc_b200.simulation import DeviceEvents, problem
    P, M0, ev = _case(1, True, phase=0.5)
    up = lambda a: torch.as_tensor(np.ascontiguousarray(a)).cuda()
    dP, dM, dS, dev = up(P), up(M0), up(np.ones((2, 3))), DeviceEvents(ev)
    got = []
    for mode in (_lib.TANGENTS_AUTO, _lib.TANGENTS_FORWARD):
        _lib.check(_lib.lib().bmc_set_tangent_mode(mode))
        try:
            for mz in (2, 5):
                z = torch.empty((3, 5), dtype=torch.float64, device="cuda")
                j = torch.empty((2, 3, 5), dtype=torch.float64, device="cuda")
                tg = _lib.Tangents()
                tg.n_tangents, tg.d_seed, tg.d_dm0 = 2, dS.data_ptr(), None
                tg.field_row[0], tg.field_row[1] = 3, 1
                _lib.check(_lib.lib().bmc_simulate_jvp(problem(3, 5, 2, 1, mz, _lib.F64), _lib.ptr(dP), dev.struct,
                                                       _lib.ptr(dM), None, tg, _lib.ptr(z), _lib.ptr(j), _lib.stream_handle()))
                got.append((z.cpu().numpy(), j.cpu().numpy()))
        finally:
            _lib.check(_lib.lib().bmc_set_tangent_mode(_lib.TANGENTS_AUTO))
    for (z, j), (zf, jf) in zip(got[:2], got[2:]):
        assert np.abs(z - zf).max() < 1e-11 and np.abs(j - jf).max() <= 1e-9 * np.abs(jf).max() + 1e-12
