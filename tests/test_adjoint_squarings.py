"""The adjoint kernel's trial points (exp(X) alone, no derivative; with four pools the squarings of a warp's two chains go
through the tensor cores together while both have some left) against forward mode, through a fit that compares its
costs. Ten chains of two saturation powers in two lengths: an odd one out, and chains of a warp with unequal squarings."""
import numpy as np
import pytest

from test_adjoint import _batch
import bmc_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc,offsets", [(2, 5), (3, 5), (4, 1), (4, 5), (4, 7), (5, 5)])
def test_trial_points_equal_forward_mode(cuda, nc, offsets):
    """z agrees to 1e-11 and the Jacobians to 1e-9 of their largest value (the tangent tests' bounds), and the scaled
    normal matrix of the two rates is conditioned below 1e2: 1e-7 of the values found, 1e-9 of the
    residual or, where two samples leave none, z's 1e-11."""
    from bmc_b200 import settings
    from bmc_b200.fitting import Experiment, FitSpec, FreeParam, fit
    from bmc_b200.sequences import cw_saturation
    from bmc_b200.simulation import SimParams, initial_state
    pb = _batch(1, nc, 5)
    jp = SimParams(*[np.asarray(x)[0] for x in pb])
    m0 = initial_state(jp)
    ppm = np.linspace(-4.1, 3.7, offsets) if offsets > 1 else np.array([3.5])
    ladder = Experiment.stack([Experiment(jp, cw_saturation(ppm, b, tp, 3.0), m0, O.mz_loc(nc))
                               for b, tp in ((0.8, 1.0), (4.0, 6.0))])
    z = np.asarray(ladder.simulate())
    z = z[None, :] + 0.002 * np.random.default_rng(3).standard_normal((3, z.size))
    k = float(np.asarray(pb.cest_k)[0, 0])
    spec = FitSpec([FreeParam("k", "cest_k", 0, scale=k, lo=0.1 * k, hi=10 * k, x0=0.8 * k),
                    FreeParam("r2", "water_r2", None, scale=10.0, lo=1.0, hi=100.0, x0=15.0)])
    out = {}
    for mode in ("auto", "forward"):
        settings.use_tangents(mode)
        try:
            out[mode] = fit(ladder, spec, z, n_per_block=len(ppm), n_iter=6)
        finally:
            settings.use_tangents("auto")
    np.testing.assert_allclose(out["auto"].x, out["forward"].x, rtol=1e-7)
    np.testing.assert_allclose(out["auto"].rms, out["forward"].rms, rtol=1e-9, atol=1e-11)
