"""The adjoint superposition over the edges of the interpolation in rSigma (the cases of
the forward's test): <g, D w> = <w, D^T g> for gradients on interleaved slices of the
grid, all of one sign, so that no error cancels against another.

Tolerance, relative: the forward's total agrees with its definition to 1e-6, the adjoint's
interpolation to 1.2e-6 per source; the single-precision sums of the adjoint (a ray over
its steps, a lattice cell over its rays, a few hundred positive terms each) stay within
sqrt(300) * 6e-8 = 1e-6 each. The sum is below 1e-5."""
import numpy as np
import pytest

from _parity import run_gpu
from test_gpu_superpose_nodes import _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["one_layer", "forty_layers", "fine_rays", "finest_rays", "coarse_rays", "density_step",
                                  "density_step_across"])
def test_dot_product_by_slices(name):
    case = _case(name)
    eng = run_gpu(case, keep_debug=False)
    dose = eng.read_dose64()
    w = np.asarray(case["beam"]["spot_weights"], np.float64)
    rng = np.random.Generator(np.random.PCG64(7))
    g = rng.lognormal(0.0, 0.5, dose.shape)
    for axis in range(3):
        for odd in (0, 1):
            part = np.zeros_like(g)
            at = tuple(slice(odd, None, 2) if i == axis else slice(None) for i in range(3))
            part[at] = g[at]
            want = float((part * dose).sum())
            assert want > 0.0
            got = float(w @ eng.adjoint_beam(case["beam"], part).astype(np.float64))
            assert abs(got - want) <= 1e-5 * want, (axis, odd, got / want - 1.0)
    eng.close()
