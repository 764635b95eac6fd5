"""The FP64 totals that a rollout starts from (the device widens FP32 to FP64 by integer operations)
against the oracle's, with zeros, denormals, tiny and large velocities in the state. 1e-11 of the
sum of magnitudes: up to 1e4 terms added in FP64 in different orders (2^-53 each)."""
import numpy as np
import pytest

from helpers import fluid
from watercube_gb300.fluid import dam_break_params, finalize, generate_dam_break
from watercube_gb300.local import WC_LOCAL_STALE, rollout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 10000])
def test_totals(gpu, oracle, n):
    p = finalize(dam_break_params(n))
    st = generate_dam_break(p, 3)
    v = np.random.default_rng(1).normal(0, 0.2, (n, 3)).astype(np.float32)
    v[0:8, 0] = [0.0, -0.0, 1e-45, -1e-40, 1.1754944e-38, -1e-30, 30.0, -30.0]
    st["velocity"] = v
    with fluid(p, st) as f:
        got = np.array(rollout(f, 1e-4, 1, mode=WC_LOCAL_STALE)["diag_start"])
    d = oracle.diagnostics(p, st)
    ref = np.array([d["mass"], *d["momentum"], d["kinetic"], d["potential"]])
    m, a = float(p.particle_mass), np.abs(v.astype(np.float64))
    scale = np.array([m * n, *(m * a.sum(0)), abs(d["kinetic"]), abs(d["potential"])])
    assert (np.abs(got - ref) <= 1e-11 * scale).all(), (got, ref)
