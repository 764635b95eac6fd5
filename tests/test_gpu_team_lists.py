"""Stage calls on a fluid with the team passes after calls that sort for the lane passes (a rollout's
judge, a surface): they see the cell tables that those calls left, as after a sort of their own."""
import numpy as np
import pytest

from helpers import fluid
from watercube_gb300 import _abi
from watercube_gb300.fluid import dam_break_params, finalize, generate_dam_break
from watercube_gb300.local import WC_LOCAL_STALE, rollout
from watercube_gb300.surface import Surface

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("before", ["rollout", "surface"])
def test_stages_after_a_lane_sort(gpu, before):
    p = dam_break_params(3000)
    p.flags |= _abi.WC_FLAG_CELL_TEAMS | _abi.WC_FLAG_TRACK_IDS
    p = finalize(p)
    st = generate_dam_break(p, 1)
    st["velocity"] = np.random.default_rng(0).normal(0, 0.3, (3000, 3))
    out = []
    for sort in (False, True):
        with fluid(p, st) as f, Surface(20) as s:
            if before == "rollout":
                rollout(f, 1e-3, 8, mode=WC_LOCAL_STALE)
            else:
                s.extract(f)
            start = f.particles()
            if sort:
                f.sort()
            f.density()
            f.integrate(1e-3)
            out.append(f.particles())
            assert (out[-1]["velocity"] != start["velocity"]).any(axis=1).sum() > 2900
    assert out[0].tobytes() == out[1].tobytes()
