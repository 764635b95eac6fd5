"""The neighbour count of a particle whose position is not a number: every particle of the 27 cells
around its own (it passes every test), and no place of their padding."""
import numpy as np
import pytest

from helpers import fluid
from watercube_gb300 import _abi
from watercube_gb300.fluid import dam_break_params, finalize, generate_dam_break

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3000, 200000])  # one and two targets per lane
@pytest.mark.parametrize("axes", [[0, 1, 2], [1]])
def test_count_of_a_particle_at_nan(gpu, n, axes):
    p = dam_break_params(n)
    p.flags |= _abi.WC_FLAG_NEIGHBOR_COUNTS
    p = finalize(p)
    st = generate_dam_break(p, 1)
    st["position"][7, axes] = np.nan
    with fluid(p, st) as f:
        f.sort()
        f.density()
        with pytest.raises(_abi.WatercubeError):
            f.synchronize()
        slot = int(np.flatnonzero(f.permutation() == 7)[0])
        got = int(f.neighbor_counts()[slot])
        R = p.grid_res
        cells = f.cell_counts().reshape(R, R, R)
        z, y, x = np.unravel_index(int(f.keys()[7]), (R, R, R))
    around = cells[max(z - 1, 0):z + 2, max(y - 1, 0):y + 2, max(x - 1, 0):x + 2].sum()
    assert got == around - 1


def test_count_after_a_judges_pass(gpu):
    """The same from the judge step's density pass (predict leaves its sorted buffer and counts)."""
    from watercube_gb300.local import LocalNet

    p = dam_break_params(3000)
    p.flags |= _abi.WC_FLAG_NEIGHBOR_COUNTS | _abi.WC_FLAG_TRACK_IDS
    p = finalize(p)
    st = generate_dam_break(p, 1)
    st["position"][7, 0] = np.nan
    with fluid(p, st) as f, LocalNet(ages=3, seed=1) as net:
        with pytest.raises(_abi.WatercubeError):
            net.predict(f, 1e-3)
        slot = int(np.flatnonzero(f.permutation() == 7)[0])
        got = int(f.neighbor_counts()[slot])
        R = p.grid_res
        cells = f.cell_counts().reshape(R, R, R)
        z, y, x = np.unravel_index(int(f.keys()[7]), (R, R, R))
    assert got == cells[max(z - 1, 0):z + 2, max(y - 1, 0):y + 2, max(x - 1, 0):x + 2].sum() - 1
