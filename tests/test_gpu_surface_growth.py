"""A surface of more triangles than the buffer holds from the start (8 grid_res^2): the buffer grows
and the mesh is the oracle's bit for bit, also when the next one is smaller."""
import numpy as np
import pytest

from helpers import fluid
from oracle import surface_ref as R
from watercube_gb300.fluid import dam_break_params, finalize, generate_dam_break

G = 20


def cloud(n=400, seed=2):
    p = finalize(dam_break_params(n))
    st = generate_dam_break(p, seed)
    rng = np.random.default_rng(seed)
    st["position"] = rng.uniform(0.05, 0.95, (n, 3)).astype(np.float32) * np.float32(p.size)
    return p, st


def mesh(oracle, p, st, iso):
    srt, _, _, _, offsets = oracle.sort(p, st)
    phi = R.field(srt["position"].astype(np.float32), np.append(offsets, np.uint32(len(st))), p.bin_size, p.grid_res,
                  p.size, G, p.kernel_radius, p.particle_mass, p.rest_density)
    return R.march(phi, p.size, iso)


def test_the_cloud_needs_more(oracle):
    p, st = cloud()
    assert mesh(oracle, p, st, 0.02).shape[0] > 8 * G * G


@pytest.mark.gpu
def test_growth(gpu, oracle):
    from watercube_gb300.surface import Surface

    p, st = cloud()
    few = st.copy()
    few["position"] *= np.float32(0.3)
    with fluid(p, st) as f, Surface(G, iso=0.02) as s:
        for state in (few, st, few):
            f.set_particles(state)
            ref = mesh(oracle, p, state, 0.02)
            assert s.extract(f) == ref.shape[0] and np.array_equal(s.triangles(), ref)
