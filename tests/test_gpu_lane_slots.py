"""The lane passes' padded slots: pairs of targets per lane, ragged cells, blocks beyond the entry
space and a sorted buffer that the caller rewrites between the passes."""
import numpy as np
import pytest

from helpers import case, fluid
from oracle.oracle import to64
from watercube_gb300 import _abi
from watercube_gb300.batch import Batch
from watercube_gb300.fluid import dam_break_params, finalize

pytestmark = pytest.mark.gpu


def ragged(n, seed, side=0.6, flags=0):
    """n particles uniform in a box of the rest volume's size: cells of 0 to ~25 particles."""
    p = dam_break_params(n)
    p.flags |= flags
    p = finalize(p)
    rng = np.random.default_rng(seed)
    st = _abi.particles(n)
    st["position"] = (0.002 + rng.random((n, 3)) * side * np.float32([1.0, 0.6, 0.95])).astype(np.float32)
    st["velocity"] = rng.normal(0.0, 0.3, (n, 3)).astype(np.float32)
    return p, st


# one target per lane (61 and 50,001), pairs in one wave (200,003) and in several (500,001)
@pytest.mark.parametrize("n", [61, 50001, 200003, 500001])
def test_ragged_cells_against_fp64(gpu, oracle, n):
    p, st = ragged(n, n, flags=_abi.WC_FLAG_NEIGHBOR_COUNTS)
    with fluid(p, st) as f:
        f.sort()
        f.density()
        srt, nc = f.particles(_abi.WC_BUFFER_SORTED), f.neighbor_counts()
    o_sorted, _, _, counts, offsets = oracle.sort(p, st)
    assert np.array_equal(nc, oracle.density(p, o_sorted, counts, offsets))
    s64 = to64(srt)
    oracle.density(p, s64, counts, offsets)
    rel = np.abs(srt["density"] - s64["density"]) / s64["density"]
    assert rel.max() <= 1e-5, f"max relative density error {rel.max():.2e}"


def test_pairs_equal_single_targets(gpu):
    """A batch large enough for pairs; each of its scenes alone runs one target per lane."""
    scenes = [ragged(100003, 1), ragged(80002, 2, side=0.5)]
    with Batch([p for p, _ in scenes], [s for _, s in scenes]) as b:
        b.step(1e-3, 3)
        out = b.particles()
        for k, (p, st) in enumerate(scenes):
            with fluid(p, st) as f:
                f.step(1e-3, 3)
                assert b.scene(k, out).tobytes() == f.particles().tobytes()


@pytest.mark.parametrize("name", ["dam16k", "compressed16k"])
def test_rewritten_sorted_buffer(gpu, oracle, name):
    """Velocities and densities that the caller writes into the sorted buffer between the density
    and the force pass are the ones the force pass uses, for the neighbours too."""
    p, st = case(name)
    q = p.copy()
    q.flags |= _abi.WC_FLAG_CELL_TEAMS
    out = []
    for prm in (p, q):
        with fluid(prm, st) as f:
            f.sort()
            f.density()
            srt = f.particles(_abi.WC_BUFFER_SORTED)
            rng = np.random.default_rng(5)
            srt["velocity"] += rng.normal(0.0, 0.5, srt["velocity"].shape).astype(np.float32)
            srt["density"] *= rng.uniform(0.8, 1.25, len(srt)).astype(np.float32)
            f.set_particles(srt, _abi.WC_BUFFER_SORTED)
            f.integrate(1e-3)
            out.append((srt, f.particles()))
    # both variants sum the same terms in another order: FP32 rounding of sums of ~30 to ~500
    # terms, 500 x 2^-24 = 3e-5 of the largest change
    dv = np.abs(out[1][1]["velocity"] - out[1][0]["velocity"]).max()
    assert np.abs(out[0][1]["velocity"] - out[1][1]["velocity"]).max() <= 1e-4 * dv


@pytest.mark.parametrize("G", [2, 5, 8, 33])
@pytest.mark.parametrize("flags", [0, _abi.WC_FLAG_CELL_TEAMS])
def test_surface_grid_edges(gpu, oracle, G, flags):
    """The field's vertex blocks at ragged grids, on a fluid of either pass variant, bit for bit; the
    same surface object then takes a larger and again the smaller mesh."""
    from oracle import surface_ref as R
    from watercube_gb300.surface import Surface

    p, small = ragged(3001, 4, flags=flags)
    big = small.copy()
    big["position"] *= np.float32([1.6, 1.6, 1.0])
    with fluid(p, small) as f, Surface(G, iso=0.3) as s:
        for state in (small, big, small):
            f.set_particles(state)
            n = s.extract(f)
            srt, _, _, counts, offsets = oracle.sort(p, state)
            phi = R.field(srt["position"].astype(np.float32), np.append(offsets, np.uint32(len(state))), p.bin_size,
                          p.grid_res, p.size, G, p.kernel_radius, p.particle_mass, p.rest_density)
            assert np.array_equal(s.field(), phi)
            ref = R.march(phi, p.size, 0.3)
            assert n == ref.shape[0] and np.array_equal(s.triangles(), ref)
