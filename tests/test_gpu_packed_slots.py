"""Dilute states, whose padded cells would not fit the lane passes' slots: the passes take the sorted slots
instead and mask what a load reads beside its row. Neighbours and densities against the FP64 oracle;
the same bits as the padded layout (a dilute scene in a batch that is padded as a whole), also for
targets with more candidates than their entries hold; the judge's sums; the surface's field; and the
memory that such a state takes."""
import numpy as np
import pytest

from helpers import fluid
from oracle import local_ref as L
from oracle.oracle import to64
from watercube_gb300 import _abi
from watercube_gb300.batch import Batch
from watercube_gb300.fluid import dam_break_params, finalize

pytestmark = pytest.mark.gpu

COUNTS, IDS = _abi.WC_FLAG_NEIGHBOR_COUNTS, _abi.WC_FLAG_TRACK_IDS


def dilute(n, box, seed, flags=0, clump=0):
    """n particles uniform in the box of a dam break of `box`, `clump` of them in the eight cells around a corner."""
    p = dam_break_params(box)
    p.num_particles = n
    p.flags |= flags
    p = finalize(p)
    rng = np.random.default_rng(seed)
    st = _abi.particles(n)
    st["position"] = rng.uniform(0.0, p.size, (n, 3)).astype(np.float32)
    h = float(p.kernel_radius)
    corner = p.grid_res // 2 * p.bin_size
    st["position"][:clump] = (corner + rng.uniform(-0.45 * h, 0.45 * h, (clump, 3))).astype(np.float32)
    st["velocity"] = rng.normal(0.0, 0.3, (n, 3)).astype(np.float32)
    return p, st


def padded_slots(f):
    return int(((f.cell_counts().astype(np.int64) + 3) // 4 * 4).sum())


# cells without any, one and several particles; the last one in more than one wave of warps
@pytest.mark.parametrize("n,box", [(1, 1000), (5, 1000), (61, 1000), (3001, 16384), (50001, 100000), (300001, 524288)])
def test_neighbours_against_fp64(gpu, oracle, n, box):
    p, st = dilute(n, box, n, COUNTS)
    with fluid(p, st) as f:
        f.sort()
        f.density()
        srt, nc = f.particles(_abi.WC_BUFFER_SORTED), f.neighbor_counts()
        assert n < 61 or padded_slots(f) > 1.5 * n + 16
    o_sorted, _, _, counts, offsets = oracle.sort(p, st)
    assert np.array_equal(nc, oracle.density(p, o_sorted, counts, offsets))
    s64 = to64(srt)
    oracle.density(p, s64, counts, offsets)
    assert (np.abs(srt["density"] - s64["density"]) / s64["density"]).max() <= 1e-5


@pytest.mark.parametrize("clump", [0, 2600])
def test_same_bits_as_padded(gpu, clump):
    """The clump: up to 2,600 candidates in blocks of 32 by row, more than a target's entries hold."""
    thin = dilute(12001, 100000, 3, clump=clump)
    small = dilute(4000, 30000, 4)
    p = finalize(dam_break_params(60000))
    rng = np.random.default_rng(5)
    thick = _abi.particles(60000)
    thick["position"] = (0.01 + 0.4 * p.size * rng.random((60000, 3))).astype(np.float32)
    out = {}
    for name, scenes in (("alone", [thin]), ("packed batch", [thin, small]), ("padded batch", [thin, (p, thick)])):
        with Batch([q for q, _ in scenes], [s for _, s in scenes]) as b:
            b.step(1e-4, 3)
            out[name] = b.scene(0, b.particles()).tobytes()
    with fluid(*thin) as f:
        f.sort()
        assert padded_slots(f) > 1.5 * 12001 + 16
        f.step(1e-4, 3)
        assert f.particles().tobytes() == out["alone"] == out["packed batch"] == out["padded batch"]


def test_judge_sums(gpu, oracle):
    from watercube_gb300.local import LocalNet

    p, st = dilute(6000, 16384, 7, IDS)
    dt = 1e-3  # the step that the scale of the density rate is stated for
    with fluid(p, st) as f, LocalNet(ages=3, seed=5) as net:
        x, _ = net.predict(f, dt)
        srt = f.particles(_abi.WC_BUFFER_SORTED)
        f.sort()
        assert padded_slots(f) > 1.5 * 6000 + 16
    acc, jerk, rate = L.pair_sums(p, to64(srt), oracle.cull_threshold(float(p.kernel_radius)))
    ref = L.inputs(p, srt, acc, jerk, rate, dt)
    for cols in (slice(0, 3), slice(3, 6), slice(6, 7)):  # acceleration, J dt, density rate: BF16 of FP32 sums
        assert np.linalg.norm(x[:, cols] - ref[:, cols]) <= 5e-3 * np.linalg.norm(ref[:, cols])


@pytest.mark.parametrize("G", [5, 33])
def test_surface_field(gpu, oracle, G):
    from oracle import surface_ref as R
    from watercube_gb300.surface import Surface

    p, st = dilute(5001, 16384, 9)
    with fluid(p, st) as f, Surface(G, iso=0.05) as s:
        n = s.extract(f)
        srt, _, _, _, offsets = oracle.sort(p, st)
        phi = R.field(srt["position"].astype(np.float32), np.append(offsets, np.uint32(len(st))), p.bin_size,
                      p.grid_res, p.size, G, p.kernel_radius, p.particle_mass, p.rest_density)
        assert np.array_equal(s.field(), phi)
        ref = R.march(phi, p.size, 0.05)
        assert n == ref.shape[0] and np.array_equal(s.triangles(), ref)


def test_memory(gpu):
    """Two states, sort tables, 512 bytes of entries, 1.5 slots of 48 bytes and the staging buffer per
    particle, four tables per cell: 800 and 20 bytes at most (four slots per particle would make 890)."""
    torch = pytest.importorskip("torch")
    p, st = dilute(2000000, 2000000, 1)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    with fluid(p, st) as f:
        f.synchronize()
        used = free - torch.cuda.mem_get_info()[0]
        assert used <= 800 * 2000000 + 20 * f.num_cells + (32 << 20), used / 2000000
