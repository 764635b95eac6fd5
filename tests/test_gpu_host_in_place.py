"""Page-locked host records are read and written in place by the kernels (wc_fluid_update_host,
wc_batch_step_host); a buffer that does not start on a 32-byte boundary, and pageable memory, go
through the staging buffer. Both give the bytes of set_particles + update + particles()."""
import numpy as np
import pytest

from helpers import fluid
from watercube_gb300.batch import Batch, batch_specs, scene_params, scene_particles
from watercube_gb300.fluid import PinnedBuffer, finalize, generate_reference_lattice, reference_params

pytestmark = pytest.mark.gpu


def records(buf, n, offset, dtype):
    raw = buf.particles(n + 2).view(np.uint8)
    return raw[offset:offset + n * dtype.itemsize].view(dtype)


@pytest.mark.parametrize("n", [1, 33, 4097])
@pytest.mark.parametrize("at", [(0, 0), (32, 64), (16, 32), (32, 16), (16, 48)])
def test_fluid(gpu, n, at):
    p = reference_params()
    p.num_particles = n
    p = finalize(p)
    st = generate_reference_lattice(p, 0)
    bufs = [PinnedBuffer(32 * (n + 2)) for _ in range(2)]
    try:
        a_in, a_out = (records(b, n, o, st.dtype) for b, o in zip(bufs, at))
        with fluid(p, st) as a, fluid(p, st) as b:
            a_in[:] = st
            for _ in range(3):
                a.update_host(1.0 / 60.0, a_in, a_out)
                b.set_particles(a_in.copy())
                b.update(1.0 / 60.0)
                assert a_out.tobytes() == b.particles().tobytes()
                a_in[:] = a_out
                a_in["velocity"] *= 0.5
            b.set_particles(a_in.copy())
            b.update(1.0 / 60.0)
            a.update_host(1.0 / 60.0, a_in, a_in)  # one buffer both ways
            assert a_in.tobytes() == b.particles().tobytes()
    finally:
        for buf in bufs:
            buf.free()


@pytest.mark.parametrize("offset", [0, 16])
def test_batch(gpu, offset):
    specs = batch_specs(9, 600, 3000, seed=5)
    params = [scene_params(s) for s in specs]
    states = [scene_particles(s, p) for s, p in zip(specs, params)]
    with Batch(params, states) as a, Batch(params, states) as b:
        n = a.num_particles
        buf = PinnedBuffer(32 * (n + 2))
        try:
            both = records(buf, n, offset, states[0].dtype)
            both[:] = a.particles()
            for _ in range(3):
                cur = both.copy()
                a.step_host(1e-3, both, both)
                b.set_particles(cur)
                b.step(1e-3, 1)
                assert both.tobytes() == b.particles().tobytes()
        finally:
            buf.free()
