"""An extraction that fails leaves the mesh of the one before as it was: the triangles go out before the
host has read the error word, so the kernel that writes them has to look at it."""
import numpy as np
import pytest

from helpers import fluid
from watercube_gb300 import _abi
from watercube_gb300.fluid import dam_break_params, finalize, generate_dam_break

pytestmark = pytest.mark.gpu


def test_mesh_survives_a_collapsed_state(gpu):
    from watercube_gb300.surface import Surface

    p = finalize(dam_break_params(9000))
    good = generate_dam_break(p, 1)
    bad = good.copy()
    bad["position"] = bad["position"] * np.float32(0.9) + np.float32(0.05)  # another surface
    bad["position"][:6500] = 0.5 * p.bin_size  # and more particles in a row of cells than are evaluated
    with fluid(p, good) as f, Surface(40) as s:
        count = s.extract(f)
        mesh = s.triangles()
        assert count > 500
        for _ in range(2):
            f.set_particles(bad)
            with pytest.raises(_abi.WatercubeError) as e:
                s.extract(f)
            assert e.value.status == _abi.WC_ERR_NUMERIC
            assert np.array_equal(s.triangles(), mesh)
        f.set_particles(good)
        assert s.extract(f) == count and np.array_equal(s.triangles(), mesh)


def test_mesh_survives_a_scan_that_gives_up(gpu, wclib):
    """Its list of cubes is incomplete (the bounded-wait test hook makes the look-back run out)."""
    from watercube_gb300.surface import Surface

    p = finalize(dam_break_params(9000))
    st = generate_dam_break(p, 1)
    with fluid(p, st) as f, Surface(40) as s:
        count = s.extract(f)
        mesh = s.triangles()
        _abi.check(wclib.wc_debug_scan_stall(1, 64))
        try:
            with pytest.raises(_abi.WatercubeError) as e:
                s.extract(f)
            assert e.value.status == _abi.WC_ERR_TIMEOUT
        finally:
            _abi.check(wclib.wc_debug_scan_stall(0, 0))
        assert np.array_equal(s.triangles(), mesh)
        with pytest.raises(_abi.WatercubeError):
            f.synchronize()  # the fluid's own sort gave up as well
        f.set_particles(st)
        assert s.extract(f) == count and np.array_equal(s.triangles(), mesh)
