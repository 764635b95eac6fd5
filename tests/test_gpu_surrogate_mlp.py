"""Inference runs an edge or encoder block (two layers and their LayerNorm) as one kernel: its
predictions against the training forward's separate layers at edge counts of less than one tile of
128 rows, a ragged few, and several tiles per block. Both round the same values to BF16 (2^-9
relative) and differ by the FP32 summation order of the LayerNorm, which can move single roundings:
1e-2 of the norm, the bound of the two forwards elsewhere."""
import numpy as np
import pytest

from test_gpu_surrogate import perturbed_params, scene
from watercube_gb300.fluid import Fluid
from watercube_gb300.surrogate import Surrogate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers,n", [(1, 8), (2, 27), (1, 129), (2, 1000), (1, 30000)])
def test_inference_matches_training_forward(gpu, layers, n):
    p, state, hist, target = scene(n, seed=layers)
    with Surrogate(layers=layers, seed=7) as s, Fluid("mlp", p) as f:
        s.set_params(perturbed_params(s, seed=5))
        f.setup(state)
        s.sample(f, 1e-3, hist, target)
        s.forward_backward(True)
        a = s.predictions()[:, :3]
        s.forward_backward(False)
        b = s.predictions()[:, :3]
        s.forward_backward(False)
        assert np.array_equal(b, s.predictions()[:, :3])
    d = np.linalg.norm(b - a) / np.linalg.norm(a)
    assert d <= 1e-2, d
