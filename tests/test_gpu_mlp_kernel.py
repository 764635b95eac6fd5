"""The kernel that runs two layers and their LayerNorm (wc_nn_mlp) is the one that inference takes: it
launches (it stands aside without a word where the compiler gave it another number of registers),
and its rows are those of the layers one after the other, bit for bit, from a single row to several
ragged tiles per block, with and without the gathered rows."""
import ctypes as C

import pytest

from test_gpu_nn import rnd, torch  # noqa: F401  (torch: the module's fixture)
from watercube_gb300 import _abi

pytestmark = pytest.mark.gpu


def call(lib, fn, desc, torch, *more):  # noqa: F811
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert getattr(lib, fn)(C.byref(desc), err.data_ptr(), None, *more) == _abi.WC_OK, lib.wc_last_error().decode()
    torch.cuda.synchronize()
    assert int(err.item()) == 0


def describe(cls, **kw):
    d = cls()
    for k, v in kw.items():
        setattr(d, k, v.data_ptr() if hasattr(v, "data_ptr") else v)
    return d


@pytest.mark.parametrize("m", [1, 127, 129, 152 * 128 * 2 + 77])
@pytest.mark.parametrize("k,gather,bias", [(16, False, True), (32, False, False), (128, False, True), (128, True, True), (128, True, False)])
def test_rows_of_the_layers_in_turn(wclib, torch, m, k, gather, bias):  # noqa: F811
    g = torch.Generator().manual_seed(m + k)
    a, w1, w2 = rnd(torch, m, k, seed=1), rnd(torch, 128, k, seed=2) * 0.2, rnd(torch, 128, 128, seed=3) * 0.1
    b1, b2, gamma, beta = (torch.randn(128, generator=g).cuda() for _ in range(4))
    rows = {}
    if gather:
        n = 700
        rows = dict(add1=rnd(torch, n, 128, seed=4), add2=rnd(torch, n, 128, seed=5),
                    add1_idx=torch.randint(0, n, (m,), generator=g).sort().values.int().cuda(),
                    add2_idx=torch.randint(0, n, (m,), generator=g).int().cuda())
    hidden = torch.zeros(m, 128, dtype=torch.bfloat16, device="cuda")
    ref, out = torch.zeros_like(hidden), torch.full((m + 8, 128), 3.0, dtype=torch.bfloat16, device="cuda")
    layer = dict(m=m, n=128, lda=128, ldb=128, ldc=128)
    first = describe(_abi.GemmDesc, **{**layer, "lda": k, "ldb": k}, k=k, k_chunk=128, a=a, b=w1, relu=1, c_bf16=hidden,
                     ld_add=128, **rows, **({"bias": b1} if bias else {}))
    second = describe(_abi.GemmDesc, **layer, k=128, k_chunk=128, a=hidden, b=w2, c_bf16=ref, ln_gamma=gamma, ln_beta=beta,
                      **({"bias": b2} if bias else {}), **({"ln_resid": a} if gather else {}))
    call(wclib, "wc_nn_gemm", first, torch)
    call(wclib, "wc_nn_gemm", second, torch)
    launched = C.c_int(0)
    mlp = describe(_abi.MlpDesc, m=m, k=k, a=a, w1=w1, w2=w2, gamma=gamma, beta=beta, out=out, **rows,
                   **({"b1": b1, "b2": b2} if bias else {}))
    call(wclib, "wc_nn_mlp", mlp, torch, C.byref(launched))
    assert launched.value == 1
    assert torch.equal(out[:m], ref)
    assert bool((out[m:] == 3.0).all())


def test_operands_it_leaves_to_the_layers(wclib, torch):  # noqa: F811
    a, out = rnd(torch, 64, 136), torch.zeros(64, 128, dtype=torch.bfloat16, device="cuda")
    w1, w2, v = rnd(torch, 128, 136), rnd(torch, 128, 128), torch.zeros(132, device="cuda")
    for kw in (dict(k=136, gamma=v), dict(k=128, gamma=v[1:])):  # too wide; not aligned
        launched = C.c_int(1)
        call(wclib, "wc_nn_mlp", describe(_abi.MlpDesc, **{**dict(m=64, a=a, w1=w1, w2=w2, beta=v, out=out), **kw}), torch,
             C.byref(launched))
        assert launched.value == 0
    assert not out.any()
