"""The TMA GEMM's epilogue (results and row operands through shared memory) at the edges of its
tiles: ragged row counts, fewer than 128 columns, each output form, FP32 accumulation, one and two
gathered rows, more k than the operand ring holds, and results whose rows TMA cannot address."""
import pytest

from test_gpu_nn import close, rnd, run, torch  # noqa: F401  (torch: the module's fixture)

pytestmark = pytest.mark.gpu

BF16 = 1e-3 + 2.0 ** -8  # FP32 sums in another order, then one BF16 rounding (half an ulp of 2^-8)


@pytest.mark.parametrize("m", [1, 31, 33, 127, 129, 19457, 40001])
@pytest.mark.parametrize("form", ["bf16", "f32", "accumulate", "both"])
@pytest.mark.parametrize("n,k", [(128, 128), (16, 64), (72, 32)])
def test_outputs(wclib, torch, m, form, n, k):  # noqa: F811
    a, wt, bias = rnd(torch, m, k, seed=1), rnd(torch, n, k, seed=2), torch.randn(n, device="cuda")
    ref = a.float() @ wt.float().t() + bias
    guard = 64  # rows past the matrix stay untouched
    c = torch.full((m + guard, n), 3.0, device="cuda")
    c16 = torch.full((m + guard, n), 3.0, dtype=torch.bfloat16, device="cuda")
    kw = dict(m=m, n=n, k=k, a=a, lda=k, b=wt, ldb=k, bias=bias, ldc=n)
    if form != "f32":
        ref = torch.relu(ref)
        kw["relu"] = 1
    if form != "bf16":
        kw["c_f32"] = c
    if form in ("bf16", "both"):
        kw["c_bf16"] = c16
    if form == "accumulate":
        kw["accumulate"] = 1
    run(wclib, torch, **kw)
    if form != "bf16":
        close(c[:m], ref + (3.0 if form == "accumulate" else 0.0))
    if form in ("bf16", "both"):
        close(c16[:m], ref, rel=BF16)
    assert bool((c[m:] == 3.0).all()) and bool((c16[m:] == 3.0).all())


@pytest.mark.parametrize("m", [5, 128, 20000, 39000])
@pytest.mark.parametrize("k", [128, 256, 384])
@pytest.mark.parametrize("which", ["first", "second", "both"])
def test_gathered_rows(wclib, torch, m, k, which):  # noqa: F811
    n = 128
    a, wt = rnd(torch, m, k, seed=1), rnd(torch, n, k, seed=2)
    ref = a.float() @ wt.float().t()
    kw, held = dict(m=m, n=n, k=k, a=a, lda=k, b=wt, ldb=k, ld_add=136, relu=1, ldc=n), []
    for q, name in enumerate(("add1", "add2")):
        if which in ("both", ("first", "second")[q]):
            rows = rnd(torch, 777, 136, seed=3 + q)
            idx = torch.randint(0, 777, (m,), device="cuda", dtype=torch.int32)
            kw[name], kw[name + "_idx"] = rows, idx
            held += [rows, idx]
            ref = ref + rows[idx.long(), :n].float()
    c16 = torch.zeros(m, n, dtype=torch.bfloat16, device="cuda")
    run(wclib, torch, c_bf16=c16, **kw)
    close(c16, torch.relu(ref), rel=BF16)


def test_unaligned_result(wclib, torch):  # noqa: F811
    m, n, k = 300, 128, 128
    a, wt = rnd(torch, m, k, seed=1), rnd(torch, n, k, seed=2)
    c = torch.zeros(m * 131 + 1, device="cuda")  # rows of 131 floats from an odd address
    run(wclib, torch, m=m, n=n, k=k, a=a, lda=k, b=wt, ldb=k, c_f32=c[1:], ldc=131)
    close(c[1:].view(m, 131)[:, :n], a.float() @ wt.float().t())


@pytest.mark.parametrize("m,n", [(128, 128), (16, 128), (128, 16), (72, 40), (8, 8)])
@pytest.mark.parametrize("k,chunk", [(1, 64), (63, 64), (65, 64), (1000, 128), (40003, 192)])
def test_weight_gradient_splits(wclib, torch, m, n, k, chunk):  # noqa: F811
    """X^T dY per split of the rows, the last one ragged; the tolerance is close()'s, of FP32 sums of
    exact products in another order."""
    x, dy = rnd(torch, k, m, seed=1), rnd(torch, k, n, seed=2)
    parts = -(-k // chunk)
    out = torch.full((parts + 1, m, n), 7.0, device="cuda")
    run(wclib, torch, m=m, n=n, k=k, k_chunk=chunk, a=x, lda=m, a_transposed=1, b=dy, ldb=n, b_rowmajor=1, c_f32=out,
        ldc=n, split_stride=m * n)
    ref = torch.stack([p.float().t() @ q.float() for p, q in zip(x.split(chunk), dy.split(chunk))])
    close(out[:parts], ref)
    assert bool((out[parts] == 7.0).all())


@pytest.mark.parametrize("m", [1, 129, 20001])
@pytest.mark.parametrize("split,k", [(128, 256), (64, 200), (40, 128)])  # 40: inside a slice, the cp.async kernel
def test_two_sources(wclib, torch, m, split, k):  # noqa: F811
    n = 128
    x, y, wt = rnd(torch, m, split, seed=1), rnd(torch, m, k - split, seed=2), rnd(torch, n, k, seed=3)
    c16 = torch.zeros(m, n, dtype=torch.bfloat16, device="cuda")
    run(wclib, torch, m=m, n=n, k=k, a=x, lda=split, a2=y, lda2=k - split, k_split=split, b=wt, ldb=k, relu=1, c_bf16=c16,
        ldc=n)
    close(c16, torch.relu(torch.cat([x, y], 1).float() @ wt.float().t()), rel=BF16)
