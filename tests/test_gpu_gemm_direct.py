"""The forms of the TMA GEMM that write their results from the registers (few columns, rows of gathered
operands that are not whole or not aligned, results that TMA cannot address or shared memory cannot
hold) at the edges of its tiles. Tolerances: those of the epilogue through shared memory."""
import pytest

from test_gpu_gemm_epilogue import BF16
from test_gpu_nn import close, rnd, run, torch  # noqa: F401  (torch: the module's fixture)

pytestmark = pytest.mark.gpu

FORMS = {  # n, k, gathered operands, ld_add, ldc, outputs
    "n8": (8, 16, 0, 0, 8, "both"),
    "n5": (5, 64, 0, 0, 8, "f32"),
    "n32": (32, 128, 0, 0, 32, "bf16"),
    "gather_n64": (64, 128, 2, 64, 64, "bf16"),
    "gather_n16": (16, 64, 1, 24, 16, "both"),
    "gather_k384": (128, 384, 2, 128, 128, "bf16"),
    "gather_f32": (128, 256, 2, 128, 128, "f32"),
    "gather_both": (128, 128, 2, 128, 128, "both"),
    "gather_rows_132": (128, 128, 2, 132, 128, "bf16"),
    "rows_131": (128, 128, 0, 0, 131, "both"),
    "two_sources_n8": (8, 192, 0, 0, 8, "bf16"),
}


@pytest.mark.parametrize("m", [1, 129, 20001])
@pytest.mark.parametrize("form", FORMS)
def test_written_from_registers(wclib, torch, form, m):  # noqa: F811
    n, k, adds, ld_add, ldc, outputs = FORMS[form]
    a, wt, bias = rnd(torch, m, k, seed=1), rnd(torch, n, k, seed=2), torch.randn(n, device="cuda")
    ref, held = a.float() @ wt.float().t() + bias, []
    kw = dict(m=m, n=n, k=k, b=wt, ldb=k, bias=bias, relu=1, ldc=ldc)
    if form.startswith("two_sources"):
        parts = a[:, :64].contiguous(), a[:, 64:].contiguous()
        kw.update(a=parts[0], lda=64, a2=parts[1], lda2=k - 64, k_split=64)
    else:
        kw.update(a=a, lda=k)
    for q in range(adds):
        rows, idx = rnd(torch, 777, ld_add, seed=3 + q), torch.randint(0, 777, (m,), device="cuda", dtype=torch.int32)
        kw.update({f"add{q + 1}": rows, f"add{q + 1}_idx": idx, "ld_add": ld_add})
        held += [rows, idx]
        ref = ref + rows[idx.long(), :n].float()
    ref = torch.relu(ref)
    c, c16 = torch.full((m + 8, ldc), 3.0, device="cuda"), torch.full((m + 8, ldc), 3.0, dtype=torch.bfloat16, device="cuda")
    if outputs in ("f32", "both"):
        kw["c_f32"] = c
    if outputs in ("bf16", "both"):
        kw["c_bf16"] = c16
    run(wclib, torch, **kw)
    for out, used, rel in ((c, "c_f32" in kw, None), (c16, "c_bf16" in kw, BF16)):
        if used:
            close(out[:m, :n], ref, **({"rel": rel} if rel else {}))
        assert bool((out[m:] == 3.0).all()) and bool((out[:, n:] == 3.0).all())
