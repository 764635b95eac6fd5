"""GEMMs in a row on one stream start before the previous one has ended (its results are waited for
inside): chains in which each reads what the one before wrote, a weight gradient over them and a
copy in between, give the bits of the same calls with a synchronisation after each; likewise
replayed from a captured graph."""
import ctypes as C

import pytest

from watercube_gb300 import _abi

pytestmark = pytest.mark.gpu


def calls(torch, m, n=128):
    g = torch.Generator().manual_seed(m)
    x = (torch.randn(m, n, generator=g)).to(torch.bfloat16).cuda()
    w = (torch.randn(n, n, generator=g) * 0.12).to(torch.bfloat16).cuda()
    gamma, beta = torch.ones(n, device="cuda"), torch.zeros(n, device="cuda")
    bufs = [torch.zeros(m, n, dtype=torch.bfloat16, device="cuda") for _ in range(3)]
    chunk = 192
    part = torch.zeros((m + chunk - 1) // chunk, n, n, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    descs = []

    def add(**kw):
        d = _abi.GemmDesc()
        for k, v in kw.items():
            setattr(d, k, v.data_ptr() if hasattr(v, "data_ptr") else v)
        descs.append(d)

    layer = dict(m=m, n=n, k=n, k_chunk=n, lda=n, b=w, ldb=n, ldc=n)
    for _ in range(4):
        add(a=bufs[0], relu=1, c_bf16=bufs[1], **layer)
        add(a=bufs[1], c_bf16=bufs[2], ln_gamma=gamma, ln_beta=beta, ln_resid=bufs[1], **layer)
        add(a=bufs[2], c_bf16=bufs[0], **layer)  # overwrites what the first of the three reads
    add(m=n, n=n, k=m, k_chunk=chunk, a=bufs[1], lda=n, a_transposed=1, b=bufs[0], ldb=n, b_rowmajor=1, c_f32=part,
        ldc=n, split_stride=n * n)
    return x, w, gamma, beta, bufs, part, err, descs


@pytest.mark.parametrize("m", [1, 257, 20000, 100000])
def test_chain(wclib, m):
    import torch

    x, w, gamma, beta, bufs, part, err, descs = calls(torch, m)
    stream = torch.cuda.Stream()

    def run(sync, s):
        with torch.cuda.stream(s):
            bufs[0].copy_(x)
            for d in descs:
                assert wclib.wc_nn_gemm(C.byref(d), err.data_ptr(), C.c_void_p(s.cuda_stream)) == _abi.WC_OK
                if sync:
                    s.synchronize()

    def result():
        torch.cuda.synchronize()
        assert int(err.item()) == 0
        return [t.clone() for t in (*bufs, part)]

    torch.cuda.synchronize()
    run(True, stream)
    ref = result()
    for _ in range(3):
        for t in (*bufs, part):
            t.zero_()
        torch.cuda.synchronize()
        run(False, stream)
        assert all(torch.equal(a, b) for a, b in zip(result(), ref))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run(False, torch.cuda.current_stream())
    for _ in range(2):
        for t in (*bufs, part):
            t.zero_()
        graph.replay()
        assert all(torch.equal(a, b) for a, b in zip(result(), ref))
