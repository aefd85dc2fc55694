"""Lists that mix ops of few rows, which are launched early, with ops of more rows, which are not: the same bits as the ops one by one."""
import ctypes as C
import random

import pytest
import torch

pytestmark = pytest.mark.gpu
W, ROWS = 1024, 4


def chain(rows_of, x, w32, w, seg):
    """Each op reads rows that the one in front wrote: products, norms, and grouped products of four rows behind any of them."""
    from qwen3_tts_cuda_graphs_b200 import codec as K

    bufs, ops = [x], []
    for kind, M in rows_of:
        a, o = bufs[-1], K.Op()
        y = a.clone()      # (rows that the op does not write)
        o.M, o.N, o.A, o.lda, o.C, o.ldc, o.flags = M, W, a.data_ptr(), W, y.data_ptr(), W, K.F_OUT_F32
        if kind == "product":
            o.kind, o.K, o.taps, o.cin, o.a_rows, o.col_mod, o.B, o.reserved, o.flags = K.K_GEMM, W, 1, W, ROWS, W, w32.data_ptr(), 1, o.flags | K.F_F32
        elif kind == "norm":
            o.kind, o.i0, o.f0 = K.K_GNORM, 1, 1e-6
        else:
            o.kind, o.K, o.i0, o.B, o.p0, o.flags = K.K_GGEMM, W, 2, w.data_ptr(), seg.data_ptr(), o.flags | K.F_A_F32
        ops.append(o)
        bufs.append(y)
    return ops, bufs


LINE = [("product", 2), ("norm", 3), ("product", 2), ("norm", 1), ("experts", 4), ("norm", 2), ("product", 3), ("product", 1), ("norm", 4), ("norm", 2), ("experts", 4), ("product", 1)]


@pytest.mark.parametrize("seed", range(6))
def test_same_bits_as_one_by_one(seed):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    lib, r = K.load_lib(), random.Random(seed)
    rows_of = LINE if seed == 0 else [("experts", 4) if r.random() < 0.2 else (r.choice(["product", "norm"]), r.randint(1, 4)) for _ in range(40)]
    g = torch.Generator(device="cuda").manual_seed(seed)
    x, w32 = torch.randn(ROWS, W, device="cuda", generator=g), torch.randn(2, W, W, device="cuda", generator=g) / W ** 0.5
    w = w32.bfloat16()
    seg = torch.tensor([0, 2, 4], device="cuda", dtype=torch.int32)
    ops, bufs = chain(rows_of, x, w32, w, seg)
    stream = torch.cuda.current_stream().cuda_stream
    for o in ops:
        assert lib.fq3c_run((K.Op * 1)(o), 1, stream) == 0, lib.fq3c_last_error()
        torch.cuda.synchronize()
    want = [b.clone() for b in bufs]
    assert all(b.isfinite().all() for b in want)
    arr, graph = (K.Op * len(ops))(*ops), C.c_void_p()
    assert lib.fq3c_graph_create(arr, len(ops), C.byref(graph)) == 0, lib.fq3c_last_error()
    for turn in range(20):
        for b, (_, M) in zip(bufs[1:], rows_of):
            b[:M] = 100.0 + turn      # what an op writes is wrong until it has
        assert (lib.fq3c_graph_launch(graph, stream) if turn % 2 else lib.fq3c_run(arr, len(ops), stream)) == 0, lib.fq3c_last_error()
        torch.cuda.synchronize()
        assert all(torch.equal(b, ref) for b, ref in zip(bufs, want))
    lib.fq3c_graph_destroy(graph)
