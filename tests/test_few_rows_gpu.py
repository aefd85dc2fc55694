"""Products of one row, whose entries go straight to the lanes: the same bits as that row among others, which are staged."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("N,Kd", [(1, 8), (7, 16), (130, 1024), (33, 1032), (64, 3072), (9, 4100), (1024, 2048)])
@pytest.mark.parametrize("off", [0, 1])      # entries in front of the rows: 0 whole 16-byte pieces, 1 staged
def test_one_row_as_among_others(N, Kd, f32, off):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    lib, dt = K.load_lib(), torch.float32 if f32 else torch.bfloat16
    g = torch.Generator(device="cuda").manual_seed(N + Kd)
    w = (torch.randn(N, Kd, device="cuda", generator=g) / Kd ** 0.5).to(dt)
    x = torch.randn(3 * (Kd + 8), device="cuda", generator=g).to(dt)
    out = []
    for M in (1, 2):
        y = torch.full((M, N), 9.0, device="cuda")
        for early in (0, 1):
            o = K.Op()
            o.kind, o.flags, o.M, o.N, o.K, o.taps, o.cin, o.a_rows, o.lda, o.ldc, o.col_mod = K.K_GEMM, K.F_OUT_F32 | K.F_NOROUND | (K.F_F32 if f32 else 0), M, N, Kd, 1, Kd, M, Kd + 8, N, N
            o.A, o.B, o.C, o.reserved = x.data_ptr() + off * x.element_size(), w.data_ptr(), y.data_ptr(), early
            assert lib.fq3c_run((K.Op * 1)(o), 1, torch.cuda.current_stream().cuda_stream) == 0, lib.fq3c_last_error()
            out.append(y[0].clone())
    assert all(torch.equal(out[0], t) for t in out)
    ref = w.double() @ x[off:off + Kd].double()
    # sums of Kd products in 32 bits, in 32 chains and a tree: at most Kd / 32 + 8 roundings of partial sums
    bound = (Kd / 32 + 8) * 2.0 ** -24 * (w.double().abs() @ x[off:off + Kd].double().abs())
    assert ((out[0].double() - ref).abs() <= bound).all()
