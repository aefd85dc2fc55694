"""SnakeBeta's sin^2 against float64, past the bf16 rounding of its outputs: with v = -1 and 1 / beta = 1 / sin^2 the sum v + sin^2 / beta is the error itself."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("magnitude", [1.6, 30.0, 1e3, 6e4, 2.49e5, 3e5, 2e6])
@pytest.mark.parametrize("fused", [False, True])
def test_sin_squared(magnitude, fused):
    from qwen3_tts_cuda_graphs_b200 import codec as K
    from test_gemm_gpu import launch, make_op

    N, M = 4096, 130
    g = torch.Generator(device="cuda").manual_seed(7)
    ea = (torch.rand(N, device="cuda", generator=g) * 2 - 1) * magnitude
    sq = torch.sin(ea.double()) ** 2
    ea = torch.where(sq > 0.02, ea, torch.full_like(ea, 1.0))      # (the quotient below magnifies the error)
    sq = torch.sin(ea.double()) ** 2
    ib = (1.0 / sq).float()
    out, out2 = torch.zeros(M, N, device="cuda", dtype=torch.bfloat16), torch.zeros(M, N, device="cuda", dtype=torch.bfloat16)
    if fused:      # the GEMM's second output: products of a single -1 x 1
        A, B = torch.zeros(M, 64, device="cuda", dtype=torch.bfloat16), torch.zeros(N, 64, device="cuda", dtype=torch.bfloat16)
        A[:, 0], B[:, 0] = -1.0, 1.0
        o = make_op(A, B, out, M, N, 64, flags=K.F_SNAKE2)
        o.C2, o.p0, o.p1 = out2.data_ptr(), ea.data_ptr(), ib.data_ptr()
    else:
        x = torch.full((M, N), -1.0, device="cuda", dtype=torch.bfloat16)
        o = K.Op()
        o.kind, o.M, o.N, o.A, o.lda, o.a_rows, o.C, o.ldc, o.col_mod = K.K_SNAKE, M, N, x.data_ptr(), N, M, out2.data_ptr(), N, N
        o.p0, o.p1 = ea.data_ptr(), ib.data_ptr()
    launch([o])
    err = (out2.double() - (ib.double() * sq - 1.0)).abs() / ib.double()
    # 1.2e-7 of sin^2; the sum's own rounding to f32 where it is not fused (2^-24 of 1 and of the product); sinf's 2 ulp beyond 2.5e5
    assert float(err.max()) < (1.2e-7 if magnitude < 2.5e5 else 2.8e-7) + (0.0 if fused else 2.0 ** -23)
    assert float((err ** 2).mean().sqrt()) < 4e-8 + (0.0 if fused else 2.0 ** -24)
