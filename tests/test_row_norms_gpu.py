"""RMSNorm of bf16 rows, a warp per row: long and short rows, pitches, and rows without whole 16-byte pieces."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,pad", [(1, 8, 0), (3, 64, 0), (5, 1016, 8), (39, 1024, 0), (7, 1032, 0), (4, 2048, 24), (2, 5000, 0), (261, 1024, 0), (9, 100, 3)])
def test_rows(M, N, pad):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    g = torch.Generator(device="cuda").manual_seed(N)
    x, w = torch.randn(M, N + pad, device="cuda", generator=g).bfloat16(), torch.rand(N, device="cuda", generator=g) + 0.5
    out = torch.full((M + 1, N + pad), 9.0, device="cuda", dtype=torch.bfloat16)
    o = K.Op()
    o.kind, o.M, o.N, o.A, o.lda, o.a_rows, o.C, o.ldc, o.col_mod, o.scale, o.f0 = K.K_RMSNORM, M, N, x.data_ptr(), N + pad, M, out.data_ptr(), N + pad, N, w.data_ptr(), 1e-5
    lib = K.load_lib()
    assert lib.fq3c_run((K.Op * 1)(o), 1, torch.cuda.current_stream().cuda_stream) == 0, lib.fq3c_last_error()
    r = x[:, :N].double()
    want = r / torch.sqrt((r * r).mean(-1, keepdim=True) + 1e-5) * w.double()
    # two roundings to bf16 (half a unit is 2^-8 at most: the scaled row, the result) and f32 sums
    assert ((out[:M, :N].double() - want).abs() <= (2.02 * 2.0 ** -8 + N * 2.0 ** -24) * want.abs() + 1e-30).all()
    assert (out[M] == 9).all() and (out[:M, N:] == 9).all()
