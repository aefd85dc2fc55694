"""RMSNorm of bf16 rows, a warp per row: long and short rows, pitches, and rows without whole 16-byte pieces, alone and behind a product."""
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


def norm_op(x, w, out, M, N):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    o = K.Op()
    o.kind, o.M, o.N, o.A, o.lda, o.a_rows, o.C, o.ldc, o.col_mod, o.scale, o.f0 = K.K_RMSNORM, M, N, x.data_ptr(), x.stride(0), M, out.data_ptr(), out.stride(0), N, w.data_ptr(), 1e-6
    return o


@pytest.mark.parametrize("M,N", [(3, 8), (5, 248), (33, 512), (17, 1016), (300, 1024), (4, 1288), (300, 2048), (2, 5000)])
def test_both_kernels_have_the_same_bits(M, N):
    """Rows of whole pieces (a warp each) and the same rows at an odd pitch (a block each): one order of sums, so that a list's results do not move with its buffers."""
    from test_gemm_gpu import launch

    g = torch.Generator(device="cuda").manual_seed(N)
    x, w = (3 * torch.randn(M, N, device="cuda", generator=g)).bfloat16(), torch.rand(N, device="cuda", generator=g) + 0.5
    odd = torch.zeros(M, N + 3, device="cuda", dtype=torch.bfloat16)
    odd[:, :N] = x
    whole, apart = torch.zeros_like(x), torch.zeros_like(odd)
    launch([norm_op(x, w, whole, M, N), norm_op(odd, w, apart, M, N)])
    assert torch.equal(whole, apart[:, :N])


@pytest.mark.parametrize("M,N,cin,offs,split", [(70, 1024, 264, (-1, 0), True), (70, 1024, 264, (-1, 0), False), (39, 1024, 2048, (0,), True), (300, 1024, 256, (0,), False), (70, 1000, 72, (-1, 0), False)])
def test_norm_behind_a_product_has_the_bits_of_the_op(M, N, cin, offs, split):
    """Every kernel that a product with a norm behind it comes to: split sums through a workspace, tcgen05 tiles split and whole, rows without whole k-blocks."""
    from test_gemm_gpu import launch, make_op

    g = torch.Generator(device="cuda").manual_seed(N + cin)
    A, w = torch.randn(M, cin, device="cuda", generator=g).bfloat16(), torch.rand(N, device="cuda", generator=g) + 0.5
    B = (torch.randn(N, len(offs) * cin, device="cuda", generator=g) / (len(offs) * cin) ** 0.5).bfloat16()
    ws = torch.zeros(8 * M * N, device="cuda") if split else None
    got = []
    for fused in (True, False):
        out, normed = (torch.zeros(M, N, device="cuda", dtype=torch.bfloat16) for _ in range(2))
        o = make_op(A, B, out, M, N, cin, offs, ws=ws)
        if fused:
            o.norm_out, o.norm_w, o.norm_ld, o.norm_eps = normed.data_ptr(), w.data_ptr(), N, 1e-6
        launch([o] if fused else [o, norm_op(out, w, normed, M, N)])
        got.append((out, normed))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
