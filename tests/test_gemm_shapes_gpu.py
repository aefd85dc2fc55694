"""The tcgen05 GEMM on both sides of the lines between its launch shapes (few rows, one wide CTA per SM, two CTAs per SM, split sums)."""
import pytest
import torch

from test_gemm_gpu import SEVEN, launch, make_op, product

pytestmark = pytest.mark.gpu

# rows, columns, inputs per tap, taps, split allowed | of the f32 launch: its shape, the columns of a tile, the parts of its sums (held to the plan in test_gemm_plan_cpu.py)
WIDE, EIGHT, TWO = 0, 1, 2      # one CTA per SM with sixteen or eight epilogue warps, two with eight each
CASES = [(64, 6144, 1024, (0,), False, EIGHT, 64, 1), (65, 6144, 1024, (0,), False, WIDE, 64, 1),      # eight and sixteen epilogue warps
         (64, 512, 256, (0,), False, TWO, 16, 1), (65, 512, 256, (0,), False, TWO, 16, 1), (700, 208, 192, (0,), False, TWO, 16, 1), (1900, 176, 64, (0,), False, TWO, 16, 1),      # one piece a tile
         (20000, 96, 96, (0,), False, TWO, 32, 1), (9600, 192, 256, (0,), False, TWO, 64, 1), (9600, 192, 320, (0,), False, WIDE, 64, 1), (20000, 96, 48, (-1, 0), False, TWO, 32, 1),      # up to four k-blocks
         (20000, 96, 40, (-1, 0), False, None, None, None),      # c_in of 8 modulo 16: another kernel
         # 3, 5, 7 and 13 column pieces, which four groups of warps share unevenly
         (2500, 256, 128, (0,), False, WIDE, 48, 1), (6000, 208, 512, (0,), False, WIDE, 80, 1), (9600, 112, 512, (0,), False, WIDE, 112, 1), (3000, 1200, 512, (0,), False, WIDE, 208, 1),
         (64, 1024, 1536, (0,), True, EIGHT, 32, 1), (64, 1024, 2048, (0,), True, EIGHT, 64, 8), (100, 1024, 3072, (0,), True, EIGHT, 64, 8), (130, 1024, 3072, (0,), True, EIGHT, 64, 4),
         (40, 2048, 1024, (0,), True, EIGHT, 32, 1), (17, 48, 2048, (0,), True, EIGHT, 32, 8), (200, 512, 512, SEVEN, True, EIGHT, 64, 8), (130, 2048, 6144, (0,), True, EIGHT, 64, 2),
         (200, 2048, 6144, (0,), True, EIGHT, 64, 2)]


@pytest.mark.parametrize("M,N,cin,offs,split", [c[:5] for c in CASES])
def test_product_residual_snake_and_units(M, N, cin, offs, split):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    g = torch.Generator(device="cuda").manual_seed(M * 31 + N)
    A = torch.randn(M, cin, device="cuda", generator=g).bfloat16()
    B = (torch.randn(N, len(offs) * cin, device="cuda", generator=g) / (len(offs) * cin) ** 0.5).bfloat16()
    ws = torch.zeros(8 * M * (N + 8), device="cuda") if split else None
    want, mag = product(A, B, M, cin, offs)
    sums = len(offs) * cin * 2.0 ** -24 * mag      # f32 sums in any order
    out = torch.full((M + 1, N), 7.0, device="cuda")
    launch([make_op(A, B, out, M, N, cin, offs, K.F_OUT_F32 | K.F_NOROUND, ws=ws)])
    assert ((out[:M].double() - want).abs() <= sums).all() and (out[M] == 7).all()
    # residual and SnakeBeta: the sum is rounded, its sum with the residual is rounded, and the second output is that value's own, rounded
    res, freq, inv = torch.randn(M, N, device="cuda", generator=g).bfloat16(), torch.rand(N, device="cuda", generator=g) + 0.5, torch.rand(N, device="cuda", generator=g)
    out, out2 = (torch.zeros(M, N, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    o = make_op(A, B, out, M, N, cin, offs, K.F_SNAKE2, res=res, ws=ws)
    o.p0, o.p1, o.C2 = freq.data_ptr(), inv.data_ptr(), out2.data_ptr()
    launch([o])
    exact = want + res.double()
    assert ((out.double() - exact).abs() <= 1.01 * 2.0 ** -8 * (want.abs() + exact.abs()) + 2 * sums).all()
    snake = out.double() + inv.double() * torch.sin(out.double() * freq.double()) ** 2
    assert ((out2.double() - snake).abs() <= 1.01 * 2.0 ** -8 * snake.abs() + 2.0 ** -20).all()
    out = torch.zeros(M, N // 2, device="cuda", dtype=torch.bfloat16)
    launch([make_op(A, B, out, M, N, cin, offs, K.F_SWIGLU | K.F_NOROUND, ws=ws)])
    gate, up = want[:, 0::2], want[:, 1::2]
    unit = gate * torch.sigmoid(gate) * up
    slack = 1.1 * sums[:, 0::2] * up.abs() + (gate * torch.sigmoid(gate)).abs() * sums[:, 1::2]      # silu's slope is at most 1.1
    assert ((out.double() - unit).abs() <= 1.01 * 2.0 ** -8 * unit.abs() + slack + 2.0 ** -20 * unit.abs() + 1e-6).all()


# rows, columns, inputs, parts: two to eight of them, one and two to a CTA, runs of k-blocks of unequal length, the last CTA with one part less
@pytest.mark.parametrize("M,N,K,parts", [(39, 1024, 2048, 8), (90, 1024, 2048, 8), (73, 1024, 3072, 8), (128, 1024, 3072, 8), (33, 1024, 1792, 7), (33, 1024, 1536, 6), (17, 1024, 1280, 5), (140, 1024, 3072, 4), (64, 2048, 6144, 4),
                                         (262, 1024, 8192, 3), (33, 4096, 2048, 2), (200, 2048, 6144, 2), (8, 40, 1536, 6), (5, 1000, 2000, 8)])
def test_sums_come_in_parts_and_in_their_order(M, N, K, parts):
    """A split product is the f32 sum, in order, of the whole products of its runs of 64 inputs."""
    g = torch.Generator(device="cuda").manual_seed(M + K)
    A, B = torch.randn(M, K, device="cuda", generator=g).bfloat16(), (torch.randn(N, K, device="cuda", generator=g) / K ** 0.5).bfloat16()
    flags = 64 | 1024      # f32, as it is
    split, whole = torch.zeros(M, N, device="cuda"), torch.zeros(M, N, device="cuda")
    launch([make_op(A, B, split, M, N, K, flags=flags, ws=torch.zeros(8 * M * (N + 8), device="cuda"))])
    blocks = (K + 63) // 64
    for p in range(parts):
        lo, hi = 64 * (p * blocks // parts), min(K, 64 * ((p + 1) * blocks // parts))
        part = torch.zeros(M, N, device="cuda")
        launch([make_op(A[:, lo:hi].contiguous(), B[:, lo:hi].contiguous(), part, M, N, hi - lo, flags=flags)])
        whole += part
    assert torch.equal(split, whole)
