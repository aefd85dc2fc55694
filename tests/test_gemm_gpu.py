"""The tcgen05 GEMM of the op lists at the edges of its tiles, taps, splits and vector epilogues, against float64 products of the same bf16 operands."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def make_op(A, B, out, M, N, cin, offs=(0,), flags=0, res=None, bias=None, scale=None, ws=None, m_begin=0):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    o = K.Op()
    o.kind, o.flags, o.M, o.N, o.K, o.taps, o.cin = K.K_GEMM, flags, M, N, len(offs) * cin, len(offs), cin
    (o.a_rows, o.lda), o.ldc, o.col_mod, o.reserved, o.m_begin = A.shape, out.stride(0), N, 1, m_begin
    for i, t in enumerate(offs):
        o.tap_off[i] = t
    o.A, o.B, o.C = A.data_ptr(), B.data_ptr(), out.data_ptr()
    if res is not None:
        o.flags |= K.F_RESID
        o.res, o.ldr = res.data_ptr(), res.stride(0)
    if bias is not None:
        o.flags |= K.F_BIAS
        o.bias = bias.data_ptr()
    if scale is not None:
        o.flags |= K.F_SCALE
        o.scale = scale.data_ptr()
    if ws is not None:
        o.ws, o.ws_bytes = ws.data_ptr(), ws.numel() * 4
    return o


def launch(ops):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    lib = K.load_lib()
    arr = (K.Op * len(ops))(*ops)
    assert lib.fq3c_run(arr, len(ops), torch.cuda.current_stream().cuda_stream) == 0, lib.fq3c_last_error()
    torch.cuda.synchronize()
    assert lib.fq3c_wait_errors() == 0


def product(A, B, M, cin, offs):
    """float64 sums, and the sums of the products' magnitudes (f32 sums in any order are within K 2^-24 of them)."""
    y = torch.zeros(M, B.shape[0], device="cuda", dtype=torch.float64)
    mag = torch.zeros_like(y)
    for j, t in enumerate(offs):
        i = torch.arange(M, device="cuda") + t
        ok = (i >= 0) & (i < A.shape[0])
        X = torch.zeros(M, cin, device="cuda", dtype=torch.float64)
        X[ok] = A[i[ok], :cin].double()
        w = B[:, j * cin:(j + 1) * cin].double()
        y += X @ w.T
        mag += X.abs() @ w.abs().T
    return y, mag


SEVEN = tuple(range(-6, 1))
SHAPES = {"one row": (1, 16, 64, (0,), False), "few rows, split": (39, 1024, 2048, (0,), True), "rows behind a tile": (129, 1000, 200, (0,), False), "three tiles, split": (262, 1024, 3072, (0,), True),
          "many tiles": (1900, 4096, 256, (0,), False), "last k-block of 32": (300, 96, 96, SEVEN, False), "last k-block of 16": (130, 48, 80, (-2, 0), False), "narrow, K of 72": (300, 40, 72, (0,), False),
          "two taps": (513, 192, 192, (0, -1), False), "taps, split": (130, 768, 768, SEVEN, True), "eight rows, split": (8, 1024, 1024, (0,), True), "taps of 8 modulo 16": (70, 64, 72, (-1, 0), False)}


@pytest.mark.parametrize("name", SHAPES)
def test_product_and_epilogues(name):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    M, N, cin, offs, split = SHAPES[name]
    g = torch.Generator(device="cuda").manual_seed(len(name))
    A = torch.randn(M, cin, device="cuda", generator=g).bfloat16()
    B = (torch.randn(N, len(offs) * cin, device="cuda", generator=g) / (len(offs) * cin) ** 0.5).bfloat16()
    ws = torch.zeros(8 * M * (N + 8), device="cuda") if split else None
    want, mag = product(A, B, M, cin, offs)
    out = torch.full((M + 1, N), 7.0, device="cuda")
    launch([make_op(A, B, out, M, N, cin, offs, K.F_OUT_F32 | K.F_NOROUND, ws=ws)])
    assert ((out[:M].double() - want).abs() <= len(offs) * cin * 2.0 ** -24 * mag).all() and (out[M] == 7).all()
    # bf16 rows with bias, scale and residual: the sum's error, then four roundings of values below |sum| + |bias| and their sum with the residual
    res, bias, scale = torch.randn(M, N, device="cuda", generator=g).bfloat16(), torch.randn(N, device="cuda", generator=g), torch.rand(N, device="cuda", generator=g)
    out = torch.zeros(M, N, device="cuda", dtype=torch.bfloat16)
    launch([make_op(A, B, out, M, N, cin, offs, res=res, bias=bias, scale=scale, ws=ws)])
    exact = (want + bias.double()) * scale.double() + res.double()
    assert ((out.double() - exact).abs() <= 2.0 ** -8 * (2 * (want + bias.double()).abs() * scale.double() + exact.abs()) + 2.0 ** -20 * mag + 1e-6).all()
    if N % 4 == 0:      # gated units, on unrounded sums and on rounded ones
        for flags in (K.F_SWIGLU | K.F_NOROUND, K.F_SWIGLU):
            out = torch.zeros(M, N // 2, device="cuda", dtype=torch.bfloat16)
            launch([make_op(A, B, out, M, N, cin, offs, flags, ws=ws)])
            gate, up = want[:, 0::2], want[:, 1::2]
            unit = gate * torch.sigmoid(gate) * up
            # silu's slope is at most 1.1; rounded sums: gate, silu, up and the product are each rounded, else the result alone
            sums = len(offs) * cin * 2.0 ** -24 * (1.1 * mag[:, 0::2] * up.abs() + (gate * torch.sigmoid(gate)).abs() * mag[:, 1::2])
            rounds = unit.abs() if flags & K.F_NOROUND else 1.1 * (gate * up).abs() + 4 * unit.abs()
            assert ((out.double() - unit).abs() <= 1.01 * 2.0 ** -8 * rounds + sums + 2.0 ** -20 * unit.abs() + 1e-6).all()


def test_rows_from_m_begin_on_are_the_full_products_rows():
    A, B = torch.randn(400, 64, device="cuda").bfloat16(), torch.randn(96, 7 * 64, device="cuda").bfloat16()
    full, tail = (torch.full((400, 96), 3.0, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    launch([make_op(A, B, full, 400, 96, 64, SEVEN)])
    launch([make_op(A, B, tail, 400, 96, 64, SEVEN, m_begin=211)])
    assert torch.equal(full[211:], tail[211:]) and (tail[:211] == 3).all()


def test_a_chain_of_products_reads_what_the_one_in_front_wrote():
    """Launches of a list may begin before the ones in front have ended: forty dependent products, each held against its own input."""
    from qwen3_tts_cuda_graphs_b200 import codec as K

    ws = torch.zeros(8 * 39 * 520, device="cuda")
    W = [(torch.randn(512, 512, device="cuda") / 512 ** 0.5).bfloat16() for _ in range(40)]
    for rows in (39, 300):
        x = [torch.randn(rows, 512, device="cuda").bfloat16()] + [torch.zeros(rows, 512, device="cuda", dtype=torch.bfloat16) for _ in W]
        ops = [make_op(x[i], W[i], x[i + 1], rows, 512, 512, ws=ws if rows == 39 and i % 2 else None) for i in range(40)]
        for _ in range(3):
            for t in x[1:]:
                t.zero_()
            launch(ops)
            for i in range(40):
                want, mag = product(x[i], W[i], rows, 512, (0,))
                assert ((x[i + 1].double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -15 * mag).all(), i


@pytest.mark.parametrize("M, N, K", [(9, 643, 256), (33, 20, 128), (701, 1286, 192), (260, 17, 64), (1501, 385, 72)])
@pytest.mark.parametrize("scratch", [True, False])
def test_widths_between_whole_pieces(M, N, K, scratch):
    """A product whose width is no multiple of 16: with scratch columns behind it only those are written, without none."""
    from qwen3_tts_cuda_graphs_b200 import codec as C

    torch.manual_seed(M)
    A, B = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(N, K, device="cuda").bfloat16()
    want, mag = product(A, B, M, K, (0,))
    wide = (N + 15) // 16 * 16
    for dtype, flags in ((torch.float32, C.F_OUT_F32 | C.F_NOROUND), (torch.bfloat16, 0)):
        out = torch.full((M + 1, wide + 16), 7.0, device="cuda", dtype=dtype)
        o = make_op(A, B, out, M, N, K, flags=flags)
        o.reserved = 9 if scratch else 1
        launch([o])
        err = K * 2.0 ** -24 * mag + (2.0 ** -8 * want.abs() if dtype == torch.bfloat16 else 0)
        assert ((out[:M, :N].double() - want).abs() <= err).all()
        assert (out[:, wide if scratch else N:] == 7).all() and (out[M] == 7).all()


# 39 rows: staged, from shared memory; 9000 rows of 768 columns: a CTA goes on to another column tile; 300 x 200: a last piece of eight columns
@pytest.mark.parametrize("M, N, cin, col_mod", [(39, 384, 128, 384), (300, 200, 64, 200), (300, 768, 64, 192), (9000, 768, 64, 256)])
@pytest.mark.parametrize("what", ["gelu", "silu", "clamp", "relu2", "snake"])
def test_vector_epilogues(M, N, cin, col_mod, what):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    g = torch.Generator(device="cuda").manual_seed(M + N)
    A, B = torch.randn(M, cin, device="cuda", generator=g).bfloat16(), (torch.randn(N, cin, device="cuda", generator=g) / cin ** 0.5).bfloat16()
    bias, res = torch.randn(col_mod, device="cuda", generator=g), torch.randn(M, N, device="cuda", generator=g).bfloat16()
    want, mag = product(A, B, M, cin, (0,))
    z = want + bias.double().repeat(N // col_mod)
    err = 2.0 ** -20 * mag + 1e-6
    out = torch.zeros(M, N, device="cuda", dtype=torch.float32 if what == "relu2" else torch.bfloat16)
    flags = dict(gelu=K.F_GELU, silu=K.F_SILU, clamp=K.F_CLAMP, relu2=K.F_RELU2 | K.F_OUT_F32 | K.F_NOROUND, snake=K.F_SNAKE2)[what]
    o = make_op(A, B, out, M, N, cin, flags=flags, bias=bias, res=res if what == "snake" else None)
    o.col_mod = col_mod
    if what == "snake":
        out2 = torch.zeros_like(out)
        ea, ib = torch.rand(col_mod, device="cuda", generator=g) * 4, torch.rand(col_mod, device="cuda", generator=g)
        ea[3], ea[7] = 2e5, 1e6      # far from zero, and beyond the range of the reduction
        o.C2, o.p0, o.p1 = out2.data_ptr(), ea.data_ptr(), ib.data_ptr()
    launch([o])
    r = 1.01 * 2.0 ** -8      # bf16 keeps 8 bits: half of the last one
    if what == "gelu":
        y = torch.nn.functional.gelu(z)
        assert ((out.double() - y).abs() <= r * (1.13 * z.abs() + y.abs()) + err).all()
    elif what == "silu":
        y = z * torch.sigmoid(z)
        assert ((out.double() - y).abs() <= r * (1.1 * z.abs() + y.abs()) + err).all()
    elif what == "clamp":
        assert ((out.double() - z.clamp(-1, 1)).abs() <= r * z.abs() + err).all()
    elif what == "relu2":
        y = z.clamp(min=0)
        assert ((out.double() - y * y).abs() <= 2 * y * err + err ** 2 + 2.0 ** -23 * y * y).all()
    else:
        y = z + res.double()
        assert ((out.double() - y).abs() <= r * (z.abs() + y.abs()) + err).all()
        x = (out.float() * ea.repeat(N // col_mod)).double()      # what the kernel takes the sine of
        y = out.double() + ib.double().repeat(N // col_mod) * torch.sin(x) ** 2
        assert ((out2.double() - y).abs() <= r * y.abs() + 4e-7).all()


@pytest.mark.parametrize("M, m_begin", [(1, 0), (255, 0), (256, 0), (257, 0), (257, 256), (700, 130)])
@pytest.mark.parametrize("offs", [SEVEN, tuple(9 * t for t in SEVEN), (1, 0), (-3, 4)])
def test_one_output_channel(M, m_begin, offs):
    """The convolution to a single channel: last blocks, rows in front of and behind the input, spread taps, rows from m_begin on."""
    from qwen3_tts_cuda_graphs_b200 import codec as K

    g = torch.Generator(device="cuda").manual_seed(M)
    for cin in (8, 96, 128):
        A, B = torch.randn(M, cin, device="cuda", generator=g).bfloat16(), (torch.randn(1, len(offs) * cin, device="cuda", generator=g) / 20).bfloat16()
        bias = torch.randn(1, device="cuda", generator=g)
        want, mag = product(A, B, M, cin, offs)
        out = torch.full((M + 1, 1), 7.0, device="cuda")
        launch([make_op(A, B, out, M, 1, cin, offs, K.F_OUT_F32 | K.F_CLAMP, bias=bias, m_begin=m_begin)])
        z = want + bias.double()
        assert ((out[:M].double() - z.clamp(-1, 1)).abs() <= 1.01 * 2.0 ** -8 * z.abs() + 2.0 ** -20 * mag + 1e-6)[m_begin:].all()
        assert (out[:m_begin] == 7).all() and out[M] == 7
