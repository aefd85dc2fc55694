"""Attention of few rows or a short window (one CTA stages what its rows see), alone and together with the q / k norm, rotation and cache rows in front of it."""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu


def attn_op(x, out, M, H, G, d, window, hist=0, known=None, flags=0):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    o = K.Op()
    o.kind, o.flags, o.M, o.N, o.A, o.lda, o.a_rows = K.K_ATTN, flags, M, H * d, x.data_ptr(), x.stride(0), M
    o.C, o.ldc, o.col_mod, o.i0, o.i1, o.i2, o.K, o.taps = out.data_ptr(), out.stride(0), H * d, H, G, d, window, hist
    if known is not None:
        o.p0 = known.data_ptr()
    return o


def launch(*ops):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    lib = K.load_lib()
    arr = (K.Op * len(ops))(*ops)
    before = lib.fq3c_launch_count()
    assert lib.fq3c_run(arr, len(ops), torch.cuda.current_stream().cuda_stream) == 0, lib.fq3c_last_error()
    torch.cuda.synchronize()
    return lib.fq3c_launch_count() - before


def exact(x, M, H, G, d, window, hist=0, first=0):
    """float64 without roundings, and what the two roundings of a score to bf16 and the output's can do to it."""
    x = x.double()
    q, k, v = x[hist:hist + M, :H * d].view(M, H, d), x[:hist + M, H * d:(H + G) * d].view(-1, G, d), x[:hist + M, (H + G) * d:(H + 2 * G) * d].view(-1, G, d)
    k, v = (t.repeat_interleave(H // G, 1) for t in (k, v))
    t, j = torch.arange(hist, hist + M, device=x.device)[:, None], torch.arange(hist + M, device=x.device)[None]
    s = torch.einsum("ihd,jhd->hij", q, k) * d ** -0.5
    s = s.masked_fill((j > t) | (j <= t - window) | (j < first), float("-inf"))
    p = s.softmax(-1)
    out = torch.einsum("hij,jhd->ihd", p, v).reshape(M, H * d)
    # a score moves by 2 x 2^-9 of itself (and f32 sums' 2^-17 of its magnitude): weights by that much relative to each other, twice with the sum's share
    moved = torch.expm1(2.1 * 2.0 ** -8 * s.masked_fill(s.isinf(), 0).abs().amax() + 2.0 ** -14)
    return out, moved * torch.einsum("hij,jhd->ihd", p, v.abs()).reshape(M, H * d) + 1.01 * 2.0 ** -8 * out.abs() + 1e-6


# rows, query heads, key / value heads, entries, window, rows of history, of which known
CASES = [(1, 16, 16, 64, 72, 0, None), (33, 16, 16, 64, 72, 0, None), (256, 16, 16, 64, 72, 0, None), (40, 2, 1, 64, 8, 0, None), (9, 16, 16, 64, 72, 71, 0), (9, 16, 16, 64, 72, 71, 30), (75, 4, 2, 64, 72, 71, 500),
         (17, 16, 8, 128, 2048, 0, None), (112, 6, 2, 128, 2048, 0, None), (70, 5, 1, 128, 33, 0, None), (65, 8, 8, 128, 1, 0, None), (600, 3, 3, 128, 32, 0, None)]


@pytest.mark.parametrize("M,H,G,d,window,hist,known", CASES)
def test_windows_and_history(M, H, G, d, window, hist, known):
    g = torch.Generator(device="cuda").manual_seed(M + d)
    x = torch.randn(hist + M, (H + 2 * G) * d + 8, device="cuda", generator=g).bfloat16()
    n = None if known is None else torch.tensor([known], dtype=torch.int32, device="cuda")
    first = 0 if known is None else hist - min(known, hist)
    x[:first] = float("nan")      # rows before the stream's begin: never read into a sum
    out = torch.full((M + 1, H * d), 5.0, device="cuda", dtype=torch.bfloat16)
    launch(attn_op(x, out, M, H, G, d, window, hist, n))
    want, bound = exact(x.nan_to_num(0.0), M, H, G, d, window, hist, first)
    assert ((out[:M].double() - want).abs() <= bound).all() and (out[M] == 5).all()
    if hist == 0 and M > 20:      # the rows behind a cut, with the ones before it as history: the same bits
        cut, tail = M - 7, torch.zeros(7, H * d, device="cuda", dtype=torch.bfloat16)
        launch(attn_op(x, tail, 7, H, G, d, window, cut))
        assert torch.equal(tail, out[cut:M])


@pytest.mark.parametrize("M,H,G,pos0", [(1, 16, 8, 0), (17, 16, 8, 0), (39, 16, 8, 3), (64, 4, 4, 0), (84, 16, 8, 0), (85, 16, 8, 0), (90, 14, 2, 0), (91, 14, 2, 0), (112, 8, 8, 0), (113, 4, 4, 0), (64, 32, 8, 0), (65, 32, 8, 0), (100, 14, 2, 0), (101, 16, 8, 0), (102, 16, 8, 0), (130, 9, 1, 0), (144, 4, 4, 0), (145, 4, 4, 0), (30, 3, 1, 0)])
def test_norm_rotation_and_cache_in_the_same_launch(M, H, G, pos0):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    g = torch.Generator(device="cuda").manual_seed(M * H)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=g).bfloat16()  # noqa: E731
    x, gq, gk, rope = rand(M, (H + 2 * G) * 128), rand(128), rand(128), torch.rand(pos0 + M, 256, device="cuda", generator=g) * 6.28
    rope = torch.cat([rope[:, :64], rope[:, :64]], -1)
    cos, sin = rope.cos().bfloat16(), rope.sin().bfloat16()
    got = []
    for scratch in (0, 1):
        rows, ck, cv, out = x.clone(), *(torch.full((G, pos0 + M + 2, 128), 3.0, device="cuda", dtype=torch.bfloat16) for _ in range(2)), torch.zeros(M, H * 128, device="cuda", dtype=torch.bfloat16)
        n = K.Op()
        n.kind, n.M, n.N, n.A, n.lda, n.a_rows, n.i0, n.i1, n.i2, n.f0, n.reserved = 8, M, x.shape[1], rows.data_ptr(), x.shape[1], M, H, G, pos0, 1e-6, scratch
        n.p0, n.p1, n.B, n.bias, n.C, n.C2, n.ldc, n.col_mod = (*(t.data_ptr() for t in (gq, gk, cos, sin, ck, cv)), ck.shape[1], x.shape[1])
        launches = launch(n, attn_op(rows, out, M, H, G, 128, 4096, flags=1))
        assert launches == (1 if scratch and (M <= 64 or (M <= 112 and M * M * H <= 115000)) else 2)      # behind that line tcgen05 takes the rows, scratch or not
        got.append((rows, ck, cv, out))
    (turned, ck, cv, apart), (_, ck1, cv1, out) = got
    assert torch.equal(ck, ck1) and torch.equal(cv, cv1) and torch.equal(apart, out)
    want, bound = exact(turned, M, H, G, 128, 4096)
    assert ((out.double() - want).abs() <= bound).all()


def streamed(x, M, H, G, d, window, chunk):
    """The rows in chunks, each behind the window's earlier rows, as a stateful stream decodes them."""
    out = torch.zeros(M, H * d, device="cuda", dtype=torch.bfloat16)
    for at in range(0, M, chunk):
        hist, rows = min(window - 1, at), min(chunk, M - at)
        launch(attn_op(x[at - hist:at + rows], out[at:at + rows], rows, H, G, d, window, hist))
    return out


# windows on both sides of what a CTA's shared memory holds: whole decode and stream do not come to the same kernel at 400 (460 rows), 480 and 1024
@pytest.mark.parametrize("M,H,G,d,window,chunk", [(100, 16, 16, 64, 72, 1), (256, 16, 16, 64, 72, 9), (460, 16, 16, 64, 400, 33), (256, 16, 16, 64, 480, 8), (300, 16, 16, 64, 1024, 33), (90, 4, 2, 64, 8, 3),
                                                  (260, 8, 8, 128, 130, 20), (300, 8, 2, 128, 300, 50)])
def test_a_stream_has_the_bits_of_the_whole_decode(M, H, G, d, window, chunk):
    g = torch.Generator(device="cuda").manual_seed(M + window)
    x = (1.5 * torch.randn(M, (H + 2 * G) * d, device="cuda", generator=g)).bfloat16()
    out = torch.zeros(M, H * d, device="cuda", dtype=torch.bfloat16)
    launch(attn_op(x, out, M, H, G, d, window))
    assert torch.equal(out, streamed(x, M, H, G, d, window, chunk))


@pytest.mark.parametrize("M,H,G,d,window,hist,known", [c for c in CASES if c[0] * c[1] * c[3] <= 400000] + [(33, 16, 16, 64, 72, 71, 71), (100, 16, 8, 128, 72, 0, None)] +
                         [(8, 16, 16, 64, 72, 0, None), (9, 16, 8, 128, 72, 0, None), (33, 16, 16, 64, 9, 0, None), (300, 16, 16, 64, 15, 0, None), (300, 16, 16, 64, 16, 0, None)])      # lines between the kernels
def test_the_general_kernel_has_the_same_bits(M, H, G, d, window, hist, known):
    """Outputs one entry off an even address go through the kernel with a warp per row and head; infinite scores among the keys."""
    g = torch.Generator(device="cuda").manual_seed(M * 3 + d)
    x = (1.5 * torch.randn(hist + M, (H + 2 * G) * d, device="cuda", generator=g)).bfloat16()
    x[(hist + M) // 2, H * d:H * d + 8] = 3e38      # scores of both signs beyond bf16 (and NaN, where they meet)
    n = None if known is None else torch.tensor([known], dtype=torch.int32, device="cuda")
    out, wide = torch.zeros(M, H * d, device="cuda", dtype=torch.bfloat16), torch.zeros(M, H * d + 4, device="cuda", dtype=torch.bfloat16)
    launch(attn_op(x, out, M, H, G, d, window, hist, n))
    launch(attn_op(x, wide[:, 1:], M, H, G, d, window, hist, n))
    got, want = out.float(), wide[:, 1:1 + H * d].float()
    assert torch.equal(got.nan_to_num(7.0), want.nan_to_num(7.0)) and torch.equal(got.isnan(), want.isnan())


@pytest.mark.parametrize("M,H,G", [(17, 16, 8), (39, 16, 8), (64, 4, 4), (84, 16, 8), (30, 14, 2), (64, 4, 1), (39, 32, 8)])
def test_prompt_in_one_launch_has_the_bits_of_two(M, H, G):
    """Rows that tcgen05 does not take yet: norm, rotation, cache and attention together, and the attention behind them by itself."""
    from qwen3_tts_cuda_graphs_b200 import codec as K

    g = torch.Generator(device="cuda").manual_seed(M * H + 1)
    rand = lambda *shape: torch.randn(*shape, device="cuda", generator=g).bfloat16()  # noqa: E731
    x, gq, gk, ang = rand(M, (H + 2 * G) * 128), rand(128), rand(128), torch.rand(M, 64, device="cuda", generator=g) * 6.28
    cos, sin = torch.cat([ang, ang], -1).cos().bfloat16(), torch.cat([ang, ang], -1).sin().bfloat16()
    got = []
    for scratch in (0, 1):
        rows, ck, cv, out = x.clone(), *(torch.zeros(G, M, 128, device="cuda", dtype=torch.bfloat16) for _ in range(2)), torch.zeros(M, H * 128, device="cuda", dtype=torch.bfloat16)
        n = K.Op()
        n.kind, n.M, n.N, n.A, n.lda, n.a_rows, n.i0, n.i1, n.f0, n.reserved = 8, M, x.shape[1], rows.data_ptr(), x.shape[1], M, H, G, 1e-6, scratch
        n.p0, n.p1, n.B, n.bias, n.C, n.C2, n.ldc, n.col_mod = (*(t.data_ptr() for t in (gq, gk, cos, sin, ck, cv)), M, x.shape[1])
        assert launch(n, attn_op(rows, out, M, H, G, 128, 4096, flags=1)) == 2 - scratch
        got.append((ck, cv, out))
    assert all(torch.equal(a, b) for a, b in zip(*got))


def switched_off():
    """In a process with FQ3C_ATTN_PREFILL=0: two launches, and the attention has the bits of one that is no prompt's."""
    from qwen3_tts_cuda_graphs_b200 import codec as K

    for M, H, G in ((39, 16, 8), (100, 16, 8), (150, 4, 4)):
        g = torch.Generator(device="cuda").manual_seed(M)
        rand = lambda *shape: torch.randn(*shape, device="cuda", generator=g).bfloat16()  # noqa: E731
        x, gq, gk, cos, sin = rand(M, (H + 2 * G) * 128), rand(128), rand(128), torch.ones(M, 128, device="cuda").bfloat16(), torch.zeros(M, 128, device="cuda").bfloat16()
        ck, cv, out, want = *(torch.zeros(G, M, 128, device="cuda", dtype=torch.bfloat16) for _ in range(2)), *(torch.zeros(M, H * 128, device="cuda", dtype=torch.bfloat16) for _ in range(2))
        n = K.Op()
        n.kind, n.M, n.N, n.A, n.lda, n.a_rows, n.i0, n.i1, n.f0, n.reserved = 8, M, x.shape[1], x.data_ptr(), x.shape[1], M, H, G, 1e-6, 1
        n.p0, n.p1, n.B, n.bias, n.C, n.C2, n.ldc, n.col_mod = (*(t.data_ptr() for t in (gq, gk, cos, sin, ck, cv)), M, x.shape[1])
        assert launch(n, attn_op(x, out, M, H, G, 128, 4096, flags=1)) == 2
        launch(attn_op(x, want, M, H, G, 128, 4096))
        assert torch.equal(out, want)
    print("two launches each")


def test_the_switch_covers_the_launch_with_the_norm():
    here = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, "-c", "import sys; sys.path[:0] = [%r, %r]; import test_attention_rows_gpu as t; t.switched_off()" % (here, os.path.dirname(here))],
                       env=dict(os.environ, FQ3C_ATTN_PREFILL="0"), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "two launches each" in r.stdout, r.stderr[-2000:]
