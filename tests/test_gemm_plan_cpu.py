"""What launches of the tcgen05 GEMM look like (host arithmetic): the shapes that the GPU tests name, the parts of a split sum, and what has to hold for every size."""
import ctypes as C
import random

import pytest
from test_gemm_gpu import SHAPES
from test_gemm_shapes_gpu import CASES, EIGHT, TWO

FLAGS = {"f32": 64 | 1024, "plain": 0, "residual": 4, "gelu": 2, "units": 16, "snake": 128 | 4}


def plan(M, N, cin, taps=1, split=False, flags=64 | 1024, m_begin=0):
    """shape, columns of a tile, row tiles, column tiles, parts, CTAs of a tile, stages, CTAs; None for a product of another kernel."""
    from qwen3_tts_cuda_graphs_b200 import codec as K

    o = K.Op()
    o.kind, o.flags, o.M, o.N, o.K, o.taps, o.cin, o.a_rows, o.lda, o.ldc, o.ldr, o.col_mod = K.K_GEMM, flags, M, N, taps * cin, taps, cin, M, cin, N, N, N
    o.A = o.B = o.C = o.C2 = o.res = 1 << 20      # addresses of whole pieces; nothing is read
    o.reserved, o.m_begin = 1 | (4 if split else 0), m_begin
    lib, out = C.CDLL(K._build.build_lib("libfq3codec.so")), (C.c_int32 * 8)()
    lib.fq3c_gemm_plan.argtypes = [C.POINTER(K.Op), C.POINTER(C.c_int32)]
    return list(out) if lib.fq3c_gemm_plan(C.byref(o), out) == 0 else None


@pytest.mark.parametrize("M,N,cin,offs,split,shape,columns,parts", CASES)
def test_cases_of_the_gpu_tests_are_what_they_are_named(M, N, cin, offs, split, shape, columns, parts):
    got = plan(M, N, cin, len(offs), split)
    assert (got is None and shape is None) or (got[0], got[1], got[4]) == (shape, columns, parts)


@pytest.mark.parametrize("name", [n for n in SHAPES if "split" in n])
def test_split_cases_are_split(name):
    M, N, cin, offs, _ = SHAPES[name]
    parts = {"few rows, split": 8, "three tiles, split": 1, "taps, split": 6, "eight rows, split": 4}[name]
    assert plan(M, N, cin, len(offs), True)[4] == parts and plan(M, N, cin, len(offs), False)[4] == 1


def test_every_plan_is_whole():
    rng = random.Random(5)
    for _ in range(4000):
        M, N, cin = (max(1, int(2 ** rng.uniform(*r))) for r in ((0, 16), (4, 13.5), (4, 13)))
        taps, split = rng.choice([1, 1, 2, 3, 7]), rng.random() < 0.5
        cin = (cin + 15) // 16 * 16
        if taps * cin < 64:
            continue
        flags = rng.choice(list(FLAGS.values()))
        N = N // 2 * 2 if flags & 16 else N
        m_begin = rng.randrange(M) if rng.random() < 0.3 else 0
        shape, bn, mt, nt, parts, ctas, stages, grid = plan(M, N, cin, taps, split, flags, m_begin)
        kb = -(-cin // 64) * taps if taps > 1 else -(-taps * cin // 64)
        assert bn % 16 == 0 and 16 <= bn <= 256 and nt * bn >= N > (nt - 1) * bn and mt == -(-(M - m_begin) // 128)
        assert 1 <= parts <= min(8, max(1, kb // 4)) and ctas <= 4 and parts <= ctas * 2 and (ctas - 1) * -(-parts // ctas) < parts      # every CTA has a part
        assert stages >= 2 and (shape != TWO or bn <= 128)
        if parts > 1:      # all clusters run at once, and the parts do not follow where the rows begin
            assert split and M <= 512 and grid == mt * nt * ctas <= 148 and shape == EIGHT
        if split and M <= 512:
            assert plan(M, N, cin, taps, split, flags)[4] == parts
        assert grid <= (296 if shape == TWO else 148) or grid == mt * nt * ctas
