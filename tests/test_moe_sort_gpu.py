"""Grouping of (token, choice) pairs by expert: whole numbers, at the edges of a warp's share and with choices that have no tensors."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,top,E", [(2, 1, 1), (3, 2, 16), (31, 1, 8), (32, 1, 8), (33, 1, 8), (129, 8, 33), (701, 2, 16), (1024, 1, 64), (1025, 1, 300), (2048, 4, 32), (40, 3, 3000)])
@pytest.mark.parametrize("identity", [0, 3])
def test_segments_rows_and_positions(M, top, E, identity):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    g = torch.Generator(device="cuda").manual_seed(M * top + E)
    ids = torch.randint(0, E + identity, (M, top), device="cuda", generator=g, dtype=torch.int32)
    seg, rows, pos = (torch.full((n,), -7, device="cuda", dtype=torch.int32) for n in (E + 1, M * top, M * top))
    o = K.Op()
    o.kind, o.M, o.i0, o.i1, o.A, o.C, o.C2, o.ws, o.col_mod = K.K_MOE_SORT, M, top, E, ids.data_ptr(), seg.data_ptr(), rows.data_ptr(), pos.data_ptr(), 1
    lib = K.load_lib()
    assert lib.fq3c_run((K.Op * 1)(o), 1, torch.cuda.current_stream().cuda_stream) == 0, lib.fq3c_last_error()
    flat = ids.flatten().long().cpu()
    real = (flat < E).nonzero().flatten()
    order = real[flat[real].argsort(stable=True)]
    want = torch.full((M * top,), -1)
    want[order] = torch.arange(len(order))
    starts = torch.cat([torch.zeros(1, dtype=torch.long), torch.bincount(flat[real], minlength=E).cumsum(0)])
    assert torch.equal(seg.long().cpu(), starts) and torch.equal(pos.long().cpu(), want)
    assert torch.equal(rows[:len(order)].long().cpu(), order // top) and (rows[len(order):] == -7).all()
