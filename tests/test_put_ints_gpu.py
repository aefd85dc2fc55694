"""A step's ids as a launch's arguments (codec.put_ints): sizes around one launch's 1000, order on the stream, under capture, values that change at once."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 32, 33, 999, 1000, 1001, 2500])
def test_values_arrive(n):
    from qwen3_tts_cuda_graphs_b200 import codec as K

    dst = torch.full((n + 2,), -7, device="cuda", dtype=torch.int32)
    values = [(i * 7919) % 100003 - 50000 for i in range(n)]
    K.put_ints(K.load_lib(), values, dst[1:n + 1])
    values[:] = [0] * n
    assert dst.tolist() == [-7] + [(i * 7919) % 100003 - 50000 for i in range(n)] + [-7]


def test_in_order_and_captured():
    from qwen3_tts_cuda_graphs_b200 import codec as K

    lib, dst = K.load_lib(), torch.zeros(3, device="cuda", dtype=torch.int32)
    seen = []
    for i in range(50):      # no launch in between waits for the host
        K.put_ints(lib, torch.tensor([i, i + 1, i + 2]), dst)
        seen.append(dst.clone())
    assert [t.tolist() for t in seen] == [[i, i + 1, i + 2] for i in range(50)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        K.put_ints(lib, [4, 5, 6], dst)
    dst.zero_()
    graph.replay()
    assert dst.tolist() == [4, 5, 6]


def test_bad_arguments_are_refused():
    from qwen3_tts_cuda_graphs_b200 import codec as K

    lib = K.load_lib()
    assert lib.fq3c_put_ints(None, 1, None, None) < 0 and lib.fq3c_put_ints(None, -1, None, None) < 0 and lib.fq3c_put_ints(None, 0, None, None) == 0
