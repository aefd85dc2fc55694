"""The codec of a streamed chunk runs on the SMs that the next chunk's frame loop leaves free: it ends long before the frames do."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_a_window_ends_beside_the_frame_loop():
    from qwen3_tts_cuda_graphs_b200 import FasterQwen3TTS
    from qwen3_tts_cuda_graphs_b200.engine import SamplingPolicy, SubPolicy

    m = FasterQwen3TTS.from_pretrained("synthetic://0.6B-Base", device="cuda", dtype=torch.bfloat16, max_seq_len=1024, seed=0)
    eng, dec = m.model.engine, m.model.model.speech_tokenizer.decoder
    try:
        H = eng.cfg.talker.hidden_size
        g = torch.Generator(device="cuda").manual_seed(1)
        rows = lambda *s: (0.3 * torch.randn(*s, H, device="cuda", generator=g)).bfloat16()
        policy = SamplingPolicy(min_new_tokens=512, seed=1)
        eng.set_text_conditioning(0, rows(40), rows())
        eng.prefill(0, rows(120), 0, policy, dense=False)
        hidden, codes = rows(), torch.randint(0, 2048, (33, 16), device="cuda", generator=g)
        alone = dec.decode(codes, 25 * 1920)
        torch.cuda.synchronize()      # (a plan's buffers belong to one stream at a time)
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            for _ in range(3):      # (from the second use on a graph; the stream's memory is there too)
                dec.decode(codes, 25 * 1920)
        assert eng.reduced_grid() > 0
        for _ in range(2):
            eng.reset_stream(0)
            eng.set_loop_state(0, 5, hidden, 120, 0)
            eng.set_decode_grid(eng.reduced_grid())
            begun, frames, window = (torch.cuda.Event(enable_timing=True) for _ in range(3))
            torch.cuda.synchronize()
            begun.record()
            eng.decode_frames(1, 8, policy, SubPolicy())
            frames.record()
            side.wait_event(begun)
            with torch.cuda.stream(side):
                wav = dec.decode(codes, 25 * 1920)
                window.record()
            torch.cuda.synchronize()
            assert torch.equal(wav, alone)
            # 13 ms of frames; the window takes 0.9 alone and a few times that on 20 SMs
            assert begun.elapsed_time(window) < 0.7 * begun.elapsed_time(frames)
    finally:
        eng.set_decode_grid(0)
        eng.close()
