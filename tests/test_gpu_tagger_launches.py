"""Tagger passes on both sides of the line up to which they launch dependently (host/tagger.cc), whole units and odd ones: ordinary, dependent and the driver's own
launches give the same loss and gradients bit for bit, in passes that follow one another without a wait."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,S", [(64, 440), (64, 520), (33, 450), (128, 220), (128, 260), (256, 100), (256, 130)])
def test_launch_forms_agree(H, S):
    import torch
    from dynet_b200 import tagger
    lens, words, tags = tagger.synthetic_corpus(S, 800, 20, seed=H, lo=5, hi=100)
    got = []
    for choice in (None, 0, 1):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            m = tagger.Tagger(800, 48, H, 24, 20, max_sentences=S, max_tokens=int(lens.sum()), max_len=100, seed=1, stream=stream.cuda_stream)
            if choice is not None:
                m.ctx.dependent_launch(choice)
            for _ in range(3):
                m.grads.zero_()
                m.launch_forward_backward(lens, words, tags)
            stream.synchronize()
            assert m.device_errors() == 0
            got.append((m.loss_dev.clone(), m.grads.clone()))
            m.close()
    assert all(torch.equal(a, b) for other in got[1:] for a, b in zip(got[0], other))
