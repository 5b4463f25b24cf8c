"""Two host threads driving one GPU at the same time, each with its own layer, state and CUDA stream (ctypes releases
the interpreter lock during the library calls, so the calls do overlap).  The per-device state the calls share - the
second stream of the single-pass step with its fork and join events, the occupancy caches - must not let one
thread's step see the other's: both threads must reproduce the ids of the same workloads run one after the other."""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _decode(seed, device, stream, steps, out, key, batch=48, vocab=32768):
    from fastertransformer_b200 import DynamicDecodeLayer
    from fastertransformer_b200.workloads import make_workload
    w = make_workload("c3", batch=batch, steps=steps, vocab=vocab, seed=seed)
    with torch.cuda.stream(stream):
        layer = DynamicDecodeLayer(w.vocab, w.vocab_padded, w.dtype, device)
        layer.stream = stream
        st = w.initial_state(device)
        inputs = w.static_inputs(device)
        layer.setup(w.batch, 1, w.runtime_args)
        logits = [w.logits(w.max_input_length + s, device) for s in range(steps)]
        stream.synchronize()
        for s in range(steps):
            layer.forward(st, dict(inputs, logits=logits[s], step=w.max_input_length + s))
        stream.synchronize()
    out[key] = st["output_ids"].cpu().numpy()


def test_two_threads_one_device(cuda_device):
    steps = 24
    alone, together = {}, {}
    for i, seed in enumerate((11, 12)):
        _decode(seed, cuda_device, torch.cuda.Stream(device=cuda_device), steps, alone, i)
    threads = [threading.Thread(target=_decode, args=(seed, cuda_device, torch.cuda.Stream(device=cuda_device), steps,
                                                      together, i)) for i, seed in enumerate((11, 12))]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=300)
    assert set(together) == {0, 1}
    for i in (0, 1):
        assert np.array_equal(alone[i], together[i]), "thread %d differs from its run alone" % i


def test_two_threads_with_different_vocabularies(cuda_device):
    """Batches of the single-pass kernels (more columns than the split kernel takes) whose needs of shared memory differ: a
    launch of one thread must not find the limit that the other one's smaller call set."""
    steps, shapes = 12, {0: (600, 32768), 1: (300, 100352)}
    alone, together = {}, {}
    for i, (batch, vocab) in shapes.items():
        _decode(21 + i, cuda_device, torch.cuda.Stream(device=cuda_device), steps, alone, i, batch, vocab)
    threads = [threading.Thread(target=_decode, args=(21 + i, cuda_device, torch.cuda.Stream(device=cuda_device), steps, together,
                                                      i, batch, vocab)) for i, (batch, vocab) in shapes.items()]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=300)
    assert set(together) == {0, 1}
    for i in shapes:
        assert np.array_equal(alone[i], together[i]), "thread %d differs from its run alone" % i
