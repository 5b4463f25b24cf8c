"""A layer set up under one stream and run under others: the steps have to see the finished set-up, and the layer's memory
must not be handed out again while a step on another stream than the allocating one is still in flight.  Streams are held
by a sleeping host function: nothing on the GPU waits, and each drains by itself."""
import ctypes as C
import gc
import time

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

HOSTFN = C.CFUNCTYPE(None, C.c_void_p)


def _sleep(_):
    time.sleep(0.2)


HOLD = HOSTFN(_sleep)


def hold(stream):
    rt = C.CDLL("libcudart.so.12")
    rt.cudaLaunchHostFunc.argtypes = [C.c_void_p, HOSTFN, C.c_void_p]
    assert rt.cudaLaunchHostFunc(C.c_void_p(stream.cuda_stream), HOLD, None) == 0


B, V = 24, 20011
ARGS = {"runtime_top_k": np.where(np.arange(B) % 3 == 0, 0, 20).astype(np.uint32),
        "runtime_top_p": np.asarray([0.9], np.float32), "repetition_penalty": np.asarray([1.2], np.float32),
        "random_seed": np.arange(B).astype(np.uint64)}


def state(device):
    g = torch.Generator(device=device)
    g.manual_seed(5)
    x = torch.randn(B, V, generator=g, device=device) * 3
    st = {"output_ids": torch.ones(12, B, dtype=torch.int32, device=device),
          "finished": torch.zeros(B, dtype=torch.bool, device=device),
          "sequence_length": torch.full((B,), 8, dtype=torch.int32, device=device)}
    return st, {"logits": x, "step": 8, "max_input_length": 8, "end_id": torch.full((B,), V - 1, dtype=torch.int32, device=device)}


@pytest.mark.parametrize("kind", ["layer", "shards"])
def test_set_up_on_a_busy_stream_run_on_another(kind, cuda_device):
    from fastertransformer_b200 import DynamicDecodeLayer, VocabParallelSampler

    def run(set_up_on, run_on, busy):
        st, inputs = state(cuda_device)
        torch.cuda.synchronize()
        with torch.cuda.stream(set_up_on):
            if busy:
                hold(set_up_on)
            if kind == "layer":
                layer = DynamicDecodeLayer(V, V, torch.float32, cuda_device)
            else:
                layer = VocabParallelSampler(V, (V + 1) // 2, 2, torch.float32, cuda_device)
            layer.setup(B, 1, ARGS)
        with torch.cuda.stream(run_on):
            if kind == "layer":
                layer.forward(st, inputs)
            else:
                w = (V + 1) // 2
                x = torch.nn.functional.pad(inputs["logits"], (0, 2 * w - V))
                layer.forward_shards(st, inputs, [x[:, :w].contiguous(), x[:, w:].contiguous()])
        torch.cuda.synchronize()
        return st["output_ids"][8].cpu(), layer.topk.curand.cpu(), layer.topp.curand.cpu()

    a, b = torch.cuda.Stream(device=cuda_device), torch.cuda.Stream(device=cuda_device)
    for want, got in zip(run(a, a, False), run(a, b, True)):
        assert torch.equal(want, got)


def test_memory_of_a_dropped_layer_is_not_reused_early(cuda_device):
    from fastertransformer_b200 import DynamicDecodeLayer
    a, b = torch.cuda.Stream(device=cuda_device), torch.cuda.Stream(device=cuda_device)
    st, inputs = state(cuda_device)
    with torch.cuda.stream(a):
        layer = DynamicDecodeLayer(V, V, torch.float32, cuda_device)
        layer.setup(B, 1, ARGS)
        layer.forward(st, inputs)  # (the workspace too belongs to the first stream)
    torch.cuda.synchronize()
    hold(b)
    with torch.cuda.stream(b):
        layer.forward(st, dict(inputs, step=9))
    held = {t.untyped_storage().data_ptr(): t.untyped_storage().nbytes() for t in layer._memory()}
    assert len(held) >= 2
    del layer
    gc.collect()
    with torch.cuda.stream(a):
        again = [torch.empty(n, dtype=torch.uint8, device=cuda_device) for n in held.values() for _ in range(3)]
        assert not b.query()  # the step on the other stream has not run yet
        assert not {t.data_ptr() for t in again} & set(held)
    torch.cuda.synchronize()
