"""Rows of the split kernel that start between two 16-byte boundaries, loaded column by column a batch ahead: vocabularies around the
edges of the loop (a CTA's columns are whole chunks of 1024 over 8, 4 or 2 CTAs, 2048 of them a batch), against the general kernel."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def step(general, x, V, bias, temperature, device):
    from fastertransformer_b200 import DynamicDecodeLayer, lib
    B = x.shape[0]
    layer = DynamicDecodeLayer(V, x.shape[1], x.dtype, device)
    args = {"random_seed": np.arange(B).astype(np.uint64), "runtime_top_k": np.resize(np.asarray([0, 1, 50], np.uint32), B),
            "runtime_top_p": np.asarray([0.8], np.float32)}
    if temperature is not None:
        args["temperature"] = np.asarray([temperature], np.float32)
    layer.setup(B, 1, args)
    st = {"output_ids": torch.ones(6, B, dtype=torch.int32, device=device),
          "finished": torch.zeros(B, dtype=torch.bool, device=device),
          "sequence_length": torch.full((B,), 4, dtype=torch.int32, device=device)}
    inputs = {"logits": x, "step": 4, "max_input_length": 4, "end_id": torch.full((B,), V - 1, dtype=torch.int32, device=device)}
    if bias is not None:
        inputs["embedding_bias"] = bias
    lib.ftb200_set_single_pass(0 if general else 1)
    try:
        layer.forward(st, inputs)
        torch.cuda.synchronize()
    finally:
        lib.ftb200_set_single_pass(1)
    return [v.cpu().numpy() for v in (st["output_ids"], st["sequence_length"], layer.topk.curand, layer.topp.curand)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,V,padded", [(5, 1025, 1025), (5, 2047, 2049), (5, 16383, 16383), (5, 16385, 16387), (5, 17409, 17409),
                                        (60, 8191, 8193), (100, 4097, 4097), (3, 208295, 208295)])
@pytest.mark.parametrize("biased,temperature", [(False, None), (False, 0.7), (True, None), (True, 1.3)])
def test_rows_between_two_boundaries(dtype, B, V, padded, biased, temperature, cuda_device):
    g = torch.Generator(device=cuda_device)
    g.manual_seed(V + B)
    x = (torch.randn(B, padded, generator=g, device=cuda_device) * 2.5).to(dtype)
    bias = (torch.randn(padded, generator=g, device=cuda_device) * 0.5).to(dtype) if biased else None
    for want, got in zip(step(True, x, V, bias, temperature, cuda_device), step(False, x, V, bias, temperature, cuda_device)):
        np.testing.assert_array_equal(got, want)
