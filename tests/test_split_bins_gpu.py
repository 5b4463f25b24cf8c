"""Nuclei of bfloat16 rows in the split kernel, whose owners order their keys bin by bin or leave them to the sort, against the general
kernel: peaked and flat rows, bins of a few, of up to 32 and of more keys, near zero and far from it, with penalised columns."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def step(general, x, history, temperature, device):
    from fastertransformer_b200 import DynamicDecodeLayer, lib
    B, V = x.shape
    n = history.shape[0]
    layer = DynamicDecodeLayer(V, V, x.dtype, device)
    layer.setup(B, 1, {"random_seed": np.arange(B).astype(np.uint64), "runtime_top_p": np.asarray([0.97], np.float32),
                       "repetition_penalty": np.asarray([1.2], np.float32), "temperature": np.asarray([temperature], np.float32)})
    st = {"output_ids": torch.cat([history, torch.zeros(2, B, dtype=torch.int32, device=device)]),
          "finished": torch.zeros(B, dtype=torch.bool, device=device),
          "sequence_length": torch.full((B,), n, dtype=torch.int32, device=device)}
    lib.ftb200_set_single_pass(0 if general else 1)
    try:
        layer.forward(st, {"logits": x, "step": n, "max_input_length": n,
                           "end_id": torch.full((B,), V - 1, dtype=torch.int32, device=device)})
        torch.cuda.synchronize()
    finally:
        lib.ftb200_set_single_pass(1)
    return [v.cpu().numpy() for v in (st["output_ids"], st["sequence_length"], st["finished"], layer.topp.curand)]


@pytest.mark.parametrize("B,V", [(16, 17001), (16, 50264), (8, 128256)])
@pytest.mark.parametrize("sigma", [0.3, 1.0, 1.5, 2.5])
@pytest.mark.parametrize("shift,temperature", [(0.0, 1.0), (0.0, 1.4), (5.0, 0.7), (-3.0, 1.0)])
def test_nuclei_of_bfloat16_rows(B, V, sigma, shift, temperature, cuda_device):
    g = torch.Generator(device=cuda_device)
    g.manual_seed(V)
    x = (torch.randn(B, V, generator=g, device=cuda_device) * sigma + shift).to(torch.bfloat16)
    history = torch.randint(1, V, (300, B), generator=g, device=cuda_device, dtype=torch.int32)
    for want, got in zip(step(True, x, history, temperature, cuda_device), step(False, x, history, temperature, cuda_device)):
        np.testing.assert_array_equal(got, want)
