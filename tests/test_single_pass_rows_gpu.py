"""The single-pass kernels against the general kernel, which serves the same rows one after the other: what a top-p row does behind its
first pass (special columns filed by chunk, the ragged end, counts above and below zero, the class found from either end), and
steps whose last row ends the step for a host that waits, with rows left to the general kernel among them."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

F16, BF16 = torch.float16, torch.bfloat16


def steps(general, dtype, V, B, device, *, kinds, history, sigma, shift=0.0, temperature=None, penalty=1.1, waits=False, n=2):
    from fastertransformer_b200 import DynamicDecodeLayer, lib
    g = torch.Generator(device=device)
    g.manual_seed(V + 7 * B + history)
    args = {"random_seed": np.arange(B).astype(np.uint64), "repetition_penalty": np.resize(np.asarray(penalty, np.float32), B)}
    args["runtime_top_p"] = np.resize(np.asarray([0.3, 0.95, 0.6, 0.99], np.float32), B)
    if kinds == "both":
        args["runtime_top_k"] = np.resize(np.asarray([0, 1, 0, 40, 700], np.uint32), B)
    if temperature is not None:
        args["temperature"] = np.asarray([temperature], np.float32)
    layer = DynamicDecodeLayer(V, V, dtype, device)
    layer.setup(B, 1, args)
    st = {"output_ids": torch.randint(1, V, (history + n + 1, B), generator=g, device=device, dtype=torch.int32),
          "finished": torch.arange(B, device=device) % 11 == 5,
          "sequence_length": torch.full((B,), history, dtype=torch.int32, device=device)}
    extra = {}
    if waits:
        limit = torch.full((B,), history + n - 1, dtype=torch.int32, device=device)
        words = torch.zeros(B, 2, 1, dtype=torch.int32, device=device)
        words[:, 0], words[:, 1] = 9, 1
        extra = {"sequence_limit_length": limit, "stop_words_list": words}
    stops = []
    lib.ftb200_set_single_pass(0 if general else 1)
    try:
        for s in range(n):
            x = torch.randn(B, V, generator=g, device=device) * sigma + shift
            if waits:
                x[::4, 9] += 20.0
            stops.append(layer.forward(st, {"logits": x.to(dtype), "step": history + s, "max_input_length": history,
                                            "end_id": torch.full((B,), V - 1, dtype=torch.int32, device=device), **extra}))
            if waits:
                assert stops[-1] == bool(st["finished"].all())
        torch.cuda.synchronize()
    finally:
        lib.ftb200_set_single_pass(1)
    out = {k: v.cpu().numpy() for k, v in st.items()}
    out["curand"] = np.concatenate([layer.topk.curand.cpu().numpy(), layer.topp.curand.cpu().numpy()])
    out["stops"] = np.asarray(stops)
    return out


def same(want, got):
    for k, v in want.items():
        np.testing.assert_array_equal(got[k], v, err_msg=k)


@pytest.mark.parametrize("dtype,V,B,history,sigma,shift,temperature", [
    (BF16, 17408, 560, 40, 2.0, 0.0, None),     # whole chunks, an odd number of them
    (F16, 18440, 520, 40, 2.5, 0.0, 0.8),       # an even number, and a ragged end of eight columns
    (BF16, 51200, 300, 900, 2.5, 0.0, None),    # more listed columns than threads: ordered by bins
    (F16, 51200, 300, 700, 1.2, 0.0, 1.1),      # a wide nucleus of half rows
    (BF16, 51200, 300, 40, 1.0, 0.0, None),     # a cut below zero: patterns of both signs counted
    (F16, 32000, 300, 40, 1.5, -9.0, None),     # every value below zero
    (BF16, 128256, 80, 2900, 2.5, 0.0, 0.9),    # a table of 4096 places
    (BF16, 250000, 40, 300, 2.0, 0.0, None)])   # more buckets than threads
def test_nucleus_rows(dtype, V, B, history, sigma, shift, temperature, cuda_device):
    kw = dict(kinds="topp", history=history, sigma=sigma, shift=shift, temperature=temperature)
    same(steps(True, dtype, V, B, cuda_device, **kw), steps(False, dtype, V, B, cuda_device, **kw))


@pytest.mark.parametrize("dtype,V,B,penalty", [
    (BF16, 32768, 560, [1.1]),         # every row served
    (F16, 32768, 560, [1.1, 0.9, 1.0]),  # rows whose penalty raises values are left
    (BF16, 17000, 4500, [1.1, 1.1, 1.1, 1.1, 0.8])])
@pytest.mark.parametrize("waits", [False, True])
def test_rows_of_both_layers(dtype, V, B, penalty, waits, cuda_device):
    kw = dict(kinds="both", history=30, sigma=2.0, penalty=penalty, waits=waits)
    same(steps(True, dtype, V, B, cuda_device, **kw), steps(False, dtype, V, B, cuda_device, **kw))


@pytest.mark.parametrize("dtype,V,B,kinds", [
    (BF16, 17001, 600, "topp"), (F16, 30003, 350, "topp"), (BF16, 128257, 75, "topp"),
    (F16, 17001, 1000, "both"), (BF16, 50257, 954, "both"), (BF16, 50257, 956, "both")])  # (either side of the line for both kinds)
@pytest.mark.parametrize("waits", [False, True])
def test_rows_off_a_16_byte_boundary(dtype, V, B, kinds, waits, cuda_device):
    kw = dict(kinds=kinds, history=30, sigma=2.5, waits=waits, n=1 if B * V > 40e6 else 2)
    same(steps(True, dtype, V, B, cuda_device, **kw), steps(False, dtype, V, B, cuda_device, **kw))


@pytest.mark.parametrize("dtype,V,B,sigma,temperature", [
    (BF16, 126959, 60, 1.5, 1.2),           # nuclei of most columns: beyond the first launch's areas, within the second's
    (torch.float32, 128256, 12, 0.6, 1.0),  # an owner's 14000 keys, stretch by stretch
    (F16, 131072, 20, 0.5, 1.0),            # as many columns as the areas hold, and rows that go to the general kernel
    (BF16, 240000, 24, 1.2, 1.0)])          # areas of half a slice
def test_flat_rows(dtype, V, B, sigma, temperature, cuda_device):
    """A step that waits and whose widest nuclei the first launch leaves."""
    kw = dict(kinds="topp", history=20, sigma=sigma, temperature=temperature, waits=True)
    same(steps(True, dtype, V, B, cuda_device, **kw), steps(False, dtype, V, B, cuda_device, **kw))
