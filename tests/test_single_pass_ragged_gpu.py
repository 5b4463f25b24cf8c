"""Top-p rows of the single-pass kernel whose vocabulary ends inside a 16-byte vector (vocab < vocab_padded), against the general kernel:
the columns behind the last whole vector are listed, counted and found once, whichever side of the pass's threshold they lie on."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

F16, BF16 = torch.float16, torch.bfloat16


def step(general, x, V, B, device, *, top_p, history, temperature=None, decay=False):
    """One decode step over the logits x [B, padded]; everything that it writes."""
    from fastertransformer_b200 import DynamicDecodeLayer, lib
    args = {"random_seed": np.arange(B).astype(np.uint64), "repetition_penalty": np.asarray([1.1], np.float32),
            "runtime_top_p": np.asarray([top_p], np.float32)}
    if temperature is not None:
        args["temperature"] = np.asarray([temperature], np.float32)
    if decay:
        args["top_p_decay"] = torch.full((B,), 0.9, device=device)
        args["top_p_min"] = torch.full((B,), 0.1, device=device)
        args["top_p_reset_ids"] = torch.arange(B, dtype=torch.int32, device=device) % V
    layer = DynamicDecodeLayer(V, x.shape[1], x.dtype, device)
    layer.setup(B, 1, args)
    n = history.shape[0]
    ids = torch.cat([history, torch.zeros(2, B, dtype=torch.int32, device=device)])
    st = {"output_ids": ids, "finished": torch.arange(B, device=device) % 11 == 5,
          "sequence_length": torch.full((B,), n, dtype=torch.int32, device=device)}
    lib.ftb200_set_single_pass(0 if general else 1)
    try:
        layer.forward(st, {"logits": x, "step": n, "max_input_length": n,
                           "end_id": torch.full((B,), V - 1, dtype=torch.int32, device=device)})
        torch.cuda.synchronize()
    finally:
        lib.ftb200_set_single_pass(1)
    out = {k: v.cpu().numpy() for k, v in st.items()}
    out["curand"] = layer.topp.curand.cpu().numpy()
    if decay:
        out["top_p"] = layer.topp.top_ps.cpu().numpy()
    return out


def compare(x, V, B, device, **kw):
    want, got = step(True, x, V, B, device, **kw), step(False, x, V, B, device, **kw)
    for k, v in want.items():
        np.testing.assert_array_equal(got[k], v, err_msg=k)


@pytest.mark.parametrize("decay", [False, True])
@pytest.mark.parametrize("dtype,V,padded,B,temperature", [
    (F16, 17401, 17408, 560, 1.3), (F16, 17405, 17408, 560, None), (BF16, 17407, 17408, 560, 0.8),
    (BF16, 50257, 50264, 300, None), (F16, 50257, 50264, 300, 1.2)])
def test_ragged_vocabulary(dtype, V, padded, B, temperature, decay, cuda_device):
    g = torch.Generator(device=cuda_device)
    g.manual_seed(V + B)
    x = torch.randn(B, padded, generator=g, device=cuda_device) * 2
    x[:, padded - 8:] += 4.0  # (the last columns in reach of the draw, the padding above them)
    history = torch.randint(V - 40, V, (20, B), generator=g, device=cuda_device, dtype=torch.int32)
    compare(x.to(dtype), V, B, cuda_device, top_p=0.95, history=history, temperature=temperature, decay=decay)


@pytest.mark.parametrize("V,padded,B", [(17401, 17408, 560), (17404, 17408, 560), (17407, 17408, 560), (50257, 50264, 300)])
@pytest.mark.parametrize("temperature", [None, 1.3])
@pytest.mark.parametrize("penalised", [False, True])
def test_class_on_both_sides_of_the_threshold(V, padded, B, temperature, penalised, cuda_device):
    """Half values of which several have one probability: the top 3 % of a row hold the pass's threshold, one value in twenty is one of eight
    neighbouring ones, so the threshold lies among them and so does most of the draw.  The last columns are of these too."""
    g = torch.Generator(device=cuda_device)
    g.manual_seed(V + B)
    near = 0.4 + torch.randint(0, 8, (B, padded), generator=g, device=cuda_device) * 2.0 ** -12
    x = torch.randn(B, padded, generator=g, device=cuda_device) - 9.0
    x = torch.where(torch.rand(B, padded, generator=g, device=cuda_device) < 0.05, near, x)
    x[:, padded - 8:] = near[:, padded - 8:]
    x[:, 7] = 1.3
    history = torch.zeros(4, B, dtype=torch.int32, device=cuda_device)
    if penalised:
        history[:2] = torch.randint(padded - 8, V, (2, B), generator=g, device=cuda_device, dtype=torch.int32)
        history[2:] = torch.randint(1, V, (2, B), generator=g, device=cuda_device, dtype=torch.int32)
    compare(x.to(F16), V, B, cuda_device, top_p=0.98, history=history, temperature=temperature)


def test_maximum_of_two_values(cuda_device):
    """Two half values that a temperature rounds to one: the first column of either is the row's best one."""
    V, B = 17408, 560
    g = torch.Generator(device=cuda_device)
    g.manual_seed(5)
    # neighbours of [16, 32), 1 / 64 apart; divided by 1.3 they lie 0.012 apart, where half values do so by 1 / 128 and 1 / 64
    low = 24.0 + torch.arange(B, device=cuda_device) % 64 / 64.0
    x = torch.randn(B, V, generator=g, device=cuda_device) * 0.5 + 7.0
    x[:, 100], x[:, 9000] = low, low + 1 / 64.0
    scale = torch.tensor(1.0, device=cuda_device) / (torch.tensor(1.3, device=cuda_device) + 1e-6)
    y = (x.to(F16)[:, [100, 9000]] * scale.to(F16)).cpu()
    assert 50 < int((y[:, 0] == y[:, 1]).sum()) < B
    history = torch.zeros(4, B, dtype=torch.int32, device=cuda_device)
    compare(x.to(F16), V, B, cuda_device, top_p=0.3, history=history, temperature=1.3)
