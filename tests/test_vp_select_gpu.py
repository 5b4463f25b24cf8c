"""Exchange records of all shards from one launch (16-bit logits): ids, flags and generator states must be those of the
unsharded layer at the edges of the kernel: rows off a 16-byte boundary, shards of fewer columns than threads, rows wide
enough for the larger block, k on both sides of the two thresholds, fewer selectable columns than k, ties that overflow
the candidate area, columns touched by penalties, bans and the minimum length, temperatures that merge values."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["f16", "bf16"])
@pytest.mark.parametrize("n_shards,shard,k,form", [
    (3, 1237, 5, "plain"), (2, 40, 30, "plain"), (4, 2047, 96, "plain"), (4, 2049, 97, "plain"), (2, 8191, 256, "plain"),
    (2, 9001, 257, "plain"), (2, 60008, 64, "plain"), (2, 60001, 192, "plain"), (2, 60001, 193, "plain"), (2, 7000, 1024, "plain"),
    (4, 3000, 40, "few"), (2, 12000, 20, "flat"), (3, 5003, 33, "hot"), (3, 5003, 33, "cold")])
def test_records_of_all_shards(dtype, n_shards, shard, k, form, cuda_device):
    from fastertransformer_b200 import DynamicDecodeLayer, VocabParallelSampler
    B, V, mil, steps = 9, n_shards * shard, 40, 2
    rng = np.random.default_rng(shard + k)
    temperature = {"hot": 5.0, "cold": 0.03}.get(form, 0.7)
    args = {"runtime_top_k": np.asarray([k], np.uint32), "runtime_top_p": np.asarray([0.92], np.float32),
            "temperature": np.asarray([temperature], np.float32), "repetition_penalty": np.asarray([1.3], np.float32),
            "min_length": np.asarray([50], np.int32), "random_seed": np.arange(B).astype(np.uint64)}
    prompt = torch.from_numpy(rng.integers(0, V, size=(mil, B)).astype(np.int32)).to(cuda_device)
    words = torch.from_numpy(np.stack([np.stack([rng.integers(1, V, 4), np.asarray([1, 2, 4, -1])]) for _ in range(B)])
                             .astype(np.int32)).to(cuda_device)

    def state():
        ids = torch.zeros(mil + steps, B, dtype=torch.int32, device=cuda_device)
        ids[:mil] = prompt
        done = torch.zeros(B, dtype=torch.bool, device=cuda_device)
        done[3] = True
        return {"output_ids": ids, "finished": done, "sequence_length": torch.full((B,), mil, dtype=torch.int32, device=cuda_device)}

    full = DynamicDecodeLayer(V, V, dtype, cuda_device)
    vp = VocabParallelSampler(V, shard, n_shards, dtype, cuda_device, cap_extra=3000 if form == "flat" else 64)
    full.setup(B, 1, args)
    vp.setup(B, 1, args)
    a, b = state(), state()
    g = torch.Generator(device=cuda_device)
    for s in range(steps):
        g.manual_seed(70 + s)
        x = torch.randn(B, V, generator=g, device=cuda_device) * 3.0
        x[:, 7] += 30.0  # (the end token, masked until the minimum length)
        x[torch.arange(B), prompt[0].long()] += 12.0
        if form == "few":  # one column in a thousand can be selected at all
            x[torch.rand(x.shape, generator=g, device=cuda_device) > 0.001] = -float("inf")
        if form == "flat":  # 6000 columns a shard share one value
            x[:, ::2] = 0.0
            x[:, 1::2].clamp_(max=-1.0)
            x[:, 3:40:2] = 2.0
        if form == "cold":
            x = (x * 4).round() / 4
        x = x.to(dtype)
        inp = {"step": mil + s, "max_input_length": mil, "end_id": torch.full((B,), 7, dtype=torch.int32, device=cuda_device),
               "input_lengths": torch.full((B,), mil - 3, dtype=torch.int32, device=cuda_device), "bad_words_list": words}
        full.forward(a, dict(inp, logits=x))
        vp.forward_shards(b, inp, [x[:, i * shard:(i + 1) * shard].contiguous() for i in range(n_shards)])
        torch.cuda.synchronize()
        if form == "flat":  # the class of the k-th value does not fit the records: every live row is reported
            assert vp.overflow_count() == (s + 1) * (B - 1)
            return
        assert vp.overflow_count() == 0
        for key in ("output_ids", "finished", "sequence_length"):
            assert torch.equal(a[key], b[key]), (s, key)
        assert torch.equal(full.topk.curand, vp.topk.curand)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["f16", "bf16"])
@pytest.mark.parametrize("penalised", [False, True])
@pytest.mark.parametrize("off,shard", [(1, 1237), (3, 40), (5, 2051), (7, 9001), (4, 60004)])
def test_shards_off_a_vector_boundary(dtype, penalised, off, shard, cuda_device):
    """Shards inside larger buffers, between two 16-byte boundaries: the first columns of the first row and the last ones
    of the last row do not travel with the whole vectors.  They hold the row's largest values, some of them penalised, and
    what lies around a shard would win if it were looked at."""
    from fastertransformer_b200 import DynamicDecodeLayer, VocabParallelSampler
    B, n, k, mil = 3, 2, 6, 6
    V = n * shard
    args = {"runtime_top_k": np.asarray([k], np.uint32), "random_seed": np.arange(B).astype(np.uint64)}
    if penalised:
        args["repetition_penalty"] = np.asarray([1.5], np.float32)
    g = torch.Generator(device=cuda_device)
    g.manual_seed(off * 100 + shard)
    x = torch.randn(B, V, generator=g, device=cuda_device)
    for i in range(n):
        x[0, i * shard:i * shard + 8] += 9.0 + torch.arange(8, device=cuda_device)
        x[-1, (i + 1) * shard - 8:(i + 1) * shard] += 9.0 + torch.arange(8, device=cuda_device)
    x = x.to(dtype)
    ids = torch.zeros(mil + 1, B, dtype=torch.int32, device=cuda_device)
    ids[:mil] = torch.tensor([[0, 0, V - 1], [2, 5, V - 2], [shard, 9, shard - 1], [shard + 1, 3, shard - 3], [7, 7, V - 8], [1, 1, 1]],
                             device=cuda_device)
    words = torch.tensor([[4, V - 4], [1, 2]], dtype=torch.int32, device=cuda_device)
    shards = []
    for i in range(n):
        buf = torch.full((off + B * shard + 8,), 1000.0, dtype=dtype, device=cuda_device)
        shards.append(buf[off:off + B * shard].view(B, shard))
        shards[-1].copy_(x[:, i * shard:(i + 1) * shard])
    got = []
    for layer in (DynamicDecodeLayer(V, V, dtype, cuda_device), VocabParallelSampler(V, shard, n, dtype, cuda_device)):
        layer.setup(B, 1, args)
        st = {"output_ids": ids.clone(), "finished": torch.zeros(B + 2, dtype=torch.bool, device=cuda_device)[1:B + 1],
              "sequence_length": torch.full((B,), mil, dtype=torch.int32, device=cuda_device)}
        inp = {"step": mil, "max_input_length": mil, "end_id": torch.full((B,), V // 2, dtype=torch.int32, device=cuda_device)}
        if penalised:
            inp["bad_words_list"] = words
        if isinstance(layer, VocabParallelSampler):
            layer.forward_shards(st, inp, shards)
        else:
            layer.forward(st, dict(inp, logits=x))
        torch.cuda.synchronize()
        got.append((st["output_ids"].cpu(), st["finished"].cpu(), st["sequence_length"].cpu(), layer.topk.curand.cpu()))
    for a, b in zip(*got):
        assert torch.equal(a, b)
