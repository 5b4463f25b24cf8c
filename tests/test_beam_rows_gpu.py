"""The beam step against plain PyTorch at the sizes where its passes can go wrong: vocabularies below, at and above a tile
of 4096 columns, rows that start between two 16-byte boundaries, 2K at the edges of the bound's two forms, more equal
values than are collected, a history that goes through the segments of the parent chain, finished beams."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def expected(logits, cum, K, ids, parents, step, penalty, finished, end):
    """[B, K] words and scores of the K best continuations (fp32, first index wins ties), from float64 log-softmax."""
    B, _, V = logits.shape
    x = logits.double().cpu().numpy()
    for b in range(B):
        for k in range(K):
            if penalty != 1.0:
                seen, beam = {int(ids[step - 1, b, k])}, k
                for i in range(step - 2, -1, -1):
                    beam = int(parents[i, b, beam])
                    seen.add(int(ids[i, b, beam]))
                for v in seen:
                    x[b, k, v] = x[b, k, v] / penalty if x[b, k, v] > 0 else x[b, k, v] * penalty
    m = x.max(-1, keepdims=True)
    score = x - m - np.log(np.exp(x - m).sum(-1, keepdims=True)) + cum.reshape(B, K, 1)
    for b in range(B):
        for k in range(K):
            if finished[b * K + k]:
                score[b, k] = -np.inf
                score[b, k, end] = cum[b * K + k]
    flat = score.reshape(B, K * V)
    order = np.argsort(-flat, axis=1, kind="stable")[:, :K]
    return order, np.take_along_axis(flat, order, 1)


@pytest.mark.parametrize("B,K,V,step,penalty,ended", [
    (2, 2, 300, 1, 1.0, False), (3, 4, 4095, 2, 1.2, False), (3, 4, 4096, 70, 1.2, True), (2, 8, 4097, 300, 1.1, False),
    (2, 9, 8203, 33, 1.3, True), (1, 64, 20001, 5, 1.0, False), (2, 16, 40000, 9, 1.2, False), (2, 3, 16384, 65, 1.0, True)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
def test_beam_step_against_torch(dtype, B, K, V, step, penalty, ended, cuda_device):
    from fastertransformer_b200 import DynamicDecodeLayer
    g = torch.Generator(device=cuda_device)
    g.manual_seed(V + K)
    ints = dict(dtype=torch.int32, device=cuda_device)
    # distinct values per beam, whatever the type: a permutation of an even grid (bf16 keeps only some of them apart)
    x = torch.stack([torch.linspace(-3.0, 6.0, V, device=cuda_device)[torch.randperm(V, generator=g, device=cuda_device)]
                     for _ in range(B * K)]).view(B, K, V).to(dtype)
    st = {"output_ids": torch.randint(3, V, (step + 1, B, K), generator=g, **ints),
          "parent_ids": torch.randint(0, K, (step + 1, B, K), generator=g, **ints),
          "finished": torch.zeros(B * K, dtype=torch.bool, device=cuda_device),
          "sequence_length": torch.full((B * K,), step, **ints),
          "cum_log_probs": torch.randn(B * K, generator=g, device=cuda_device) - 5.0}
    if ended:
        st["finished"][1::3] = True
    before = {k: v.cpu().numpy().copy() for k, v in st.items()}
    args = {} if penalty == 1.0 else {"repetition_penalty": np.asarray([penalty], np.float32)}
    layer = DynamicDecodeLayer(V, V, dtype, cuda_device)
    layer.setup(B, K, args)
    layer.forward(st, dict(args, logits=x, step=step, max_input_length=1, ite=0, local_batch_size=B,
                           end_id=torch.full((B,), 2, **ints), input_lengths=torch.full((B, K), 1, **ints)))
    torch.cuda.synchronize()
    words, scores = expected(x.float(), before["cum_log_probs"], K, before["output_ids"], before["parent_ids"], step, penalty,
                             before["finished"], 2)
    got = st["cum_log_probs"].view(B, K).cpu().numpy()
    np.testing.assert_allclose(got, scores, rtol=2e-5, atol=2e-5)
    ids, par = st["output_ids"][step].cpu().numpy(), st["parent_ids"][step].cpu().numpy()
    near = np.abs(np.diff(scores, axis=1)).min(initial=1.0) < 1e-4  # two candidates too close to tell apart here
    if not near:
        np.testing.assert_array_equal(par * V + ids, words)
    # every chosen continuation has the score that is reported for it
    for b in range(B):
        assert len({(int(p), int(i)) for p, i in zip(par[b], ids[b])}) == K


def hot_columns(V, K, B, step, seed):
    """Logits whose largest columns are few and far apart in any type, prompt and parents, with penalised columns among
    the largest and beside them in the same word of a bit map, and one a power of two away."""
    rng = np.random.default_rng(seed)
    x = np.round(rng.uniform(-6.0, -2.0, size=(B, K, V)) * 8) / 8
    ids, parents = rng.integers(3, V, size=(step + 1, B, K)), rng.integers(0, K, size=(step + 1, B, K))
    m = step // K  # levels of each beam's columns; every beam's ancestry goes through all of them
    for b in range(B):
        level = rng.permutation(step)
        for k in range(K):
            cols = rng.choice(np.arange(40, V - 40), size=6 * K, replace=False)  # the largest first
            x[b, k, cols] = 1.0 + np.arange(6 * K)[::-1] / (4.0 if K < 8 else 16.0)
            near = np.stack([cols[:2 * K:2], cols[1:2 * K:2] ^ 1, (cols[2 * K:3 * K] + (1 << 19)) % V], 1).reshape(-1)[:m]
            ids[level[k * m:k * m + near.size], b] = near[:, None]
    return x, ids.astype(np.int32), parents.astype(np.int32)


@pytest.mark.parametrize("dtype,V,B,K,step,seed", [
    (torch.float32, 4097, 3, 4, 40, 1), (torch.bfloat16, 4097, 3, 4, 40, 1), (torch.bfloat16, 33001, 2, 9, 130, 1),
    # the last vocabulary that has a bit for every column, and ones with a filter and a list
    (torch.float32, 983040, 1, 2, 30, 1), (torch.float32, 983041, 1, 2, 30, 1), (torch.float32, 1200003, 2, 3, 600, 1),
    (torch.bfloat16, 1245184, 1, 2, 30, 1), (torch.bfloat16, 1245192, 1, 4, 300, 2)])
def test_penalised_columns_of_a_beam(dtype, V, B, K, step, seed, cuda_device):
    from fastertransformer_b200 import DynamicDecodeLayer
    x, ids, parents = hot_columns(V, K, B, step, seed)
    cum = -5.0 - np.random.default_rng(seed).uniform(0, 1, size=B * K).astype(np.float32)
    words, scores = expected(torch.from_numpy(x.copy()), cum, K, ids, parents, step, 1.25, np.zeros(B * K, bool), 2)
    assert np.abs(np.diff(scores, axis=1)).min() > 1e-3  # (nothing that rounding could turn round)
    ints = dict(dtype=torch.int32, device=cuda_device)
    st = {"output_ids": torch.from_numpy(ids).to(cuda_device), "parent_ids": torch.from_numpy(parents).to(cuda_device),
          "finished": torch.zeros(B * K, dtype=torch.bool, device=cuda_device), "sequence_length": torch.full((B * K,), step, **ints),
          "cum_log_probs": torch.from_numpy(cum).to(cuda_device)}
    args = {"repetition_penalty": np.asarray([1.25], np.float32)}
    layer = DynamicDecodeLayer(V, V, dtype, cuda_device)
    layer.setup(B, K, args)
    layer.forward(st, dict(args, logits=torch.from_numpy(x).to(device=cuda_device, dtype=dtype), step=step, max_input_length=1, ite=0,
                           local_batch_size=B, end_id=torch.full((B,), 2, **ints), input_lengths=torch.full((B, K), 1, **ints)))
    torch.cuda.synchronize()
    np.testing.assert_array_equal(st["parent_ids"][step].cpu().numpy() * V + st["output_ids"][step].cpu().numpy(), words)
    np.testing.assert_allclose(st["cum_log_probs"].view(B, K).cpu().numpy(), scores, rtol=2e-5, atol=2e-5)
