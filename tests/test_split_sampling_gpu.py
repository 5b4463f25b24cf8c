"""The split decode-sampling kernel (a row over a cluster of CTAs) against the general kernel, which the other tests pin
to the CPU restatement and the reference: everything a step writes has to be the same, bit for bit.  The sizes are the
edges of its split: chunks of 1024 columns, two / four / eight CTAs per row, rows that start between two 16-byte
boundaries, the largest slice, one row, and batches either side of "all rows resident"."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

F32, F16, BF16 = torch.float32, torch.float16, torch.bfloat16


def run(general, dtype, V, Vp, B, ties, log_probs, device):
    from fastertransformer_b200 import DynamicDecodeLayer, lib
    rng = np.random.default_rng(V + B)
    g = torch.Generator(device=device)
    g.manual_seed(V * 7 + B)
    step, mil = 40, 32
    ids = torch.randint(1, V, (step + 4, B), generator=g, device=device, dtype=torch.int32)
    st = {"output_ids": ids, "finished": torch.zeros(B, dtype=torch.bool, device=device),
          "sequence_length": torch.full((B,), step, dtype=torch.int32, device=device)}
    st["finished"][B // 2:B // 2 + 1] = B > 2
    if log_probs:
        st["cum_log_probs"] = torch.zeros(B, device=device)
        st["output_log_probs"] = torch.zeros(step + 4 - mil, B, device=device)
    args = {"runtime_top_k": rng.choice(np.asarray([0, 1, 7, 1024], np.uint32), size=B),
            "runtime_top_p": rng.choice(np.asarray([0.3, 0.9, 0.99], np.float32), size=B),
            "temperature": rng.choice(np.asarray([0.7, 1.0], np.float32), size=B),
            "repetition_penalty": rng.choice(np.asarray([0.8, 1.2], np.float32), size=B),
            "min_length": rng.choice(np.asarray([0, 30], np.int32), size=B),
            "random_seed": np.arange(B).astype(np.uint64)}
    words = torch.from_numpy(np.tile(np.asarray([[[3, 5, 6, 9], [1, 3, 4, -1]]], np.int32), (B, 1, 1))).to(device)
    lim = torch.full((B,), step + 2, dtype=torch.int32, device=device)
    layer = DynamicDecodeLayer(V, Vp, dtype, device)
    layer.setup(B, 1, args)
    lib.ftb200_set_single_pass(0 if general else 1)
    stops = []
    try:
        for s in range(3):
            x = torch.randn(B, Vp, generator=g, device=device) * 2.5
            x[::2, rng.integers(0, V, 3)] += 9.0
            if ties:
                x = (x * 4).round() / 4
            x[1::5, ::2] = -float("inf")
            stop = layer.forward(st, {"logits": x.to(dtype), "step": step + s, "max_input_length": mil, "ite": 0,
                                      "local_batch_size": B, "end_id": torch.full((B,), V - 1, dtype=torch.int32, device=device),
                                      "input_lengths": torch.full((B,), mil - 3, dtype=torch.int32, device=device),
                                      "bad_words_list": words, "stop_words_list": words, "sequence_limit_length": lim})
            stops.append(bool(stop))
        torch.cuda.synchronize()
    finally:
        lib.ftb200_set_single_pass(1)
    out = {k: v.cpu().numpy() for k, v in st.items()}
    out["curand"] = np.concatenate([layer.topk.curand.cpu().numpy(), layer.topp.curand.cpu().numpy()])
    out["stops"] = np.asarray(stops)
    return out


@pytest.mark.parametrize("dtype,V,Vp,B,ties,log_probs", [
    (F32, 1024, 1024, 1, False, False), (F32, 1025, 1032, 5, True, True), (F16, 2047, 2047, 3, False, True),
    (BF16, 40960, 40960, 37, True, False), (F16, 40961, 40963, 38, False, False), (F32, 16384, 16384, 74, False, True),
    (F32, 16385, 16388, 75, True, False), (BF16, 32000, 32000, 150, False, False), (BF16, 65537, 65543, 20, True, False),
    (F32, 128256, 128256, 9, False, False), (F32, 128256, 128256, 40, True, True), (BF16, 128257, 128257, 4, False, True),
    (F32, 350208, 350208, 3, False, False), (F32, 352257, 352260, 2, False, False)])
def test_split_kernel_equals_general_kernel(dtype, V, Vp, B, ties, log_probs, cuda_device):
    want = run(True, dtype, V, Vp, B, ties, log_probs, cuda_device)
    got = run(False, dtype, V, Vp, B, ties, log_probs, cuda_device)
    for k, v in want.items():
        np.testing.assert_array_equal(got[k], v, err_msg=k)
    assert want["stops"].tolist() == [False, False, True]


@pytest.mark.parametrize("dtype,V,B", [(BF16, 110003, 44), (F32, 60000, 80), (F16, 36000, 150)])
def test_wide_nuclei_of_many_rows(dtype, V, B, cuda_device):
    """Flat rows whose nucleus does not fit the first launch's areas, several to a cluster of the second one."""
    from fastertransformer_b200 import DynamicDecodeLayer, lib
    got = []
    for general in (1, 0):
        g = torch.Generator(device=cuda_device)
        g.manual_seed(V)
        layer = DynamicDecodeLayer(V, V, dtype, cuda_device)
        layer.setup(B, 1, {"runtime_top_p": np.asarray([0.98], np.float32), "temperature": np.asarray([1.1], np.float32),
                           "random_seed": np.arange(B).astype(np.uint64)})
        st = {"output_ids": torch.ones(12, B, dtype=torch.int32, device=cuda_device),
              "finished": torch.arange(B, device=cuda_device) % 9 == 4,
              "sequence_length": torch.full((B,), 8, dtype=torch.int32, device=cuda_device),
              "cum_log_probs": torch.zeros(B, device=cuda_device), "output_log_probs": torch.zeros(8, B, device=cuda_device)}
        lib.ftb200_set_single_pass(1 - general)
        try:
            for s in range(2):
                x = torch.randn(B, V, generator=g, device=cuda_device) * 0.8
                layer.forward(st, {"logits": x.to(dtype), "step": 8 + s, "max_input_length": 8, "ite": 0, "local_batch_size": B,
                                   "end_id": torch.full((B,), V - 1, dtype=torch.int32, device=cuda_device)})
            torch.cuda.synchronize()
        finally:
            lib.ftb200_set_single_pass(1)
        got.append({k: v.cpu().numpy() for k, v in st.items()} | {"curand": layer.topp.curand.cpu().numpy()})
    for k, v in got[0].items():
        np.testing.assert_array_equal(got[1][k], v, err_msg=k)


@pytest.mark.parametrize("dtype,V,B,sigma,grid,log_probs", [
    (F32, 20000, 5, 0.5, 0, False),     # a nucleus of most columns, several owners, sub-buckets of a key or two
    (F32, 50257, 9, 2.5, 0, True),      # either side of what the leader takes alone
    (F32, 50257, 66, 1.5, 0, False),    # four CTAs a row, owners at and above half of their area
    (F32, 128256, 3, 1.2, 0, False),    # eight owners with more keys than half of their area: stretch by stretch
    (BF16, 128256, 4, 1.5, 8, False),   # runs of thousands of equal keys: a bin that is larger than a stretch
    (BF16, 128256, 20, 2.0, 0, True), (F16, 51200, 40, 1.8, 0, True), (F16, 40960, 12, 1.0, 16, True)])
def test_nucleus_widths(dtype, V, B, sigma, grid, log_probs, cuda_device):
    """Top-p rows of every width: candidates of the leader, keys of one to eight owners, their sort in all its forms."""
    from fastertransformer_b200 import DynamicDecodeLayer, lib
    got = []
    for general in (1, 0):
        g = torch.Generator(device=cuda_device)
        g.manual_seed(V + B)
        p = np.resize(np.asarray([0.2, 0.5, 0.8, 0.9, 0.97], np.float32), B)
        layer = DynamicDecodeLayer(V, V, dtype, cuda_device)
        layer.setup(B, 1, {"runtime_top_p": p, "repetition_penalty": np.asarray([1.05], np.float32), "random_seed": np.arange(B).astype(np.uint64)})
        st = {"output_ids": torch.randint(1, V, (44, B), generator=g, device=cuda_device, dtype=torch.int32),
              "finished": torch.zeros(B, dtype=torch.bool, device=cuda_device),
              "sequence_length": torch.full((B,), 40, dtype=torch.int32, device=cuda_device)}
        if log_probs:
            st |= {"cum_log_probs": torch.zeros(B, device=cuda_device), "output_log_probs": torch.zeros(8, B, device=cuda_device)}
        lib.ftb200_set_single_pass(1 - general)
        try:
            for s in range(3):
                x = torch.randn(B, V, generator=g, device=cuda_device) * sigma
                x = (x * grid).round() / grid if grid else x
                layer.forward(st, {"logits": x.to(dtype), "step": 40 + s, "max_input_length": 40, "ite": 0, "local_batch_size": B,
                                   "end_id": torch.full((B,), V - 1, dtype=torch.int32, device=cuda_device)})
            torch.cuda.synchronize()
        finally:
            lib.ftb200_set_single_pass(1)
        got.append({k: v.cpu().numpy() for k, v in st.items()} | {"curand": layer.topp.curand.cpu().numpy()})
    for k, v in got[0].items():
        np.testing.assert_array_equal(got[1][k], v, err_msg=k)


def one_kind(general, kind, dtype, V, B, device):
    """Two steps of a call with top-k rows or top-p rows alone; what they wrote and the launches they took."""
    from fastertransformer_b200 import DynamicDecodeLayer, lib
    g = torch.Generator(device=device)
    g.manual_seed(V + 3 * B)
    args = {"random_seed": np.arange(B).astype(np.uint64), "repetition_penalty": np.asarray([1.1], np.float32)}
    if kind == "topk":
        args["runtime_top_k"] = np.asarray([40], np.uint32)
    else:
        args["runtime_top_p"] = np.asarray([0.9], np.float32)
    layer = DynamicDecodeLayer(V, V, dtype, device)
    layer.setup(B, 1, args)
    st = {"output_ids": torch.randint(1, V, (20, B), generator=g, device=device, dtype=torch.int32),
          "finished": torch.arange(B, device=device) % 7 == 5,
          "sequence_length": torch.full((B,), 16, dtype=torch.int32, device=device)}
    lib.ftb200_set_single_pass(0 if general else 1)
    try:
        for s in range(2):
            x = (torch.randn(B, V, generator=g, device=device) * 2.5).to(dtype)
            layer.forward(st, {"logits": x, "step": 16 + s, "max_input_length": 8,
                               "end_id": torch.full((B,), V - 1, dtype=torch.int32, device=device),
                               "sequence_limit_length": torch.full((B,), 99, dtype=torch.int32, device=device)})
        torch.cuda.synchronize()
    finally:
        lib.ftb200_set_single_pass(1)
    out = {k: v.cpu().numpy() for k, v in st.items()}
    out["curand"] = np.concatenate([layer.topk.curand.cpu().numpy(), layer.topp.curand.cpu().numpy()])
    return out, layer.launches // 2


@pytest.mark.parametrize("kind,dtype,V,B", [
    ("topk", BF16, 128256, 14), ("topk", BF16, 128256, 18), ("topk", F32, 128256, 18), ("topk", F32, 32000, 33),
    ("topk", F32, 32000, 37), ("topk", F32, 32000, 71), ("topk", F32, 32000, 74), ("topp", F32, 45000, 74), ("topp", F16, 17000, 148),
    ("topp", F16, 17000, 149), ("topp", BF16, 32000, 120), ("topp", F16, 41000, 94), ("topp", F16, 41000, 95),
    ("topp", BF16, 80000, 66), ("topp", BF16, 80000, 67)])
def test_calls_of_one_kind_around_the_resident_clusters(kind, dtype, V, B, cuda_device):
    """Sizes either side of the lines of the dispatch that follow from how many clusters are resident at once."""
    want, _ = one_kind(True, kind, dtype, V, B, cuda_device)
    got, launches = one_kind(False, kind, dtype, V, B, cuda_device)
    for k, v in want.items():
        np.testing.assert_array_equal(got[k], v, err_msg=k)
    if kind == "topk" and V == 128256 and B == 18 and torch.cuda.get_device_properties(0).multi_processor_count <= 148:
        assert launches > 1  # eighteen clusters of eight CTAs are not resident with one CTA on an SM


@pytest.mark.parametrize("general", [True, False])
def test_empty_word_in_front_of_a_list(general, cuda_device):
    """A word list whose first word is empty (its end offset is 0): nothing in front of the list is a token of it."""
    from fastertransformer_b200 import DynamicDecodeLayer, lib
    B, V = 5, 6000
    # tokens 4000 and 4001 in front of the list, 7 and 11 in it
    buf = torch.tensor([4000, 4001, 7, 11, 0, 0, 0, 1, 2, -1], dtype=torch.int32, device=cuda_device)
    words = buf[2:].view(2, 4)
    x = torch.zeros(B, V, device=cuda_device)
    x[:, 7], x[:, 11], x[:, 4001], x[:, 4000] = 9.0, 8.0, 7.0, 6.0
    layer = DynamicDecodeLayer(V, V, F32, cuda_device)
    layer.setup(B, 1, {"runtime_top_k": np.asarray([1], np.uint32)})
    st = {"output_ids": torch.ones(4, B, dtype=torch.int32, device=cuda_device),
          "finished": torch.zeros(B, dtype=torch.bool, device=cuda_device),
          "sequence_length": torch.full((B,), 2, dtype=torch.int32, device=cuda_device)}
    lib.ftb200_set_single_pass(0 if general else 1)
    try:
        layer.forward(st, {"logits": x, "step": 2, "max_input_length": 2, "bad_words_list": words,
                           "end_id": torch.full((B,), V - 1, dtype=torch.int32, device=cuda_device)})
        torch.cuda.synchronize()
    finally:
        lib.ftb200_set_single_pass(1)
    assert st["output_ids"][2].tolist() == [4001] * B


@pytest.mark.parametrize("limit", [True, False])
@pytest.mark.parametrize("dtype,V,B", [(F32, 50257, 6), (BF16, 128256, 9), (BF16, 128256, 40), (F32, 200000, 3)])
def test_stop_criteria_with_rows_left_to_another_launch(dtype, V, B, limit, cuda_device):
    """Stop words, and the count behind a length limit, when some rows' nuclei leave the first launch's areas: who serves a
    row sees to its words, and the host hears of the rows that are left."""
    from fastertransformer_b200 import DynamicDecodeLayer, lib
    got = []
    for general in (1, 0):
        g = torch.Generator(device=cuda_device)
        g.manual_seed(V + B)
        layer = DynamicDecodeLayer(V, V, dtype, cuda_device)
        layer.setup(B, 1, {"runtime_top_k": np.resize(np.asarray([0, 0, 5], np.uint32), B),
                           "runtime_top_p": np.resize(np.asarray([0.99, 0.3, 0.9], np.float32), B),
                           "random_seed": np.arange(B).astype(np.uint64)})
        st = {"output_ids": torch.ones(12, B, dtype=torch.int32, device=cuda_device),
              "finished": torch.arange(B, device=cuda_device) == B // 2,
              "sequence_length": torch.full((B,), 8, dtype=torch.int32, device=cuda_device)}
        stops = []
        lib.ftb200_set_single_pass(1 - general)
        try:
            for s in range(3):
                x = torch.randn(B, V, generator=g, device=cuda_device) * 0.5
                x[B - 1, :] = 0.0
                hot = torch.arange(B, device=cuda_device) % 3 != 0  # these stop by their second word; rows 0, 3, ... are flat
                x[hot, 77] = 30.0
                words = torch.tensor([[[5, 77, 0], [1, 2, -1]]] * B, dtype=torch.int32, device=cuda_device)
                words[1::2, 0, 1] = 78 if s == 0 else 77
                kw = {"sequence_limit_length": torch.full((B,), 10, dtype=torch.int32, device=cuda_device)} if limit else {}
                stop = layer.forward(st, {"logits": x.to(dtype), "step": 8 + s, "max_input_length": 8, "ite": 0, "local_batch_size": B,
                                          "end_id": torch.full((B,), V - 1, dtype=torch.int32, device=cuda_device),
                                          "stop_words_list": words, **kw})
                stops.append(bool(stop))
                stops.append(st["finished"].cpu().numpy().copy())
            torch.cuda.synchronize()
        finally:
            lib.ftb200_set_single_pass(1)
        got.append({k: v.cpu().numpy() for k, v in st.items()} | {"stops": np.hstack([np.atleast_1d(v) for v in stops])})
    for k, v in got[0].items():
        np.testing.assert_array_equal(got[1][k], v, err_msg=k)
    assert got[0]["stops"][1 + 0:1 + B].any() and not got[0]["stops"][1:1 + B].all()


@pytest.mark.parametrize("dtype,V,B", [(F32, 16385, 5), (F16, 50257, 6), (BF16, 32001, 7), (BF16, 114514, 3), (F16, 4096, 2)])
def test_bias_beside_rows_off_a_boundary(dtype, V, B, cuda_device):
    """An embedding bias, rows that start between two 16-byte boundaries (and one size that does not)."""
    from fastertransformer_b200 import DynamicDecodeLayer, lib
    got = []
    for general in (1, 0):
        g = torch.Generator(device=cuda_device)
        g.manual_seed(V)
        layer = DynamicDecodeLayer(V, V, dtype, cuda_device)
        layer.setup(B, 1, {"runtime_top_k": np.resize(np.asarray([0, 40], np.uint32), B), "runtime_top_p": np.asarray([0.9], np.float32),
                           "temperature": np.asarray([0.7], np.float32), "random_seed": np.arange(B).astype(np.uint64)})
        st = {"output_ids": torch.ones(12, B, dtype=torch.int32, device=cuda_device),
              "finished": torch.zeros(B, dtype=torch.bool, device=cuda_device),
              "sequence_length": torch.full((B,), 8, dtype=torch.int32, device=cuda_device),
              "cum_log_probs": torch.zeros(B, device=cuda_device), "output_log_probs": torch.zeros(8, B, device=cuda_device)}
        bias = (torch.randn(V, generator=g, device=cuda_device) * 2).to(dtype)
        lib.ftb200_set_single_pass(1 - general)
        try:
            for s in range(3):
                x = torch.randn(B, V, generator=g, device=cuda_device) * 2
                layer.forward(st, {"logits": x.to(dtype), "step": 8 + s, "max_input_length": 8, "ite": 0, "local_batch_size": B,
                                   "embedding_bias": bias, "end_id": torch.full((B,), V - 1, dtype=torch.int32, device=cuda_device)})
            torch.cuda.synchronize()
        finally:
            lib.ftb200_set_single_pass(1)
        got.append({k: v.cpu().numpy() for k, v in st.items()})
    for k, v in got[0].items():
        np.testing.assert_array_equal(got[1][k], v, err_msg=k)
