"""ftb200_decode_step, the whole step in one call, where its parts can come apart: a batch in slices under a length limit (the
criteria count the whole batch, a slice's kernel serves its own rows), in each of the forms a step can take - the kernel
that does the criteria itself, the split kernel with a second launch, the single-pass kernels - and a deadline that runs
out while the stream is held by a sleeping host function (nothing on the GPU waits)."""
import ctypes as C
import gc
import time

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

F32, F16, BF16 = torch.float32, torch.float16, torch.bfloat16
MIL = 8


def build(dtype, V, B, device, stop_words, limits):
    rng = np.random.default_rng(V + B)
    from fastertransformer_b200 import DynamicDecodeLayer
    layer = DynamicDecodeLayer(V, V, dtype, device)
    layer.setup(B, 1, {"runtime_top_k": rng.choice(np.asarray([0, 1, 30], np.uint32), size=B),
                       "runtime_top_p": np.asarray([0.8], np.float32), "random_seed": np.arange(B).astype(np.uint64)})
    st = {"output_ids": torch.ones(MIL + 8, B, dtype=torch.int32, device=device),
          "finished": torch.zeros(B, dtype=torch.bool, device=device),
          "sequence_length": torch.full((B,), MIL, dtype=torch.int32, device=device)}
    inputs = {"max_input_length": MIL, "end_id": torch.full((B,), V - 1, dtype=torch.int32, device=device),
              "sequence_limit_length": torch.from_numpy(limits).to(device)}
    if stop_words:
        # [1] for every third row (its history), [0] - a token nobody draws here - for the others
        words = np.zeros((B, 2, 1), np.int32)
        words[::3, 0], words[:, 1] = 5, 1
        inputs["stop_words_list"] = torch.from_numpy(words).to(device)
    return layer, st, inputs


def logits(dtype, V, B, step, device):
    g = torch.Generator(device=device)
    g.manual_seed(step)
    x = torch.randn(B, V, generator=g, device=device) * 2
    x[:, 5] += 14.0 * (torch.arange(B, device=device) % 2 == step % 2)  # a row draws token 5 in every other step
    return x.to(dtype)


@pytest.mark.parametrize("stop_words", [False, True])
@pytest.mark.parametrize("dtype,V,B,slices", [(F32, 5003, 12, 3), (F16, 32000, 15, 5), (F32, 32000, 300, 3), (BF16, 32768, 1040, 2),
                                              (F32, 600, 9, 3)])
def test_slices_under_a_length_limit(dtype, V, B, slices, stop_words, cuda_device):
    limits = (MIL + 1 + np.arange(B) % 4).astype(np.int32)  # the last rows end in the fifth step
    limits[0] = MIL + 4
    n = B // slices
    got = []
    for whole_step in (True, False):
        layer, st, inputs = build(dtype, V, B, cuda_device, stop_words, limits)
        layer.time_kernels = not whole_step  # (then sampling, criteria and wait are calls of their own)
        stops = []
        for s in range(5):
            x = logits(dtype, V, B, MIL + s, cuda_device)
            for i in range(slices):
                stop = layer.forward(st, dict(inputs, logits=x, step=MIL + s, ite=i, local_batch_size=n))
                # what the host was told is what the flags say
                assert stop == bool(st["finished"].all()), (whole_step, s, i)
                stops.append(stop)
        got.append({k: v.cpu() for k, v in st.items()} | {"stops": torch.tensor(stops), "curand": layer.topk.curand.cpu()})
    for k in got[0]:
        assert torch.equal(got[0][k], got[1][k]), k
    assert got[0]["stops"].tolist()[:slices] == [False] * slices and got[0]["stops"][-1]


@pytest.mark.parametrize("dtype,V,B", [(F32, 5003, 6), (F32, 32000, 300), (BF16, 32768, 520)])
def test_deadline_runs_out(dtype, V, B, cuda_device):
    from fastertransformer_b200 import lib
    rt = C.CDLL("libcudart.so.12")
    HOSTFN = C.CFUNCTYPE(None, C.c_void_p)
    hold = HOSTFN(lambda _: time.sleep(0.3))
    rt.cudaLaunchHostFunc.argtypes = [C.c_void_p, HOSTFN, C.c_void_p]
    limits = np.full(B, MIL + 3, np.int32)
    xs = [logits(dtype, V, B, MIL + s, cuda_device) for s in range(4)]
    got = []
    for late in (False, True):
        layer, st, inputs = build(dtype, V, B, cuda_device, False, limits)
        stream = torch.cuda.Stream(device=cuda_device)
        stops = []
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            for s in range(4):
                if late and s == 1:
                    # the block of the step before, moved on by hand, for a deadline of its own
                    P, stop = layer._gate[0, B]["params"], C.c_int(-7)
                    P.step, P.logits = MIL + s, xs[s].data_ptr()
                    assert rt.cudaLaunchHostFunc(C.c_void_p(stream.cuda_stream), hold, None) == 0
                    assert lib.ftb200_decode_step(layer._gate[0, B]["params_ref"], layer._stop_ref, 20, C.byref(stop)) == 6
                    assert stop.value == 0 and b"deadline" in lib.ftb200_last_error_string()
                    stream.synchronize()  # the step itself was launched and ends
                    stops.append(bool(st["finished"].all()))
                    continue
                stops.append(layer.forward(st, dict(inputs, logits=xs[s], step=MIL + s)))
        torch.cuda.synchronize()
        assert stops == [False, False, False, True]
        got.append({k: v.cpu() for k, v in st.items()} | {"curand": layer.topk.curand.cpu()})
    for k in got[0]:
        assert torch.equal(got[0][k], got[1][k]), k


@pytest.mark.parametrize("one_call", [True, False])
def test_word_of_a_late_step_is_kept(one_call, cuda_device):
    """A layer that is dropped after its step missed the deadline: the step still writes its page-locked word, which must
    not have become somebody else's by then."""
    from fastertransformer_b200._lib import FtbError
    rt = C.CDLL("libcudart.so.12")
    HOSTFN = C.CFUNCTYPE(None, C.c_void_p)
    hold = HOSTFN(lambda _: time.sleep(0.3))
    rt.cudaLaunchHostFunc.argtypes = [C.c_void_p, HOSTFN, C.c_void_p]
    layer, st, inputs = build(F32, 5003, 6, cuda_device, False, np.full(6, MIL + 9, np.int32))
    layer.time_kernels = not one_call
    x = logits(F32, 5003, 6, 0, cuda_device)
    layer.forward(st, dict(inputs, logits=x, step=MIL))
    layer.deadline_ms = 20
    word = (layer._result if one_call else layer._count_host).data_ptr()
    stream = torch.cuda.Stream(device=cuda_device)
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        assert rt.cudaLaunchHostFunc(C.c_void_p(stream.cuda_stream), hold, None) == 0
        with pytest.raises(FtbError, match="deadline"):
            layer.forward(st, dict(inputs, logits=x, step=MIL + 1))
        del layer
        gc.collect()
        others = [torch.zeros(n, dtype=torch.int64).pin_memory() for n in (1, 1, 1, 1, 8, 64)]
        assert not stream.query() and word not in [t.data_ptr() for t in others]
    stream.synchronize()
    assert all(int(t.abs().sum()) == 0 for t in others)


@pytest.mark.parametrize("dtype,kind,V,B", [(F16, "topp", 41000, 37), (BF16, "topk", 128256, 18), (F32, "topk", 32000, 74),
                                            (F16, "topp", 32000, 120)])
def test_step_under_capture(dtype, kind, V, B, cuda_device):
    """A step whose size the library has not met before, recorded in a graph: the dispatch asks for occupancies then."""
    from fastertransformer_b200 import DynamicDecodeLayer

    def run(columns, capture):
        layer = DynamicDecodeLayer(columns, columns, dtype, cuda_device)
        layer.setup(B, 1, {"runtime_top_k": np.asarray([40], np.uint32)} if kind == "topk" else
                    {"runtime_top_p": np.asarray([0.9], np.float32)})
        st = {"output_ids": torch.ones(MIL + 2, B, dtype=torch.int32, device=cuda_device),
              "finished": torch.zeros(B, dtype=torch.bool, device=cuda_device),
              "sequence_length": torch.full((B,), MIL, dtype=torch.int32, device=cuda_device)}
        inputs = {"max_input_length": MIL, "step": MIL, "logits": logits(dtype, columns, B, 3, cuda_device),
                  "end_id": torch.full((B,), columns - 1, dtype=torch.int32, device=cuda_device)}
        torch.cuda.synchronize()
        if capture:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                layer.forward(st, inputs)
            assert int(st["output_ids"][MIL, 0]) == 1  # (recorded, not run)
            graph.replay()
        else:
            layer.forward(st, inputs)
        torch.cuda.synchronize()
        return st["output_ids"][MIL].cpu(), layer.topk.curand.cpu(), layer.topp.curand.cpu()

    run(V + 1024, False)  # (the kernels are loaded; the size of the recorded step is a new one)
    recorded, direct = run(V, True), run(V, False)
    for a, b in zip(recorded, direct):
        assert torch.equal(a, b)


@pytest.mark.parametrize("form", ["plain", "bias", "words", "limit", "log_probs", "all", "other_buffers"])
def test_native_step_equals_the_python_code(form, cuda_device, monkeypatch):
    """forward() through the step module and through the code beside it: every optional entry, and buffers that change from
    step to step."""
    from fastertransformer_b200 import DynamicDecodeLayer, decode_layer
    V, B, got = 9000, 5, []
    for native in (True, False):
        with monkeypatch.context() as m:
            if not native:
                m.setattr(decode_layer, "_LIBRARY", object())
            g = torch.Generator(device=cuda_device)
            g.manual_seed(3)
            layer = DynamicDecodeLayer(V, V, torch.float16, cuda_device)
            layer.setup(B, 1, {"runtime_top_k": np.asarray([0, 1, 9, 0, 64], np.uint32), "runtime_top_p": np.asarray([0.8], np.float32),
                               "repetition_penalty": np.asarray([1.1], np.float32), "random_seed": np.arange(B).astype(np.uint64)})
            st = {"output_ids": torch.ones(14, B, dtype=torch.int32, device=cuda_device),
                  "finished": torch.zeros(B, dtype=torch.bool, device=cuda_device),
                  "sequence_length": torch.full((B,), 8, dtype=torch.int32, device=cuda_device)}
            if form in ("log_probs", "all"):
                st["cum_log_probs"] = torch.zeros(B, device=cuda_device)
                st["output_log_probs"] = torch.zeros(6, B, device=cuda_device)
            extra = {}
            if form in ("bias", "all"):
                extra["embedding_bias"] = torch.randn(V, generator=g, device=cuda_device).half()
            if form in ("words", "all"):
                extra["stop_words_list"] = torch.tensor([[[7, 1, 9], [1, 3, -1]]] * B, dtype=torch.int32, device=cuda_device)
                extra["bad_words_list"] = torch.tensor([[5], [1]], dtype=torch.int32, device=cuda_device)
            if form in ("limit", "all"):
                extra["sequence_limit_length"] = torch.full((B,), 11, dtype=torch.int32, device=cuda_device)
            if form == "all":
                extra["input_lengths"] = torch.full((B,), 6, dtype=torch.int32, device=cuda_device)
            stops = []
            for s in range(4):
                x = (torch.randn(B, V, generator=g, device=cuda_device) * 3).half()
                if form == "other_buffers" and s == 2:
                    st = {k: v.clone() for k, v in st.items()}
                stops.append(bool(layer.forward(st, {"logits": x, "step": 8 + s, "max_input_length": 8, "ite": 0, "local_batch_size": B,
                                                     "end_id": torch.full((B,), V - 1, dtype=torch.int32, device=cuda_device), **extra})))
            torch.cuda.synchronize()
            assert (layer._native is not None) == native
            got.append({k: v.cpu().numpy() for k, v in st.items()} | {"stops": np.asarray(stops), "launches": np.asarray(layer.launches)})
    for k, v in got[1].items():
        np.testing.assert_array_equal(got[0][k], v, err_msg=k)


@pytest.mark.parametrize("types", [(F16, BF16, F16), (F16, F32, F16, F16), (F32, BF16, F16, F32)])
def test_logits_types_in_turn(types, cuda_device):
    """One layer whose logits change their type from call to call, against the maxima of each call's logits."""
    from fastertransformer_b200 import DynamicDecodeLayer
    V, B = 9001, 5
    layer = DynamicDecodeLayer(V, V, types[0], cuda_device)
    layer.setup(B, 1, {"runtime_top_k": np.asarray([1], np.uint32)})
    st = {"output_ids": torch.ones(MIL + 4, B, dtype=torch.int32, device=cuda_device),
          "finished": torch.zeros(B, dtype=torch.bool, device=cuda_device),
          "sequence_length": torch.full((B,), MIL, dtype=torch.int32, device=cuda_device)}
    for s, dtype in enumerate(types):
        x = torch.full((B, V), -8.0, device=cuda_device)
        want = torch.tensor([(s + 1) * (977 + b) % (V - 1) for b in range(B)], device=cuda_device)
        x[torch.arange(B), want] = 8.0  # (exact in every type)
        layer.forward(st, {"logits": x.to(dtype), "step": MIL + s, "max_input_length": MIL,
                           "end_id": torch.full((B,), V - 1, dtype=torch.int32, device=cuda_device)})
        assert torch.equal(st["output_ids"][MIL + s].long(), want), s


@pytest.mark.parametrize("dtype,V,B", [(F32, 50257, 6), (BF16, 128256, 9), (BF16, 128256, 40), (F32, 200000, 3)])
def test_deadline_runs_out_with_rows_left(dtype, V, B, cuda_device):
    """Rows that the first launch cannot hold, in a step whose deadline passes before that launch has run: the step ends by
    itself all the same - each row's token, generator and stop word, the limit, the count in the word."""
    from fastertransformer_b200 import DynamicDecodeLayer
    from fastertransformer_b200._lib import FtbError
    rt = C.CDLL("libcudart.so.12")
    HOSTFN = C.CFUNCTYPE(None, C.c_void_p)
    hold = HOSTFN(lambda _: time.sleep(0.3))
    rt.cudaLaunchHostFunc.argtypes = [C.c_void_p, HOSTFN, C.c_void_p]
    got = []
    for late in (False, True):
        g = torch.Generator(device=cuda_device)
        g.manual_seed(V + B)
        layer = DynamicDecodeLayer(V, V, dtype, cuda_device)
        layer.setup(B, 1, {"runtime_top_k": np.resize(np.asarray([0, 0, 5], np.uint32), B),
                           "runtime_top_p": np.resize(np.asarray([0.99, 0.3, 0.9], np.float32), B),
                           "random_seed": np.arange(B).astype(np.uint64)})
        st = {"output_ids": torch.full((MIL + 4, B), -1, dtype=torch.int32, device=cuda_device),
              "finished": torch.arange(B, device=cuda_device) == B - 1,
              "sequence_length": torch.full((B,), MIL, dtype=torch.int32, device=cuda_device)}
        limits = torch.full((B,), MIL + 3, dtype=torch.int32, device=cuda_device)
        limits[0] = MIL + 1
        words = torch.tensor([[[77], [1]]] * B, dtype=torch.int32, device=cuda_device)
        stream = torch.cuda.Stream(device=cuda_device)
        torch.cuda.synchronize()
        for s in range(3):
            x = torch.randn(B, V, generator=g, device=cuda_device) * 0.5  # (flat: the rows of p = 0.99 keep most of the columns)
            x[1, 77] = 30.0
            inputs = {"logits": x.to(dtype), "step": MIL + s, "max_input_length": MIL, "stop_words_list": words,
                      "end_id": torch.full((B,), V - 1, dtype=torch.int32, device=cuda_device), "sequence_limit_length": limits}
            torch.cuda.synchronize()
            with torch.cuda.stream(stream):
                if late and s == 1:
                    layer.deadline_ms = 20
                    assert rt.cudaLaunchHostFunc(C.c_void_p(stream.cuda_stream), hold, None) == 0
                    with pytest.raises(FtbError, match="deadline"):
                        layer.forward(st, inputs)
                    layer.deadline_ms = 10000
                    stream.synchronize()
                else:
                    layer.forward(st, inputs)
            # the word holds (calls so far, finished rows), whatever the host has waited for
            assert int(layer._result) == (s + 1) << 32 | int(st["finished"].sum()) and int(layer._arrived) == 0
        torch.cuda.synchronize()
        got.append({k: v.cpu() for k, v in st.items()} | {"topk": layer.topk.curand.cpu(), "topp": layer.topp.curand.cpu()})
    for k in got[0]:
        assert torch.equal(got[0][k], got[1][k]), k
    assert int(got[0]["output_ids"][MIL + 1].min()) >= 0 and int(got[0]["finished"].sum()) >= 3
