"""The end of a step that waits, single-pass kernels: once the call has returned, nothing of the step is queued that could still read its
workspace, so that the caller may use it on another stream at once."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

F16, BF16 = torch.float16, torch.bfloat16


def make(dtype, V, B, kinds, device, penalty=1.1):
    from fastertransformer_b200 import DynamicDecodeLayer
    args = {"random_seed": np.arange(B).astype(np.uint64), "repetition_penalty": np.resize(np.asarray(penalty, np.float32), B)}
    if kinds != "topk":
        args["runtime_top_p"] = np.asarray([0.9], np.float32)
    if kinds != "topp":
        args["runtime_top_k"] = np.resize(np.asarray({"both": [0, 40, 1], "wide": [0, 1024, 1], "topk": [40]}[kinds], np.uint32), B)
    layer = DynamicDecodeLayer(V, V, dtype, device)
    layer.setup(B, 1, args)
    return layer


def run(layer, x, ids, step, limit):
    B, V = x.shape
    device = x.device
    st = {"output_ids": ids, "finished": torch.zeros(B, dtype=torch.bool, device=device),
          "sequence_length": torch.full((B,), step, dtype=torch.int32, device=device)}
    inputs = {"logits": x, "step": step, "max_input_length": step, "end_id": torch.full((B,), V - 1, dtype=torch.int32, device=device)}
    if limit:
        inputs["sequence_limit_length"] = torch.full((B,), step + 9, dtype=torch.int32, device=device)
    torch.cuda.synchronize()
    assert not layer.forward(st, inputs)
    return st


@pytest.mark.parametrize("kinds,penalty,launches", [
    ("topk", 1.1, 2), ("topp", 1.1, 2), ("both", 1.1, 3),  # the header's kernel, then the rows' kernels
    ("topp", [1.1, 0.9], 3), ("both", [1.1, 1.1, 0.9, 0.9], 4),  # rows whose penalty raises values are left: sent for
    ("wide", 1.1, 4)])  # k = 1024 of few columns is always left: the general kernel is queued and ends the step
def test_nothing_behind_the_end(kinds, penalty, launches, cuda_device):
    from fastertransformer_b200 import lib
    V, B = 32768, 560
    layer = make(BF16, V, B, kinds, cuda_device, penalty)
    x = (torch.randn(B, V, device=cuda_device) * 2.5).to(BF16)
    for _ in range(2):  # (the first such step on a device queues the general kernel, which loads it)
        run(layer, x, torch.ones(12, B, dtype=torch.int32, device=cuda_device), 8, True)
    assert lib.ftb200_last_launch_count() == launches


@pytest.mark.parametrize("dtype,V,B,kinds,penalty", [
    (BF16, 32768, 560, "both", 1.1), (BF16, 128256, 200, "both", 1.1), (F16, 17408, 1024, "topp", 1.1),
    (F16, 32768, 560, "both", [1.1, 0.9, 1.1]), (BF16, 32768, 560, "wide", 1.1)])
def test_workspace_is_free_at_the_end(dtype, V, B, kinds, penalty, cuda_device):
    """Two streams take turns with one layer, ordered by nothing but the host's wait; the workspace is written over in between."""
    g = torch.Generator(device=cuda_device)
    g.manual_seed(V + B)
    rounds = 12
    xs = [(torch.randn(B, V, generator=g, device=cuda_device) * 2.5).to(dtype) for _ in range(4)]
    history = torch.randint(1, V, (20, B), generator=g, device=cuda_device, dtype=torch.int32)
    results = []
    for turns in (False, True):
        layer = make(dtype, V, B, kinds, cuda_device, penalty)
        streams = [torch.cuda.Stream(cuda_device) for _ in range(2 if turns else 1)]
        ids = [history.clone() for _ in range(rounds)]
        states = [{"output_ids": i, "finished": torch.zeros(B, dtype=torch.bool, device=cuda_device),
                   "sequence_length": torch.full((B,), 16, dtype=torch.int32, device=cuda_device)} for i in ids]
        inputs = [{"logits": x, "step": 16, "max_input_length": 16,
                   "end_id": torch.full((B,), V - 1, dtype=torch.int32, device=cuda_device),
                   "sequence_limit_length": torch.full((B,), 99, dtype=torch.int32, device=cuda_device)} for x in xs]
        torch.cuda.synchronize()
        for i in range(rounds):
            with torch.cuda.stream(streams[i % len(streams)]):
                if turns and i > 0:
                    layer._workspace[:4096].fill_(1)
                assert not layer.forward(states[i], inputs[i % 4])
        torch.cuda.synchronize()
        results.append([s[k].cpu().numpy() for s in states for k in ("output_ids", "sequence_length", "finished")])
    for want, got in zip(*results):
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("dtype,V,B,kinds", [(BF16, 32768, 560, "both"), (F16, 32768, 560, "wide"), (BF16, 17408, 1024, "topp")])
def test_kernels_side_by_side_under_capture(dtype, V, B, kinds, cuda_device):
    """The kernels that follow each other without a wait in between, recorded in a graph; the logits and everything else are written
    right in front of each replay."""
    g = torch.Generator(device=cuda_device)
    g.manual_seed(V)
    xs = [(torch.randn(B, V, generator=g, device=cuda_device) * 2.5).to(dtype) for _ in range(6)]
    results = []
    for capture in (False, True):
        layer = make(dtype, V, B, kinds, cuda_device)
        x, step = torch.zeros_like(xs[0]), 8
        st = {"output_ids": torch.ones(step + 2, B, dtype=torch.int32, device=cuda_device),
              "finished": torch.zeros(B, dtype=torch.bool, device=cuda_device),
              "sequence_length": torch.full((B,), step, dtype=torch.int32, device=cuda_device)}
        inputs = {"logits": x, "step": step, "max_input_length": step, "end_id": torch.full((B,), V - 1, dtype=torch.int32, device=cuda_device)}
        call = lambda: layer.forward(st, inputs)
        if capture:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                call()
            call = graph.replay
        got = []
        for logits in xs:
            x.copy_(logits)
            st["output_ids"][:step] = torch.arange(B, device=cuda_device, dtype=torch.int32) % 997
            call()
            got.append(st["output_ids"].clone())
        torch.cuda.synchronize()
        results.append([t.cpu().numpy() for t in got] + [layer.topk.curand.cpu().numpy(), layer.topp.curand.cpu().numpy()])
    for want, got in zip(*results):
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("kinds,penalty", [("both", [1.1, 0.9, 1.1]), ("topp", 1.1), ("wide", 1.1)])
def test_deadline_with_rows_on_the_list(kinds, penalty, cuda_device):
    """A step that misses its deadline while the stream is held sends what serves the rows left, and ends by itself."""
    import ctypes as C
    import time

    from fastertransformer_b200 import lib
    rt = C.CDLL("libcudart.so.12")
    HOSTFN = C.CFUNCTYPE(None, C.c_void_p)
    hold = HOSTFN(lambda _: time.sleep(0.3))
    rt.cudaLaunchHostFunc.argtypes = [C.c_void_p, HOSTFN, C.c_void_p]
    V, B, step = 32768, 560, 8
    g = torch.Generator(device=cuda_device)
    g.manual_seed(1)
    xs = [(torch.randn(B, V, generator=g, device=cuda_device) * 2.5).to(BF16) for _ in range(3)]
    got = []
    for late in (False, True):
        layer = make(BF16, V, B, kinds, cuda_device, penalty)
        st = {"output_ids": torch.ones(step + 4, B, dtype=torch.int32, device=cuda_device),
              "finished": torch.zeros(B, dtype=torch.bool, device=cuda_device),
              "sequence_length": torch.full((B,), step, dtype=torch.int32, device=cuda_device)}
        inputs = {"max_input_length": step, "end_id": torch.full((B,), V - 1, dtype=torch.int32, device=cuda_device),
                  "sequence_limit_length": torch.full((B,), step + 2, dtype=torch.int32, device=cuda_device)}
        stream, stops = torch.cuda.Stream(device=cuda_device), []
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            for s in range(3):
                if late and s == 1:
                    P, stop = layer._gate[0, B]["params"], C.c_int(-7)
                    P.step, P.logits = step + s, xs[s].data_ptr()
                    assert rt.cudaLaunchHostFunc(C.c_void_p(stream.cuda_stream), hold, None) == 0
                    assert lib.ftb200_decode_step(layer._gate[0, B]["params_ref"], layer._stop_ref, 20, C.byref(stop)) == 6
                    stream.synchronize()
                    stops.append(bool(st["finished"].all()))
                    continue
                stops.append(layer.forward(st, dict(inputs, logits=xs[s], step=step + s)))
        torch.cuda.synchronize()
        assert stops == [False, False, True]
        got.append([v.cpu().numpy() for v in st.values()] + [layer.topk.curand.cpu().numpy(), layer.topp.curand.cpu().numpy()])
    for want, have in zip(*got):
        np.testing.assert_array_equal(have, want)
