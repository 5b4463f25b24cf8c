"""What setup() leaves behind, without a GPU: the upload and the kernel of a set-up are on one stream, and that stream has
been waited for when setup() returns, so that a step may follow on any other stream."""
import contextlib
import types

import numpy as np
import pytest
import torch

from fastertransformer_b200 import decode_layer


@pytest.mark.parametrize("own_stream", [False, True])
def test_setup_ends_synchronised(own_stream, monkeypatch):
    log = []

    def stream(handle):
        return types.SimpleNamespace(cuda_stream=handle, synchronize=lambda: log.append(("synchronize", handle)))

    def place(pack, device):
        log.append(("place", None))
        for owner, name, dtype, _, size, _ in pack.parts:
            setattr(owner, name, torch.zeros(size, dtype=torch.uint8).view(dtype))
        return torch.zeros(1)

    def setup_sampling(block):
        log.append(("setup", block._obj.stream or 0))
        return 0

    monkeypatch.setattr(decode_layer._Pack, "place", place)
    monkeypatch.setattr(decode_layer, "lib", types.SimpleNamespace(ftb200_setup_sampling=setup_sampling))
    monkeypatch.setattr(decode_layer, "_raw_stream", lambda index: 7)
    monkeypatch.setattr(torch.cuda, "stream", lambda s: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: stream(7))
    layer = decode_layer.DynamicDecodeLayer(100, 104, torch.float16, "cuda:0", stream(5) if own_stream else None)
    layer.setup(3, 1, {"runtime_top_k": np.asarray([4], np.uint32), "random_seed": np.asarray([1, 2, 3], np.uint64)})
    on = 5 if own_stream else 7
    assert log == [("place", None), ("setup", on), ("synchronize", on)]
