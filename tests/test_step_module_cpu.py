"""The native step (host/step_module.c) on the CPU, linked to a library that records the argument blocks it is given: what
reaches the library is the call's own, whatever calls came before it."""
import ctypes as C
import os
import subprocess
import sys
import sysconfig
import types

import numpy as np
import pytest
import torch

from fastertransformer_b200 import decode_layer
from fastertransformer_b200._abi import SamplingParams

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RECORDER = r"""
#include "ftb200.h"
ftb200_sampling_params recorded[16];
int                    calls;
int ftb200_decode_step_sampling(const ftb200_sampling_params* p) { recorded[calls++] = *p; return 0; }
int ftb200_decode_step(const ftb200_sampling_params* p, ftb200_stop_params* s, int ms, int* stop) { return *stop = 0, ftb200_decode_step_sampling(p); }
int ftb200_last_launch_count(void) { return 1; }
int ftb200_setup_sampling(const ftb200_setup_params* p) { return 0; }
int ftb200_sampling_workspace_bytes(int dtype, int rows, int padded, size_t* bytes) { return *bytes = 64, 0; }
"""


@pytest.fixture(scope="module")
def recorder(tmp_path_factory):
    """The module and the recording library in one file: (module, library)."""
    import importlib.util
    at = tmp_path_factory.mktemp("step")
    (at / "recorder.c").write_text(RECORDER)
    out = at / "_ftb200_step.so"
    subprocess.check_call(["gcc", "-std=c11", "-Wno-unused-parameter", "-fPIC", "-shared", str(at / "recorder.c"),
                           os.path.join(ROOT, "fastertransformer_b200", "host", "step_module.c"),
                           "-I" + sysconfig.get_paths()["include"], "-I" + os.path.join(ROOT, "include"), "-o", str(out)])
    spec = importlib.util.spec_from_file_location("_ftb200_step", str(out))
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    return module, C.CDLL(str(out))


@pytest.fixture
def layer(recorder, monkeypatch):
    """A set-up layer of 8 rows whose memory is on the host, and the blocks that the library was given since."""
    module, library = recorder

    def place(pack, device):
        for owner, name, dtype, _, size, _ in pack.parts:
            setattr(owner, name, torch.zeros(size, dtype=torch.uint8).view(dtype))
        return torch.zeros(1)

    monkeypatch.setattr(decode_layer._Pack, "place", place)
    for name, value in (("_step", module), ("lib", library), ("_LIBRARY", library), ("_raw_stream", lambda index: 7)):
        monkeypatch.setattr(decode_layer, name, value)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: types.SimpleNamespace(synchronize=lambda: None))
    new = decode_layer.DynamicDecodeLayer(100, 104, torch.float16, torch.device("cpu", 0))
    new.setup(8, 1, {"runtime_top_k": np.asarray([4], np.uint32)})
    new._home = 7
    C.c_int.in_dll(library, "calls").value = 0
    new.recorded = lambda: list((SamplingParams * 16).in_dll(library, "recorded"))[:C.c_int.in_dll(library, "calls").value]
    return new


def call(layer, logits, **more):
    layer.forward({"output_ids": torch.zeros(9, 8, dtype=torch.int32), "finished": torch.zeros(8, dtype=torch.bool)},
                  {"logits": logits, "step": 4, "max_input_length": 4, "end_id": torch.zeros(8, dtype=torch.int32), **more})


@pytest.mark.parametrize("types_", ["hbh", "bhhfh", "fhhff"])
def test_each_call_is_of_its_own_type(types_, layer):
    kinds = {"f": torch.float32, "h": torch.float16, "b": torch.bfloat16}
    given = [torch.zeros(8, 104, dtype=kinds[t]) for t in types_]
    for x in given:
        call(layer, x)
        assert layer._native is not None
    assert [(p.dtype, p.logits) for p in layer.recorded()] == [(decode_layer._DT[x.dtype], x.data_ptr()) for x in given]


def test_block_of_a_slice_is_its_own(layer):
    """A call of other sizes for the same rows makes the layer a new argument block: the old one's memory is not the
    native step's any more."""
    x, twice = torch.zeros(8, 104, dtype=torch.float16), torch.zeros(16, 104, dtype=torch.float16)
    call(layer, x)
    old = layer._gate[(0, 8)]["params"]
    call(layer, twice, local_batch_size=8)
    C.memset(C.byref(old), 0xff, C.sizeof(old))  # (as its next owner may; the test still holds on to it)
    call(layer, x)
    call(layer, twice, local_batch_size=8)
    assert bytes(old) == b"\xff" * C.sizeof(old)
    got = layer.recorded()
    assert [(p.batch_size, p.local_batch_size, p.vocab_size, p.logits) for p in got] == [
        (8, 8, 100, x.data_ptr()), (16, 8, 100, twice.data_ptr())] * 2
    for p in got[2:]:
        for name in ("row_order", "topk_ks", "topk_states", "workspace", "workspace_bytes", "max_top_k"):
            assert getattr(p, name) == getattr(got[0], name), name


def test_package_without_the_module(layer, monkeypatch):
    """No step module was built (or only another interpreter's): the package imports, and the Python code takes every step."""
    code = ("import os; real = os.path.exists; os.path.exists = lambda p: '_ftb200_step' not in str(p) and real(p)\n"
            "import fastertransformer_b200._lib as l; assert l.step_module is None and l.STEP_MODULE_PATH.endswith(%r)"
            % sysconfig.get_config_var("EXT_SUFFIX"))
    subprocess.check_call([sys.executable, "-c", code], cwd=ROOT)
    monkeypatch.setattr(decode_layer, "_step", None)
    x = torch.zeros(8, 104, dtype=torch.float16)
    for _ in range(2):
        call(layer, x)
    assert layer._native is None and layer.launches == 2 and [p.logits for p in layer.recorded()] == [x.data_ptr()] * 2
