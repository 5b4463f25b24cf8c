"""Host-side mirror of FasterTransformer's DynamicDecodeLayer for the sampling path (beam_width == 1).

Same keys, dtypes and placement as the reference's TensorMap interface
(layers/DynamicDecodeLayer.cc:153-178 setup, :191-474 forward): runtime arguments are host arrays of
shape [1] or [batch]; logits, ids and state live on the GPU.  torch is used only to own device memory
and streams; every computation is a call into libftb200.so through the C ABI.
"""
import ctypes as C

import numpy as np
import torch

from ._lib import BeamHyps, BeamParams, SamplingParams, SetupParams, StopParams, check, lib, step_module as _step

# Page-locked words that a step which missed its deadline has still to write, with an event behind that step: the host
# allocator would hand them out again when their layer goes.
_LATE = []


def _keep_until_done(word, stream):
    """Holds on to `word` until what is on `stream` now has run."""
    done = torch.cuda.Event()
    done.record(stream)
    _LATE[:] = [(w, e) for w, e in _LATE if not e.query()] + [(word, done)]


_DT = {torch.float32: 0, torch.float16: 1, torch.bfloat16: 2}
TIMEOUT = 6  # FTB200_TIMEOUT
_LIBRARY = lib  # what the step module calls
CURAND_STATE_BYTES = 48  # sizeof(curandState_t), XORWOW


# the current stream's handle without a Stream object per call, where this torch has it
_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)


def _ptr(t):
    return None if t is None else C.c_void_p(t.data_ptr())


def _addr(t):
    return None if t is None else t.data_ptr()


_HYPS = [f for f, _ in BeamHyps._fields_[:-1]]
_BEAM_SCALARS = ("temperature", "repetition_penalty", "presence_penalty", "min_length", "beam_search_diversity_rate",
                 "len_penalty")


def _scalar(inputs, name):
    """First value of a host argument, None where it is absent."""
    v = inputs.get(name)
    return None if v is None else (v.flat[0] if isinstance(v, np.ndarray) else np.atleast_1d(np.asarray(v)).reshape(-1)[0]).item()


class _SamplingLayerState:
    """Buffers one reference sampling layer keeps (BaseSamplingLayer.cc:29-53, TopK/TopP allocateBuffer): device tensors
    curand, top_ks (uint32 payload), top_ps, skip, and skip_host."""
    active = False


class _Pack:
    """Host arrays and device-only buffers of a set-up, laid out behind each other in one device allocation; the host
    part travels in one copy from page-locked memory."""

    def __init__(self):
        self.parts, self.size = [], 0

    def add(self, owner, name, dtype, count, host=None):
        size = dtype.itemsize * count
        self.parts.append((owner, name, dtype, self.size, size, host))
        self.size += (size + 63) // 64 * 64

    def place(self, device):
        """Sets the attributes `name` of the owners to tensors; host parts have to be added first."""
        upload = max([at + size for _, _, _, at, size, host in self.parts if host is not None], default=0)
        dev = torch.empty(self.size, dtype=torch.uint8, device=device)
        if upload:
            staged = torch.empty(upload, dtype=torch.uint8, pin_memory=True)
            bytes_ = staged.numpy()
            for _, _, _, at, size, host in self.parts:
                if host is not None:
                    bytes_[at:at + size] = host.view(np.uint8)
            dev[:upload].copy_(staged, non_blocking=True)
        for owner, name, dtype, at, size, _ in self.parts:
            setattr(owner, name, dev[at:at + size].view(dtype))
        return dev


class DynamicDecodeLayer:
    """Drop-in for the sampling half of fastertransformer::DynamicDecodeLayer<T>."""

    _launches = 0
    _native = None  # the whole batch's slice in _ftb200_step, once a call has gone through forward()'s own code

    def __init__(self, vocab_size, vocab_size_padded, dtype=torch.float32, device="cuda:0", stream=None):
        self.vocab_size = int(vocab_size)
        self.vocab_size_padded = int(vocab_size_padded)
        self.dtype = dtype
        self.device = torch.device(device)
        self.stream = stream
        self._device_index = self.device.index if self.device.index is not None else torch.cuda.current_device()
        self._setup_mem = self._workspace = self._beam_ws = self._arrived = None
        self._home = None           # stream all of the layer's device memory was allocated on, see _allocated()
        self._beam_key = self._beam_blocks = None
        self._gate = {}
        self.time_kernels = False   # when set, CUDA events bracket each fused launch (kernel_events)
        self.kernel_events = []
        self.deadline_ms = 10000    # of the wait for should_stop
        self._count_dev = None
        self._count_host = None
        self._stop = None

    # ---- helpers -------------------------------------------------------------------------------
    @property
    def launches(self):
        """Kernels launched so far."""
        return self._launches + (0 if self._native is None else _step.launches(self._native))

    @launches.setter
    def launches(self, n):
        self._launches = n - (0 if self._native is None else _step.launches(self._native))

    def _drop_native(self):
        if self._native is not None:
            self._launches, self._native = self.launches, None

    def _make_native(self, logits, B, lo, lbs, P):
        """Later calls of this form go to the library through one native call (host/step_module.c)."""
        if (lo, lbs, B) != (0, self.batch_size, self.batch_size) or logits.dim() != 2 or self.stream is not None or _raw_stream is None \
                or _step is None or self._home is None or self._home < 0 or self._stream != self._home or lib is not _LIBRARY:
            return
        g, S = self._g, self._stop
        self._native = _step.make(C.addressof(P), 0 if S is None else C.addressof(S), S, logits.dtype, _DT[logits.dtype], _raw_stream,
                                  self._device_index, self._home, B, g["temp"], self.penalty_type != 2 and g["pen"], g["minlen"])

    def _stream_ptr(self):
        return C.c_void_p(self._raw_stream())

    def _raw_stream(self):
        if self.stream is not None:
            return self.stream.cuda_stream
        if _raw_stream is not None:
            return _raw_stream(self._device_index)
        return torch.cuda.current_stream(self.device).cuda_stream

    def _run_stream(self):
        return self.stream if self.stream is not None else torch.cuda.current_stream(self.device)

    # Device memory of the layer, by attribute.  The caching allocator hands a freed block out again on the stream it was
    # allocated on, without a look at the others: a call on another stream has to be noted on each of them.
    _MEMORY = ("_setup_mem", "_workspace", "_beam_ws", "_arrived", "_count_dev")

    def _allocated(self, make, *args, **kw):
        """What make(...) allocates, on the layer's own stream if it has one, else on the current one."""
        if self.device.type != "cuda":
            return make(*args, **kw)
        if self.stream is None:
            t = make(*args, **kw)
        else:
            with torch.cuda.stream(self.stream):
                t = make(*args, **kw)
        self._drop_native()  # (it holds the addresses of what there was)
        on = self._raw_stream()
        if self._home != on:
            self._home = on if self._home is None else -1  # (several streams: none of them is the home of all)
        return t

    def _away(self):
        """Before a call on another stream than the one all of the layer's memory was allocated on."""
        memory = self._memory()
        if memory:
            here = self._run_stream()
            for t in memory:
                t.record_stream(here)

    def _memory(self):
        mem = [getattr(self, name) for name in self._MEMORY] + [g["order"] for g in self._gate.values()]
        return [t for t in mem if t is not None]

    @staticmethod
    def _arg(args, key):
        v = args.get(key)
        if v is None:
            return None
        return np.atleast_1d(np.asarray(v))

    def _broadcast(self, arr, batch, dtype, default):
        if arr is None:
            arr = np.asarray([default], dtype=dtype)
        arr = arr.astype(dtype)
        if arr.size == 1:
            return np.full(batch, arr[0], dtype=dtype)
        if arr.size != batch:
            raise ValueError("runtime argument must have shape [1] or [batch_size]")
        return arr.copy()

    # ---- setup (DynamicDecodeLayer.cc:153-178 -> TopK/TopPSamplingLayer::setup) -------------------
    def setup(self, batch_size, beam_width, runtime_args):
        self.beam_width = int(beam_width)
        # hasDiffRuntimeArgs (DynamicDecodeLayer.cc:477-514): beam search then runs one batch entry at a time
        self.has_diff_runtime_args = False
        for key in ("beam_search_diversity_rate", "temperature", "len_penalty", "repetition_penalty",
                    "presence_penalty", "min_length"):
            v = self._arg(runtime_args, key)
            if v is not None and v.size > 1 and bool((v != v[0]).any()):
                self.has_diff_runtime_args = True
        if beam_width != 1:
            return  # the beam layers have no set-up (BaseBeamSearchLayer.cu:123-127)
        B, dev, st = int(batch_size), self.device, self._stream_ptr()
        self._drop_native()
        self.batch_size = B
        self._gate = {}
        a = runtime_args
        top_k = self._arg(a, "runtime_top_k")
        top_p = self._arg(a, "runtime_top_p")
        seeds = self._arg(a, "random_seed")
        if "repetition_penalty" in a and "presence_penalty" in a:
            raise RuntimeError("[FT][ERROR] Found ambiguous parameters repetition_penalty and presence_penalty "
                               "which are mutually exclusive.")
        # BaseSamplingLayer::setup (BaseSamplingLayer.cc:112-206)
        self.temperature_host = self._broadcast(self._arg(a, "temperature"), B, np.float32, 1.0)
        if "repetition_penalty" in a:
            self.penalty_type, pen = 1, self._arg(a, "repetition_penalty")
        elif "presence_penalty" in a:
            self.penalty_type, pen = 0, self._arg(a, "presence_penalty")
        else:
            self.penalty_type, pen = 2, None
        default_pen = 1.0 if self.penalty_type == 1 else 0.0
        self.penalty_default = default_pen
        self.penalty_host = self._broadcast(pen, B, np.float32, default_pen)
        self.min_length_host = self._broadcast(self._arg(a, "min_length"), B, np.int32, 0)
        # TopKSamplingLayer::setup (TopKSamplingLayer.cu:134-186), TopPSamplingLayer::setup (TopPSamplingLayer.cu:184-253):
        # the kernel writes the normalised arguments on the device; what the host side needs of them follows from the
        # same rules here, so nothing is read back.
        k_arr = top_k.astype(np.uint32) if top_k is not None else np.zeros(1, np.uint32)
        p_arr = None if top_p is None else top_p.astype(np.float32)
        for v in (k_arr, p_arr):
            if v is not None and v.size not in (1, B):
                raise RuntimeError("[FT][ERROR] runtime_top_k and runtime_top_p must be of shape [1] or [batch_size]")
        if seeds is not None and seeds.size not in (1, B):
            raise RuntimeError("[FT][ERROR] random_seeds must be of shape [1] or [batch_size]")
        zero = np.float32(0.0)
        k_all = np.broadcast_to(k_arr if k_arr.size > 1 else k_arr.max(), (B,))
        p_all = np.broadcast_to(zero if p_arr is None else (p_arr if p_arr.size > 1 else p_arr[0]), (B,))
        k_topk = np.where((k_all == 0) & (p_all == zero), np.uint32(1), k_all)
        self.topk, self.topp = _SamplingLayerState(), _SamplingLayerState()
        self.topk.skip_host, self.topk.active = k_topk == 0, True
        self.max_top_k = int(np.minimum(k_topk, 1024).max())
        cost = 1.0 + np.minimum(k_topk, 1024) / 128.0
        if p_arr is None:
            self.topp.skip_host = np.ones(B, dtype=bool)
        else:
            k_first = np.broadcast_to(k_arr if k_arr.size > 1 else k_arr[0], (B,))
            self.topp.skip_host = (k_first > 0) | (p_all == zero)
            self.topp.active = True
            cost = np.where(self.topk.skip_host, 10.0 + 8.0 * np.clip(p_all, 0.0, 1.0), cost)
        # Relative cost of a row, for the launch order: top-p rows cost most, then top-k by k.
        self._row_cost = cost
        order = np.argsort(-cost, kind="stable").astype(np.int32)

        pack = _Pack()
        per_row_seeds = seeds is not None and seeds.size > 1
        if per_row_seeds:
            pack.add(self, "_seeds", torch.int64, B, seeds.astype(np.uint64))
        pack.add(self, "temperature", torch.float32, B, self.temperature_host)
        pack.add(self, "penalty", torch.float32, B, self.penalty_host)
        pack.add(self, "min_length", torch.int32, B, self.min_length_host)
        pack.add(self, "_order", torch.int32, B, order)
        for layer in (self.topk, self.topp):
            pack.add(layer, "top_ks", torch.int32, B, k_arr if k_arr.size > 1 else None)
            pack.add(layer, "top_ps", torch.float32, B, p_arr if p_arr is not None and p_arr.size > 1 else None)
        for layer in (self.topk, self.topp):
            pack.add(layer, "skip", torch.uint8, B)
            pack.add(layer, "curand", torch.uint8, B * CURAND_STATE_BYTES)
        if self.topp.active:
            for name, dtype in (("initial", torch.float32), ("decay", torch.float32), ("min", torch.float32),
                                ("reset", torch.int32)):
                pack.add(self.topp, name, dtype, B)
        self._setup_mem = self._allocated(pack.place, dev)
        tk, tp = self.topk, self.topp
        S = SetupParams()
        S.batch = B
        S.topk_states, S.topp_states = tk.curand.data_ptr(), tp.curand.data_ptr()
        if per_row_seeds:
            S.seeds = self._seeds.data_ptr()
        elif seeds is not None:
            S.seed = int(seeds[0])
        S.topk_top_k, S.topp_top_k = int(k_arr.max()), int(k_arr[0])
        S.top_ks_size, S.top_ps_size = int(k_arr.size), 0 if p_arr is None else int(p_arr.size)
        S.top_p = 0.0 if p_arr is None else float(p_arr[0])
        S.topk_ks, S.topk_ps, S.topk_skip = tk.top_ks.data_ptr(), tk.top_ps.data_ptr(), tk.skip.data_ptr()
        if tp.active:
            S.topp_ks, S.topp_ps, S.topp_skip = tp.top_ks.data_ptr(), tp.top_ps.data_ptr(), tp.skip.data_ptr()
            S.topp_initial, S.topp_decay = tp.initial.data_ptr(), tp.decay.data_ptr()
            S.topp_min, S.topp_reset_ids = tp.min.data_ptr(), tp.reset.data_ptr()
            S.top_p_decay, S.top_p_min = _addr(a.get("top_p_decay")), _addr(a.get("top_p_min"))
            S.top_p_reset_ids = _addr(a.get("top_p_reset_ids"))
        S.stream = st.value
        check(lib.ftb200_setup_sampling(C.byref(S)))
        # The arguments, the launch order and the generators are there when this returns: steps may follow on any stream,
        # from any thread, under capture.  (An event would do for the first of these only; a request waits 10 us here once.)
        self._run_stream().synchronize()

    # ---- forward (DynamicDecodeLayer.cc:191-474, sampling branch) ---------------------------------
    def forward(self, outputs, inputs):
        if self._native is not None and self.stream is None and not self.time_kernels:
            done = _step.step(self._native, outputs, inputs, self.deadline_ms)
            if done is True or done is False:
                return done
            if done is not None:
                self._failed(done)
        logits = inputs["logits"]
        shape = logits.shape
        if len(shape) == 3 and shape[1] > 1:
            return self._forward_beam(outputs, inputs)
        B = shape[0]
        step = int(inputs["step"])
        ite = int(inputs.get("ite", 0))
        lbs = int(inputs.get("local_batch_size", B))
        mil = int(inputs["max_input_length"])
        lo, hi = ite * lbs, (ite + 1) * lbs
        g = self._gate.get((lo, hi))
        if g is None:
            g = self._gate[(lo, hi)] = {
                "topk_on": self.topk.active and not self.topk.skip_host[lo:hi].all(),
                "topp_on": self.topp.active and not self.topp.skip_host[lo:hi].all(),
                "temp": bool((self.temperature_host[lo:hi] != 1.0).any()),
                "pen": bool((self.penalty_host[lo:hi] != self.penalty_default).any()),
                "minlen": int(self.min_length_host[lo:hi].max()),
                "order": self._order if lo == 0 and hi == self.batch_size else self._allocated(
                    lambda: torch.from_numpy(np.argsort(-self._row_cost[lo:hi], kind="stable").astype(np.int32)).to(self.device)),
            }
        self._g = g
        self._stream = self._raw_stream()  # one look-up per call, used by the sampling and the criteria launch
        if self._stream != self._home:
            self._away()
        if not (g["topk_on"] or g["topp_on"]):
            return self._stop_criteria(outputs, inputs, B, step, lbs, lo)
        P = self._fill(outputs, inputs, logits, B, step, ite, lbs, mil, lo)
        sw = inputs.get("stop_words_list")
        lim = inputs.get("sequence_limit_length")
        if (sw is None and lim is None) or self.time_kernels or P.finished is None:
            self._sample(P)
            if self._native is None and P.finished is not None and not self.time_kernels:
                self._make_native(logits, B, lo, lbs, P)
            return self._stop_criteria(outputs, inputs, B, step, lbs, lo)
        # sampling, stop criteria and the wait for should_stop in one call
        S = self._stop
        if S is None:
            self._arrived = self._allocated(torch.zeros, 1, dtype=torch.int32, device=self.device)
            self._result = torch.zeros(1, dtype=torch.int64).pin_memory()
            S = self._stop = StopParams()
            S.arrived_dev, S.result_host = self._arrived.data_ptr(), self._result.data_ptr()
            self._stop_ref, self._should_stop = C.byref(S), C.c_int(0)
            self._should_stop_ref = C.byref(self._should_stop)
        if sw is None:
            S.stop_words, S.stop_words_len = None, 0
        else:
            L = sw.shape[-1]
            S.stop_words, S.stop_words_len = sw.data_ptr() + lo * 2 * L * 4, L
        S.sequence_limit_length = None if lim is None else lim.data_ptr()
        rc = lib.ftb200_decode_step(g["params_ref"], self._stop_ref, self.deadline_ms, self._should_stop_ref)
        if rc:
            self._failed(rc)
        self._launches += lib.ftb200_last_launch_count()
        if self._native is None:
            self._make_native(logits, B, lo, lbs, P)
        return bool(self._should_stop.value)

    def _failed(self, rc):
        if rc == TIMEOUT:
            _keep_until_done(self._result, self._run_stream())
        check(rc)

    # ---- beam search branch (DynamicDecodeLayer.cc:286-386 -> OnlineBeamSearchLayer::forward) -------
    def _forward_beam(self, outputs, inputs):
        logits = inputs["logits"]
        B, K, Vp = logits.shape
        step = int(inputs["step"])
        ite = int(inputs.get("ite", 0))
        lbs = int(inputs.get("local_batch_size", B))
        mil = int(inputs["max_input_length"])
        self._stream = self._raw_stream()
        if self._stream != self._home:
            self._away()
        st = C.c_void_p(self._stream)
        es = logits.element_size()
        out_ids = outputs["output_ids"]
        L = out_ids.shape[0]
        if "cum_log_probs" not in outputs:
            raise RuntimeError("[FT][ERROR] cum_log_probs should be provided in beam search.")
        bw = inputs.get("bad_words_list")
        if bw is not None:
            shared = bw.dim() == 2 or bw.shape[0] == 1
            Lw = bw.shape[-1]
            check(lib.ftb200_ban_bad_words(
                C.c_void_p(logits.data_ptr() + ite * lbs * K * Vp * es), _DT[logits.dtype],
                _ptr(out_ids), _ptr(outputs["parent_ids"]), B, lbs, K,
                C.c_void_p(bw.data_ptr() if shared else bw.data_ptr() + ite * lbs * 2 * Lw * 4), int(shared), Lw,
                ite * lbs, Vp, step, st))
            self._launches += 1

        sub = 1 if self.has_diff_runtime_args else lbs
        n_sub = lbs // sub
        hyps = outputs.get("beam_hyps")
        bias, il, olp = inputs.get("embedding_bias"), inputs.get("input_lengths"), outputs.get("output_log_probs")
        src, tgt = inputs.get("src_cache_indirection"), outputs.get("tgt_cache_indirection")
        # The argument blocks of a call (one per sub-batch) are kept between steps and filled again when one of the
        # caller's pointers or scalars changes; the step's own values are written every time.
        key = (logits.dtype, B, K, Vp, L, mil, ite, lbs, sub, self._stream, out_ids.data_ptr(), outputs["parent_ids"].data_ptr(),
               outputs["finished"].data_ptr(), outputs["sequence_length"].data_ptr(), outputs["cum_log_probs"].data_ptr(),
               inputs["end_id"].data_ptr(), _addr(bias), _addr(il), _addr(olp),
               None if hyps is None else tuple((f, _addr(hyps.get(f))) for f in _HYPS) + (int(hyps.get("early_stopping", True)),),
               tuple(_scalar(inputs, k) for k in _BEAM_SCALARS))
        if key != self._beam_key:
            self._beam_blocks = self._fill_beam(outputs, inputs, key, B, K, Vp, L, mil, ite, lbs, sub, n_sub, es)
            self._beam_key = key
        for P, ref, row0 in self._beam_blocks:
            P.step = step
            P.logits = logits.data_ptr() + row0 * Vp * es
            P.src_cache_indirection = None if src is None else src.data_ptr()
            P.tgt_cache_indirection = None if tgt is None else tgt.data_ptr()
            rc = lib.ftb200_beam_search_step(ref)
            if rc:
                check(rc)
            self._launches += lib.ftb200_last_launch_count()
        return self._stop_criteria(outputs, inputs, B, step, lbs, ite * lbs, beam=K)

    def _fill_beam(self, outputs, inputs, key, B, K, Vp, L, mil, ite, lbs, sub, n_sub, es):
        need = C.c_size_t(0)
        check(lib.ftb200_beam_workspace_bytes(sub, K, C.byref(need)))
        if self._beam_ws is None or self._beam_ws.numel() < need.value:
            self._beam_ws = self._allocated(torch.empty, need.value, dtype=torch.uint8, device=self.device)
        if "repetition_penalty" in inputs and "presence_penalty" in inputs:
            raise RuntimeError("[FT][ERROR] Found ambiguous parameters repetition_penalty and "
                               "presence_penalty which are mutually exclusive.")

        def scalar(name, default):
            v = _scalar(inputs, name)
            return default if v is None else v

        blocks = []
        for d_ite in range(ite * n_sub, (ite + 1) * n_sub):
            row0 = d_ite * sub * K          # first batch-beam row of this sub-batch
            P = BeamParams()
            P.dtype = _DT[inputs["logits"].dtype]
            P.batch_size, P.local_batch_size, P.ite, P.beam_width = B, sub, d_ite, K
            P.vocab_size, P.vocab_size_padded = self.vocab_size, Vp
            P.max_input_length, P.max_seq_len = mil, L
            P.embedding_bias = _addr(inputs.get("embedding_bias"))
            P.end_ids = inputs["end_id"].data_ptr() + d_ite * sub * 4
            il = inputs.get("input_lengths")
            P.input_lengths = None if il is None else il.data_ptr() + row0 * 4
            P.temperature = float(scalar("temperature", 1.0))
            if inputs.get("repetition_penalty") is not None:
                P.penalty_type, P.repetition_penalty = 1, float(scalar("repetition_penalty", 1.0))
            elif inputs.get("presence_penalty") is not None:
                P.penalty_type, P.repetition_penalty = 0, float(scalar("presence_penalty", 0.0))
            else:
                P.penalty_type, P.repetition_penalty = 2, 1.0
            P.min_length = int(scalar("min_length", 0))
            P.diversity_rate = float(scalar("beam_search_diversity_rate", 0.0))
            P.length_penalty = float(scalar("len_penalty", 0.0))
            P.output_ids = outputs["output_ids"].data_ptr()
            P.parent_ids = outputs["parent_ids"].data_ptr()
            P.finished = outputs["finished"].data_ptr() + row0
            P.sequence_length = outputs["sequence_length"].data_ptr() + row0 * 4
            P.cum_log_probs = outputs["cum_log_probs"].data_ptr() + row0 * 4
            P.output_log_probs = _addr(outputs.get("output_log_probs"))
            hyps = outputs.get("beam_hyps")
            if hyps is not None:
                H = BeamHyps()
                for f in _HYPS:
                    setattr(H, f, _addr(hyps.get(f)))
                H.early_stopping = int(hyps.get("early_stopping", True))
                P.beam_hyps = C.pointer(H)
            P.workspace = self._beam_ws.data_ptr()
            P.workspace_bytes = self._beam_ws.numel()
            P.stream = self._stream
            blocks.append((P, C.byref(P), row0))
        return blocks

    def _stop_criteria(self, outputs, inputs, B, step, lbs, lo, beam=1):
        """Stop words, length limit and should_stop (DynamicDecodeLayer.cc:447-473)."""
        sw = inputs.get("stop_words_list")
        lim = inputs.get("sequence_limit_length")
        if sw is None and lim is None:
            return False
        if self._count_dev is None:
            self._count_dev = self._allocated(torch.zeros, 1, dtype=torch.int32, device=self.device)
            self._count_host = torch.zeros(1, dtype=torch.int32).pin_memory()
        L = 0 if sw is None else sw.shape[-1]
        st = C.c_void_p(self._stream)
        check(lib.ftb200_stop_criteria(
            _ptr(outputs["output_ids"]), _ptr(outputs.get("parent_ids")),
            None if sw is None else C.c_void_p(sw.data_ptr() + lo * 2 * L * 4), L, _ptr(outputs["finished"]),
            _ptr(lim), lo * beam, lbs, B, beam, step, _ptr(self._count_dev),
            C.c_void_p(self._count_host.data_ptr()), st))
        self._launches += 1
        if lim is None:
            return False
        stop = C.c_int(0)
        rc = lib.ftb200_wait_should_stop(C.c_void_p(self._count_host.data_ptr()), B, beam, st, self.deadline_ms, C.byref(stop))
        if rc:
            if rc == TIMEOUT:
                _keep_until_done(self._count_host, self._run_stream())
            check(rc)
        return bool(stop.value)

    def _fill(self, outputs, inputs, logits, B, step, ite, lbs, mil, lo):
        """The argument block of a slice.  It is kept between steps: what setup() fixed (the layer's own buffers, the
        launch order, the slice) is written once, the caller's pointers when one of them changes, the step's own
        values every time."""
        Vp = self.vocab_size_padded
        g = self._g
        P = g.get("params")
        if P is None or g["params_key"] != (B, lbs, ite):
            topk_on, topp_on = g["topk_on"], g["topp_on"]
            P = SamplingParams()
            P.batch_size, P.local_batch_size, P.ite = B, lbs, ite
            P.vocab_size, P.vocab_size_padded = self.vocab_size, Vp
            P.temperature = self.temperature.data_ptr() + lo * 4
            P.repetition_penalty = self.penalty.data_ptr() + lo * 4
            P.penalty_type = self.penalty_type
            P.min_lengths = self.min_length.data_ptr() + lo * 4
            if topk_on:
                P.topk_states = self.topk.curand.data_ptr() + lo * CURAND_STATE_BYTES
                P.topk_ks = self.topk.top_ks.data_ptr() + lo * 4
                P.topk_ps = self.topk.top_ps.data_ptr() + lo * 4
                P.topk_skip = self.topk.skip.data_ptr() + lo
                P.max_top_k = self.max_top_k
            if topp_on:
                P.topp_states = self.topp.curand.data_ptr() + lo * CURAND_STATE_BYTES
                P.topp_ps = self.topp.top_ps.data_ptr() + lo * 4
                P.topp_skip = self.topp.skip.data_ptr() + lo
                P.topp_initial_ps = self.topp.initial.data_ptr() + lo * 4
                P.topp_decay = self.topp.decay.data_ptr() + lo * 4
                P.topp_min = self.topp.min.data_ptr() + lo * 4
                P.topp_reset_ids = self.topp.reset.data_ptr() + lo * 4
            P.row_order = g["order"].data_ptr()
            g["params"], g["params_key"], g["params_ref"], g["ptrs"] = P, (B, lbs, ite), C.byref(P), None
        P.step = step
        P.logits = logits.data_ptr() + lo * Vp * logits.element_size()
        bias, il, bw = inputs.get("embedding_bias"), inputs.get("input_lengths"), inputs.get("bad_words_list")
        seq, fin = outputs.get("sequence_length"), outputs.get("finished")
        cum, olp = outputs.get("cum_log_probs"), outputs.get("output_log_probs")
        ptrs = (logits.dtype, mil, inputs["end_id"].data_ptr(), outputs["output_ids"].data_ptr(), self._stream,
                None if bias is None else bias.data_ptr(), None if il is None else il.data_ptr(),
                None if bw is None else (bw.data_ptr(), bw.shape), None if seq is None else seq.data_ptr(),
                None if fin is None else fin.data_ptr(), None if cum is None else cum.data_ptr())
        if ptrs != g["ptrs"]:
            P.dtype = _DT[logits.dtype]
            P.max_input_length = mil
            P.embedding_bias = None if bias is None else bias.data_ptr()
            P.end_ids = inputs["end_id"].data_ptr() + lo * 4
            P.input_lengths = None if il is None else il.data_ptr() + lo * 4
            P.output_ids = outputs["output_ids"].data_ptr()
            if bw is not None:
                shared = bw.dim() == 2 or bw.shape[0] == 1
                L = bw.shape[-1]
                P.bad_words = bw.data_ptr() if shared else bw.data_ptr() + lo * 2 * L * 4
                P.bad_words_len, P.bad_words_shared = L, int(shared)
            else:
                P.bad_words, P.bad_words_len, P.bad_words_shared = None, 0, 0
            P.apply_temperature = int(bias is not None or g["temp"])
            P.sequence_length = None if seq is None else seq.data_ptr() + lo * 4
            P.finished = None if fin is None else fin.data_ptr() + lo
            P.cum_log_probs = None if cum is None else cum.data_ptr() + lo * 4
            if self._workspace is None or self._ws_key != (P.dtype, lbs, Vp):
                need = C.c_size_t(0)
                check(lib.ftb200_sampling_workspace_bytes(P.dtype, lbs, Vp, C.byref(need)))
                if self._workspace is None or self._workspace.numel() < need.value:
                    self._workspace = self._allocated(torch.empty, need.value, dtype=torch.uint8, device=self.device)
                self._ws_key = (P.dtype, lbs, Vp)
            P.stream = self._stream
            g["ptrs"] = ptrs
        P.workspace = self._workspace.data_ptr()
        P.workspace_bytes = self._workspace.numel()
        # host-side gating of the penalty kernels (BaseSamplingLayer.cc:302-349)
        P.apply_repetition = int(step > 1 and self.penalty_type != 2 and g["pen"])
        P.apply_min_length = int(g["minlen"] > step - mil)
        # [request_output_len, batch] sliced at (step - max_input_length) (DynamicDecodeLayer.cc:427-435)
        P.output_log_probs = None if olp is None else olp.data_ptr() + ((step - mil) * B + lo) * 4
        return P

    def _sample(self, P):
        if self.time_kernels:
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            check(lib.ftb200_decode_step_sampling(C.byref(P)))
            e1.record()
            self.kernel_events.append((e0, e1))
        else:
            check(lib.ftb200_decode_step_sampling(self._g["params_ref"]))
        self._launches += lib.ftb200_last_launch_count()
