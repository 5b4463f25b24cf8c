"""Timed cases of the decode-sampling framework: what a serving or generation program has it do.

A case is a dict of plain values; its "kind" says which public entry points it goes through:

  decode            one token for every row of a batch: DynamicDecodeLayer.forward, beam width 1
  generate          a short request from set-up to its last token: setup, then `steps` forward calls
  beam              one beam-search step: DynamicDecodeLayer.forward, beam width > 1
  vocab_parallel    one token from column shards of the logits: VocabParallelSampler.forward_shards
  context_logprob   scoring of given texts: log_prob_from_logits
  finish            end of a beam generation: gather tree, or archive of the live beams and ranking of the archive

Logits are seeded normal draws; "spikes" > 0 raises that many columns of each row by `spike_height` (a model's
logits are peaked; one of the raised columns is a token that the row has already seen), 0 leaves the row flat.
The end token's logit is lowered so that no sequence ends while it is being timed, however often a pass is
repeated; rows that have ended already are asked for with "ended".
"""
import ctypes as C

import numpy as np
import torch

from fastertransformer_b200 import DynamicDecodeLayer, VocabParallelSampler, check, lib, log_prob_from_logits
from fastertransformer_b200 import BeamHyps, GatherTreeParams

DEVICE = "cuda:0"
DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
SIZE = {"f32": 4, "f16": 2, "bf16": 2}
END_LOGIT = -60.0

# What a decode step's options are when a case does not name them.
DECODE = {
    "kind": "decode", "batch": 8, "vocab": 32000, "padded": 32000, "dtype": "f16",
    "rows": "topk",        # topk: k (and p) for all | topp: p for all | mixed: k in {0, 1, 40, 1024}, p in {0, 0.5, 0.95} per row
    "k": 1, "p": 0.0, "temperature": 1.0,
    "penalty": "none",     # none | repetition | presence
    "penalty_value": 1.0,
    "prompt": 64, "step": 80,   # prompt length (rows may be shorter) and the position being generated
    "ragged": False,       # prompts of different lengths, padded to `prompt`
    "min_length": 0,
    "bad_words": 0,        # banned words of 1 to 3 tokens per row
    "stop_words": 0,       # stop words of 2 or 3 tokens per row (a single one is the end token)
    "limit": True,         # a length limit: forward() then says whether the whole batch is done
    "log_probs": False,    # cum_log_probs and output_log_probs wanted
    "bias": False,         # an embedding bias on every logit
    "sigma": 2.0, "spikes": 4, "spike_height": 8.0,
    "ended": 0.0,          # share of rows that have ended already
}


def _decode(**kw):
    return dict(DECODE, **kw)


def listed():
    return [
        # one chat user, greedy, on a small half-precision vocabulary: the smallest call, all latency
        _decode(name="greedy_1x32000_f16"),
        # the top-k configuration of the benchmark: fp32 logits of an odd vocabulary, a small batch
        _decode(name="topk_8x50257_f32", batch=8, vocab=50257, padded=50264, dtype="f32", k=50, penalty="repetition",
                penalty_value=1.2, prompt=64, step=64, spikes=0, limit=False),
        # the top-p configuration of the benchmark: half logits, temperature, presence penalty, minimum length
        _decode(name="topp_256x51200_f16", batch=256, vocab=51200, padded=51200, rows="topp", p=0.9, temperature=0.8,
                penalty="presence", penalty_value=0.5, prompt=128, step=136, min_length=16, sigma=3.0, limit=False),
        # the headline configuration of the benchmark: per-row arguments, a large vocabulary, bad words, length limit
        _decode(name="mixed_1024x128256_bf16", batch=1024, vocab=128256, padded=128256, dtype="bf16", rows="mixed",
                penalty="repetition", penalty_value=1.1, prompt=512, step=544, bad_words=8, sigma=2.5, spikes=0),
        # models hand fp32 logits to this path by default: nucleus sampling of a mid-sized batch, ragged prompts
        _decode(name="topp_64x50257_f32", batch=64, vocab=50257, padded=50257, dtype="f32", rows="topp", p=0.9,
                temperature=0.7, prompt=256, step=300, ragged=True),
        # a service that returns log-probabilities with its tokens, and biases some logits
        _decode(name="logprobs_48x51200_f16", batch=48, vocab=51200, padded=51200, rows="mixed", penalty="repetition",
                penalty_value=1.2, prompt=128, step=160, log_probs=True, bias=True),
        # long conversations: thousands of tokens of history, stop words, a batch in which some have ended
        _decode(name="history_96x128256_bf16", batch=96, vocab=128256, padded=128256, dtype="bf16", rows="mixed",
                temperature=0.8, penalty="repetition", penalty_value=1.1, prompt=1800, step=2500, ragged=True,
                stop_words=4, ended=0.25),
        # a request from set-up to its last token: 24 greedy-or-sampled tokens for 16 rows, penalised as they come
        dict(_decode(name="generate_16x128256_bf16", batch=16, vocab=128256, padded=128256, dtype="bf16", rows="mixed",
                     penalty="repetition", penalty_value=1.1, prompt=128, step=128), kind="generate", steps=24),
        # the beam-search configuration of the benchmark
        {"name": "beam_64x4x32000_f16", "kind": "beam", "batch": 64, "beams": 4, "vocab": 32000, "dtype": "f16",
         "step": 64, "prompt": 16, "len_penalty": 1.0, "penalty": 1.0, "temperature": 1.0, "archive": False, "sigma": 2.0},
        # the vocabulary-parallel configuration of the benchmark, all shards on one GPU
        {"name": "vocab_parallel_2048x256000", "kind": "vocab_parallel", "batch": 2048, "shard": 32000, "shards": 8,
         "dtype": "bf16", "k": 64, "p": 0.92, "temperature": 0.7, "sigma": 3.0},
        # scoring of a batch of texts: every position's logits at once
        {"name": "context_logprob_512x32x50257", "kind": "context_logprob", "length": 512, "batch": 32, "vocab": 50257,
         "padded": 50257, "dtype": "f16", "batch_first": False, "sigma": 2.0},
        # end of a long beam generation: the sequences are read back through their parents
        {"name": "gather_tree_64x4x2048", "kind": "finish", "form": "gather_tree", "batch": 64, "beams": 4, "time": 2048,
         "prompt": 256, "log_probs": False},
    ]


# ---- drawn cases ------------------------------------------------------------------------------------------------
def _log_int(rng, lo, hi):
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def _draw_decode(rng):
    dtype = rng.choice(["f32", "f16", "bf16"])
    vocab = _log_int(rng, 4000, 256000)
    padded = rng.choice([vocab, (vocab + 7) // 8 * 8])
    # up to the headline's bytes for 16-bit logits; callers with fp32 logits run smaller batches
    most = (1024 * 128256 * 2 if dtype != "f32" else 128 * 128256 * 4) // (padded * SIZE[dtype])
    batch = _log_int(rng, 1, max(1, min(1024, most)))
    prompt = _log_int(rng, 8, 2000)
    step = prompt + _log_int(rng, 1, 1000)
    rows = rng.choice(["topk", "topk", "topp", "mixed"])
    pen = rng.choice(["none", "repetition", "presence"])
    return _decode(
        batch=batch, vocab=vocab, padded=padded, dtype=dtype, rows=rows,
        k=rng.choice([1, _log_int(rng, 2, 1024)]), p=round(rng.uniform(0.3, 0.98), 3) if rows == "topp" or rng.random() < 0.5 else 0.0,
        temperature=rng.choice([1.0, round(rng.uniform(0.5, 1.3), 2)]), penalty=pen,
        penalty_value={"none": 1.0, "repetition": round(rng.uniform(1.02, 1.4), 2), "presence": round(rng.uniform(0.1, 1.0), 2)}[pen],
        prompt=prompt, step=step, ragged=rng.random() < 0.5, min_length=rng.choice([0, 0, step - prompt + 8]),
        bad_words=rng.choice([0, 0, rng.randint(1, 16)]), stop_words=rng.choice([0, 0, rng.randint(1, 8)]),
        limit=rng.random() < 0.7, log_probs=rng.random() < 0.25, bias=rng.random() < 0.15,
        sigma=round(rng.uniform(1.5, 3.0), 2), spikes=rng.choice([0, 4, 4, rng.randint(1, 64)]),
        spike_height=round(rng.uniform(4.0, 12.0), 1), ended=rng.choice([0.0, 0.0, round(rng.uniform(0.05, 0.6), 2)]))


def draw(rng):
    kind = rng.choice(["decode"] * 10 + ["generate", "beam", "beam", "vocab_parallel", "context_logprob", "finish"])
    if kind == "decode":
        return _draw_decode(rng)
    if kind == "generate":
        c = _draw_decode(rng)
        most = 16 * 128256 * 4 // (c["padded"] * SIZE[c["dtype"]])
        return dict(c, kind="generate", batch=_log_int(rng, 1, max(1, min(64, most))), steps=rng.randint(4, 48), ended=0.0,
                    step=c["prompt"], limit=True)
    dtype = rng.choice(["f32", "f16", "bf16"])
    if kind == "beam":
        beams, vocab = rng.choice([2, 3, 4, 4, 5, 8]), _log_int(rng, 4000, 128000)
        prompt = _log_int(rng, 4, 500)
        return {"kind": "beam", "batch": _log_int(rng, 1, max(1, min(256, 32_000_000 // (beams * vocab)))), "beams": beams,
                "vocab": vocab, "dtype": dtype, "step": prompt + _log_int(rng, 1, 500), "prompt": prompt,
                "len_penalty": rng.choice([0.0, 1.0]), "penalty": rng.choice([1.0, 1.2]),
                "temperature": rng.choice([1.0, 0.8]), "archive": rng.random() < 0.5, "sigma": round(rng.uniform(1.5, 3.0), 2)}
    if kind == "vocab_parallel":
        shards, dtype = rng.choice([2, 4, 8]), rng.choice(["f16", "bf16"])
        shard = _log_int(rng, 4000, 64000) // 8 * 8
        return {"kind": "vocab_parallel", "batch": _log_int(rng, 1, max(1, min(2048, 2048 * 256000 // (shard * shards)))),
                "shard": shard, "shards": shards, "dtype": dtype, "k": rng.choice([1, _log_int(rng, 2, 256)]),
                "p": round(rng.uniform(0.5, 0.98), 2), "temperature": rng.choice([1.0, 0.7]), "sigma": round(rng.uniform(1.5, 3.0), 2)}
    if kind == "context_logprob":
        length, vocab = _log_int(rng, 16, 1024), _log_int(rng, 4000, 256000)
        padded = rng.choice([vocab, (vocab + 7) // 8 * 8])
        most = 1_600_000_000 // (length * padded * SIZE[dtype])
        return {"kind": "context_logprob", "length": length, "batch": _log_int(rng, 1, max(1, min(64, most))), "vocab": vocab,
                "padded": padded, "dtype": dtype, "batch_first": rng.random() < 0.5, "sigma": round(rng.uniform(1.5, 3.0), 2)}
    time = _log_int(rng, 32, 2048)
    return {"kind": "finish", "form": rng.choice(["gather_tree", "archive"]), "batch": _log_int(rng, 1, 64),
            "beams": rng.choice([2, 3, 4, 5, 8]), "time": time, "prompt": max(1, int(time * rng.uniform(0.05, 0.5))),
            "log_probs": rng.random() < 0.5}


# ---- inputs -----------------------------------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _normal(shape, sigma, dtype, g):
    return torch.randn(shape, generator=g, device=DEVICE, dtype=torch.float32).mul_(sigma).to(DTYPES[dtype])


def _logits(case, rows, g, seen=None):
    """[rows, padded] logits of one step; `seen` [rows]: a token of each row's history, the first raised column."""
    x = torch.randn((rows, case["padded"]), generator=g, device=DEVICE, dtype=torch.float32).mul_(case["sigma"])
    n = case["spikes"]
    if n:
        cols = torch.randint(0, case["vocab"], (rows, n), generator=g, device=DEVICE)
        if seen is not None:
            cols[:, 0] = seen
        x.scatter_add_(1, cols, torch.full(cols.shape, case["spike_height"], device=DEVICE))
    x[:, case["vocab"] - 1] = END_LOGIT
    return x.to(DTYPES[case["dtype"]])


def _words(rng, batch, n, vocab, shortest):
    """[batch, 2, L] word lists: the tokens of `n` words of up to 3 tokens, then the end offset of each, padded with -1."""
    size = rng.integers(shortest, 4, size=(batch, n))
    ends = np.cumsum(size, axis=1)
    out = np.zeros((batch, 2, 3 * n), np.int32)
    out[:, 1] = -1
    out[:, 1, :n] = ends
    tokens = rng.integers(1, vocab - 1, size=(batch, 3 * n))
    out[:, 0] = np.where(np.arange(3 * n)[None, :] < ends[:, -1:], tokens, 0)
    return torch.from_numpy(out).to(DEVICE)


def _runtime_args(case, rng):
    B = case["batch"]
    a = {"random_seed": (np.arange(B) * 3 + 1 + rng.integers(1 << 20)).astype(np.uint64)}
    if case["rows"] == "mixed":
        a["runtime_top_k"] = rng.choice(np.asarray([0, 1, 40, 1024], np.uint32), size=B)
        a["runtime_top_p"] = rng.choice(np.asarray([0.0, 0.5, 0.95], np.float32), size=B)
    elif case["rows"] == "topp":
        a["runtime_top_p"] = np.asarray([case["p"]], np.float32)
    else:
        a["runtime_top_k"] = np.asarray([case["k"]], np.uint32)
        if case["p"]:
            a["runtime_top_p"] = np.asarray([case["p"]], np.float32)
    if case["temperature"] != 1.0:
        a["temperature"] = np.asarray([case["temperature"]], np.float32)
    if case["penalty"] != "none":
        a[case["penalty"] + "_penalty"] = np.asarray([case["penalty_value"]], np.float32)
    if case["min_length"]:
        a["min_length"] = np.asarray([case["min_length"]], np.int32)
    return a


def _prepare_decode(case, seed):
    g, rng = _generator(seed), np.random.default_rng(int(seed))
    B, V, step, prompt = case["batch"], case["vocab"], case["step"], case["prompt"]
    steps = case.get("steps", 1)
    ids = torch.zeros(step + steps + 1, B, dtype=torch.int32, device=DEVICE)
    ids[:step] = torch.randint(1, V - 1, (step, B), generator=g, device=DEVICE, dtype=torch.int32)
    lengths = torch.full((B,), prompt, dtype=torch.int32, device=DEVICE)
    if case["ragged"]:
        lengths = torch.randint((prompt + 1) // 2, prompt + 1, (B,), generator=g, device=DEVICE, dtype=torch.int32)
    inputs = {"max_input_length": prompt, "ite": 0, "local_batch_size": B, "input_lengths": lengths, "step": step,
              "end_id": torch.full((B,), V - 1, dtype=torch.int32, device=DEVICE)}
    if case["bad_words"]:
        inputs["bad_words_list"] = _words(rng, B, case["bad_words"], V, 1)
    if case["stop_words"]:
        inputs["stop_words_list"] = _words(rng, B, case["stop_words"], V, 2)
    if case["limit"]:
        limit = step + steps + 1 if case["kind"] == "generate" else step + 100
        inputs["sequence_limit_length"] = torch.full((B,), limit, dtype=torch.int32, device=DEVICE)
    if case["bias"]:
        inputs["embedding_bias"] = _normal((case["padded"],), 0.5, case["dtype"], g)
        inputs["embedding_bias"][V - 1] = 0
    outputs = {"output_ids": ids,
               "finished": torch.rand(B, generator=g, device=DEVICE) < case["ended"],
               "sequence_length": torch.full((B,), step, dtype=torch.int32, device=DEVICE)}
    if case["log_probs"]:
        outputs["cum_log_probs"] = -3.0 * (step - prompt + 1) * torch.rand(B, generator=g, device=DEVICE)
        outputs["output_log_probs"] = torch.zeros(step - prompt + steps + 1, B, dtype=torch.float32, device=DEVICE)
    pool = [_logits(case, B, g, ids[step - 1].long()) for _ in range(min(steps, 4))]
    args = _runtime_args(case, rng)
    layer = DynamicDecodeLayer(V, case["padded"], DTYPES[case["dtype"]], DEVICE)
    layer.setup(B, 1, args)
    return {"case": case, "layer": layer, "args": args, "inputs": inputs, "outputs": outputs, "pool": pool,
            "start_scores": torch.zeros(B, dtype=torch.float32, device=DEVICE)}


def _prepare_beam(case, seed):
    g = _generator(seed)
    B, K, V, step, prompt = case["batch"], case["beams"], case["vocab"], case["step"], case["prompt"]
    L = step + 2
    ints = dict(dtype=torch.int32, device=DEVICE)
    logits = torch.randn((B, K, V), generator=g, device=DEVICE).mul_(case["sigma"])
    logits[:, :, 2] = END_LOGIT
    outputs = {"output_ids": torch.randint(3, V, (L, B, K), generator=g, **ints),
               "parent_ids": torch.randint(0, K, (L, B, K), generator=g, **ints),
               "finished": torch.zeros(B * K, dtype=torch.bool, device=DEVICE),
               "sequence_length": torch.full((B * K,), step, **ints),
               "cum_log_probs": torch.randn(B * K, generator=g, device=DEVICE) - 5.0,
               "tgt_cache_indirection": torch.zeros(B, K, L, **ints)}
    if case["archive"]:
        f = dict(dtype=torch.float32, device=DEVICE)
        outputs["beam_hyps"] = {
            "output_ids_tgt": torch.zeros(B, 2 * K, L, **ints), "sequence_lengths_tgt": torch.zeros(B, 2 * K, **ints),
            "cum_log_probs": torch.zeros(B, 2 * K, **f), "normed_scores": torch.zeros(B, 2 * K, **f),
            "min_normed_scores": torch.zeros(B, **f), "num_beams": torch.zeros(B, **ints),
            "is_done": torch.zeros(B, dtype=torch.bool, device=DEVICE)}
    args = {"len_penalty": np.asarray([case["len_penalty"]], np.float32)}
    if case["penalty"] != 1.0:
        args["repetition_penalty"] = np.asarray([case["penalty"]], np.float32)
    if case["temperature"] != 1.0:
        args["temperature"] = np.asarray([case["temperature"]], np.float32)
    inputs = dict(args, logits=logits.to(DTYPES[case["dtype"]]), step=step, max_input_length=prompt, ite=0, local_batch_size=B,
                  end_id=torch.full((B,), 2, **ints), input_lengths=torch.full((B, K), prompt, **ints),
                  src_cache_indirection=torch.randint(0, K, (B, K, L), generator=g, **ints))
    layer = DynamicDecodeLayer(V, V, DTYPES[case["dtype"]], DEVICE)
    layer.setup(B, K, args)
    return {"case": case, "layer": layer, "inputs": inputs, "outputs": outputs}


def _prepare_vocab_parallel(case, seed):
    g = _generator(seed)
    B, V, prompt = case["batch"], case["shard"] * case["shards"], 8
    ints = dict(dtype=torch.int32, device=DEVICE)
    shards = [_normal((B, case["shard"]), case["sigma"], case["dtype"], g) for _ in range(case["shards"])]
    shards[-1][:, -1] = END_LOGIT
    sampler = VocabParallelSampler(V, case["shard"], case["shards"], DTYPES[case["dtype"]], torch.device(DEVICE))
    sampler.setup(B, 1, {"runtime_top_k": np.asarray([case["k"]], np.uint32), "runtime_top_p": np.asarray([case["p"]], np.float32),
                         "temperature": np.asarray([case["temperature"]], np.float32),
                         "random_seed": np.asarray([int(seed) % (1 << 31)], np.uint64)})
    outputs = {"output_ids": torch.zeros(prompt + 2, B, **ints), "finished": torch.zeros(B, dtype=torch.bool, device=DEVICE),
               "sequence_length": torch.full((B,), prompt, **ints)}
    inputs = {"step": prompt, "max_input_length": prompt, "end_id": torch.full((B,), V - 1, **ints)}
    return {"case": case, "sampler": sampler, "shards": shards, "inputs": inputs, "outputs": outputs}


def _prepare_context_logprob(case, seed):
    g = _generator(seed)
    B, T = case["batch"], case["length"]
    order = (B, T) if case["batch_first"] else (T, B)
    return {"case": case, "logits": _normal(order + (case["padded"],), case["sigma"], case["dtype"], g),
            "ids": torch.randint(0, case["vocab"], order, generator=g, device=DEVICE, dtype=torch.int32),
            "lengths": torch.randint((T + 1) // 2, T + 1, (B,), generator=g, device=DEVICE, dtype=torch.int32)}


def _prepare_finish(case, seed):
    g = _generator(seed)
    B, K, T, prompt = case["batch"], case["beams"], case["time"], case["prompt"]
    ints, floats = dict(dtype=torch.int32, device=DEVICE), dict(dtype=torch.float32, device=DEVICE)
    s = {"case": case, "ids": torch.randint(3, 32000, (T + 1, B, K), generator=g, **ints),
         "parents": torch.randint(0, K, (T + 1, B, K), generator=g, **ints),
         "lengths": torch.randint((prompt + T) // 2, T, (B, K), generator=g, **ints)}
    s["ids"][:prompt] = s["ids"][:prompt, :, :1]
    if case["form"] == "gather_tree":
        s.update(beams=torch.zeros(T, B, K, **ints), output_ids=torch.zeros(B, K, T, **ints),
                 end=torch.full((B,), 2, **ints), input_lengths=torch.full((B, K), prompt, **ints))
        s["params"] = GatherTreeParams(
            beams=s["beams"].data_ptr(), max_sequence_lengths=s["lengths"].data_ptr(), max_sequence_length_final_step=0,
            input_lengths=s["input_lengths"].data_ptr(), response_input_lengths=None, max_time=T, batch_size=B, beam_width=K,
            step_ids=s["ids"].data_ptr(), parent_ids=s["parents"].data_ptr(), end_tokens=s["end"].data_ptr(),
            max_input_length=prompt, prefix_soft_prompt_lengths=None, p_prompt_tuning_prompt_lengths=None,
            max_input_without_prompt_length=prompt, max_prefix_soft_prompt_length=0, output_ids=s["output_ids"].data_ptr())
        return s
    lp = case["log_probs"]
    s.update(log_probs=torch.randn((T + 1, B, K), generator=g, device=DEVICE) if lp else None,
             finished=torch.zeros(B * K, dtype=torch.bool, device=DEVICE),
             scores=-20.0 * torch.rand(B * K, generator=g, device=DEVICE),
             hyp_ids=torch.zeros(B, 2 * K, T + 1, **ints), hyp_lengths=torch.zeros(B, 2 * K, **ints),
             hyp_cum=torch.zeros(B, 2 * K, **floats), hyp_normed=torch.zeros(B, 2 * K, **floats),
             hyp_log_probs=torch.zeros(B, 2 * K, T + 1, **floats) if lp else None,
             hyp_count=torch.zeros(B, **ints), done=torch.zeros(B, dtype=torch.bool, device=DEVICE),
             output_ids=torch.zeros(B, K, T, **ints), output_lengths=torch.zeros(B, K, **ints),
             output_cum=torch.zeros(B, K, **floats), output_log_probs=torch.zeros(B, K, T, **floats) if lp else None)
    s["hyps"] = BeamHyps(output_ids_tgt=s["hyp_ids"].data_ptr(), sequence_lengths_tgt=s["hyp_lengths"].data_ptr(),
                         cum_log_probs=s["hyp_cum"].data_ptr(), normed_scores=s["hyp_normed"].data_ptr(),
                         log_probs=s["hyp_log_probs"].data_ptr() if lp else None, num_beams=s["hyp_count"].data_ptr(),
                         is_done=s["done"].data_ptr(), early_stopping=1)
    return s


def prepare(case, seed):
    return {"decode": _prepare_decode, "generate": _prepare_decode, "beam": _prepare_beam,
            "vocab_parallel": _prepare_vocab_parallel, "context_logprob": _prepare_context_logprob,
            "finish": _prepare_finish}[case["kind"]](case, seed)


# ---- one pass ---------------------------------------------------------------------------------------------------
def _ptr(t):
    return None if t is None else t.data_ptr()


def _run_decode(s):
    stop = s["layer"].forward(s["outputs"], dict(s["inputs"], logits=s["pool"][0]))
    return dict(s["outputs"], should_stop=bool(stop))


def _run_generate(s):
    c, out = s["case"], s["outputs"]
    B = c["batch"]
    check(lib.ftb200_decoding_initialize(_ptr(out["finished"]), _ptr(out["sequence_length"]), None, _ptr(s["start_scores"]), 0,
                                         None, B, 1, c["step"], torch.cuda.current_stream().cuda_stream))
    s["layer"].setup(B, 1, s["args"])
    for i in range(c["steps"]):
        if s["layer"].forward(out, dict(s["inputs"], logits=s["pool"][i % len(s["pool"])], step=c["step"] + i)):
            break
    return out


def _run_beam(s):
    out, inputs = s["outputs"], s["inputs"]
    s["layer"].forward(out, inputs)
    # the next step reads what this one wrote
    inputs["src_cache_indirection"], out["tgt_cache_indirection"] = out["tgt_cache_indirection"], inputs["src_cache_indirection"]
    return dict(out, src_cache_indirection=inputs["src_cache_indirection"])


def _run_vocab_parallel(s):
    s["sampler"].forward_shards(s["outputs"], s["inputs"], s["shards"])
    return s["outputs"]


def _run_context_logprob(s):
    return log_prob_from_logits(s["logits"], s["ids"], s["lengths"], s["case"]["vocab"], s["case"]["batch_first"])


def _run_finish(s):
    c = s["case"]
    B, K, T = c["batch"], c["beams"], c["time"]
    stream = torch.cuda.current_stream().cuda_stream
    if c["form"] == "gather_tree":
        s["params"].stream = stream
        check(lib.ftb200_gather_tree(C.byref(s["params"])))
        return {"beams": s["beams"], "output_ids": s["output_ids"], "lengths": s["lengths"]}
    s["hyp_count"].zero_()  # an archive starts empty
    check(lib.ftb200_insert_unfinished_path(C.byref(s["hyps"]), _ptr(s["ids"]), _ptr(s["parents"]), _ptr(s["lengths"]),
                                            _ptr(s["log_probs"]), T, 1.0, _ptr(s["finished"]), _ptr(s["scores"]), B, K, stream))
    check(lib.ftb200_finalize(_ptr(s["output_ids"]), _ptr(s["output_lengths"]), _ptr(s["output_cum"]), _ptr(s["output_log_probs"]),
                              _ptr(s["hyp_ids"]), _ptr(s["hyp_lengths"]), _ptr(s["hyp_normed"]), _ptr(s["hyp_cum"]),
                              _ptr(s["hyp_log_probs"]), _ptr(s["hyp_count"]), K, T, B, stream))
    return [s[k] for k in ("output_ids", "output_lengths", "output_cum", "output_log_probs", "hyp_ids", "hyp_lengths", "hyp_normed",
                           "hyp_log_probs", "hyp_count")]


RUN = {"decode": _run_decode, "generate": _run_generate, "beam": _run_beam, "vocab_parallel": _run_vocab_parallel,
       "context_logprob": _run_context_logprob, "finish": _run_finish}


def run(state):
    return RUN[state["case"]["kind"]](state)


# ---- what a pass cannot do without, and how close two correct passes are ------------------------------------------------
def work(case):
    kind, es = case["kind"], SIZE.get(case.get("dtype"), 4)
    if kind in ("decode", "generate"):
        # every logit of a live row once, its history where a penalty reads it, word lists, generator state and flags
        live = case["batch"] * (1.0 - case["ended"])
        row = case["padded"] * es + (4 * case["step"] if case["penalty"] != "none" else 0)
        row += 24 * (case["bad_words"] + case["stop_words"]) + 128 + (16 if case["log_probs"] else 0)
        n = case.get("steps", 1)
        return {"bytes": n * (live * row + (case["padded"] * es if case["bias"] else 0)), "flops": n * live * case["padded"] * 2}
    if kind == "beam":
        rows = case["batch"] * case["beams"]
        hist = 8 * case["step"] if case["penalty"] != 1.0 else 0  # ids and parents
        return {"bytes": rows * (case["vocab"] * es + hist + 8 * (case["step"] + 2) + 64), "flops": rows * case["vocab"] * 4}
    if kind == "vocab_parallel":
        rows = case["batch"]
        return {"bytes": rows * (case["shard"] * case["shards"] * es + 128), "flops": rows * case["shard"] * case["shards"] * 2}
    if kind == "context_logprob":
        rows = case["batch"] * case["length"] * 0.75  # lengths are spread over the upper half
        return {"bytes": rows * (case["vocab"] * es + 4), "flops": rows * case["vocab"] * 4}
    entries = case["batch"] * case["beams"] * (case["time"] * 0.75 + case["prompt"] * 0.25)
    if case["form"] == "gather_tree":  # ids and parents in, the tree and its transposed form out
        return {"bytes": 8 * entries + 8 * case["batch"] * case["beams"] * case["time"], "flops": entries}
    return {"bytes": entries * ((8 + 4 + 4) + (12 if case["log_probs"] else 0)), "flops": entries}


def tolerance(case):
    if case["kind"] in ("decode", "generate") and not case["log_probs"]:
        return "exact"  # ids, lengths and flags
    if case["kind"] in ("decode", "generate"):
        return {"rel": 1e-5, "max": 1e-4}  # log-probabilities are 32-bit; the ids stay the same
    if case["kind"] == "vocab_parallel" or (case["kind"] == "finish" and case["form"] == "gather_tree"):
        return "exact"
    if case["kind"] == "beam":
        # scores are 32-bit sums; two candidates whose scores are that close may change places
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.001}
    return {"rel": 1e-5, "max": 1e-4}
