"""ftb200_log_prob_from_logits against the reference's invokeLogProbFromLogits (oracle/_ref), the CPU
restatement and the committed outputs of the reference kernel.  Shapes are the reference test's own
(tests/unittests/test_logprob_kernels.cu:265-303) plus ragged, padded and unaligned rows."""
import json
import os
import sys

import numpy as np
import pytest
import torch

import ft_reference
from ft_oracle import oracle_log_prob_from_logits

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(HERE, "golden"))
from make_logprob_fixture import CASES, logprob_case  # noqa: E402

# log-probs are floating point: 1e-3 absolute per scored token is the bar; sums over n tokens get n times that
TOL = 1e-3


def run_ours(logits, ids, lengths, vocab, bf):
    from fastertransformer_b200 import log_prob_from_logits
    max_len = logits.shape[1] if bf else logits.shape[0]
    batch = logits.shape[0] if bf else logits.shape[1]
    ws = torch.zeros(max_len * batch, dtype=torch.float32, device="cuda")
    cum = log_prob_from_logits(logits, ids, lengths, vocab_size=vocab, batch_first=bf, workspace=ws)
    torch.cuda.synchronize()
    return cum.cpu().numpy(), ws[:(max_len - 1) * batch].cpu().numpy()


def run_ref(logits, ids, lengths, vocab, bf):
    lib = ft_reference.ref_lib()
    max_len = logits.shape[1] if bf else logits.shape[0]
    batch = logits.shape[0] if bf else logits.shape[1]
    ws = torch.zeros(max_len * batch, dtype=torch.float32, device="cuda")
    cum = torch.zeros(batch, dtype=torch.float32, device="cuda")
    rc = lib.ftref_log_prob_from_logits(cum.data_ptr(), logits.data_ptr(), 0 if logits.dtype == torch.float32 else 1,
                                        ids.data_ptr(), lengths.data_ptr(), max_len, batch, vocab,
                                        logits.shape[2], ws.data_ptr(), ws.numel() * 4, None, int(bf))
    torch.cuda.synchronize()
    assert rc == 0
    return cum.cpu().numpy(), ws[:(max_len - 1) * batch].cpu().numpy()


def valid_mask(lengths, max_len, bf):
    steps = np.arange(max_len - 1)
    m = steps[None, :] < (lengths[:, None] - 1) if bf else steps[:, None] < (lengths[None, :] - 1)
    return m.ravel()


@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
def test_committed_reference_outputs(case):
    name, max_len, batch, vocab, vp, dtype, bf = case
    with open(os.path.join(HERE, "golden", "logprob_ref.json")) as f:
        g = json.load(f)[name]
    logits, ids, lengths = logprob_case(*case)
    cum, lp = run_ours(torch.from_numpy(logits).cuda(), torch.from_numpy(ids).cuda(),
                       torch.from_numpy(lengths).cuda(), vocab, bf)
    m = valid_mask(lengths, max_len, bf)
    np.testing.assert_allclose(np.where(m, lp, 0.0), np.array(g["log_probs"], np.float32), rtol=0, atol=TOL)
    np.testing.assert_allclose(cum, np.array(g["cum_log_probs"], np.float32), rtol=0, atol=TOL * max_len)


REF_SHAPES = [(1, 32, 16), (129, 8, 50211), (1023, 8, 5001), (4096, 8, 5001)]


@pytest.mark.skipif(not ft_reference.available(), reason="oracle/_ref not built")
@pytest.mark.parametrize("bf", [False, True], ids=["step_major", "batch_first"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16], ids=["f32", "f16"])
@pytest.mark.parametrize("shape", REF_SHAPES, ids=[f"len{s[0]}_b{s[1]}_v{s[2]}" for s in REF_SHAPES])
def test_reference_test_shapes(shape, dtype, bf):
    max_input_length, batch, vocab = shape
    max_len = max_input_length + 1        # the reference test scores max_input_length tokens (:140)
    g = torch.Generator(device="cuda").manual_seed(max_len * 7 + batch)
    full = (batch, max_len, vocab) if bf else (max_len, batch, vocab)
    logits = (torch.rand(full, generator=g, device="cuda") * 6 - 3).to(dtype)
    ids = torch.randint(0, vocab, (batch, max_len) if bf else (max_len, batch), generator=g, device="cuda",
                        dtype=torch.int32)
    lengths = torch.randint(1, max_len + 1, (batch,), generator=g, device="cuda", dtype=torch.int32)
    lengths[0] = max_len
    cum, lp = run_ours(logits, ids, lengths, vocab, bf)
    rcum, rlp = run_ref(logits, ids, lengths, vocab, bf)
    m = valid_mask(lengths.cpu().numpy(), max_len, bf)
    assert np.abs(np.where(m, lp - rlp, 0.0)).max() <= 2e-5       # same arithmetic up to summation order
    n = lengths.cpu().numpy().astype(np.float64)
    assert (np.abs(cum - rcum) <= 1e-6 * np.abs(rcum) + 2e-5 * np.sqrt(n) + 1e-4).all()
    # the reference test's own check, against its host computation (gtest_utils.h:39-102)
    atol, rtol = (1e-4, 1e-2) if dtype == torch.float32 else (1e-3, 1e-1)
    x = logits.float().double()
    if bf:
        x = x.transpose(0, 1)
        idm = ids.t()
    else:
        idm = ids
    lsm = torch.log_softmax(x[:-1], dim=2)
    tok = torch.gather(lsm, 2, idm[1:].long().unsqueeze(2))[:, :, 0]
    steps = torch.arange(max_len - 1, device="cuda")[:, None]
    want = torch.where(steps < (lengths[None, :] - 1), tok, torch.zeros_like(tok)).sum(0).cpu().numpy()
    assert (np.abs(cum - want) <= atol + rtol * np.abs(want)).all()


@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16"])
@pytest.mark.parametrize("bf", [False, True], ids=["step_major", "batch_first"])
def test_padded_unaligned_rows_against_restatement(dtype, bf):
    # vocab_padded odd: rows start at every 2- or 4-byte phase of a 16-byte line; vocab < padded
    max_len, batch, vocab, vp = 7, 5, 1003, 1011
    rng = np.random.default_rng(17)
    shape = (batch, max_len, vp) if bf else (max_len, batch, vp)
    x = rng.uniform(-6, 6, size=shape).astype(np.float32)
    x[..., vocab:] = 50.0                       # padding must not be counted
    ids = rng.integers(0, vocab, size=(batch, max_len) if bf else (max_len, batch)).astype(np.int32)
    lengths = np.array([7, 1, 2, 5, 7], np.int32)
    tdt = {"float32": torch.float32, "float16": torch.float16, "bfloat16": torch.bfloat16}[dtype]
    d = torch.from_numpy(x).cuda().to(tdt)
    if dtype == "bfloat16":
        host = d.view(torch.int16).cpu().numpy().view(np.uint16)
    else:
        host = d.cpu().numpy()
    cum, lp = run_ours(d, torch.from_numpy(ids).cuda(), torch.from_numpy(lengths).cuda(), vocab, bf)
    ocum, olp = oracle_log_prob_from_logits(host, ids, lengths, vocab, batch_first=bf, dtype_name=dtype)
    m = valid_mask(lengths, max_len, bf)
    np.testing.assert_allclose(np.where(m, lp, 0.0), np.where(m, olp.ravel(), 0.0), rtol=0, atol=2e-5)
    np.testing.assert_allclose(cum, ocum, rtol=0, atol=1e-4)
    assert cum[1] == 0.0


def test_argument_checks():
    from fastertransformer_b200 import lib
    x = torch.zeros(2, 2, 8, device="cuda")
    i = torch.zeros(2, 2, dtype=torch.int32, device="cuda")
    n = torch.ones(2, dtype=torch.int32, device="cuda")
    c = torch.zeros(2, device="cuda")
    ws = torch.zeros(4, device="cuda")
    f = lib.ftb200_log_prob_from_logits
    assert f(c.data_ptr(), x.data_ptr(), 0, i.data_ptr(), n.data_ptr(), 2, 2, 8, 8, ws.data_ptr(), 8, None, 0) == 4
    assert f(c.data_ptr(), x.data_ptr(), 0, i.data_ptr(), n.data_ptr(), 2, 2, 9, 8, ws.data_ptr(), 16, None, 0) == 1
    assert f(c.data_ptr(), x.data_ptr(), 9, i.data_ptr(), n.data_ptr(), 2, 2, 8, 8, ws.data_ptr(), 16, None, 0) == 1
    assert f(c.data_ptr(), None, 0, i.data_ptr(), n.data_ptr(), 2, 2, 8, 8, ws.data_ptr(), 16, None, 0) == 1


def test_single_position_sequences_score_nothing():
    from fastertransformer_b200 import log_prob_from_logits
    x = torch.randn(1, 5, 64, device="cuda")
    ids = torch.zeros(1, 5, dtype=torch.int32, device="cuda")
    n = torch.ones(5, dtype=torch.int32, device="cuda")
    cum = log_prob_from_logits(x, ids, n)
    assert cum.shape == (5,) and bool((cum == 0).all())


@pytest.mark.parametrize("batch", [1, 31, 256, 1024, 1025])
@pytest.mark.parametrize("bf", [False, True], ids=["step_major", "batch_first"])
def test_ragged_lengths_of_many_sequences(batch, bf):
    """The counted rows are dealt out from a table of the sequences' counts (up to 1024 of them): lengths from 0 to the
    longest, a run of empty sequences in front and at the end, against the restatement."""
    rng = np.random.default_rng(batch)
    max_len, vocab = 9, 515
    lengths = rng.integers(0, max_len + 1, batch).astype(np.int32)
    lengths[: batch // 4] = 1
    lengths[batch - batch // 8:] = 0
    lengths[batch // 2] = max_len
    shape = (batch, max_len) if bf else (max_len, batch)
    logits = (rng.standard_normal(shape + (vocab,)) * 2).astype(np.float32)
    ids = rng.integers(0, vocab, shape).astype(np.int32)
    cum, lp = run_ours(torch.from_numpy(logits).cuda(), torch.from_numpy(ids).cuda(), torch.from_numpy(lengths).cuda(), vocab, bf)
    want_cum, want_lp = oracle_log_prob_from_logits(logits, ids, lengths, vocab, bf)
    live = valid_mask(lengths, max_len, bf)
    assert np.abs(lp - np.asarray(want_lp).ravel()[: lp.size])[live].max() < TOL
    assert np.abs(cum - want_cum).max() < TOL * max_len


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("vocab,vp", [(1, 8), (7, 8), (2049, 2056), (8195, 8195), (50257, 50257)])
def test_extreme_values_of_16_bit_rows(dtype, vocab, vp):
    """-infinity, the type's lowest value, its largest and values of very different size, at each remainder of the pairs."""
    max_len, batch = 6, 4
    g = torch.Generator().manual_seed(vocab)
    x = torch.randn(max_len, batch, vp, generator=g) * 4
    low = torch.finfo(dtype).min
    x[1, :, ::2] = -float("inf")
    x[2, :, 1::3] = low
    x[3] = x[3] * 100
    x[4, 0], x[4, 1, 0], x[4, 2] = low, torch.finfo(dtype).max, 0.0
    for t in range(max_len):
        x[t, :, vocab - 1] = 1.5  # (the token that is scored below)
    x = x.to(dtype)
    ids = torch.full((max_len, batch), vocab - 1, dtype=torch.int32)
    lengths = torch.full((batch,), max_len, dtype=torch.int32)
    cum, lp = run_ours(x.cuda(), ids.cuda(), lengths.cuda(), vocab, False)
    want = torch.log_softmax(x[:max_len - 1, :, :vocab].double(), -1)[..., vocab - 1].numpy()
    # fp32 sums of the exponentials (2^-24 relative per term of a tree) and a result rounded to fp32
    tol = 1e-6 * 8 + np.abs(want) * 2.0 ** -22
    assert (np.abs(lp.reshape(max_len - 1, batch) - want) <= tol).all()
    assert (np.abs(cum - want.sum(0)) <= tol.sum(0) * 2).all()


@pytest.mark.parametrize("mask", [-1e4, -1e9, -1e10, -1e12, -1e20])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("vocab", [515, 8195, 50257])
def test_masked_columns_and_large_maxima(vocab, dtype, mask):
    """A thread's running maximum is the mask's value until it meets a column that is not masked, and rows whose maximum
    itself is large: all but a few columns at the end masked, every second one, all of them."""
    g = torch.Generator().manual_seed(vocab)
    peaks = [0.0, -300.0, 3e3, 8160.0, 8192.0, -8192.0, 1e4, 6e4, 1e5, 3e5, 1e6, 1e7, -1e9, 1e10, 1e12]
    max_len, batch = len(peaks) + 1, 4
    limit = 65504.0 if dtype == torch.float16 else 3e38
    x = torch.randn(max_len, batch, vocab, generator=g) * 4
    x[:-1] += torch.tensor(peaks).clamp(-limit, limit)[:, None, None]
    x[:, 0, : vocab - 7] = mask
    x[:, 1, ::2] = mask
    x[:, 2] = mask
    x = x.clamp(-limit, limit).to(dtype)
    best = x.float().argmax(-1).int()  # (scored: the differences that count are small)
    ids = torch.cat([torch.zeros(1, batch, dtype=torch.int32), best[:-1]])
    lengths = torch.full((batch,), max_len, dtype=torch.int32)
    _, lp = run_ours(x.cuda(), ids.cuda(), lengths.cuda(), vocab, False)
    want = torch.log_softmax(x[:-1].double(), -1).gather(2, best[:-1, :, None].long())[..., 0].numpy()
    # the bound of the test above: fp32 sums, and a result rounded to fp32
    assert (np.abs(lp.reshape(max_len - 1, batch) - want) <= 8e-6 + np.abs(want) * 2.0 ** -22).all()
