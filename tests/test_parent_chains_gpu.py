"""Gather tree and archive of unfinished beams by parallel parent chains, against the CPU restatement: one and two levels,
level counts either side of a square (the segments' edges), one beam, more segments' threads than a block, chains that
break off, beams of different prompt lengths, positions past the register batches, and tables that do not fit shared memory."""
import numpy as np
import pytest

import decoding_cases as dc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw,uneven", [
    (dict(seed=101, B=3, K=4, T=2, M=1, final_step=0), False), (dict(seed=102, B=2, K=1, T=3, M=1, final_step=1), False),
    (dict(seed=103, B=5, K=5, T=65, M=3, final_step=1), False), (dict(seed=104, B=5, K=5, T=66, M=3, bad_parents=True), False),
    (dict(seed=105, B=3, K=4, T=90, M=12, prefix=True, virtual=True, with_response=True), True),
    (dict(seed=106, B=2, K=7, T=200, M=20, bad_parents=True), True), (dict(seed=107, B=2, K=4, T=5000, M=9), False),
    (dict(seed=108, B=2, K=33, T=1800, M=30, bad_parents=True), False)])
def test_gather_tree_chains(kw, uneven):
    c = dc.gather_tree_case(**kw)
    if uneven:
        lo = int(c["input_lengths"].min())
        c["input_lengths"] = np.random.default_rng(1).integers(lo, kw["M"] + 1, size=c["input_lengths"].shape).astype(np.int32)
        c["input_lengths"] = np.maximum(c["input_lengths"], 6)  # prompts longer than any prefix
    dc.same(dc.run_gather_tree("ours", c), dc.run_gather_tree("oracle", c))


@pytest.mark.parametrize("kw", [dict(seed=111, B=3, K=4, L=1), dict(seed=112, B=4, K=3, L=63), dict(seed=113, B=4, K=3, L=65),
                                dict(seed=114, B=2, K=100, L=300), dict(seed=115, B=2, K=40, L=1500, with_log_probs=False)])
def test_insert_unfinished_path_chains(kw):
    c = dc.insert_case(**kw)
    dc.same(dc.run_insert("ours", c), dc.run_insert("oracle", c), float_keys=("normed",))


@pytest.mark.parametrize("kw", [
    dict(seed=121, B=3, K=1, T=1023, M=7), dict(seed=122, B=4, K=4, T=1024, M=9, final_step=1),
    dict(seed=123, B=4, K=4, T=1025, M=64, bad_parents=True), dict(seed=124, B=2, K=7, T=2047, M=30, bad_parents=True),
    dict(seed=125, B=2, K=5, T=4096, M=100, prefix=True, with_response=True), dict(seed=126, B=2, K=4, T=4097, M=20),
    dict(seed=127, B=5, K=7, T=37, M=36), dict(seed=128, B=3, K=8, T=300, M=12), dict(seed=129, B=3, K=6, T=4096, M=5),
    dict(seed=130, B=6, K=3, T=40, M=12, virtual=True, prefix=True), dict(seed=131, B=2, K=2, T=2048, M=2047, final_step=1)])
def test_gather_tree_by_maps(kw):
    """The form that composes the levels' maps: one to four levels a thread and one more, the most beams a map holds and one
    more, tables that just fit and just do not, broken parents, sequences that end inside the prompt or behind the time."""
    c = dc.gather_tree_case(**kw)
    dc.same(dc.run_gather_tree("ours", c), dc.run_gather_tree("oracle", c))
    c["seq_lengths"] = c["seq_lengths"] + kw["T"] // 3  # (some now end behind max_time)
    dc.same(dc.run_gather_tree("ours", c), dc.run_gather_tree("oracle", c))
    c["seq_lengths"][:] = np.maximum(kw["M"] - 2, 1)
    dc.same(dc.run_gather_tree("ours", c), dc.run_gather_tree("oracle", c))
