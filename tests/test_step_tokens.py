"""An entry's token ids, checked and copied as an array: the same answers as one by one."""
import numpy as np
import pytest
import torch

import boring_llm_b200                                                   # noqa: F401
from boring_llm_b200.engine import runner

VOCAB = 1000


@pytest.mark.parametrize("n", [1, runner.ARRAY_MIN_TOKENS - 1, runner.ARRAY_MIN_TOKENS, 257])
@pytest.mark.parametrize("put", [None, -1, VOCAB, VOCAB - 1, 2 ** 31, -2 ** 40, 3.0, "7", True, np.int64(5), np.int64(VOCAB), torch.tensor(6)])
@pytest.mark.parametrize("kind", [list, tuple, np.array, bytes])
def test_token_ids_as_an_array(n, put, kind):
    ids = [(7 * i) % (256 if kind is bytes else VOCAB) for i in range(n)]
    if put is not None:
        if kind is bytes or (kind is np.array and not isinstance(put, (int, np.int64))):
            return
        ids[n // 2] = put
    tokens = kind(ids)
    got = runner._token_array(tokens, VOCAB)
    if got is not None:
        assert all(0 <= int(t) < VOCAB for t in tokens) and got.dtype == np.int32
        assert got.tolist() == np.asarray([int(t) for t in tokens], dtype=np.int32).tolist()
    plain = all(isinstance(t, (int, np.int64)) and 0 <= t < VOCAB for t in ids)
    assert (got is not None) == (kind in (list, tuple) and n >= runner.ARRAY_MIN_TOKENS and (plain or isinstance(put, torch.Tensor)))


def test_a_batch_is_filled_alike_from_arrays_and_from_lists():
    class Cached:
        def __init__(self, slot, held):
            self.slot, self.num_tokens, self.tables = slot, held, [[slot, slot + 1]]

    entries = [runner.StepEntry("a", list(range(40)), [3, 39]), runner.StepEntry("b", [5], [0]), runner.StepEntry("c", tuple(range(100, 150)))]
    rcs = [Cached(2, 0), Cached(1, 7), Cached(0, 3)]
    q_lens = [len(e.tokens) for e in entries]
    filled = []
    for ids in (None, [runner._token_array(e.tokens, VOCAB) for e in entries]):
        f = {k: np.full(n, -9, np.int32) for k, n in (("token_ids", 91), ("positions", 91), ("tok_req", 91), ("cu_q", 4), ("ctx_len", 3), ("slots", 3),
                                                      ("logit_rows", 3))}
        f["tables"] = np.full((1, 3, 4), -9, np.int32)
        assert runner._fill_batch(f, entries, rcs, q_lens, [40, 8, 53], ids) == [2, 1, 0]
        filled.append(f)
    for k in filled[0]:
        assert np.array_equal(filled[0][k], filled[1][k]) and not (filled[0][k] == -9).any(), k
