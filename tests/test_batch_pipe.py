"""The mixed batch's choice of pipe for its contexts (no GPU)."""

import pytest


class _Context:
    def __init__(self, words, fp64):
        self.words, self.fp64 = words, fp64

    def set_fp64(self, enable):
        self.fp64 = enable


class _Entry:
    def __init__(self, words, fp64):
        self.ctx = _Context(words, fp64)


@pytest.mark.parametrize("tuned,before,after", [
    (True, 0, 1), (True, 1, 1), (True, 2, 2),  # 2 also moves the server's products: the caller's choice
    (False, 0, 0), (False, 1, 0), (False, 2, 0),
    (None, 0, 0), (None, 1, 1), (None, 2, 2),  # widths that were not tuned
])
def test_select_pipe_leaves_contexts_that_are_on_it(tuned, before, after):
    from cuhepy_b200.batch import MixedBatch

    batch = MixedBatch.__new__(MixedBatch)
    batch.paillier_fp64 = {} if tuned is None else {64: tuned}
    entries = [_Entry(64, before), _Entry(128, before)]
    batch._select_pipe(entries)
    assert [e.ctx.fp64 for e in entries] == [after, before]
