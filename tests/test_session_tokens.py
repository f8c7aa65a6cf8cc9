"""What ``Session.feed`` takes as tokens, on a stand-in generator."""
from types import SimpleNamespace

import pytest
import torch

from rpeg_b200.engine.generation import PAGE, Generator, PagePool
from rpeg_b200.engine.session import Session


def _session():
    seen = []
    gen = SimpleNamespace(pool=PagePool(9), page_table=torch.zeros(2, 4, dtype=torch.int32), zero_cache=False, max_slots=2, dev=torch.device("cpu"),
                          cfg=SimpleNamespace(vocab=100), max_seq_len=4 * PAGE, pages_per_row=4, cached_prefill=True, first_visible_key=None)
    gen._upload = lambda arrays: Generator._upload(gen, arrays)

    def prefill_hidden(pieces, slots, starts):
        seen.extend(p.tolist() for p in pieces)
        return None, None

    gen.prefill_hidden = prefill_hidden
    return Session(gen), seen


@pytest.mark.parametrize("tokens,want", [([5, 0, 99], [5, 0, 99]), ((True, 3), [1, 3]), ([1.0, 2.7], [1, 2]), (torch.tensor([4, 7]), [4, 7])])
def test_tokens_that_are_taken(tokens, want):
    session, seen = _session()
    session.feed([("a", tokens, [])])
    assert seen == [want]


@pytest.mark.parametrize("tokens", [[], [100], [-1, 3], [3, 2 ** 40], [1.0, -3.0], [1.0, 100.0], [1.0, float("nan"), 3.0], [float("nan")], [1.0, float("inf")],
                                    [1, float("nan")], torch.tensor([4.0, 7.9])])
def test_tokens_that_are_refused(tokens):
    """Nothing that is no token of the vocabulary reaches the embedding, and a refused call starts no request."""
    session, seen = _session()
    with pytest.raises((ValueError, RuntimeError, TypeError)):
        session.feed([("a", tokens, [])])
    assert not seen and not session.requests and len(session.free_slots) == 2
