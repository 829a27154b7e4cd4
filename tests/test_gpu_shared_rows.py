"""Several sessions over one host array of exact rows: whichever made the mapping and whichever ends first, the others' rows stay mapped."""
import numpy as np
import pytest

import oracle
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 4])   # mapped, hybrid
def test_rows_stay_mapped_for_the_last_session(psb, mode):
    ix = synth.make_index(4000, 32, 16, 8, seed=5)
    q = synth.make_queries(ix, 200, seed=6)
    want = oracle.ivfpq_search(ix, q, 4, 10, 40)

    def check(s):
        got = s.search(q, 4, 10)
        assert np.array_equal(got["indices"], want["indices"]) and np.array_equal(got["distances"], want["distances"])

    first, second, third = [psb.Session(ix, n_rerank=40, exact_mode=mode, max_batch=200) for _ in range(3)]
    check(first)
    first.close()
    check(second)
    check(third)
    third.close()
    check(second)
    second.close()
    with psb.Session(ix, n_rerank=40, exact_mode=mode, max_batch=200) as s:   # mapped anew
        check(s)


def test_parts_of_a_mapped_array(psb):
    """A session over part of an array that is mapped whole shares the mapping; one that would need more of it than is mapped is refused."""
    ix = synth.make_index(4000, 32, 16, 8, seed=5)
    half = int(ix["offsets"][8])
    part = dict(ix, nlist=8, centroids=ix["centroids"][:8], offsets=ix["offsets"][:9], codes=ix["codes"][:half], vectors=ix["vectors"][:half],
                reordered_ids=np.arange(half, dtype=np.int64))
    q = synth.make_queries(ix, 50, seed=7)
    want = oracle.ivfpq_search(part, q, 4, 10, 40)
    whole = psb.Session(ix, n_rerank=40, max_batch=200)
    s = psb.Session(part, n_rerank=40, max_batch=200)
    whole.close()
    got = s.search(q, 4, 10)
    assert np.array_equal(got["indices"], want["indices"]) and np.array_equal(got["distances"], want["distances"])
    s.close()
    with psb.Session(part, n_rerank=40, max_batch=200):
        with pytest.raises(psb.PsbError):
            psb.Session(ix, n_rerank=40, max_batch=200)
        with psb.Session(ix, n_rerank=40, max_batch=200, exact_mode=psb.EXACT_HOST_STAGED) as t:
            t.search(q, 4, 10)
    with psb.Session(ix, n_rerank=40, max_batch=200) as t:
        t.search(q, 4, 10)
