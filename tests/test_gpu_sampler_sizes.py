"""The sampler at the edges of its slices (a row is spread over eight CTAs, csrc/sample.cu): rows shorter than
the cluster, slices with a remainder, slices too long for shared memory, ties across slices -- against the same
walk restated with whole numbers: p as c/sample.h:91-180 defines it, mass in 2^-60 steps, tokens ordered by
(p descending, index ascending).  The token is compared exactly."""
import numpy as np
import pytest

from _gpu import P, lib

pytestmark = pytest.mark.gpu
ONE = 1 << 60


def pick(lg, temp, top_p, u):
    x = ((lg - lg.max()).astype(np.float32) / np.float32(temp)).astype(np.float32)
    e = np.exp(x.astype(np.float64)).astype(np.float32)
    p = (e.astype(np.float64) / e.astype(np.float64).sum()).astype(np.float32)
    order = np.lexsort((np.arange(p.size), -p.astype(np.float64)))
    inc = np.cumsum((p[order].astype(np.float64) * ONE).astype(np.uint64))

    def first(m):                                        # the first place whose inclusive mass exceeds m
        return int(np.searchsorted(inc, np.uint64(m), side="right"))
    cut = first(int(np.float32(top_p).astype(np.float64) * ONE))
    kept = int(inc[min(cut, p.size - 1)])
    return int(order[first(min(int(u * float(kept)), kept - 1))])


@pytest.mark.parametrize("n", [1, 7, 9, 1023, 8193, 129283, 327681])
@pytest.mark.parametrize("top_p", [0.3, 0.95, 1.0])
def test_token_is_the_one_of_the_whole_number_walk(n, top_p):
    L, rng = lib(), np.random.default_rng(n)
    rows = 6
    lg = (rng.standard_normal((rows, n)) * 2).astype(np.float32)
    lg[1] = np.round(lg[1] * 2) / 2                      # ties in every slice
    lg[2] = 1.25                                         # one value everywhere
    lg[3, n - 1] = 30.0                                  # nearly all the mass on the last token
    u = rng.random(rows)
    u[4], u[5] = 0.0, 1.0 - 2.0 ** -53
    tok = np.empty(rows, np.int32)
    assert L.apus_cuda_sample_logits_u(P(lg), n, 0.8, top_p, P(u), P(tok), rows) == 0, L.apus_cuda_last_error()
    assert tok.tolist() == [pick(lg[r], 0.8, top_p, u[r]) for r in range(rows)]
