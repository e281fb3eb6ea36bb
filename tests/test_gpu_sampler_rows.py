"""The sampler on both sides of the line where a row goes to one CTA or to a cluster of eight, few rows and many: a
row's token does not depend on its neighbours and is the one of the whole-number walk."""
import numpy as np
import pytest

from _gpu import P, lib
from test_gpu_sampler_sizes import pick

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 2047, 2048, 2049])
@pytest.mark.parametrize("rows", [1, 40])
def test_one_cta_or_a_cluster_per_row(n, rows):
    L, rng = lib(), np.random.default_rng(n + rows)
    lg = (rng.standard_normal((rows, n)) * 2).astype(np.float32)
    lg[rows // 2] = np.round(lg[rows // 2] * 2) / 2          # ties
    u = rng.random(rows)
    tok = np.empty(rows, np.int32)
    assert L.apus_cuda_sample_logits_u(P(lg), n, 0.8, 0.95, P(u), P(tok), rows) == 0, L.apus_cuda_last_error()
    assert tok.tolist() == [pick(lg[r], 0.8, 0.95, u[r]) for r in range(rows)]
