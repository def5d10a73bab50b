"""Few rows per expert: the one-block routing against the oracle, at the sizes where it can go wrong.  Needs a B200: ``-m gpu``."""
import numpy as np
import pytest

from oracle import moe_oracle as oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,experts,top_k", [(1, 1, 1), (1, 256, 8), (31, 33, 4), (33, 32, 3), (128, 256, 8), (128, 64, 6), (129, 64, 6), (97, 5, 5)])
def test_one_block_routing_matches_the_oracle(tokens, experts, top_k):
    """Both sides of the token limit, every width of a lane's expert list, ties, and scores of the lowest values."""
    from gpu_util import RouteTables, check_route_against_oracle, to_device

    rng = np.random.default_rng(tokens * 3 + experts)
    scores = rng.standard_normal((tokens, experts)).astype(np.float32)
    scores[:, ::3] = np.round(scores[:, ::3])                                 # ties, zeros of both signs among them
    scores[tokens // 2] = -0.0
    scores[-1, : experts // 2] = np.finfo(np.float32).min
    tables = RouteTables(tokens, experts, top_k)
    tables.run(to_device(scores, "float32"))
    check_route_against_oracle(tables, oracle.routing(scores, top_k))
    # readers of the per-block probability sums add them over the blocks
    sums = tables.host("block_colsum", (-1, experts)).sum(axis=0)
    assert np.abs(sums - tables.host("probs", (tokens, experts)).sum(axis=0)).max() <= 1e-5 * tokens
