"""The shares of a pass's tokens over CTA pairs, where they can go wrong: an odd number of tokens, one more than fill a pair, a last CTA with fewer than the
others, one to four occupied quadrants of 32 rows; splits without keys; a cache that ends half way through a tile of keys."""
import pytest

from tests.helpers import assert_close
from tests.test_gpu_tc import _run_tc
from yasakani_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fused", [False, True], ids=["workspace", "fused"])
@pytest.mark.parametrize("shape,ctx,M,splits", [
    (synth.C2, 90, 9, 3),                                  # 5 + 4 tokens: 30 and 24 rows; the cache ends at 192
    (synth.C2, 64, 11, 9),                                 # 36 rows: a second quadrant of four rows; more splits than tiles
    (synth.C2, 190, 43, 2),                                # two pairs of 11 tokens a CTA, the last one 10
    (synth.C1, 33, 33, 2),                                 # hd 128, eight heads: one row more than a pair holds
    (synth.Shape(4, 4, 256, 64, 1e4), 130, 33, 1),         # one head per kv-head: 17 rows in a tile of 128
    (synth.Shape(4, 4, 128, 32, 1e4), 5, 257, 2),          # the same over more than one pair
])
def test_token_shares_match_exact_oracle(oracle, shape, ctx, M, splits, fused):
    from yasakani_b200 import kv4
    got, want = _run_tc(kv4, oracle, shape, ctx, M, splits, seed=77, fused=fused)
    assert_close(got, want, f"{shape} ctx {ctx} M {M} splits {splits} fused {fused}")
