"""The merge of attention splits with 12 and with 24 partial outputs in flight (tree_attn.cu): around both counts of splits, more splits than key
tiles, and on both sides of the number of rows from which 24 are taken for few splits; against fp32 like the other passes."""
import pytest

from test_kernels_gpu import test_tree_attention_matches_fp32 as attention

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("splits", [2, 11, 12, 13, 24, 25, 32])
@pytest.mark.parametrize("tq,hq,hkv", [(1, 32, 2), (37, 32, 2), (38, 32, 2), (64, 16, 4)])
def test_splits(tq, hq, hkv, splits):
    attention((tq, hq, hkv, 1900, "causal", splits))
