"""Prefill-sized stage-1 scores (sparse_stage1.cu: more than 64 query rows, 16 query heads per key head): ragged last token tile, ragged
last chunks of compressed keys, both kinds of log-sum-exp keys, caches of several sizes, up to one that is full; the checks of
the decode-sized kernels."""
import pytest

from test_sparse_gpu import test_block_selection_matches_oracle as check_selection

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,hq,hkv,L,top,sink,window,lse,budget", [
    (65, 16, 1, 5000, 64, 1, 4, True, None), (100, 32, 2, 3000, 16, 1, 8, False, None), (131, 32, 2, 2064, 8, 2, 2, True, 65536),
    (72, 16, 1, 8256, 30, 1, 2, True, 131072), (67, 16, 1, 2048, 7, 0, 1, False, None), (80, 48, 3, 16300, 64, 1, 32, True, 16384 + 128)])
def test_block_selection(T, hq, hkv, L, top, sink, window, lse, budget):
    check_selection(T, hq, hkv, L, top, sink, window, lse, budget)
