"""GPU: few query rows of full-int8 where the splits of a K/V head are a cluster of CTAs (scores in shared memory, maxima and results
through distributed shared memory): 1 to 8 CTAs, the last one with one key or all of its keys, one and two row halves, many heads."""
import pytest

import test_gpu_decode as base

pytestmark = pytest.mark.gpu

CASES = [
    # B, Hkv, ratio, Nq, Nk, D, G, causal, scales
    (1, 1, 1, 1, 7, 128, 128, True, "fp32"),
    (1, 1, 4, 1, 512, 128, 128, True, "fp16"),                # one CTA
    (1, 2, 4, 2, 513, 128, 128, True, "fp32"),                # two, the second with one key
    (1, 1, 8, 1, 1537, 64, 64, True, "fp16"),
    (1, 1, 1, 5, 2500, 128, 64, False, "fp32"),
    (1, 1, 2, 3, 3583, 64, 128, True, "fp32"),                # seven
    (1, 1, 2, 1, 4096, 128, 128, True, "fp16"),               # eight, all full
    (1, 1, 4, 4, 4000, 128, 128, True, "fp32"),               # eight, 16 rows
    (1, 2, 4, 5, 1025, 64, 64, True, "fp32"),                 # 20 rows: two tiles
    (16, 20, 1, 1, 2113, 64, 64, True, "fp32"),               # as many heads as fill a wave: the scores decide the number of CTAs
    (3, 2, 2, 6, 2047, 64, 128, True, "fp16"),
]


@pytest.mark.parametrize("B,Hkv,ratio,Nq,Nk,D,G,causal,scales", CASES)
def test_splits_as_a_cluster(B, Hkv, ratio, Nq, Nk, D, G, causal, scales, pkg, oracle):
    base.test_few_rows_against_a_cache("full", B, Hkv, ratio, Nq, Nk, D, G, causal, scales, pkg, oracle)
