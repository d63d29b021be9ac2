"""The BCH check at batch sizes on both sides of each step of its cluster-size
rule (eight, four, two and one CTA a codeword)."""
import pytest

from test_gpu_bch_clusters import test_bch_check_clusters as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rate,n,nblk", [
    ("2/15", 16200, 37), ("2/15", 16200, 38), ("13/15", 16200, 100), ("13/15", 16200, 101),
    ("6/15", 64800, 222), ("6/15", 64800, 223)])
def test_cluster_rule(rate, n, nblk):
    check(rate, n, nblk)
