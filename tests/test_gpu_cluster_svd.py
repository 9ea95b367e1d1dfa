"""k_svd where it changes form: one CTA below m = 40 and from m = 64, a cluster of CTAs between, at sizes
that divide the cluster's columns evenly and that do not.  The tolerances are the one-CTA form's."""
import pytest

from test_gpu_svd import _check, _graded

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k", [(39, 10), (40, 1), (41, 39), (47, 10), (48, 24), (49, 16), (55, 8), (63, 31), (64, 8)])
def test_sizes_around_the_cluster_form(m, k):
    _check(_graded(m, 7 + m, decades=4.0), k)
