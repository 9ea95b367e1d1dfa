"""k_svd at the largest sizes of its cluster form, 56 to 62 columns, and the first beyond, where the exchange
buffers no longer fit beside the work and one CTA runs.  The tolerances are the one-CTA form's."""
import pytest

from test_gpu_svd import _check, _graded

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k", [(56, 20), (57, 28), (60, 20), (61, 30), (62, 31), (63, 20)])
def test_largest_cluster_sizes(m, k):
    _check(_graded(m, 11 + m, decades=4.0), k)
