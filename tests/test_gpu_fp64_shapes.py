"""FP64 self-sums on both sides of the sizes where their launch shape changes (128 x 1 targets split up to 1,280 points,
128 x 2 up to 2,304, the Laplacian's up to 4,096, then whole tiles)."""
import pytest

import test_gpu_fp64_sums

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n,name', [(1280, 'gauss'), (1281, 'gauss'), (2304, 'gauss'), (1280, 'laplacian'),
                                    (1281, 'laplacian'), (4096, 'laplacian'), (4097, 'laplacian')])
def test_fp64_self_sums_at_shape_changes(n, name):
    test_gpu_fp64_sums.test_fp64_self_sums_at_block_edges(n, name)
