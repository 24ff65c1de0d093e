"""The FP64 sweep on the longest lines a grid may have (3000 rows) and on the
first length whose three line arrays at four columns exceed a block's shared
memory (2134 rows): backward error of the correction, as for shorter lines."""
import pytest

import test_fp64_lines_gpu as lines

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(5, 2134, 3), (6, 3000, 3)])
def test_backward_error(gpu_ctx, dims):
    lines.test_long_lines_backward_error(gpu_ctx, dims)
