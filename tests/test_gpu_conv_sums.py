"""Weight and bias gradient sums of the convolution layers over grids that fill the bias
kernel's grid and exceed it, with a voxel count that no block divides, and over one voxel.
Bar: FP32 sums of partial sums against FP64, relative L2 1e-5."""
import pytest

from test_gpu_learned import test_conv3d_kernels_match_oracle as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cin,cout,shape,relu", [(3, 5, (1, 1, 1), 0), (5, 3, (21, 43, 43), 1), (1, 1, (3, 7, 3), 1),
                                                 (2, 16, (32, 37, 32), 0)])
def test_conv3d_gradient_sums(gpu_lib, cin, cout, shape, relu):
    check(gpu_lib, cin, cout, shape, relu)
