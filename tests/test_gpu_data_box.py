"""The data box of a view (mvd::dev_data_box): the bounds of image > 0 or weight > 0."""
import ctypes

import pytest

from spim_registration_gb300 import native

pytestmark = pytest.mark.gpu


def test_rows_of_nearly_2_to_the_31_voxels():
    """A row's last step of 128 voxels passes 2^31."""
    torch = pytest.importorskip("torch")
    nx = 2**31 - 10
    if torch.cuda.mem_get_info()[0] < 12 * 2**30:
        pytest.skip("needs 9 GB")
    box_of = native.load()._ZN3mvd12dev_data_boxEPKfS1_iiiPiP11CUstream_st
    box_of.argtypes, box_of.restype = [ctypes.c_void_p] * 2 + [ctypes.c_int] * 3 + [ctypes.c_void_p] * 2, None
    img = torch.zeros(nx, device="cuda")
    img[7] = img[nx - 2] = 1.0
    box = torch.tensor([2**31 - 1] * 3 + [-1] * 3, dtype=torch.int32, device="cuda")
    box_of(img.data_ptr(), img.data_ptr(), nx, 1, 1, box.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert box.tolist() == [7, 0, 0, nx - 2, 0, 0]
