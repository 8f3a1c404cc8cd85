"""What the Python binding refuses before it hands a pointer to the library.  Runs without a GPU: nothing is launched."""
import pytest

import fp8_quant_matmul_b200 as f

torch = pytest.importorskip("torch")


class OnDevice:
    """As much of a CUDA tensor as an argument check looks at."""
    is_cuda = True

    def __init__(self, index):
        self.index = index

    def get_device(self):
        return self.index


@pytest.mark.parametrize("src,dst", [(torch.zeros(32, dtype=torch.uint8), None),
                                     (torch.zeros(32, dtype=torch.uint8, device="meta"), None),
                                     (torch.zeros(32, dtype=torch.uint8), torch.zeros(32, dtype=torch.uint8)),
                                     (OnDevice(0), torch.zeros(32, dtype=torch.uint8)),
                                     (OnDevice(0), OnDevice(1))],
                         ids=["cpu", "meta", "both cpu", "dst on the cpu", "two devices"])
def test_reencoding_refuses_tensors_that_are_not_on_one_gpu(src, dst):
    before = f.launch_count()
    with pytest.raises(ValueError):
        f.fnuz_to_fn_device(src, dst)
    assert f.launch_count() == before
