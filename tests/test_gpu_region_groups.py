"""xnor_b200_region_activate on both sides of the group size that fits shared memory, against fp64."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import synth  # noqa: E402
from darknet_b200 import capi  # noqa: E402


@pytest.mark.parametrize("batch,anchors,classes,hw", [(1, 1, 1, 1), (2, 3, 127, 33), (1, 2, 150, 165), (1, 2, 150, 166), (2, 1, 1000, 50), (70, 5, 3, 169),
                                                      (3, 5, 80, 169), (2, 2, 7, 256), (1, 2, 9, 257), (1, 1, 30, 512), (1, 1, 30, 513), (2, 1, 2, 64)])
def test_class_softmax(batch, anchors, classes, hw):
    x = torch.from_numpy(synth.bell(classes + hw, (batch, anchors, 5 + classes, hw), 3.0)).cuda()
    out = torch.full_like(x, float("nan"))
    capi.check(capi.lib().xnor_b200_region_activate(x.data_ptr(), out.data_ptr(), batch, anchors, 4, classes, 1, hw,
                                                   torch.cuda.current_stream().cuda_stream), "region_activate")
    want = x.double()
    want[:, :, [0, 1, 4]] = torch.sigmoid(want[:, :, [0, 1, 4]])
    want[:, :, 5:] = torch.softmax(want[:, :, 5:], 2)
    assert (out.double() - want).abs().max().item() <= 2e-6
