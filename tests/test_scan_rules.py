"""What the scans' bindings decide on the host: which views go to the kernels as they are, and which kernels a size takes."""
import pytest
import torch

from linear_moe_b200.ops import cuda as K


@pytest.mark.parametrize("name,view,copied", [
    ("dense", lambda x: x, False),
    ("a third of a projection", lambda x: x[..., 128:256], False),
    ("transposed heads", lambda x: x.transpose(1, 2)[..., :128], False),
    ("one head for all", lambda x: x[:, :, :1, :128].expand(-1, -1, 4, -1), True),
    ("one sequence for all", lambda x: x[:1, ..., :128].expand(3, -1, -1, -1), True),
    ("a single head with any stride", lambda x: x[:, :, :1, :128].as_strided((2, 6, 1, 128), (6 * 4 * 384, 4 * 384, 0, 1)), False),
    ("two bytes behind a boundary", lambda x: x[..., 1:129], True),
    ("rows off a boundary", lambda x: x.flatten()[:2 * 6 * 4 * 132].view(2, 6, 4, 132)[..., :128], True),
    ("channels apart", lambda x: x[..., ::3], True)])
def test_views_for_tensor_maps(name, view, copied):
    """Repeated rows, other strides along the channels, rows or starts off 16 bytes are copied, anything else is read where it is; the values stay."""
    x = torch.randn(2, 6, 4, 384).bfloat16()
    t = view(x)
    out = K._tma_view(t)
    assert (out.data_ptr() != t.data_ptr()) == copied and torch.equal(out, t)
    if copied:
        assert out.is_contiguous() and out.data_ptr() % 16 == 0
