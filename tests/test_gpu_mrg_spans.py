"""The MRG32k3a stream does not depend on how a call cuts it: pieces with short
spans per lane against a whole with longer ones, bit for bit, at both sides of
the lines between the spans and far along the stream."""
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu

LINE = 152 * 32 * 32       # lanes of one fill of 152 SMs


def _call(kind, first, count):
    import torch
    P = pkg()
    out = torch.empty(count, dtype=torch.float32 if kind == "normals_f32" else torch.float64, device="cuda")
    fn = getattr(P, "mrg32k3a_%s_device" % kind)
    args = (12345, first, count, out.data_ptr())
    fn(*args)
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("kind,count", [("uniforms", 2 * LINE * 64 - 1), ("uniforms", 2 * LINE * 64), ("normals_f32", 2 * LINE * 64 + 5),
                                        ("normals_f64", 8 * LINE * 32 - 1), ("normals_f64", 8 * LINE * 32)])
@pytest.mark.parametrize("first", [0, (1 << 62) + 12345])
def test_pieces_equal_the_whole(kind, count, first):
    import torch
    whole = _call(kind, first, count)
    for at, n in ((0, 1), (1, 33), (511, 4097), (count // 3, 100_001), (count - 65_537, 65_537), (count - 1, 1)):
        assert torch.equal(whole[at:at + n], _call(kind, first + at, n))
