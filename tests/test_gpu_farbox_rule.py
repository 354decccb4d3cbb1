"""The rule between boxes and direct loop where calls have few samples a box: the
boxes' cost counts a share for every block of node sums and every target, so
such calls take the direct loop, which is the faster there (measured on one
B200, direct loop and boxes: 205,379 x 1,509 in a cube 255 and 321 us, 420,000 x
738 in a channel 299 and 483; with four and six times the samples 757 and 495 us
in the cube, 1,097 and 577 in the channel)."""
import pytest

from test_gpu_farbox_forms import make, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,every,boxes", [((59, 59, 59), 136, False), ((59, 59, 59), 32, True),
                                               ((1000, 21, 20), 569, False), ((1000, 21, 20), 88, True)])
def test_route(cuda, shape, every, boxes):
    ps, solver, _ = make(shape=shape, keep=1.0, every=every)
    assert run(ps, solver)[1] == boxes
