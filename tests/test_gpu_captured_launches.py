"""The kernels that a captured step launches, as the library counts them (the benchmark's gpu_launches):
dt with the ghost fill, Phase1 + stress, the sweeps, the second Phase1, whichever of them a form and a
grid's size put into one launch."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,prec,form,want", [
    ((20, 10, 12), "fp64", None, 4),     # the three sweeps in one launch
    ((256, 128, 96), "fp64", None, 4),   # eight waves of them
    ((256, 128, 128), "fp64", None, 6),  # eleven: three launches
    ((20, 10, 12), "fp64", "1", 5),      # one sweep kernel, behind its own ghost fill
    ((20, 10, 12), "fp32", None, 4),     # x1 and x3 folded in, the seams with the x2 sweep
    ((20, 10, 12), "fp32", "0", 4),
    ((512, 128, 64), "fp32", None, 6),   # the two seam kernels beside the x2 sweep
    ((512, 128, 64), "fp32", "0", 6),    # three sweeps of more than a few waves
])
def test_captured_launches(ark, monkeypatch, C, prec, form, want):
    if form is not None:
        monkeypatch.setenv("ARK_PHASE2_FUSED", form)
    p = ark.make_params(*C, precision=ark.FP64 if prec == "fp64" else ark.FP32)
    with ark.Context(p) as c:
        c.upload(ark.channel_init(p, seed=3, amp=0.1))
        assert c.captured_launches() == want
        c.step(72)  # graphs of eight steps where the grid is small enough
        c.sync()
        assert c.captured_launches() == want
        c.set_averaging(True)
        assert c.captured_launches() == want + 1
