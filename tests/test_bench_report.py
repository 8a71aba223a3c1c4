"""What bench.py reports beside its times belongs to the kernel that ran."""
import glob
import os

import pytest

import bench

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_measured_traffic_is_that_of_the_kernel():
    sources = "".join(open(f).read() for f in glob.glob(os.path.join(ROOT, "smallframework_b200", "csrc", "*.cu")))
    assert bench.MEASURED_TRAFFIC
    for (layer, batch, kernel), (nbytes, profile, _) in bench.MEASURED_TRAFFIC.items():
        assert "\n" + kernel + "(" in sources                     # a kernel that exists
        text = open(os.path.join(ROOT, "profiles", profile)).read()
        assert kernel in text and "%.1f MB" % (nbytes / 1e6) in text and layer in text
        assert bench.measured_traffic(layer, batch, kernel + " (tcgen05 kind::f16)") == bench.MEASURED_TRAFFIC[layer, batch, kernel]
        assert bench.measured_traffic(layer, batch, "another_kernel (FFMA)") is None
        assert bench.measured_traffic(layer, batch + 1, kernel) is None


def test_kernels_are_named_as_the_library_names_them():
    """The report takes a kernel's name from the launch (small_b200_last_kernel); what it adds is keyed by names that are launched."""
    sources = "".join(open(f).read() for f in glob.glob(os.path.join(ROOT, "smallframework_b200", "csrc", "*.cu")))
    for name in bench.KERNELS:
        assert any('"%s"' % name in line for line in sources.splitlines() if "launched(" in line), name
    assert bench.kernel_class("conv_f16x3_kernel", ["maxpool"]) == ("conv_f16x3_kernel (tcgen05 kind::f16, two-word operands) + maxpool", "f16x3")
    assert bench.kernel_class("softmax_f32") == ("softmax_f32", "stream")


@pytest.mark.gpu
def test_last_kernel_is_this_threads():
    import threading

    from smallframework_b200 import _lib
    from smallframework_b200 import interface as S
    names = {}

    def run(key, call):
        names[key, 0] = _lib.last_kernel()
        call()
        names[key, 1] = _lib.last_kernel()

    I, O = S.FloatBuffer(16 * 8 * 8), S.FloatBuffer(16 * 8 * 8)
    t = threading.Thread(target=run, args=("other", lambda: S.ReLUActivation(16, 8, 8, I, O)))
    S.MaxPool2D(2, 2, 2, 0, 0, 0, 0, 16, 8, 8, I, O)
    t.start()
    t.join()
    assert names == {("other", 0): "", ("other", 1): "relu_f32"} and _lib.last_kernel() == "maxpool2d_f32"
