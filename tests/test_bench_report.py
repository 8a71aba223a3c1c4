"""What bench.py reports beside its times belongs to the kernel that ran."""
import glob
import os

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
