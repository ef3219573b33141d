"""A renderer's streams do not order against the legacy default stream (cudaStreamNonBlocking), and
a blocking copy from pageable host memory may return before its transfer has reached the device.
So whatever a renderer's kernels read is written on the renderer's own stream: in the source of the
renderer no blocking host-to-device copy and no blocking fill occurs before the stand-alone BSDF
calls, whose kernels run on the default stream, too."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "xenon_b200", "csrc", "renderer.cu")


def test_renderer_writes_device_memory_on_its_stream():
    text = open(SRC).read()
    assert text.count("\nint xb_bsdf_eval(") == 1
    renderer = text[:text.index("\nint xb_bsdf_eval(")]
    calls = re.findall(r"\bcudaMemcpy\([^;]*;|\bcudaMemset\([^;]*;", renderer)
    assert [c for c in calls if "cudaMemcpyDeviceToHost" not in c] == []
