"""CPU: uploads go through the stream that reads them.

The library's streams do not wait for the default stream, and a copy from pageable memory on
the default stream may return before its last part has reached the device, so nothing would
order such a copy (or a copy or memset within the device) before the kernels that read it."""
import glob
import os
import re

from conftest import REPO


def test_no_write_of_device_memory_on_the_default_stream():
    found = []
    for path in sorted(glob.glob(os.path.join(REPO, "b12_b200", "csrc", "*.cu*"))):
        text = open(path).read()
        for m in re.finditer(r"\b(cudaMemcpy|cudaMemset|cudaMemcpy2D|cudaMemset2D)\s*\(([^;]*);", text):
            if m.group(1).startswith("cudaMemset") or "DeviceToHost" not in m.group(2):
                found.append((os.path.basename(path), text.count("\n", 0, m.start()) + 1, m.group(0)))
    assert not found, found
