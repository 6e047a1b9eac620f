"""Every host-to-device copy and memset of the library is ordered before the
kernels that read its destination: on a handle's stream, or complete when the
call returns (upload_sync, zero_sync).  A plain cudaMemcpy from pageable memory
may return while its transfer to the device is pending, a plain cudaMemset does
return at once, and the handles' non-blocking streams wait for neither; no run
shows that reliably, so the sources are read."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fvs2d_gb300", "csrc")
HELPER = re.compile(r"inline cudaError_t (?:upload|zero)_sync\(.*?\n}\n", re.S)
PLAIN = re.compile(r"cudaMemcpy(?:2D|3D)?\s*\([^;]*?cudaMemcpy(?:HostToDevice|DeviceToDevice|Default)|cudaMemset(?:2D|3D)?\s*\(", re.S)


def test_no_plain_upload_or_memset():
    found, helpers = [], 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*"))):
        if not path.endswith((".cu", ".cuh", ".cpp", ".hpp")):
            continue
        text = open(path).read()
        helpers += len(HELPER.findall(text))
        text = HELPER.sub("", text)
        text = re.sub(r"//[^\n]*", "", text)
        found += [f"{os.path.basename(path)}: {m.group(0)[:70]}" for m in PLAIN.finditer(text)]
    assert not found, found
    assert helpers == 2
