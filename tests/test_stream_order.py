"""Device memory is written on the stream of the launches that read it.

The engine's streams are non-blocking: they do not wait for the legacy stream,
and cudaMemcpy from pageable memory may return while its last part is still on
the way (cudaMemset returns at once).  So a plain cudaMemcpy to the device or
cudaMemset is only sound where the whole device is waited for before anything is
launched: in the making of a context, which ends with cudaDeviceSynchronize."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "brain-match_b200", "csrc")


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu"))), ids=os.path.basename)
def test_no_unordered_writes(path):
    text = open(path).read()
    end = text.find("cudaDeviceSynchronize") if path.endswith("bm_engine.cu") else 0
    assert end >= 0
    late = [m.group(0) for m in re.finditer(r"\bcuda(Memcpy|Memset)\([^;]*;", text)
            if m.start() > end and "DeviceToHost" not in m.group(0)]
    assert not late, late
