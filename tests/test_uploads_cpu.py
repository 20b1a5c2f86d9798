"""Copies of the C layer to the device are ordered before the kernels that read
them.  The systems' streams are not ordered after the legacy stream, on which
cudaMemcpy runs: from pageable memory, and between device arrays, it may return
before its copy is done.  Read from the source, since whether a kernel overtakes
such a copy is left to chance."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "maglua_b200", "csrc")
UNITS = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h")))


@pytest.mark.parametrize("unit", UNITS)
def test_no_device_write_on_the_legacy_stream(unit):
    src = open(os.path.join(CSRC, unit)).read()
    src = re.sub(r"//[^\n]*", "", src)
    calls = [m.group(0) for m in re.finditer(r"\bcudaMemcpy\s*\([^;]*;", src)]
    assert [c for c in calls if "HostToDevice" in c or "DeviceToDevice" in c] == []


def _body(name):
    src = open(os.path.join(CSRC, "capi.cu")).read()
    at = src.index(name)
    return src[at:src.index("\n}\n", at)]


@pytest.mark.parametrize("name", ["mlb_system* make_system(int", "int mlb_ensemble_create(", "int mlb_system_status(",
                                  "int mlb_ensemble_status("])
def test_clears_in_stream_order(name):
    assert not re.search(r"\bcudaMemset\s*\(", _body(name))


# the constant tables and a surrogate's arrays: written anywhere, waited for at the end
@pytest.mark.parametrize("name", ["int mlb_init(", "int mlb_surrogate_create("])
def test_set_up_waits(name):
    assert "cudaDeviceSynchronize()" in _body(name).rsplit("configure", 1)[-1].rsplit("cudaMemset", 1)[-1]
